// Rows of the operator for one cell, shared by the CG kernels that take a cell per
// thread (cg_flat.cu, cg_cluster.cu), and the Jacobi 1/diag.
#pragma once
#include "cg_common.cuh"

namespace mb {
namespace fcg {

// ---- operator rows ------------------------------------------------------------

// A 7-point row gathered for one cell: the field at the cell and at the six
// neighbours (-x, +x, -y, +y, -z, +z), the code byte, and for kind 1 the six
// face coefficients.  Neighbour indices are clamped into the grid, so every
// load of the row is issued at once, independent of the code byte; values
// of faces that do not couple are discarded by row_apply.
template <typename T, int KIND>
struct Row7 {
    T pc, p[6];
    T c[KIND == 1 ? 6 : 1];
    unsigned m;
};

template <typename T, int KIND, typename PF>
__device__ __forceinline__ Row7<T, KIND> gather7(const mb_stencil_dev &st, uint32_t g, PF pf) {
    Row7<T, KIND> R;
    const uint32_t sy = (uint32_t)st.nx, sz = (uint32_t)st.nx * (uint32_t)st.ny, n = sz * (uint32_t)st.nz;
    const uint32_t i0 = g > 0u ? g - 1u : g, i1 = g + 1u < n ? g + 1u : g;
    const uint32_t i2 = g >= sy ? g - sy : g, i3 = g + sy < n ? g + sy : g;
    const uint32_t i4 = g >= sz ? g - sz : g, i5 = g + sz < n ? g + sz : g;
    R.m = __ldg(st.code + g);
    R.pc = pf(g);
    R.p[0] = pf(i0);
    R.p[1] = pf(i1);
    R.p[2] = pf(i2);
    R.p[3] = pf(i3);
    R.p[4] = pf(i4);
    R.p[5] = pf(i5);
    if constexpr (KIND == 1) {
        R.c[0] = T(__ldg(st.fx + i0));
        R.c[1] = T(__ldg(st.fx + g));
        R.c[2] = T(__ldg(st.fy + i2));
        R.c[3] = T(__ldg(st.fy + g));
        R.c[4] = T(__ldg(st.fz + i4));
        R.c[5] = T(__ldg(st.fz + g));
    }
    return R;
}

// (A p)_c = alpha p_c + sum over coupled faces of c (p_c - p_n).
template <typename T, int KIND>
__device__ __forceinline__ T row_apply(const mb_stencil_dev &st, const Row7<T, KIND> &R) {
    T acc = T(st.alpha) * R.pc;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        T c;
        if constexpr (KIND == 0) c = T(q < 2 ? st.cx : (q < 4 ? st.cy : st.cz));
        else c = R.c[q];
        if ((R.m >> q) & 1u) acc += c * (R.pc - R.p[q]);
    }
    return acc;
}

// 27-point rows (kind 2) from the per-plane class table; the product is
// formed while gathering.  Missing neighbours have zero coefficients in the
// table and are not loaded; entries that are zero in every row of the table
// (st.nzmask) are not read at all.
template <typename T>
struct Row27 {
    T pc, ap;
    unsigned m;
};

template <typename T, typename PF>
__device__ __forceinline__ Row27<T> gather27(const mb_stencil_dev &st, uint32_t g, PF pf) {
    Row27<T> R;
    R.m = ACTIVE;
    R.pc = pf(g);
    const int sy = st.nx, sz = st.nx * st.ny;
    const size_t row = (size_t)__ldg(st.rowid + g) * 27;
    T acc = T(0);
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                const int q = (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1);
                if (!((st.nzmask >> q) & 1u)) continue;     // zero in every row
                const T c = sizeof(T) == 8 ? T(__ldg(st.table + row + q)) : T(__ldg(st.table32 + row + q));
                if (q == 13) acc += c * R.pc;
                else if (c != T(0)) acc += c * pf((uint32_t)((int)g + dx + sy * dy + sz * dz));
            }
    R.ap = acc;
    return R;
}

template <typename T, int KIND, typename PF>
__device__ __forceinline__ auto gather(const mb_stencil_dev &st, uint32_t g, PF pf) {
    if constexpr (KIND == 2) return gather27<T>(st, g, pf);
    else return gather7<T, KIND>(st, g, pf);
}

template <typename T, int KIND, typename R>
__device__ __forceinline__ T product(const mb_stencil_dev &st, const R &row) {
    if constexpr (KIND == 2) return row.ap;
    else return row_apply<T, KIND>(st, row);
}

template <bool MIXED>
struct Prec { using T = double; };
template <>
struct Prec<true> { using T = float; };

template <bool MIXED>
__device__ __forceinline__ typename Prec<MIXED>::T inv_d(const Args &a, uint32_t g) {
    if constexpr (MIXED) return a.inv_diag32[g];
    else return a.inv_diag64[g];
}

// Jacobi 1/diag of a cell: with constant coefficients (kind 0) it depends on
// the code byte only and comes from the block's 64-entry table (filled by
// fill_inv_table as k_inv_diag forms it), otherwise from the per-cell array.
template <bool MIXED, int KIND>
__device__ __forceinline__ typename Prec<MIXED>::T inv_of(const Args &a, const typename Prec<MIXED>::T *tab,
                                                         uint32_t g, unsigned m) {
    if constexpr (KIND == 0) return tab[m & 63u];
    else return inv_d<MIXED>(a, g);
}

// Fills the block's table; a block may have as few as 32 threads (the host
// sizes blocks to whole rounds of cells).
template <bool MIXED>
__device__ __forceinline__ void fill_inv_table(const mb_stencil_dev &st, typename Prec<MIXED>::T *tab) {
    for (unsigned m = threadIdx.x; m < 64; m += blockDim.x) {
        const double c[6] = {st.cx, st.cx, st.cy, st.cy, st.cz, st.cz};
        double d64 = st.alpha;
        float d32 = (float)st.alpha;
        for (int q = 0; q < 6; ++q)
            if ((m >> q) & 1u) {
                d64 += c[q];
                d32 += (float)c[q];
            }
        if constexpr (MIXED) tab[m] = 1.0f / d32;
        else tab[m] = 1.0 / d64;
    }
}

}  // namespace fcg
}  // namespace mb
