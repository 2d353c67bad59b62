// Jacobi-PCG of a small tissue inside one thread-block cluster: the vectors stay in
// the shared memory of its blocks for the whole solve, neighbours across
// blocks are read through distributed shared memory, and the iteration
// synchronises with cluster barriers instead of grid reductions through L2.
//
// Why: below about 100 k cells an iteration of the grid-wide two-pass kernel (cg_flat.cu)
// is its two grid reductions, 6.5 - 7 us with 148 blocks whether the tissue has 400
// cells or 65 k, and of the fused one 5 us.  Here it takes 2.5 us for a 400-cell cable (a solve of 10 iterations
// 34 us, 66 us grid-wide) and 3.8 us for 12.7 k cells in 16 blocks (61 against 98
// us for 13), bound by the latency of the reduction's and the rows' FP64
// chains; with 4 k cells per block (65 k, FP64) a block's work is 5 us and the fused
// grid-wide kernel is faster (80 against 111 us): the host times clusters to 32 k cells.
//
// One reduction per iteration: with q = A p and z = M r (M the Jacobi
// preconditioner) the pass sums p.q, q.z, q.Mq, q.r, q.q, r.z and r.r; then
// alpha = r.z / p.q, and after r' = r - alpha q
//     r'.z' = r.z - 2 alpha q.z + alpha^2 q.Mq,  r'.r' = r.r - 2 alpha q.r + alpha^2 q.q,
// so beta and the stopping test need no second reduction.  alpha comes from the stored
// r's own sums every iteration, so nothing accumulates; where the new sum would be a small
// difference of large ones (below GUARD of the old) it is taken from the
// updated r with a reduction of its own.  Same iterates and stopping rule as
// cg_flat.cu (linear_system_solver.c:47-183), mixed precision and its FP64
// refinement included.
#include <cooperative_groups.h>
#include "cg_rows.cuh"

namespace cg = cooperative_groups;

namespace mb {
namespace ccg {

using fcg::ACTIVE;
using fcg::Args;
using fcg::fill_inv_table;
using fcg::gather;
using fcg::inv_of;
using fcg::Prec;
using fcg::product;

constexpr int NT = 512;           // threads per block: 16 warps to reduce, 128 registers each
constexpr int MAXC = 16;          // largest cluster
constexpr double GUARD = 1e-4;    // leaves 12 digits of a recurred FP64 sum, all of an FP32 one

// Cluster-wide sums of 8 values per thread, the same bits in every thread.  A warp
// exchanges halves, so that each lane carries one value after three steps
// (18 shuffles, not 80); the warps' sums are added by the first warp, which leaves
// the block's 8 totals with every block of the cluster; after the barrier each
// warp adds the blocks' totals itself.  part alternates between two buffers.
__device__ __forceinline__ void cluster_sum(cg::cluster_group &cl, double (&v)[8], double (*part)[MAXC][8],
                                            double (*wsum)[8], int &red) {
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned C = cl.num_blocks(), me = cl.block_rank();
    const double s = fcg::warp_sum8(v);
    if ((lane & 3u) == 0u) wsum[warp][lane >> 2] = s;
    __syncthreads();
    const int buf = red & 1;
    red++;
    if (warp == 0) {
        // lanes: value lane & 7, warps of the quarter lane >> 3
        constexpr int W = NT / 32 / 4;
        double w[W];
#pragma unroll
        for (int k = 0; k < W; ++k) w[k] = wsum[(lane >> 3) * W + k][lane & 7u];
#pragma unroll
        for (int h = W / 2; h > 0; h /= 2)
#pragma unroll
            for (int k = 0; k < h; ++k) w[k] += w[k + h];
        double t = w[0];
        t += __shfl_xor_sync(0xffffffffu, t, 8);
        t += __shfl_xor_sync(0xffffffffu, t, 16);
        for (unsigned d = lane >> 3; d < C; d += 4) cl.map_shared_rank(&part[buf][me][0], d)[lane & 7u] = t;
    }
    cl.sync();
    double w[MAXC / 4];
#pragma unroll
    for (int k = 0; k < MAXC / 4; ++k) {
        const unsigned b = (lane >> 3) + 4 * k;
        w[k] = b < C ? part[buf][b][lane & 7u] : 0.0;
    }
    double t = (w[0] + w[1]) + (w[2] + w[3]);
    t += __shfl_xor_sync(0xffffffffu, t, 8);
    t += __shfl_xor_sync(0xffffffffu, t, 16);
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = __shfl_sync(0xffffffffu, t, q);
}

// The row of a cell whose neighbours all lie in this block, without the clamps
// of gather: f at l and at the strides o (0 where the grid has one plane or one row,
// which reads the cell itself; its code couples no such face).
template <typename F, int KIND>
__device__ __forceinline__ fcg::Row7<F, KIND> row_in_block(const mb_stencil_dev &st, uint32_t g, const F *f, uint32_t l,
                                                           uint32_t oy, uint32_t oz) {
    fcg::Row7<F, KIND> R;
    R.m = __ldg(st.code + g);
    R.pc = f[l];
    R.p[0] = f[l - 1];
    R.p[1] = f[l + 1];
    R.p[2] = f[l - oy];
    R.p[3] = f[l + oy];
    R.p[4] = f[l - oz];
    R.p[5] = f[l + oz];
    if constexpr (KIND == 1) {
        R.c[0] = F(__ldg(st.fx + g - 1));
        R.c[1] = F(__ldg(st.fx + g));
        R.c[2] = F(__ldg(st.fy + g - oy));
        R.c[3] = F(__ldg(st.fy + g));
        R.c[4] = F(__ldg(st.fz + g - oz));
        R.c[5] = F(__ldg(st.fz + g));
    }
    return R;
}

// f at grid index g from the block that holds it.
template <typename F>
struct Field {
    const F *own;
    uint32_t base, chunk;
    __device__ __forceinline__ F operator()(uint32_t g) const {
        const uint32_t l = g - base;
        if (l < chunk) return own[l];
        const uint32_t rank = g / chunk;
        return cg::this_cluster().map_shared_rank(own, rank)[g - rank * chunk];
    }
};

template <bool MIXED, int KIND>
__global__ void __launch_bounds__(NT, 1) k_ccg(Args a, uint32_t chunk) {
    using T = typename Prec<MIXED>::T;
    extern __shared__ __align__(16) unsigned char ccg_smem[];
    __shared__ double part[2][MAXC][8];
    __shared__ double wsum[NT / 32][8];
    __shared__ T itab[64];
    cg::cluster_group cl = cg::this_cluster();
    double *xs = reinterpret_cast<double *>(ccg_smem);
    T *ps = reinterpret_cast<T *>(xs + chunk), *rs = ps + chunk, *qs = rs + chunk;
    const mb_stencil_dev &st = a.st;
    const uint32_t n = (uint32_t)st.nx * st.ny * st.nz;
    const uint32_t base = cl.block_rank() * chunk;
    const uint32_t mine = base < n ? min(chunk, n - base) : 0u;
    mb_ctrl *c = a.ctrl;
    const bool pre = c->use_precond != 0;
    const double tol = c->tol, ratio = c->refine_ratio, floor_ = c->refine_floor;
    const int max_its = c->max_its;
    int red = 0;
    if constexpr (KIND == 0) fill_inv_table<MIXED>(st, itab);
    for (uint32_t l = threadIdx.x; l < mine; l += NT) {
        xs[l] = a.x[base + l];
        ps[l] = rs[l] = qs[l] = T(0);
    }
    cl.sync();

    // kinds 0, 1: whether every index a row reads lies in the block
    const uint32_t oy = st.ny > 1 ? (uint32_t)st.nx : 0u, oz = st.nz > 1 ? (uint32_t)st.nx * st.ny : 0u;
    const uint32_t reach = max(1u, max(oy, oz));
    auto in_block = [&](uint32_t l) { return KIND != 2 && l >= reach && l + reach < mine; };
    auto code = [&](uint32_t g) -> unsigned { return KIND == 2 ? ACTIVE : (unsigned)__ldg(st.code + g); };
    auto inv = [&](uint32_t g, unsigned m) -> T { return pre ? inv_of<MIXED, KIND>(a, itab, g, m) : T(1); };

    double v[8];
    // FP64 true residual r = b - A x, p = z; v: r.z, r.r of the stored r, the FP64 r.r
    auto residual = [&]() {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = 0.0;
        const Field<double> fx{xs, base, chunk};
        for (uint32_t l = threadIdx.x; l < mine; l += NT) {
            const uint32_t g = base + l;
            const auto row = gather<double, KIND>(st, g, fx);
            if (!(row.m & ACTIVE)) continue;
            const double r64 = (a.b ? a.b[g] : st.alpha * a.vstar[g]) - product<double, KIND>(st, row);
            const T rt = (T)r64, z = inv(g, row.m) * rt;
            rs[l] = rt;
            ps[l] = z;
            v[0] += (double)rt * (double)z;
            v[1] += (double)rt * (double)rt;
            v[2] += r64 * r64;
        }
        cluster_sum(cl, v, part, wsum, red);
    };

    residual();
    double rz = v[0], rr = v[1], error = v[2], rr_ref = v[2], alpha = 0.0, beta = 0.0;
    int its = 1, refinements = MIXED ? 1 : 0;
    bool done = !(error >= tol) || !(1 < max_its), first = true, updated = false;
    const Field<T> fp{ps, base, chunk};
    while (!done) {
        if (!first) {
            // r and x of the last direction, the new direction
            const T al = (T)alpha, bt = (T)beta;
            for (uint32_t l = threadIdx.x; l < mine; l += NT) {
                const unsigned m = code(base + l);
                if (!(m & ACTIVE)) continue;
                const T po = ps[l], r = updated ? rs[l] : rs[l] - al * qs[l];
                xs[l] += alpha * (double)po;
                rs[l] = r;
                ps[l] = inv(base + l, m) * r + bt * po;
            }
        }
        cl.sync();
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = 0.0;
        auto use = [&](uint32_t l, const auto &row) {
            if (!(row.m & ACTIVE)) return;
            const T qt = product<T, KIND>(st, row), r = rs[l], id = inv(base + l, row.m);
            qs[l] = qt;
            const double q = (double)qt, z = (double)(id * r), rd = (double)r;
            v[0] += (double)row.pc * q;
            v[1] += q * z;
            v[2] += q * (double)(id * qt);
            v[3] += q * rd;
            v[4] += q * q;
            v[5] += rd * z;
            v[6] += rd * rd;
        };
        if constexpr (KIND == 2) {
            for (uint32_t l = threadIdx.x; l < mine; l += NT) use(l, gather<T, KIND>(st, base + l, fp));
        } else {
            // U rows' loads in flight together
            constexpr int U = KIND == 0 ? 4 : 2;
            for (uint32_t l0 = threadIdx.x; l0 < mine; l0 += U * NT) {
                if (in_block(l0) && l0 + (U - 1) * NT + reach < mine) {
                    fcg::Row7<T, KIND> rows[U];
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        rows[u] = row_in_block<T, KIND>(st, base + l0 + u * NT, ps, l0 + u * NT, oy, oz);
#pragma unroll
                    for (int u = 0; u < U; ++u) use(l0 + u * NT, rows[u]);
                } else {
#pragma unroll 1
                    for (uint32_t l = l0; l < mine && l < l0 + U * NT; l += NT) {
                        if (in_block(l)) use(l, row_in_block<T, KIND>(st, base + l, ps, l, oy, oz));
                        else use(l, gather<T, KIND>(st, base + l, fp));
                    }
                }
            }
        }
        cluster_sum(cl, v, part, wsum, red);
        rz = v[5];
        rr = v[6];
        alpha = (pre ? rz : rr) / v[0];
        const T al = (T)alpha;
        const double ad = (double)al;
        double rzn = rz - ad * (2.0 * v[1] - ad * v[2]), rrn = rr - ad * (2.0 * v[3] - ad * v[4]);
        its += 1;
        updated = false;
        if (!(rrn > GUARD * rr && rzn > GUARD * rz)) {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = 0.0;
            for (uint32_t l = threadIdx.x; l < mine; l += NT) {
                const unsigned m = code(base + l);
                if (!(m & ACTIVE)) continue;
                const T r = rs[l] - al * qs[l];
                rs[l] = r;
                v[0] += (double)r * (double)(inv(base + l, m) * r);
                v[1] += (double)r * (double)r;
            }
            cluster_sum(cl, v, part, wsum, red);
            rzn = v[0];
            rrn = v[1];
            updated = true;
        }
        const bool last = its >= max_its;
        if (!MIXED) {
            error = rrn;
            done = rrn <= tol || last;
            beta = pre ? rzn / rz : rrn / rr;
            first = false;
            if (done) {
                rz = rzn;
                rr = rrn;
                for (uint32_t l = threadIdx.x; l < mine; l += NT) xs[l] += alpha * (double)ps[l];
            }
        } else if (rrn <= fmax(floor_, ratio * rr_ref) || last) {
            // FP64 true residual replaces the FP32 recurrence; restart from it
            for (uint32_t l = threadIdx.x; l < mine; l += NT) xs[l] += alpha * (double)ps[l];
            cl.sync();
            residual();
            refinements += 1;
            error = v[2];
            rr_ref = v[2];
            rz = v[0];
            rr = v[1];
            first = true;
            done = error <= tol || last;
        } else {
            beta = pre ? rzn / rz : rrn / rr;
            error = rrn;
            first = false;
        }
    }
    for (uint32_t l = threadIdx.x; l < mine; l += NT) a.x[base + l] = xs[l];
    if (cl.block_rank() == 0 && threadIdx.x == 0) {
        c->its = its;
        c->error = error;
        c->refinements = refinements;
        c->rz = rz;
        c->rr = rr;
        c->done = 1;
        if (a.end.on) fcg::step_end(c, a.end);
    }
    cl.sync();        // no block leaves while another may still read its memory
}

static const void *kernel_of(int mixed, int kind) {
    static const void *const t[2][3] = {
        {(const void *)k_ccg<false, 0>, (const void *)k_ccg<false, 1>, (const void *)k_ccg<false, 2>},
        {(const void *)k_ccg<true, 0>, (const void *)k_ccg<true, 1>, (const void *)k_ccg<true, 2>}};
    return t[mixed ? 1 : 0][kind];
}

static uint32_t chunk_of(uint32_t n, int C) { return ((n + C - 1) / C + 31u) & ~31u; }
static size_t smem_of(int mixed, uint32_t chunk) { return (size_t)chunk * (8 + 3 * (mixed ? 4 : 8)); }

static cudaLaunchConfig_t config(int C, size_t smem, cudaStream_t s, cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = C;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace ccg
}  // namespace mb

using namespace mb::ccg;

// Variant v is a cluster of 2^v blocks.
extern "C" int mbk_ccg_variants(void) { return 5; }

// Whether variant v can run this tissue: its vectors fit the cluster's shared
// memory, no block is left nearly empty, and the device can place the cluster.
extern "C" int mbk_ccg_usable(const mb_pcg_dev *p, int v) {
    const unsigned long long n = (unsigned long long)p->st.nx * p->st.ny * p->st.nz;
    const int C = 1 << v;
    if (v < 0 || v >= 5 || p->st.kind > 2 || n > (1ULL << 20)) return 0;
    if (C > 1 && n < 128ULL * C) return 0;
    int dev = 0, lim = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return 0;
    const uint32_t chunk = chunk_of((uint32_t)n, C);
    const size_t smem = smem_of(p->mixed, chunk);
    if (smem + 8192 > (size_t)lim) return 0;      // the reduction's own arrays
    const void *fn = kernel_of(p->mixed, p->st.kind);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, lim - 8192) != cudaSuccess ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = config(C, smem, 0, attr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return clusters > 0;
}

extern "C" int mbk_ccg_launch(const mb_pcg_dev *p, cudaStream_t s) {
    Args a{};
    a.st = p->st;
    a.x = p->x; a.vstar = p->vstar; a.b = p->b;
    a.inv_diag64 = p->inv_diag64; a.inv_diag32 = p->inv_diag32;
    a.ctrl = p->ctrl; a.status = p->status;
    a.end = p->end;
    const int C = 1 << p->cc_variant;
    uint32_t chunk = chunk_of((uint32_t)p->st.nx * p->st.ny * p->st.nz, C);
    void *args[] = {&a, &chunk};
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = config(C, smem_of(p->mixed, chunk), s, attr);
    return (int)cudaLaunchKernelExC(&cfg, kernel_of(p->mixed, p->st.kind), args);
}
