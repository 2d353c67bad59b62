// Pieces shared by the persistent CG kernels (cg_flat.cu, cg_resident.cu):
// the launch arguments and the bounded grid-wide reduction.
#pragma once
#include <cstdint>
#include <cuda/atomic>
#include <cuda_runtime.h>
#include "mb_internal.h"

namespace mb {
namespace fcg {

constexpr long long SPIN_LIMIT = 1LL << 24;   // bounded waits (about a second)

struct Args {
    mb_stencil_dev st;
    double *x;
    const double *vstar;
    const double *b;
    double *r64, *pa64, *pb64, *z64;
    float *r32, *pa32, *pb32, *z32;
    double *ap64;              // A p of the current direction (stored by Q, read by U)
    float *ap32;
    float *ap32b;              // second A p buffer (z-march fused pass, flat fused kernel)
    double *ap64b;             // the same in FP64 (flat fused kernel)
    double *w;                 // the z-march fused solve's stored A x (FP64), or NULL
    const double *inv_diag64;  // Jacobi 1/diag per cell (FP64 form)
    const float *inv_diag32;   // Jacobi 1/diag per cell (mixed form)
    double *partials;          // 2 x 8 x gridDim.x partials
    mb_ctrl *ctrl;
    unsigned *bar;             // [0] arrivals since launch (zeroed before each launch)
    int *status;
    mb_step_end end;           // the loop step's end, by the thread that writes the result
};

// The end of a loop step: the solve's record, the NaN flag, periodic stimuli and
// the clock (monodomain_solver.c:746,907-908).
__device__ __forceinline__ void step_end(mb_ctrl *c, const mb_step_end &e) {
    if (e.log && c->count >= 0 && c->count < e.log_len) {
        mb_step_stats s;
        s.cg_iterations = c->its;
        s.refinements = c->refinements;
        s.cg_error = c->error;
        e.log[c->count] = s;
    }
    if (isnan(c->error)) c->nan_flag = 1;
    double time = c->cur_time;
    for (int j = 0; j < e.num_steps; ++j) time += e.dt_ode;
    for (int k = 0; k < c->num_stims; ++k) {
        if (c->stim_period[k] > 0.0 && time >= c->stim_start[k] + c->stim_period[k])
            c->stim_start[k] = c->stim_start[k] + c->stim_period[k];
    }
    c->count += 1;
    c->cur_time += e.dt_pde;
}

// Grid-wide sum of NV per-thread values.  Every block reduces its threads
// (warp shuffles, then one warp over the per-warp sums), stores its partials
// and counts its arrival (release).  The arrival counter only grows during a
// launch: the r-th reduction is complete when it reaches (r + 1) x blocks.
// Each block then adds all partials itself, in block order and with the same
// shuffle tree, so every block holds bit-identical totals without a second
// hand-off.  Partials alternate between two buffers, so a fast block never
// overwrites values a slow block has still to read.  Waits are bounded: after
// SPIN_LIMIT polls the block records MB_ERR_CUDA in the status word and
// returns false (the caller leaves the kernel).
template <int NV, int NT>
__device__ __forceinline__ bool grid_reduce(const Args &a, double (&v)[NV], double (&out)[NV], int &red) {
    static_assert(NV >= 1 && NV <= 8, "the partials hold up to 8 values per block");
    // partials loaded per lane before the adds (fewer for many values)
    constexpr int J = NV <= 4 ? 8 : 4;
    __shared__ double sm[NV][NT / 32];
    __shared__ double tot[NV];
    __shared__ int flag;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *part = a.partials + (size_t)(red & 1) * 8 * gridDim.x;
    const unsigned target = (unsigned)(red + 1) * gridDim.x;
    red++;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
        if (lane == 0) sm[q][warp] = v[q];
    }
    __syncthreads();
    if (warp == 0) {
        cuda::atomic_ref<unsigned, cuda::thread_scope_device> arrive(a.bar[0]);
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            double s = lane < (int)(blockDim.x >> 5) ? sm[q][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) part[(size_t)q * gridDim.x + blockIdx.x] = s;
        }
        int ok = 1;
        if (lane == 0) {
            arrive.fetch_add(1u, cuda::memory_order_release);
            long long spins = 0;
            while (arrive.load(cuda::memory_order_acquire) < target) {
                if (++spins > SPIN_LIMIT) {
                    atomicExch(a.status, MB_ERR_CUDA);
                    ok = 0;
                    break;
                }
                if (spins > 4096) __nanosleep(32);
            }
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        // every lane that reads the partials orders its reads after the
        // arrivals lane 0 observed
        cuda::atomic_thread_fence(cuda::memory_order_acquire, cuda::thread_scope_device);
        if (ok) {
            // every partial of a chunk of up to 32 J blocks is loaded before
            // any is added, so the reads cost one L2 round trip, not one per value
            double s[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) s[q] = 0.0;
            for (unsigned base = 0; base < gridDim.x; base += 32 * J) {
                double vals[NV][J];
#pragma unroll
                for (int q = 0; q < NV; ++q)
#pragma unroll
                    for (int j = 0; j < J; ++j) {
                        const unsigned bk = base + lane + 32 * j;
                        vals[q][j] = bk < gridDim.x ? __ldcg(&part[(size_t)q * gridDim.x + bk]) : 0.0;
                    }
#pragma unroll
                for (int q = 0; q < NV; ++q)
#pragma unroll
                    for (int j = 0; j < J; ++j) s[q] += vals[q][j];
            }
#pragma unroll
            for (int q = 0; q < NV; ++q) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
                if (lane == 0) tot[q] = s[q];
            }
        }
        if (lane == 0) flag = ok;
    }
    __syncthreads();
    if (!flag) return false;
    // tot, sm and flag are next written only after the next reduction's first
    // __syncthreads, which every thread reaches after reading them here
#pragma unroll
    for (int q = 0; q < NV; ++q) out[q] = tot[q];
    return true;
}

// The sum of 8 values over a warp: halves are exchanged, so that a lane carries one
// value after three steps (18 shuffles, not 80).  Returns, in lanes 4 i .. 4 i + 3,
// the sum of value i.
__device__ __forceinline__ double warp_sum8(const double (&v)[8]) {
    const unsigned lane = threadIdx.x & 31u;
    double a4[4], a2[2];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const bool up = (lane & 16u) != 0u;
        const double keep = up ? v[q + 4] : v[q], give = up ? v[q] : v[q + 4];
        a4[q] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const bool up = (lane & 8u) != 0u;
        const double keep = up ? a4[q + 2] : a4[q], give = up ? a4[q] : a4[q + 2];
        a2[q] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
    }
    const bool up = (lane & 4u) != 0u;
    const double keep = up ? a2[1] : a2[0], give = up ? a2[0] : a2[1];
    double s = keep + __shfl_xor_sync(0xffffffffu, give, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    return s;
}

// grid_reduce for 8 values: the same arrivals, partials (8 per block, together)
// and bounded wait; the warps' sums by warp_sum8 and the blocks' partials read with a
// value per lane, so that the shuffles do not grow with the number of values.
template <int NT>
__device__ __forceinline__ bool grid_reduce8(const Args &a, double (&v)[8], int &red) {
    __shared__ double sm[NT / 32][8];
    __shared__ double tot[8];
    __shared__ int flag;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    double *part = a.partials + (size_t)(red & 1) * 8 * gridDim.x;
    const unsigned target = (unsigned)(red + 1) * gridDim.x;
    red++;
    const double s = warp_sum8(v);
    if ((lane & 3) == 0) sm[warp][lane >> 2] = s;
    __syncthreads();
    if (warp == 0) {
        const int q = lane & 7, h = lane >> 3;
        constexpr int W = (NT / 32 + 3) / 4;
        double w[W];
#pragma unroll
        for (int k = 0; k < W; ++k) w[k] = h + 4 * k < warps ? sm[h + 4 * k][q] : 0.0;
#pragma unroll
        for (int k = 1; k < W; ++k) w[0] += w[k];
        double t = w[0];
        t += __shfl_xor_sync(0xffffffffu, t, 8);
        t += __shfl_xor_sync(0xffffffffu, t, 16);
        if (h == 0) part[(size_t)blockIdx.x * 8 + q] = t;
        __syncwarp();
        cuda::atomic_ref<unsigned, cuda::thread_scope_device> arrive(a.bar[0]);
        int ok = 1;
        if (lane == 0) {
            // the 8 lanes' partials are ordered before lane 0's release
            cuda::atomic_thread_fence(cuda::memory_order_acq_rel, cuda::thread_scope_device);
            arrive.fetch_add(1u, cuda::memory_order_release);
            long long spins = 0;
            while (arrive.load(cuda::memory_order_acquire) < target) {
                if (++spins > SPIN_LIMIT) {
                    atomicExch(a.status, MB_ERR_CUDA);
                    ok = 0;
                    break;
                }
                if (spins > 4096) __nanosleep(32);
            }
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
        cuda::atomic_thread_fence(cuda::memory_order_acquire, cuda::thread_scope_device);
        if (ok) {
            constexpr int J = 10;           // 40 blocks' partials in flight per value
            double acc[J];
#pragma unroll
            for (int j = 0; j < J; ++j) acc[j] = 0.0;
            for (unsigned base = h; base < gridDim.x; base += 4 * J) {
                double vals[J];
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    const unsigned bk = base + 4 * j;
                    vals[j] = bk < gridDim.x ? __ldcg(&part[(size_t)bk * 8 + q]) : 0.0;
                }
#pragma unroll
                for (int j = 0; j < J; ++j) acc[j] += vals[j];
            }
            double u = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7])) + (acc[8] + acc[9]);
            u += __shfl_xor_sync(0xffffffffu, u, 8);
            u += __shfl_xor_sync(0xffffffffu, u, 16);
            if (h == 0) tot[q] = u;
        }
        if (lane == 0) flag = ok;
    }
    __syncthreads();
    if (!flag) return false;
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = tot[q];
    return true;
}

// bit 6 of a cell's code byte: the cell is active
constexpr unsigned ACTIVE = 64u;

}  // namespace fcg
}  // namespace mb
