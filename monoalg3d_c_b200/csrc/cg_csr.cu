// Jacobi-PCG on a general CSR matrix as one cooperative kernel per solve
// (mb_csr_solve): the iteration and stopping rule of cpu_conjugate_gradient
// (linear_system_solver.c:47-183), one reduction and one barrier per iteration.
//
// Why: with a kernel per phase (cg_kernels.cu:k_csr_*) an iteration is three launches
// with their gaps, and the host reads the stopping flag back every 16 iterations: 30 us
// an iteration on a 200 k-row 7-point matrix whose 17 MB stay in L2, 16 us here.
//
// A part of a warp (LANES lanes) takes a row, so that its entries are read
// as whole sectors, R rows at a time: bound by the latency of row pointer, entry and
// vector value, one after the other.  R = 4 takes 108
// registers, one block per SM: 16 us an iteration at 200 k rows, 22 us with one row at a
// time, 18 and 17 us with R = 2 and 8.  Bound to 64 registers, two blocks per SM, it is
// faster on large matrices (600 k rows 26 us, 33 here) and slower on small ones (50 k rows 12
// us, 9 here).  Once matrix and vectors leave L2 a thread per row in the phases' kernels
// keeps more rows in flight (mbk_csr_in_l2).
// Per iteration: x, r and p of the rows, a grid barrier (p of
// other rows is read next), then q = A p and the sums p.q, q.z, q.Mq, q.r, q.q,
// r.z, r.r for the next r.z and r.r (cg_cluster.cu, with its guard).
#include <type_traits>
#include "cg_common.cuh"

namespace mb {
namespace csr {

using fcg::Args;
using fcg::grid_reduce8;
using fcg::SPIN_LIMIT;

constexpr int NT = 512;
constexpr int R = 4;
constexpr double GUARD = 1e-4;

// Grid-wide barrier on the reductions' arrival counter.
__device__ __forceinline__ bool grid_barrier(const Args &a, int &red) {
    __shared__ int flag;
    const unsigned target = (unsigned)(red + 1) * gridDim.x;
    red++;
    __syncthreads();
    if (threadIdx.x == 0) {
        cuda::atomic_ref<unsigned, cuda::thread_scope_device> arrive(a.bar[0]);
        cuda::atomic_thread_fence(cuda::memory_order_acq_rel, cuda::thread_scope_device);
        arrive.fetch_add(1u, cuda::memory_order_release);
        long long spins = 0;
        int ok = 1;
        while (arrive.load(cuda::memory_order_acquire) < target) {
            if (++spins > SPIN_LIMIT) {
                atomicExch(a.status, MB_ERR_CUDA);
                ok = 0;
                break;
            }
            if (spins > 4096) __nanosleep(32);
        }
        flag = ok;
    }
    __syncthreads();
    cuda::atomic_thread_fence(cuda::memory_order_acquire, cuda::thread_scope_device);
    return flag != 0;
}

template <int LANES>
__device__ __forceinline__ int row_max(int e) {
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    return e;
}

template <int LANES>
__device__ __forceinline__ double row_sum(double s) {
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

template <int LANES>
__global__ void __launch_bounds__(NT) k_csr_pcg(mb_csr_dev m, Args a) {
    mb_ctrl *c = a.ctrl;
    const bool pre = c->use_precond != 0;
    const double tol = c->tol;
    const int max_its = c->max_its;
    const int lane = threadIdx.x % LANES;
    const int per = gridDim.x * NT / LANES;
    const int first_row = (blockIdx.x * NT + threadIdx.x) / LANES;
    int red = 0;
    double v[8];
    auto zero = [&]() {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = 0.0;
    };
    // f(row, lane 0 of an existing row, the row's product with x).  R rows of a thread
    // at once, so that their entries are in flight together; every warp runs the same
    // number of rounds (the row sums' shuffles).
    auto rows = [&](const double *x, auto with_diag, auto f) {
        constexpr bool diag = decltype(with_diag)::value;
        for (int row0 = first_row; row0 - first_row % (32 / LANES) < m.n; row0 += R * per) {
            int e[R], e1[R], at[R];     // at: the row's diagonal entry (the last one, if it has several)
            double s[R];
            bool more = false;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int row = row0 + k * per;
                const bool in = row < m.n;
                e[k] = in ? m.row_ptr[row] + lane : 0;
                e1[k] = in ? m.row_ptr[row + 1] : 0;
                s[k] = 0.0;
                at[k] = -1;
            }
#pragma unroll
            for (int k = 0; k < R; ++k) more |= e[k] < e1[k];
            while (more) {
                int col[R];
                double val[R];
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    const bool in = e[k] < e1[k];
                    col[k] = in ? m.col[e[k]] : 0;
                    val[k] = in ? m.val[e[k]] : 0.0;
                }
                more = false;
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    if (e[k] < e1[k]) {
                        s[k] += val[k] * __ldcg(x + col[k]);
                        if (diag && col[k] == row0 + k * per) at[k] = e[k];
                    }
                    e[k] += LANES;
                    more |= e[k] < e1[k];
                }
            }
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int row = row0 + k * per;
                const double sum = row_sum<LANES>(s[k]);
                const int d = diag ? row_max<LANES>(at[k]) : -1;
                if (lane == 0 && row < m.n) f(row, sum, d >= 0 ? m.val[d] : 0.0);
            }
        }
    };
    zero();
    rows(m.x, std::true_type{}, [&](int row, double ax, double d) {
        const double id = 1.0 / (d == 0.0 ? 1.0 : d), r = m.b[row] - ax, z = pre ? id * r : r;
        m.inv_diag[row] = id;
        m.r[row] = r;
        m.p[row] = z;
        v[0] += r * z;
        v[1] += r * r;
    });
    if (!grid_reduce8<NT>(a, v, red)) return;
    double rz = v[0], rr = v[1], error = v[1], alpha = 0.0, beta = 0.0;
    int its = 1;
    bool done = !(error >= tol) || !(1 < max_its), first = true, updated = false;
    // the rows a thread owns in the streaming parts
    const int t0 = blockIdx.x * NT + threadIdx.x, step = gridDim.x * NT;
    while (!done) {
        if (!first) {
            for (int row = t0; row < m.n; row += step) {
                const double p = m.p[row];
                m.x[row] += alpha * p;
                double r = m.r[row];
                if (!updated) {
                    r -= alpha * m.q[row];
                    m.r[row] = r;
                }
                m.p[row] = (pre ? m.inv_diag[row] * r : r) + beta * p;
            }
            if (!grid_barrier(a, red)) return;
        }
        zero();
        rows(m.p, std::false_type{}, [&](int row, double q, double) {
            const double r = __ldcg(m.r + row), id = pre ? __ldcg(m.inv_diag + row) : 1.0, z = id * r;
            m.q[row] = q;
            v[0] += __ldcg(m.p + row) * q;
            v[1] += q * z;
            v[2] += q * (id * q);
            v[3] += q * r;
            v[4] += q * q;
            v[5] += r * z;
            v[6] += r * r;
        });
        if (!grid_reduce8<NT>(a, v, red)) return;
        rz = v[5];
        rr = v[6];
        alpha = (pre ? rz : rr) / v[0];
        double rzn = rz - alpha * (2.0 * v[1] - alpha * v[2]), rrn = rr - alpha * (2.0 * v[3] - alpha * v[4]);
        its += 1;
        updated = false;
        if (!(rrn > GUARD * rr && rzn > GUARD * rz)) {
            zero();
            for (int row = t0; row < m.n; row += step) {
                const double r = m.r[row] - alpha * __ldcg(m.q + row);
                m.r[row] = r;
                v[0] += r * (pre ? m.inv_diag[row] * r : r);
                v[1] += r * r;
            }
            if (!grid_reduce8<NT>(a, v, red)) return;
            rzn = v[0];
            rrn = v[1];
            updated = true;
        }
        error = rrn;
        done = rrn <= tol || its >= max_its;
        beta = pre ? rzn / rz : rrn / rr;
        first = false;
    }
    if (!first)
        for (int row = t0; row < m.n; row += step) m.x[row] += alpha * m.p[row];
    if (t0 == 0) {
        c->its = its;
        c->error = error;
        c->done = 1;
    }
}

}  // namespace csr
}  // namespace mb

using namespace mb::csr;

// Lanes per row: its entries in a few sectors each.
static int lanes_of(int32_t n, int32_t nnz) { return nnz / n <= 16 ? 4 : 16; }
static const void *kernel_of(int32_t n, int32_t nnz) {
    return lanes_of(n, nnz) == 4 ? (const void *)k_csr_pcg<4> : (const void *)k_csr_pcg<16>;
}

// Blocks of the cooperative launch: all that fit at once, no more than the rows
// give work.
extern "C" int mbk_csr_pcg_blocks(int32_t n, int32_t nnz) {
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel_of(n, nnz), NT, 0) != cudaSuccess || per < 1) return -1;
    const long long want = ((long long)n * lanes_of(n, nnz) + NT - 1) / NT;
    const int most = sms * (per > 2 ? 2 : per);
    return want < most ? (int)want : most;
}

// Whether the one-launch solve is the faster: while the matrix (12 B an entry) and the
// vectors (56 B a row) stay in L2.  Measured per iteration, here and by phases: 600 k rows
// of 7 entries (84 MB) 34 and 43 us, 50 k rows of 152 (94 MB) 37 and 58 us, but 200 k
// rows of 38 (105 MB) 60 and 56 us, 900 k rows of 7 (125 MB) 76 and 64 us, 2 M rows 186 and
// 116 us.
extern "C" int mbk_csr_in_l2(int32_t n, int32_t nnz) {
    return 12LL * nnz + 56LL * n <= (96LL << 20);
}

// bar: 2 words; partials: 16 values per block.
extern "C" int mbk_csr_pcg(const mb_csr_dev *m, int32_t nnz, int blocks, mb_ctrl *ctrl, double *partials, unsigned *bar,
                           int *status, cudaStream_t s) {
    Args a{};
    a.partials = partials;
    a.ctrl = ctrl;
    a.bar = bar;
    a.status = status;
    cudaError_t e = cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), s);
    if (e != cudaSuccess) return (int)e;
    mb_csr_dev dev = *m;
    void *args[] = {&dev, &a};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(NT);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return (int)cudaLaunchKernelExC(&cfg, kernel_of(m->n, nnz), args);
}
