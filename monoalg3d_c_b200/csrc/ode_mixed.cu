// Mixed-precision cell-model kernels: right-hand sides in FP32 with the
// hardware exp2/log2 approximations (this file is compiled with
// MB_FAST_FP32_MATH, -ftz=true, -prec-div=false), V and the ion
// concentrations accumulated in FP64.
#include "ode_common.cuh"

using namespace mb;

extern "C" int mbk_ode_step_mixed(const mb_ode_dev *o, mb_ctrl *ctrl, const double *vin, double *vout,
                                  cudaStream_t s) {
    if (o->n == 0) return 0;
    const unsigned blocks = (o->n + ODE_THREADS - 1) / ODE_THREADS;
    const mb_ode_dev &a = *o;
#define MB_STAGED(KERNEL, N64, N32)                                                       \
    do {                                                                                  \
        const size_t sm = staged_smem(N64, N32);                                          \
        auto *kfn = KERNEL;                                                               \
        const unsigned gb = staged_grid((const void *)kfn, sm, blocks);                   \
        if (!gb) return (int)cudaErrorInvalidConfiguration;                               \
        kfn<<<gb, ODE_THREADS, sm, s>>>(a, ctrl, vin, vout);                              \
    } while (0)
    if (o->model == MB_MODEL_TT2006) {
#define L(MB) k_tt2006_mixed<MB><<<blocks, ODE_THREADS, 0, s>>>(a, ctrl, vin, vout)
#define LS(MB) MB_STAGED(k_tt2006_mixed_s<MB>, 6, 13)
        MB_VARIANT_SWITCH(o->variant, L, LS)
#undef L
#undef LS
    } else {
        // Variants 0 and 1 keep the state in registers (any number of
        // sub-steps), 2..5 copy it to shared memory first, 6..9 are staged
        // persistent launches; several sub-steps per call take 0 or 1.
#define L(R, K, MB) k_torord_mixed##K<R, MB><<<blocks, ODE_THREADS, 0, s>>>(a, ctrl, vin, vout)
#define LS(R, MB) MB_STAGED((k_torord_mixed_s<R, MB>), TOR_N64, TOR_N32)
#define ALL(R)                                                        \
    switch (o->num_steps > 1 && o->variant > 1 ? 1 : o->variant) {    \
    case 0: L(R, , 1); break;                                         \
    case 1: L(R, , 4); break;                                         \
    case 2: L(R, _slots, 4); break;                                   \
    case 3: L(R, _slots, 5); break;                                   \
    case 4: L(R, _slots, 6); break;                                   \
    case 5: L(R, _slots, 7); break;                                   \
    case 6: LS(R, 1); break;                                          \
    case 7: LS(R, 2); break;                                          \
    case 8: LS(R, 3); break;                                          \
    default: LS(R, 4); break;                                         \
    }
        if (o->rl_rule == MB_RL_TRUE) {
            ALL(MB_RL_TRUE)
        } else {
            ALL(MB_RL_REFERENCE_CPU)
        }
#undef ALL
#undef L
#undef LS
    }
#undef MB_STAGED
    return (int)cudaGetLastError();
}
