// Kernels of the discrete adjoint of the monodomain step (ten Tusscher 2006,
// per-cell conductivity, FP64).
//
// One loop step maps (v_n, s_n) to v_{n+1} through
//     (V*, s_{n+1}) = Phi(v_n, s_n; theta)       Rush-Larsen sub-step
//     A(sigma) v_{n+1} = alpha V*                implicit diffusion
// and its adjoint, run backwards, maps (lambda_{n+1} = dL/dv_{n+1},
// mu_{n+1} = dL/ds_{n+1}) to (lambda_n, mu_n):
//     A w = lambda_{n+1}                          (A is symmetric: the same PCG)
//     dL/dsigma += -(w_a - w_b)(v_a - v_b) dF_ab/dsigma  over faces ab
//     (lambda_n, mu_n, dL/dtheta) = J_Phi^T (alpha w, mu_{n+1})
// J_Phi^T g is formed by one reverse sweep over the model's expression graph
// (adj_cell): the gates' steady states and time constants, functions of V
// alone, are differentiated by one forward-mode dual pass through the model
// code the forward kernels run (tt2006_gate_rates), everything else by hand.
#include <cstdint>
#include <cuda_runtime.h>
#include "mb_internal.h"
#include "ode_common.cuh"

MB_NS_BEGIN

// ---- dual numbers (value and derivative with respect to one input) ---------------

// value type T: double for the FP64 forward, float for the mixed one
template <typename T = double>
struct Dual {
    T v, d;
    __device__ __forceinline__ Dual() {}
    __device__ __forceinline__ Dual(double x) : v((T)x), d(T(0)) {}
    __device__ __forceinline__ Dual(T x, T dx) : v(x), d(dx) {}
};

#define MB_DUAL template <typename T> __device__ __forceinline__
MB_DUAL Dual<T> operator+(const Dual<T> &a, const Dual<T> &b) { return Dual<T>(a.v + b.v, a.d + b.d); }
MB_DUAL Dual<T> operator-(const Dual<T> &a, const Dual<T> &b) { return Dual<T>(a.v - b.v, a.d - b.d); }
MB_DUAL Dual<T> operator*(const Dual<T> &a, const Dual<T> &b) { return Dual<T>(a.v * b.v, a.d * b.v + a.v * b.d); }
MB_DUAL Dual<T> operator-(const Dual<T> &a) { return Dual<T>(-a.v, -a.d); }
MB_DUAL bool operator<(const Dual<T> &a, const Dual<T> &b) { return a.v < b.v; }
// the value-type functions of mb_math.cuh
MB_DUAL Dual<T> mrcp(const Dual<T> &a) {
    const T y = mrcp(a.v);
    return Dual<T>(y, -y * y * a.d);
}
MB_DUAL Dual<T> mdiv(const Dual<T> &a, const Dual<T> &b) {
    const T q = mdiv(a.v, b.v);
    return Dual<T>(q, (a.d - q * b.d) * mrcp(b.v));
}
MB_DUAL Dual<T> mexp(const Dual<T> &a) {
    const T e = mexp(a.v);
    return Dual<T>(e, e * a.d);
}
MB_DUAL Dual<T> msqrt(const Dual<T> &a) {
    const T s = msqrt(a.v);
    return Dual<T>(s, mdiv(T(0.5), s) * a.d);
}
#undef MB_DUAL

// ---- ODE adjoint ----------------------------------------------------------------

constexpr int ADJ_THREADS = 128;
constexpr int ADJ_IN = TT_NEQ + 1;      // the 19 states and the gKr scaling

// res = J_Phi^T g for one cell: Phi the Rush-Larsen sub-step of
// tt2006_rhs at state y, res[j] = sum_i g_i d(out_i)/d(in_j) with inputs 0..18
// the states (0 = V) and input 19 the gKr scaling.  T is the arithmetic of the
// forward step (double; float for the mixed form, whose right-hand side is
// FP32): model values and local derivatives are in T, the adjoint values they
// are contracted with are FP64.
//
// What bounds it is the FP64 pipe and the latency of its chains (254 registers, two
// warps per scheduler).  The sweep costs about three evaluations
// of the model: 21 us per step on a 256 x 256 sheet in FP64 and 18 us on a
// 97 x 131 sheet in FP32, against 1876 and 239 us for J column block by column
// block with forward-mode duals (the model and two tangents, ten times).
template <typename T>
__device__ __forceinline__ void adj_cell(const T (&y)[TT_NEQ], const TTScale<T> &sc, T dt, const double (&g)[TT_NEQ],
                                         double (&res)[ADJ_IN]) {
    const T V = y[TT_V];
    const T Ca_i = y[TT_CAI], Ca_SR = y[TT_CASR], Ca_ss = y[TT_CASS], Rp = y[TT_RPRIME];
    const T Na_i = y[TT_NAI], K_i = y[TT_KI];
    const T R = T(8314.472), Tk = T(310.0), F = T(96485.3415f), RTF = (R * Tk) / F, FRT = F / (R * Tk);
    const T Cm = T(0.185), V_c = T(0.016404), V_sr = T(0.001094f), V_ss = T(5.468e-05f);
    const T Ko = T(5.4), Nao = T(140.0), Cao = T(2.0);
    const double dtd = (double)dt;

    // Euler states pass their own adjoint on; a = adjoint of the derivatives
    double bV = g[TT_V], bcai = g[TT_CAI], bsr = g[TT_CASR], bss = g[TT_CASS], brp = g[TT_RPRIME];
    double bnai = g[TT_NAI], bki = g[TT_KI];
    const double aV = dtd * g[TT_V], aCai = dtd * g[TT_CAI], aSR = dtd * g[TT_CASR], aSS = dtd * g[TT_CASS];
    const double aRp = dtd * g[TT_RPRIME], aNai = dtd * g[TT_NAI], aKi = dtd * g[TT_KI];

    // buffers and their derivatives
    const T K_buf_c = T(0.001f), K_buf_sr = T(0.3f), K_buf_ss = T(0.00025f);
    const T qc = T(0.2f) * K_buf_c, qsr = T(10.0f) * K_buf_sr, qss = T(0.4f) * K_buf_ss;
    const T cbc = Ca_i + K_buf_c, cbs = Ca_SR + K_buf_sr, cbss = Ca_ss + K_buf_ss;
    const T ic = mrcp(cbc * cbc + qc), isr = mrcp(cbs * cbs + qsr), iss = mrcp(cbss * cbss + qss);
    const T Bc = cbc * cbc * ic, Bsr = cbs * cbs * isr, Bss = cbss * cbss * iss;

    // adjoints of the currents
    const double kNa = (double)(Cm / (V_c * F)), kCa = 0.5 * kNa * (double)Bc;
    const double kss = (double)(Cm / (T(2) * V_ss * F) * Bss);
    const double bK = -aV - aKi * kNa;                  // IK1, Ito, IKr, IKs, IpK
    const double bNa = -aV - aNai * kNa;                // INa, IbNa
    const double bNaK = -aV - 3.0 * aNai * kNa + 2.0 * aKi * kNa;
    const double bNaCa = -aV - 3.0 * aNai * kNa + 2.0 * aCai * kCa;
    const double bCa = -aV - aCai * kCa;                // IbCa, IpCa
    const double bCaL = -aV - aSS * kss;

    // potassium currents
    const T vek = V - RTF * mlog(mdiv(Ko, K_i));
    {
        const T e1 = mexp(T(0.0002f) * (vek + T(100))), e2 = mexp(T(0.1f) * (vek - T(10))), e3 = mexp(T(-0.5f) * vek);
        const T ea = mexp(T(0.06f) * (vek - T(200)));
        const T d3 = mrcp(T(1) + e3), da = mrcp(T(1) + ea);
        const T be = (T(3) * e1 + e2) * d3, al = T(0.1f) * da;
        const T dbe = (T(3) * T(0.0002f) * e1 + T(0.1f) * e2) * d3 + T(0.5f) * e3 * d3 * be;
        const T dal = -T(0.06f) * ea * da * al;
        const T s = mrcp(al + be), x = al * s;
        const T dx = (dal * be - al * dbe) * s * s;
        const T xr1 = y[TT_XR1], xr2 = y[TT_XR2], xs = y[TT_XS], r = y[TT_R], sg = y[TT_S];
        const T gto = T(0.294), gpk = T(0.0146), gkr0 = T(0.153) * T(TT_SQRT_KO), gkr = gkr0 * sc.gKr;
        const T ep = mexp(MB_OVER(T(25) - V, (double)5.98f)), dp = mrcp(T(1) + ep);
        const double bvek = bK * (double)(T(5.405) * sc.gK1 * (x + vek * dx) + gto * r * sg + gkr * xr1 * xr2 + gpk * dp);
        bV += bvek + bK * (double)(gpk * vek * MB_OVER(ep, (double)5.98f) * dp * dp);
        bki += bvek * (double)mdiv(RTF, K_i);
        res[TT_R] = bK * (double)(gto * sg * vek);
        res[TT_S] = bK * (double)(gto * r * vek);
        res[TT_XR1] = bK * (double)(gkr * xr2 * vek);
        res[TT_XR2] = bK * (double)(gkr * xr1 * vek);
        res[TT_NEQ] = bK * (double)(gkr0 * xr1 * xr2 * vek);
        const T gks = T(0.098) * sc.gKs, ks = K_i + T(0.03) * Na_i;
        const T iks = mrcp(ks), vks = V - RTF * mlog(mdiv(Ko + T(0.03) * Nao, ks));
        res[TT_XS] = bK * (double)(gks * T(2) * xs * vks);
        const double t = bK * (double)(gks * xs * xs);
        bV += t;
        bki += t * (double)(RTF * iks);
        bnai += t * (double)(RTF * T(0.03) * iks);
    }
    // sodium currents
    {
        const T m = y[TT_M], h = y[TT_H], j = y[TT_J], gna = T(14.838) * sc.gNa;
        const T vna = V - RTF * mlog(mdiv(Nao, Na_i));
        res[TT_M] = bNa * (double)(gna * T(3) * m * m * h * j * vna);
        res[TT_H] = bNa * (double)(gna * (m * m * m) * j * vna);
        res[TT_J] = bNa * (double)(gna * (m * m * m) * h * vna);
        const double t = bNa * (double)(gna * (m * m * m) * h * j + T(0.00029));
        bV += t;
        bnai += t * (double)mdiv(RTF, Na_i);
    }
    // sodium-potassium pump
    {
        const T e1 = mexp(T(-0.1f) * V * FRT), e2 = mexp(-V * FRT);
        const T D = mrcp(T(1) + T(0.1245f) * e1 + T(0.0353f) * e2);
        const T P = T(2.724) * Ko / (Ko + T(1)), na = mrcp(Na_i + T(40));
        bnai += bNaK * (double)(P * T(40) * na * na * D);
        bV += bNaK * (double)(P * Na_i * na * D * D * FRT * (T(0.1245f) * T(0.1f) * e1 + T(0.0353f) * e2));
    }
    // sodium-calcium exchanger
    T INaCa;
    {
        const T n = T(0.35), nm1 = n - T(1), na3 = Na_i * Na_i * Na_i, nao3 = Nao * Nao * Nao;
        const T ep = mexp(n * V * FRT), em = mexp(nm1 * V * FRT);
        const T C = (T(87.5) * T(87.5) * T(87.5) + nao3) * (T(1.38) + Cao);
        const T D = mrcp(T(1) + T(0.1) * em), k = T(1000) / C * D;
        const T in = ep * na3 * Cao, out = em * nao3 * Ca_i * T(2.5);
        INaCa = k * (in - out);
        bnai += bNaCa * (double)(k * T(3) * ep * (Na_i * Na_i) * Cao);
        bcai -= bNaCa * (double)(k * em * nao3 * T(2.5));
        bV += bNaCa * (double)(k * FRT * ((n * in - nm1 * out) - (in - out) * T(0.1) * nm1 * em * D));
    }
    // calcium background, pump and L-type currents
    {
        const double t = bCa * (double)T(0.000592);
        bV += t;
        bcai += t * (double)mdiv(T(0.5f) * RTF, Ca_i);
        const T kp = mrcp(Ca_i + T(0.0005));
        bcai += bCa * (double)(T(0.1238) * T(0.0005) * kp * kp);
        const T v15 = V - T(15.0f), d = y[TT_D], f = y[TT_F], f2 = y[TT_F2], fc = y[TT_FCASS];
        const T gca = T(3.98e-05) * sc.gCaL;
        T G, GV, Gc;
        if (V < T(15.0f - 1.0e-5f) || V > T(15.0f + 1.0e-5f)) {
            const T k = T(2) * FRT, e = mexp(k * v15), im = mrcp(mexpm1(k * v15)), c = T(4) * F * FRT;
            const T A = T(0.25f) * Ca_ss * e - Cao;
            G = c * v15 * A * im;
            Gc = c * v15 * T(0.25f) * e * im;
            GV = c * im * (A + v15 * k * e * (T(0.25f) * Ca_ss - A * im));
        } else {                                        // the band's limit value does not depend on V
            G = T(2) * F * (T(0.25f) * Ca_ss - Cao);
            Gc = T(2) * F * T(0.25f);
            GV = T(0);
        }
        const T gd = gca * d * f * f2 * fc;
        bV += bCaL * (double)(gd * GV);
        bss += bCaL * (double)(gd * Gc);
        res[TT_D] = bCaL * (double)(gca * f * f2 * fc * G);
        res[TT_F] = bCaL * (double)(gca * d * f2 * fc * G);
        res[TT_F2] = bCaL * (double)(gca * d * f * fc * G);
        res[TT_FCASS] = bCaL * (double)(gca * d * f * f2 * G);
        // the buffered compartments: what multiplies Bc, Bsr and Bss
        const T K_up2 = T(0.00025) * T(0.00025), V_rel = T(0.102), k3 = T(0.06), k4 = T(0.005f);
        const T iu = mrcp(Ca_i * Ca_i + K_up2), i_up = T(0.006375) * (Ca_i * Ca_i * iu);
        const T i_leak = T(0.00036f) * (Ca_SR - Ca_i), i_xfer = T(0.0038f) * (Ca_ss - Ca_i);
        const T iq = mrcp(Ca_SR * Ca_SR + T(1.5) * T(1.5));
        const T kc = T(2.5) - T(1.5) * (Ca_SR * Ca_SR * iq), ikc = mrcp(kc), k1 = T(0.15) * ikc;
        const T w = k1 * Ca_ss * Ca_ss, iw = mrcp(k3 + w), O = w * Rp * iw, grad = Ca_SR - Ca_ss;
        const T Irel = V_rel * O * grad;
        const T IbCa = T(0.000592) * (V - T(0.5f) * RTF * mlog(mdiv(Cao, Ca_i))), IpCa = T(0.1238) * Ca_i * kp;
        const T sc_ = (i_leak - i_up) * (V_sr / V_c) + i_xfer - (IbCa + IpCa - T(2) * INaCa) * (Cm / (T(2) * V_c * F));
        const T ssr = i_up - (Irel + i_leak);
        const T sss = -gd * G * (Cm / (T(2) * V_ss * F)) + Irel * (V_sr / V_ss) - i_xfer * (V_c / V_ss);
        bcai += aCai * (double)(sc_ * T(2) * qc * cbc * ic * ic);
        bsr += aSR * (double)(ssr * T(2) * qsr * cbs * isr * isr);
        bss += aSS * (double)(sss * T(2) * qss * cbss * iss * iss);
        // fluxes
        const double uc = aCai * (double)Bc, us = aSR * (double)Bsr, uss = aSS * (double)Bss;
        const double vr = (double)(V_sr / V_c);
        const double bup = us - uc * vr, bleak = uc * vr - us, bx = uc - uss * (double)(V_c / V_ss);
        const double brel = uss * (double)(V_sr / V_ss) - us;
        bcai += bup * (double)(T(0.006375) * T(2) * K_up2 * Ca_i * iu * iu);
        bsr += bleak * (double)T(0.00036f);
        bcai -= bleak * (double)T(0.00036f);
        bss += bx * (double)T(0.0038f);
        bcai -= bx * (double)T(0.0038f);
        // release: O and R'
        const double bO = brel * (double)(V_rel * grad);
        bsr += brel * (double)(V_rel * O);
        bss -= brel * (double)(V_rel * O);
        const double bw = bO * (double)(Rp * k3 * iw * iw);
        const T k2 = T(0.045f) * kc;
        brp += bO * (double)(w * iw) - aRp * (double)(k2 * Ca_ss + k4);
        bss += bw * (double)(T(2) * k1 * Ca_ss) - aRp * (double)(k2 * Rp);
        const double bkc = -aRp * (double)(T(0.045f) * Ca_ss * Rp) - bw * (double)(w * ikc);
        bsr -= bkc * (double)(T(1.5) * T(2) * T(1.5) * T(1.5) * Ca_SR * iq * iq);
    }
    // gates: inf + (y - inf) exp(-dt rate)
    {
        Dual<T> inf[12], rate[12];
        tt2006_gate_rates<Dual<T>>(Dual<T>(V, T(1)), Dual<T>(Ca_ss, T(0)), inf, rate);
        // fCass follows Ca_ss: inf = 0.6 / (1 + c^2) + 0.4, 1/rate = 80 / (1 + c^2) + 2, c = Ca_ss / 0.05
        const T c = MB_OVER(Ca_ss, (double)0.05f), fc = mrcp(T(1) + c * c), dc = -T(2) * MB_OVER(c, (double)0.05f) * fc * fc;
        inf[9].d = T(0.6f) * dc;
        rate[9].d = -T(80.0f) * dc * rate[9].v * rate[9].v;
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            const T E = mexp(-dt * rate[k].v);
            const double b = g[1 + k] * (double)((T(1) - E) * inf[k].d - (y[1 + k] - inf[k].v) * E * (dt * rate[k].d));
            if (k == 9) bss += b;
            else bV += b;
            res[1 + k] += g[1 + k] * (double)E;
        }
    }
    res[TT_V] = bV;
    res[TT_CAI] = bcai;
    res[TT_CASR] = bsr;
    res[TT_CASS] = bss;
    res[TT_RPRIME] = brp;
    res[TT_NAI] = bnai;
    res[TT_KI] = bki;
}

// Per compact cell t: y = (v_n, s_n) from a snapshot, g = (alpha w, mu_in);
// writes lambda_n (grid), mu_out (state rows 1..18) and adds dL/dgKr.
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_tt2006(mb_ode_dev o, const double *__restrict__ v_n,
                                                            const double *__restrict__ sv_n,
                                                            const double *__restrict__ w, double alpha,
                                                            const double *__restrict__ mu_in, double *mu_out,
                                                            double *lam_out, double *gth) {
    exp_table_fill();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= o.n) return;
    const uint32_t g = o.cell ? o.cell[t] : t;
    const size_t ld = o.ld;
    double y[TT_NEQ], gi[TT_NEQ];
    y[0] = v_n[g];
    gi[0] = alpha * w[g];
#pragma unroll
    for (int s = 1; s < TT_NEQ; ++s) {
        y[s] = sv_n[s * ld + t];
        gi[s] = mu_in[s * ld + t];
    }
    const TTScale<double> sc = load_tt_scale<double>(o, t);
    double res[ADJ_IN];
    adj_cell<double>(y, sc, o.dt, gi, res);
    lam_out[g] = res[0];
#pragma unroll
    for (int s = 1; s < TT_NEQ; ++s) mu_out[s * ld + t] = res[s];
    gth[t] += res[TT_NEQ];
}

// The same for the mixed forward (k_tt2006_mixed): the state from the mixed
// rows of the snapshot (FP64 rows 1..5 = Ca_i, Ca_SR, Ca_ss, Na_i, K_i; FP32
// rows 0..11 = the gates, row 12 = R'), the local derivatives in FP32,
// contracted and accumulated in FP64.
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_tt2006_mixed(mb_ode_dev o, const double *__restrict__ v_n,
                                                                  const double *__restrict__ sv64_n,
                                                                  const float *__restrict__ sv32_n,
                                                                  const double *__restrict__ w, double alpha,
                                                                  const double *__restrict__ mu_in, double *mu_out,
                                                                  double *lam_out, double *gth) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= o.n) return;
    const uint32_t g = o.cell ? o.cell[t] : t;
    const size_t ld = o.ld;
    float y[TT_NEQ];
    double gi[TT_NEQ];
    y[TT_V] = (float)v_n[g];
#pragma unroll
    for (int k = 0; k < 12; ++k) y[1 + k] = sv32_n[k * ld + t];
    y[TT_CAI] = (float)sv64_n[1 * ld + t];
    y[TT_CASR] = (float)sv64_n[2 * ld + t];
    y[TT_CASS] = (float)sv64_n[3 * ld + t];
    y[TT_NAI] = (float)sv64_n[4 * ld + t];
    y[TT_KI] = (float)sv64_n[5 * ld + t];
    y[TT_RPRIME] = sv32_n[12 * ld + t];
    gi[0] = alpha * w[g];
#pragma unroll
    for (int s = 1; s < TT_NEQ; ++s) gi[s] = mu_in[s * ld + t];
    const TTScale<float> sc = load_tt_scale<float>(o, t);
    double res[ADJ_IN];
    adj_cell<float>(y, sc, (float)o.dt, gi, res);
    lam_out[g] = res[0];
#pragma unroll
    for (int s = 1; s < TT_NEQ; ++s) mu_out[s * ld + t] = res[s];
    gth[t] += res[TT_NEQ];
}

// ---- conductivity gradient ---------------------------------------------------

// dL/dsigma_c += sum over the coupled faces of c of -(w_c - w_n)(v_c - v_n)
// m dH/dsigma_c, with H = 2 s_c s_n / (s_c + s_n) the face conductivity
// (fill_discretization_matrix_elements, assembly_common.c:969-991) and m the
// face's area / distance.
__global__ void k_adj_face_grad(mb_stencil_dev st, const double *__restrict__ sigma, const double *__restrict__ w,
                                const double *__restrict__ v, double mx, double my, double mz, double *gsig) {
    const uint32_t n = (uint32_t)st.nx * st.ny * st.nz;
    const uint32_t sy = st.nx, sz = (uint32_t)st.nx * st.ny;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
        const unsigned m = st.code[g];
        if (!(m & 64u)) continue;
        const double sa = sigma[g], wa = w[g], va = v[g];
        const uint32_t nb[6] = {g - 1, g + 1, g - sy, g + sy, g - sz, g + sz};
        const double mult[6] = {mx, mx, my, my, mz, mz};
        double acc = 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            if (!((m >> q) & 1u)) continue;
            const double sb = sigma[nb[q]];
            if (sa == 0.0 || sb == 0.0) continue;
            const double s = sa + sb;
            const double dh = 2.0 * sb * sb / (s * s);
            acc += -(wa - w[nb[q]]) * (va - v[nb[q]]) * mult[q] * dh;
        }
        gsig[g] += acc;
    }
}

// ---- sensors, tolerance ----------------------------------------------------------

__global__ void k_adj_gather(const double *v, const int64_t *cells, int ns, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ns) out[i] = v[cells[i]];
}

__global__ void k_adj_scatter(double *lam, const int64_t *cells, int ns, const double *gsrc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ns) atomicAdd(&lam[cells[i]], gsrc[i]);
}

// tol of the transposed solve: rel^2 x (lambda . lambda), floored so that an all-zero
// right-hand side stops at once.  Every block leaves its partial sum, the last one
// to finish adds them in block order (part: TOL_BLOCKS values and, after them, the
// arrival count, zero between calls).  One block alone took 13 us on 65 k cells.
constexpr int TOL_BLOCKS = 64;

__global__ void __launch_bounds__(256) k_adj_tol(const double *lam, int64_t n, double rel2, mb_ctrl *c, double *part) {
    __shared__ double sm[8];
    __shared__ bool last;
    unsigned *count = reinterpret_cast<unsigned *>(part + TOL_BLOCKS);
    double s = 0.0;
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n; g += (int64_t)gridDim.x * blockDim.x)
        s += lam[g] * lam[g];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += sm[w];
        part[blockIdx.x] = t;
        __threadfence();
        last = atomicAdd(count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x >= 32) return;
    __threadfence();
    s = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += 32) s += __ldcg(part + b);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) {
        *count = 0;
        c->tol = c->refine_floor = fmax(rel2 * s, 1e-300);
    }
}

// A snapshot of the loop state, or one put back: up to four arrays of 16-byte
// words in one launch (a copy each cost a launch each).
struct CopyList {
    const uint4 *src[4];
    uint4 *dst[4];
    int64_t words[4];
};
__global__ void __launch_bounds__(256) k_copy4(CopyList l) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        for (int64_t i = t0; i < l.words[q]; i += step) l.dst[q][i] = l.src[q][i];
}

MB_NS_END

using namespace mb;

extern "C" int mbk_adj_tt2006(const mb_ode_dev *o, const double *v_n, const double *sv_n,
                              const double *w, double alpha, const double *mu_in, double *mu_out, double *lam_out,
                              double *gth, cudaStream_t s) {
    const unsigned blocks = (o->n + ADJ_THREADS - 1) / ADJ_THREADS;
    k_adj_tt2006<<<blocks, ADJ_THREADS, 0, s>>>(*o, v_n, sv_n, w, alpha, mu_in, mu_out, lam_out, gth);
    return (int)cudaGetLastError();
}

extern "C" int mbk_adj_tt2006_mixed(const mb_ode_dev *o, const double *v_n,
                                    const double *sv64_n, const float *sv32_n, const double *w, double alpha,
                                    const double *mu_in, double *mu_out, double *lam_out, double *gth, cudaStream_t s) {
    const unsigned blocks = (o->n + ADJ_THREADS - 1) / ADJ_THREADS;
    k_adj_tt2006_mixed<<<blocks, ADJ_THREADS, 0, s>>>(*o, v_n, sv64_n, sv32_n, w, alpha, mu_in, mu_out,
                                                        lam_out, gth);
    return (int)cudaGetLastError();
}

extern "C" int mbk_adj_face_grad(const mb_stencil_dev *st, const double *sigma, const double *w, const double *v,
                                 double mx, double my, double mz, double *gsig, cudaStream_t s) {
    k_adj_face_grad<<<592, 256, 0, s>>>(*st, sigma, w, v, mx, my, mz, gsig);
    return (int)cudaGetLastError();
}

extern "C" int mbk_adj_gather(const double *v, const int64_t *cells, int ns, double *out, cudaStream_t s) {
    k_adj_gather<<<(ns + 255) / 256, 256, 0, s>>>(v, cells, ns, out);
    return (int)cudaGetLastError();
}

extern "C" int mbk_adj_scatter(double *lam, const int64_t *cells, int ns, const double *gsrc, cudaStream_t s) {
    k_adj_scatter<<<(ns + 255) / 256, 256, 0, s>>>(lam, cells, ns, gsrc);
    return (int)cudaGetLastError();
}

extern "C" size_t mbk_adj_tol_bytes(void) { return (TOL_BLOCKS + 1) * sizeof(double); }

extern "C" int mbk_adj_tol(const double *lam, int64_t n, double rel2, mb_ctrl *c, double *part, cudaStream_t s) {
    k_adj_tol<<<TOL_BLOCKS, 256, 0, s>>>(lam, n, rel2, c, part);
    return (int)cudaGetLastError();
}

// Copies of `arrays` (at most 4) device arrays, each 16-byte aligned and a multiple of
// 16 bytes long.
extern "C" int mbk_copy4(int arrays, void *const *dst, const void *const *src, const size_t *bytes, cudaStream_t s) {
    CopyList l{};
    int64_t most = 0;
    for (int q = 0; q < arrays && q < 4; ++q) {
        l.dst[q] = (uint4 *)dst[q];
        l.src[q] = (const uint4 *)src[q];
        l.words[q] = (int64_t)(bytes[q] / 16);
        if (l.words[q] > most) most = l.words[q];
    }
    if (!most) return 0;
    int64_t blocks = (most + 1023) / 1024;      // four words of the longest array per thread
    if (blocks > 1184) blocks = 1184;
    k_copy4<<<(unsigned)blocks, 256, 0, s>>>(l);
    return (int)cudaGetLastError();
}
