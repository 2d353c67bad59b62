// ten Tusscher & Panfilov 2006 human ventricular myocyte, epicardial variant
// with the constants of the reference model library
// (src/models_library/ten_tusscher/ten_tusscher_2006_RS_CPU.c:137-351).
//
// One Rush-Larsen sub-step: gates 1..12 advance with
//     y <- y_inf + (y - y_inf) * exp(-dt / tau)
// (the reference's RL update, _RS_CPU.c:337-348); V and the six
// concentration-like states advance with explicit Euler (_RS_CPU.c:112,128-133).
//
// The arithmetic type T is double for the plain method and float for the
// mixed-precision form.  Every literal keeps the reference's spelling: a
// constant written with an `f` suffix there is the float value promoted to
// double here too, which the FP64 parity bar depends on.
#pragma once
#include "mb_math.cuh"

MB_NS_BEGIN

constexpr int TT_NEQ = 19;

// sqrt(Ko / 5.4f) with Ko = 5.4 a double (the two differ in the 8th digit)
constexpr double TT_SQRT_KO = 1.0 + 0.5 * (5.4 / (double)5.4f - 1.0);

// Indices of the state rows (the reference sv[] order, _RS_CPU.c:140-158).
enum TTIdx {
    TT_V = 0, TT_XR1, TT_XR2, TT_XS, TT_M, TT_H, TT_J, TT_D, TT_F, TT_F2, TT_FCASS,
    TT_S, TT_R, TT_CAI, TT_CASR, TT_CASS, TT_RPRIME, TT_NAI, TT_KI
};

// Default initial state (_RS_CPU.c:27-45); the literals are floats there.
__host__ __device__ inline double tt2006_default_state(int i) {
    switch (i) {
    case 0: return -85.23f;   case 1: return 0.00621f;  case 2: return 0.4712f;
    case 3: return 0.0095f;   case 4: return 0.00172f;  case 5: return 0.7444f;
    case 6: return 0.7045f;   case 7: return 3.373e-5f; case 8: return 0.7888f;
    case 9: return 0.9755f;   case 10: return 0.9953f;  case 11: return 0.999998f;
    case 12: return 2.42e-8f; case 13: return 0.000126f; case 14: return 3.64f;
    case 15: return 0.00036f; case 16: return 0.9073f;  case 17: return 8.604f;
    default: return 136.89f;
    }
}

// Conductance scalings applied to gNa, gKr, gKs, gCaL, gK1 (1 = reference).
template <typename T>
struct TTScale { T gNa, gKr, gKs, gCaL, gK1; };

// Outputs of one evaluation: dV/dt, the six Euler derivatives and the twelve
// already-advanced gate values.
template <typename T>
struct TTUpdate {
    T dV;
    T gate[12];          // new values of states 1..12
    T dCai, dCaSR, dCaSS, dRprime, dNai, dKi;
};

// Steady states and rates 1/tau of gates 1..12 (state order): functions of V,
// for fCass of Ca_ss.
template <typename T>
__device__ __forceinline__ void tt2006_gate_rates(const T V, const T Ca_ss, T (&inf)[12], T (&rate)[12]) {
    inf[0] = sigm(MB_OVER(T(-26.0f) - V, 7.0f));
    rate[0] = (T(1.0f) + mexp(MB_OVER(T(-45.0f) - V, 10.0f))) * (T(1.0f) + mexp(MB_OVER(V + T(30.0f), 11.5f))) *
              T(1.0 / (450.0f * 6.0f));
    inf[1] = sigm(MB_OVER(V + T(88.0f), 24.0f));
    rate[1] = (T(1.0f) + mexp(MB_OVER(T(-60.0f) - V, 20.0f))) * (T(1.0f) + mexp(MB_OVER(V - T(60.0f), 20.0f))) *
              T(1.0 / (3.0 * (double)1.12f));
    inf[2] = sigm(MB_OVER(T(-5.0f) - V, 14.0f));
    {
        // 1400 / (sqrt(e1) e2) + 80
        const T e = msqrt(T(1.0f) + mexp(MB_OVER(T(5.0f) - V, 6.0f))) * (T(1.0f) + mexp(MB_OVER(V - T(35.0f), 15.0f)));
        rate[2] = mrcp(T(1400.0f) * mrcp(e) + T(80.0f));
    }
    const T em = sigm(MB_OVER(T(-56.86f) - V, 9.03f));
    inf[3] = em * em;
    {
        // 1 / (a (0.1 / b + 0.1 / c)) with b = 1 + exp((V + 35) / 5) as its reciprocal, because b c
        // overflows from 400 mV on in FP32 and 3.4 V in FP64
        const T c = T(1.0f) + mexp(MB_OVER(V - T(50.0f), 200.0f));
        rate[3] = (T(1.0f) + mexp(MB_OVER(T(-60.0f) - V, 5.0f))) * MB_OVER(c, (double)0.1f) *
                  mrcp(T(1.0f) + c * sigm(MB_OVER(V + T(35.0f), 5.0f)));
    }
    const T eh = sigm(MB_OVER(V + T(71.55f), 7.43f));
    inf[4] = eh * eh;
    inf[5] = inf[4];
    if (V < T(-40.0f)) {
        const T alpha_h = T(0.057f) * mexp(MB_OVER(-(V + T(80.0f)), 6.8f));
        const T beta_h = (T(2.7f) * mexp(T(0.079f) * V)) + (T(310000.0f) * mexp(T(0.3485f) * V));
        const T alpha_j = mdiv((((T(-25428.0f)) * mexp(T(0.2444f) * V)) - (T(6.948e-06f) * mexp(T(-0.04391f) * V))) *
                                   (V + T(37.78f)),
                               T(1.0f) + mexp(T(0.311f) * (V + T(79.23f))));
        const T beta_j = mdiv(T(0.02424f) * mexp(T(-0.01052f) * V), T(1.0f) + mexp(T(-0.1378f) * (V + T(40.14f))));
        rate[4] = alpha_h + beta_h;
        rate[5] = alpha_j + beta_j;
    } else {
        rate[4] = mdiv(T(0.77f), T(0.13f) * (T(1.0f) + mexp(MB_OVER(V + T(10.66f), -11.1f))));
        rate[5] = mdiv(T(0.6f) * mexp(T(0.057f) * V), T(1.0f) + mexp(T(-0.1f) * (V + T(32.0f))));
    }
    inf[6] = sigm(MB_OVER(T(-8.0f) - V, 7.5f));
    rate[6] = mrcp((T(1.4f) * sigm(MB_OVER(T(-35.0f) - V, 13.0f)) + T(0.25f)) * (T(1.4f) * sigm(MB_OVER(V + T(5.0f), 5.0f))) +
                   sigm(MB_OVER(T(50.0f) - V, 20.0f)));
    const T e30 = sigm(MB_OVER(V + T(30.0f), 10.0f));
    const T v27 = V + T(27.0f);
    inf[7] = sigm(MB_OVER(V + T(20.0f), 7.0f));
    rate[7] = mrcp((T(1102.5f) * mexp(MB_OVER(-(v27 * v27), 225.0f))) + T(200.0f) * sigm(MB_OVER(T(13.0f) - V, 10.0f)) +
                   T(180.0f) * e30 + T(20.0f));
    inf[8] = T(0.67f) * sigm(MB_OVER(V + T(35.0f), 7.0f)) + T(0.33f);
    rate[8] = mrcp((T(562.0f) * mexp(MB_OVER(-(v27 * v27), 240.0f))) + T(31.0f) * sigm(MB_OVER(T(25.0f) - V, 10.0f)) +
                   T(80.0f) * e30);
    const T cr = MB_OVER(Ca_ss, (double)0.05f);
    const T fc = mrcp(T(1.0f) + cr * cr);
    inf[9] = T(0.6f) * fc + T(0.4f);
    rate[9] = mrcp(T(80.0f) * fc + T(2.0f));
    inf[10] = sigm(MB_OVER(V + T(20.0f), 5.0f));
    const T v45 = V + T(45.0f);
    rate[10] = mrcp((T(85.0f) * mexp(MB_OVER(-(v45 * v45), 320.0f))) + T(5.0f) * sigm(MB_OVER(V - T(20.0f), 5.0f)) + T(3.0f));
    inf[11] = sigm(MB_OVER(T(20.0f) - V, 6.0f));
    const T v40 = V + T(40.0f);
    rate[11] = mrcp((T(9.5f) * mexp(MB_OVER(-(v40 * v40), 1800.0f))) + T(0.8f));
}

// y: the 19 state values (in T), stim: merged stimulus current.
template <typename T>
__device__ __forceinline__ void tt2006_rhs(const T *y, T stim, T dt, const TTScale<T> &sc,
                                           TTUpdate<T> &u) {
    const T V = y[TT_V];
    const T Xr1 = y[TT_XR1], Xr2 = y[TT_XR2], Xs = y[TT_XS];
    const T m = y[TT_M], h = y[TT_H], j = y[TT_J];
    const T d = y[TT_D], f = y[TT_F], f2 = y[TT_F2], fCass = y[TT_FCASS];
    const T s = y[TT_S], r = y[TT_R];
    const T Ca_i = y[TT_CAI], Ca_SR = y[TT_CASR], Ca_ss = y[TT_CASS];
    const T R_prime = y[TT_RPRIME], Na_i = y[TT_NAI], K_i = y[TT_KI];

    // physical constants and cell geometry
    const T R = T(8314.472), Tk = T(310.0), F = T(96485.3415f);
    const T Cm = T(0.185), V_c = T(0.016404);
    const T Ko = T(5.4), Nao = T(140.0), Cao = T(2.0);
    const T P_kna = T(0.03), K_mNa = T(40.0), K_pCa = T(0.0005);
    // calcium handling
    const T V_rel = T(0.102), k1_prime = T(0.15), max_sr = T(2.5), min_sr = T(1.0);
    const T EC = T(1.5), Vmax_up = T(0.006375);
    // Na/Ca exchanger
    const T n_alpha = T(2.5), n_gamma = T(0.35), K_sat = T(0.1), Km_Ca = T(1.38);
    const T Km_Nai = T(87.5), K_NaCa = T(1000.0);
    // maximal conductances
    const T g_to = T(0.294), g_Kr = T(0.153) * sc.gKr, g_Ks = T(0.098) * sc.gKs;
    const T g_CaL = T(3.98e-05) * sc.gCaL, g_Na = T(14.838) * sc.gNa, g_pK = T(0.0146);
    const T g_bca = T(0.000592), g_pCa = T(0.1238), g_K1 = T(5.405) * sc.gK1, g_bna = T(0.00029);

    const T RTF = (R * Tk) / F;
    const T EK = RTF * mlog(mdiv(Ko, K_i));
    const T EKs = RTF * mlog(mdiv(Ko + (P_kna * Nao), K_i + (P_kna * Na_i)));
    const T ENa = RTF * mlog(mdiv(Nao, Na_i));
    const T ECa = ((T(0.5f) * R * Tk) / F) * mlog(mdiv(Cao, Ca_i));

    // inward rectifier
    const T vek = V - EK;
    const T beta_K1 = mdiv((T(3.0f) * mexp(T(0.0002f) * (vek + T(100.0f)))) + mexp(T(0.1f) * (vek - T(10.0f))),
                           T(1.0f) + mexp(T(-0.5f) * vek));
    const T alpha_K1 = T(0.1f) * sigm(T(0.06f) * (vek - T(200.0f)));
    const T xK1_inf = mdiv(alpha_K1, alpha_K1 + beta_K1);

    const T IK1 = g_K1 * xK1_inf * vek;
    const T Ito = g_to * r * s * vek;
    const T IKr = g_Kr * Xr1 * Xr2 * vek * T(TT_SQRT_KO);
    const T IKs = g_Ks * (Xs * Xs) * (V - EKs);
    const T IpK = (g_pK * vek) * sigm(MB_OVER(T(25.0f) - V, (double)5.98f));

    // L-type calcium current; the removable singularity at V = 15 mV uses
    // the limit value inside a +-1e-5 mV band (_RS_CPU.c:221)
    const T FRT = F / (R * Tk);
    T ICaL;
    const T v15 = V - T(15.0f);
    if (V < T(15.0f - 1.0e-5f) || V > T(15.0f + 1.0e-5f)) {
        const T ea = T(2.0f) * v15 * FRT;
        ICaL = mdiv((g_CaL * d * f * f2 * fCass * T(4.0f) * v15 * F * FRT) * ((T(0.25f) * Ca_ss * mexp(ea)) - Cao),
                    mexpm1(ea));
    } else {
        ICaL = g_CaL * d * f * f2 * fCass * T(2.0f) * F * (T(0.25f) * Ca_ss - Cao);
    }
    const T IbCa = g_bca * (V - ECa);
    const T IpCa = mdiv(g_pCa * Ca_i, Ca_i + K_pCa);

    // P_NaK Ko / (Ko + K_mk) = 2.724 x 5.4 / 6.4
    const T INaK = mdiv(T(2.724 * 5.4 / (5.4 + 1.0)) * Na_i,
                        (Na_i + K_mNa) * (T(1.0f) + (T(0.1245f) * mexp(T(-0.1f) * V * FRT)) +
                                          (T(0.0353f) * mexp(-V * FRT))));
    const T INa = g_Na * (m * m * m) * h * j * (V - ENa);
    const T IbNa = g_bna * (V - ENa);
    const T e_gm1 = mexp((n_gamma - T(1.0f)) * V * FRT);
    const T INaCa = mdiv(K_NaCa * ((mexp(n_gamma * V * FRT) * (Na_i * Na_i * Na_i) * Cao) -
                                   (e_gm1 * (Nao * Nao * Nao) * Ca_i * n_alpha)),
                         ((Km_Nai * Km_Nai * Km_Nai) + (Nao * Nao * Nao)) * (Km_Ca + Cao) *
                             (T(1.0f) + (K_sat * e_gm1)));

    T inf[12], rate[12];
    tt2006_gate_rates<T>(V, Ca_ss, inf, rate);

    // calcium dynamics
    // x / (x + c) in place of 1 / (1 + c / x)
    const T sr2 = Ca_SR * Ca_SR;
    const T kcasr = max_sr - (max_sr - min_sr) * mdiv(sr2, sr2 + EC * EC);
    const T k1 = mdiv(k1_prime, kcasr);
    const T k3 = T(0.06);
    const T css2 = Ca_ss * Ca_ss;
    const T O = mdiv(k1 * css2 * R_prime, k3 + (k1 * css2));
    const T Irel = V_rel * O * (Ca_SR - Ca_ss);
    const T K_up = T(0.00025);
    const T ci2 = Ca_i * Ca_i;
    const T i_up = Vmax_up * mdiv(ci2, ci2 + K_up * K_up);
    const T i_leak = T(0.00036f) * (Ca_SR - Ca_i);
    const T i_xfer = T(0.0038f) * (Ca_ss - Ca_i);
    const T k2 = T(0.045f) * kcasr;
    const T k4 = T(0.005f);
    const T Buf_c = T(0.2f), K_buf_c = T(0.001f);
    const T cbc = Ca_i + K_buf_c;
    const T Ca_i_bufc = mdiv(cbc * cbc, cbc * cbc + Buf_c * K_buf_c);
    const T K_buf_sr = T(0.3f), Buf_sr = T(10.0f);
    const T cbs = Ca_SR + K_buf_sr;
    const T Ca_sr_bufsr = mdiv(cbs * cbs, cbs * cbs + Buf_sr * K_buf_sr);
    const T Buf_ss = T(0.4f), K_buf_ss = T(0.00025f);
    const T cbss = Ca_ss + K_buf_ss;
    const T Ca_ss_bufss = mdiv(cbss * cbss, cbss * cbss + Buf_ss * K_buf_ss);
    const T V_sr = T(0.001094f), V_ss = T(5.468e-05f);

    u.dV = -(IK1 + Ito + IKr + IKs + ICaL + INaK + INa + IbNa + INaCa + IbCa + IpK + IpCa + stim);
    u.dRprime = ((-k2) * Ca_ss * R_prime) + (k4 * (T(1.0f) - R_prime));
    u.dCai = Ca_i_bufc * (((i_leak - i_up) * (V_sr / V_c) + i_xfer) -
                          ((IbCa + IpCa) - (T(2.0f) * INaCa)) * (Cm / (T(2.0f) * V_c * F)));
    u.dCaSR = Ca_sr_bufsr * (i_up - (Irel + i_leak));
    u.dCaSS = Ca_ss_bufss * (((-ICaL) * (Cm / (T(2.0f) * V_ss * F)) + Irel * (V_sr / V_ss)) - i_xfer * (V_c / V_ss));
    u.dNai = -(INa + IbNa + (T(3.0f) * INaK) + (T(3.0f) * INaCa)) * (Cm / (V_c * F));
    u.dKi = -((IK1 + Ito + IKr + IKs + IpK + stim) - (T(2.0f) * INaK)) * (Cm / (V_c * F));

    // Rush-Larsen gate updates
#pragma unroll
    for (int k = 0; k < 12; ++k) u.gate[k] = inf[k] + (y[TT_XR1 + k] - inf[k]) * mexp(-dt * rate[k]);
}

MB_NS_END
