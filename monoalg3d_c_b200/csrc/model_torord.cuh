// ToRORd-fkatp human ventricular model (Tomek et al. 2019) with endo/mid/epi
// cell types, as the reference's Rush-Larsen library evaluates it
// (src/models_library/ToROrd/ToRORd_fkatp_mixed_endo_mid_epi_RL.common.c:1-754,
//  driver ToRORd_fkatp_mixed_endo_mid_epi.c:252-310).
//
// The 17 explicitly-integrated states (0-9, 32-38) advance by forward Euler,
// the 26 gates (10-31, 39-42), dy/dt = (y_inf - y) / tau, by
//     y <- exp(-dt/tau) (y - y_inf) + y_inf    (Rush-Larsen)
//     y <- y + (dt/tau) (y_inf - y)            (when 1/tau is "small")
// where "small" follows the reference macro (ToRORd_fkatp_mixed_endo_mid_epi.h:20):
// MB_RL_REFERENCE_CPU reproduces the CPU build, in which abs() of a double
// truncates to int, so 1/tau < 1 takes the Euler form; MB_RL_TRUE uses the
// written threshold 1/tau < 1e-8.
//
// Model features reproduced as the reference has them: the IClb multiplier is
// 1 (the reference CPU driver leaves it uninitialised), INaK has no MID
// scaling (the reference tests celltype == 2 after testing EPI == 2), and
// I_katp is identically zero (fkatp = 0).
//
// The step (torord_step) is written as a stream: each current reads its
// gates, uses them, advances them and writes them back before the next
// current starts, so that only V, the ten concentration-like states and a few
// running sums live across it.  Holding all 43 states and the 26 pairs of gate
// coefficients (the form before) took 255 registers and spilled, which left two
// warps per scheduler.
#pragma once
#include "mb_math.cuh"

MB_NS_BEGIN

constexpr int TOR_NEQ = 43;
constexpr int TOR_N64 = 9;    // mixed form: V and the 8 ion concentrations in FP64
constexpr int TOR_N32 = 34;   // mixed form: everything else in FP32

// Mixed-form row of state s: rows64 = {V, cass, nai, nass, ki, kss, cansr,
// cajsr, cai}; rows32 = {CaMKt, states 10..42}.
__host__ __device__ inline int tor_mixed_row(int s, bool &is64) {
    if (s == 0) { is64 = true; return 0; }
    if (s >= 2 && s <= 9) { is64 = true; return s - 1; }
    is64 = false;
    if (s == 1) return 0;
    return s - 9;
}

template <typename T>
struct TorScale { T INa, IKr, IKs, ICaL, IK1; };

template <typename T>
__device__ __forceinline__ void load_tor_scale(const float *scale, size_t ld, uint32_t t, TorScale<T> &sc) {
    if (scale) {
        sc.INa = T(scale[0 * ld + t]);
        sc.IKr = T(scale[1 * ld + t]);
        sc.IKs = T(scale[2 * ld + t]);
        sc.ICaL = T(scale[3 * ld + t]);
        sc.IK1 = T(scale[4 * ld + t]);
    } else {
        sc.INa = sc.IKr = sc.IKs = sc.ICaL = sc.IK1 = T(1);
    }
}

// 1.82e6 * (74 * 310)^-1.5, the Davies-equation constant of the driving-force
// activity coefficients, evaluated once in double precision.
#define MB_TOR_CONSTA 0x1.0c3201d875e3fp-1  /* 0.52381902472820474 */
// the same factors of the extracellular side (I = 0.5 (140 + 5 + 150 + 4 x 1.8) / 1000),
// and log(cli / clo) = log(24 / 150)
#define MB_TOR_GAMMA_CAO 0.6117017520062547
#define MB_TOR_GAMMA_O 0.8843718923169582
#define MB_TOR_LOG_CL -1.8325814637483102

// x / (exp(x) - 1), with its limit 1 - x/2 near x = 0.  The GHK fluxes
// divide by exp(z V F/RT) - 1, which vanishes at V = 0; in single precision
// exp(x) rounds to 1 once |V| is below a few microvolts and the quotient
// becomes 0/0, which a travelling wave crossing 0 mV in a million cells meets
// about once per beat.  The single-precision form therefore evaluates the
// flux through this function (the plain FP64 form keeps the reference's
// expression, whose singularity double precision does not reach).
__device__ __forceinline__ float ghk_b(float x) {
    if (fabsf(x) < 1e-4f) return 1.0f - 0.5f * x;
    return x / mexpm1(x);
}

// Activity-coefficient factors exp(-A z^2 (sqrt(I)/(1+sqrt(I)) - 0.3 I)) for
// z = 2 (g4) and z = 1 (g1).
template <typename T>
__device__ __forceinline__ void davies(T I, T &g4, T &g1) {
    const T s = msqrt(I);
    const T e = mexp(-T(MB_TOR_CONSTA) * (mdiv(s, T(1) + s) - T(0.3) * I));
    g1 = e;
    g4 = sq(sq(e));
}

// Na/Ca exchanger flux for one compartment (RL.common.c:364-451), times its
// allosteric factor.  The quotients h = 1 + a (1 + b) of the reference are kept
// with their reciprocals formed once; E1..E4 share one division.
template <typename T>
__device__ __forceinline__ T torord_ncx(T na, T ca, T hna, T ihna, T ihca, T nao, T cao) {
    const T kna1 = T(15.0), kna2 = T(5.0), kna3 = T(88.12), kasymm = T(12.5);
    const T wna = T(6.0e4), wca = T(6.0e4), wnaca = T(5.0e3);
    const T kcaon = T(1.5e6), kcaoff = T(5.0e3);
    const T h3 = mrcp(T(1) + na / kna3 * (T(1) + hna));
    const T h2 = na * hna * T(1.0 / 88.12) * h3;
    const T h6 = mrcp(T(1) + na / kna1 * (T(1) + na / kna2));
    const T h5 = na * na * h6 * T(1.0 / (15.0 * 5.0));
    const T h9 = mrcp(T(1) + nao / kna3 * (T(1) + ihna));
    const T h8 = nao / kna3 * ihna * h9;
    const T h10 = kasymm + T(1) + nao / kna1 * (T(1) + nao / kna2);      // constants from here
    const T h11 = nao * nao / (h10 * kna1 * kna2);
    const T k1 = T(1) / h10 * cao * kcaon;
    const T k2 = kcaoff, k5 = kcaoff;
    const T k3pp = h8 * wnaca;
    const T k3 = h9 * wca + k3pp;
    const T k4pp = h2 * wnaca;
    const T k4 = h3 * wca * ihca + k4pp;
    const T k6 = h6 * ca * kcaon;
    const T k7 = h5 * h2 * wna;
    const T k8 = h8 * h11 * wna;
    const T x1 = k2 * k4 * (k7 + k6) + k5 * k7 * (k2 + k3);
    const T x2 = k1 * k7 * (k4 + k5) + k4 * k6 * (k1 + k8);
    const T x3 = k1 * k3 * (k7 + k6) + k8 * k6 * (k2 + k3);
    const T x4 = k2 * k8 * (k4 + k5) + k3 * k5 * (k1 + k8);
    const T KmCaAct = T(150.0e-6);
    // allo = 1 / (1 + (KmCaAct / ca)^2)
    const T JncxNa = T(3.0) * (x4 * k7 - x1 * k8) + x3 * k4pp - x2 * k3pp;
    const T JncxCa = x2 * k2 - x1 * k1;
    return mdiv((JncxNa + T(2.0) * JncxCa) * (ca * ca), (x1 + x2 + x3 + x4) * (ca * ca + KmCaAct * KmCaAct));
}

// A gate's new value from y, its rate k = 1/tau and its steady state.
template <typename T, int RULE>
__device__ __forceinline__ T rl_gate(T y, T k, T inf, T dt) {
    const bool euler = (RULE == MB_RL_REFERENCE_CPU) ? (k < T(1) && k > T(-1)) : (fabs(k) < T(1e-8));
    if (euler) return y + dt * (k * (inf - y));
    return mexp(-dt * k) * (y - inf) + inf;
}
// The same for a gate whose rate is below 1 at every V (tau bounded below by
// the model's constants): Euler under the reference's CPU rule.
template <typename T, int RULE>
__device__ __forceinline__ T rl_slow(T y, T k, T inf, T dt) {
    if constexpr (RULE == MB_RL_REFERENCE_CPU) return y + dt * (k * (inf - y));
    else return rl_gate<T, RULE>(y, k, inf, dt);
}

// One sub-step of dt.  IO holds the cell's state: get(s) reads state s (in T),
// put(s, y) writes a gate, euler(s, y, d) advances an Euler state that was read as
// y by dt d, in the precision it is stored in; fence() ends a part of the step
// (nothing of the next part's reads moves above it).  celltype 0 endo, 1 mid, 2 epi.
template <typename T, int RULE, typename IO>
__device__ __forceinline__ void torord_step(IO &io, const T stim, const T dt, const int celltype, const TorScale<T> &sc) {
    const bool EPI = celltype == 2, MID = celltype == 1;
    const T nao = T(140.0), cao = T(1.8), ko = T(5.0);
    const T R = T(8314.0), Tk = T(310.0), F = T(96485.0);
    const T RTF = R * Tk / F, FRT = F / (R * Tk);
    const T cli = T(24);
    // cell geometry
    const T L = T(0.01), rad = T(0.0011);
    const T vcell = T(1000) * T(3.14) * rad * rad * L;
    const T Ageo = T(2) * T(3.14) * rad * rad + T(2) * T(3.14) * rad * L;
    const T Acap = T(2) * Ageo;
    const T vmyo = T(0.68) * vcell, vnsr = T(0.0552) * vcell, vjsr = T(0.0048) * vcell, vss = T(0.02) * vcell;

    const T v = io.get(0), cass = io.get(2), nai = io.get(3), nass = io.get(4), ki = io.get(5), kss = io.get(6);
    const T cai = io.get(9);
    const T vfrt = v * FRT;

    // CaMK; p = fINap = fINaLp = fItop = fICaLp = fJrelp = fJupp
    T p;
    {
        const T CaMKt = io.get(1);
        const T CaMKb = T(0.05) * (T(1.0) - CaMKt) * mdiv(cass, cass + T(0.0015));
        const T CaMKa = CaMKb + CaMKt;
        p = mdiv(CaMKa, CaMKa + T(0.15));
        io.euler(1, CaMKt, T(0.05) * CaMKb * CaMKa - T(0.00068) * CaMKt);
    }
    const T q = T(1.0) - p;
    const T vek = v - RTF * mlog(mdiv(ko, ki));

    // sums of the currents: all, and by the ion and compartment they load
    T Iall, Inai, Iki;

    // INa (Grandi formulation with CaMK phosphorylation), INaL
    {
        const T vna = v - RTF * mlog(mdiv(nao, nai));
        const T mss = sigm(MB_OVER(-(T(56.86) + v), 9.03));
        const T km = mrcp(T(0.1292) * mexp(-sq(MB_OVER(v + T(45.79), 15.54))) +
                          T(0.06487) * mexp(-sq(MB_OVER(v - T(4.823), 51.12))));
        T kh, kj;
        if (v >= T(-40)) {
            kh = mdiv(T(0.77), T(0.13) * (T(1) + mexp(MB_OVER(-(v + T(10.66)), 11.1))));
            kj = mdiv(T(0.6) * mexp(T(0.057) * v), T(1) + mexp(T(-0.1) * (v + T(32))));
        } else {
            kh = T(0.057) * mexp(MB_OVER(-(v + T(80)), 6.8)) +
                 (T(2.7) * mexp(T(0.079) * v) + T(3.1) * T(100000.0) * mexp(T(0.3485) * v));
            kj = mdiv((T(-2.5428) * T(10000.0) * mexp(T(0.2444) * v) - T(6.948) * T(1.0e-6) * mexp(T(-0.04391) * v)) *
                          (v + T(37.78)),
                      T(1) + mexp(T(0.311) * (v + T(79.23)))) +
                 mdiv(T(0.02424) * mexp(T(-0.01052) * v), T(1) + mexp(T(-0.1378) * (v + T(40.14))));
        }
        const T hss = sq(sigm(MB_OVER(v + T(71.55), 7.43)));
        const T hssp = sq(sigm(MB_OVER(v + T(71.55) + T(6), 7.43)));
        const T m = io.get(10), h = io.get(11), j = io.get(12), hp = io.get(13), jp = io.get(14);
        const T INa = sc.INa * T(11.7802) * vna * (m * m * m) * (q * h * j + p * hp * jp);
        // mL has m's time constant
        const T mL = io.get(15), hL = io.get(16), hLp = io.get(17);
        const T INaL = (EPI ? T(0.0279) * T(0.6) : T(0.0279)) * vna * mL * (q * hL + p * hLp);
        const T mLss = sigm(MB_OVER(-(v + T(42.85)), 5.264));
        const T hLss = sigm(MB_OVER(v + T(87.61), 7.488));
        const T hLssp = sigm(MB_OVER(v + T(93.81), 7.488));
        // 1/tau_m > 1 at every V (tau_m <= 0.195): Rush-Larsen under either rule
        const T em = mexp(-dt * km);
        io.put(10, em * (m - mss * mss) + mss * mss);
        io.put(15, em * (mL - mLss) + mLss);
        io.put(11, rl_gate<T, RULE>(h, kh, hss, dt));
        io.put(12, rl_gate<T, RULE>(j, kj, hss, dt));
        io.put(13, rl_gate<T, RULE>(hp, kh, hssp, dt));
        io.put(14, rl_gate<T, RULE>(jp, T(1.0 / 1.46) * kj, hss, dt));
        io.put(16, rl_slow<T, RULE>(hL, T(1.0 / 200.0), hLss, dt));
        io.put(17, rl_slow<T, RULE>(hLp, T(1.0 / 600.0), hLssp, dt));
        Inai = INa + INaL;
        Iall = Inai;
    }
    io.fence();
    // Ito
    {
        const T a = io.get(18), iF = io.get(19), iS = io.get(20), ap = io.get(21), iFp = io.get(22), iSp = io.get(23);
        const T AiF = sigm(MB_OVER(v - T(213.6), 151.2));
        const T AiS = T(1.0) - AiF;
        const T Ito = (EPI || MID ? T(0.16) * T(2.0) : T(0.16)) * vek *
                      (q * a * (AiF * iF + AiS * iS) + p * ap * (AiF * iFp + AiS * iSp));
        const T ass = sigm(MB_OVER(-(v - T(14.34)), 14.82));
        const T assp = sigm(MB_OVER(-(v - T(24.34)), 14.82));
        const T ka = T(1.0 / 1.0515) * (T(1.0 / 1.2089) * sigm(MB_OVER(-(v - T(18.4099)), 29.3814)) +
                                        T(3.5) * sigm(MB_OVER(v + T(100.0), 29.3814)));
        const T iss = sigm(MB_OVER(v + T(43.94), 5.711));
        T tiF = T(4.562) + mrcp(T(0.3933) * mexp(MB_OVER(-(v + T(100.0)), 100.0)) +
                                T(0.08004) * mexp(MB_OVER(v + T(50.0), 16.59)));
        T tiS = T(23.62) + mrcp(T(0.001416) * mexp(MB_OVER(-(v + T(96.52)), 59.05)) +
                                T(1.780e-8) * mexp(MB_OVER(v + T(114.1), 8.079)));
        if (EPI) {
            const T de = T(1.0) - T(0.95) * sigm(MB_OVER(v + T(70.0), 5.0));
            tiF = tiF * de;
            tiS = tiS * de;
        }
        const T dti = (T(1.354) + T(1.0e-4) * mrcp(mexp(MB_OVER(v - T(167.4), 15.89)) + mexp(MB_OVER(-(v - T(12.23)), 0.2154)))) *
                      (T(1.0) - T(0.5) * sigm(MB_OVER(v + T(70.0), 20.0)));
        const T kF = mrcp(tiF), kS = mrcp(tiS), kd = mrcp(dti);
        io.put(18, rl_gate<T, RULE>(a, ka, ass, dt));
        io.put(21, rl_gate<T, RULE>(ap, ka, assp, dt));
        io.put(19, rl_gate<T, RULE>(iF, kF, iss, dt));
        io.put(20, rl_gate<T, RULE>(iS, kS, iss, dt));
        io.put(22, rl_gate<T, RULE>(iFp, kd * kF, iss, dt));
        io.put(23, rl_gate<T, RULE>(iSp, kd * kS, iss, dt));
        Iki = Ito;
        Iall += Ito;
    }
    io.fence();
    // ICaL, ICaNa, ICaK, and the background currents of the same fluxes
    T ICaL, Icai, Icass, Inass, Ikss;
    {
        T oss, oi;          // open probabilities x conductance, subspace and myoplasm
        {
            const T d = io.get(24), ff = io.get(25), fs = io.get(26), fcaf = io.get(27), fcas = io.get(28);
            const T jca = io.get(29), ffp = io.get(30), fcafp = io.get(31), nca = io.get(32), nca_i = io.get(33);
            const T f = T(0.6) * ff + T(0.4) * fs, fp = T(0.6) * ffp + T(0.4) * fs;
            const T Af = T(0.3) + T(0.6) * sigm(MB_OVER(v - T(10.0), 10.0));
            const T fca = jca * (Af * fcaf + (T(1.0) - Af) * fcas), fcap = jca * (Af * fcafp + (T(1.0) - Af) * fcas);
            T PCa = T(8.3757e-05) * sc.ICaL;
            if (EPI) PCa = PCa * T(1.2);
            else if (MID) PCa = PCa * T(2);
            const T g = PCa * d, pp = T(1.1) * p;
            oss = g * (q * (f * (T(1.0) - nca) + fca * nca) + pp * (fp * (T(1.0) - nca) + fcap * nca));
            oi = g * (q * (f * (T(1.0) - nca_i) + fca * nca_i) + pp * (fp * (T(1.0) - nca_i) + fcap * nca_i));
            // n gate: anca = 1 / (k2n/km2n + (1 + Kmn/c)^4) with t = c / (c + Kmn), km2n = jca;
            // 0 where jca and c are both 0 (tiny is below the last place of everything else)
            const T k2n = T(500.0), tiny = T(1e-30);
            const T t4 = sq(sq(mdiv(cass, cass + T(0.002)))), u4 = sq(sq(mdiv(cai, cai + T(0.002))));
            io.euler(32, nca, k2n * mdiv(t4 * jca, k2n * t4 + (jca + tiny)) - nca * jca);
            io.euler(33, nca_i, k2n * mdiv(u4 * jca, k2n * u4 + (jca + tiny)) - nca_i * jca);
            T dss = T(1.0763) * mexp(T(-1.0070) * mexp(T(-0.0829) * v));
            if (v > T(31.4978)) dss = T(1);
            const T sd = mexp(T(-0.05) * (v + T(6.0))) + mexp(T(0.09) * (v + T(14.0)));
            io.put(24, rl_gate<T, RULE>(d, mrcp(T(0.6) + mrcp(sd)), dss, dt));
            const T fss = sigm(MB_OVER(v + T(19.58), 3.696));
            const T sf = T(0.0045) * (mexp(MB_OVER(-(v + T(20.0)), 10.0)) + mexp(MB_OVER(v + T(20.0), 10.0)));
            const T kff = mrcp(T(7.0) + mrcp(sf));
            io.put(25, rl_slow<T, RULE>(ff, kff, fss, dt));
            io.put(30, rl_slow<T, RULE>(ffp, T(1.0 / 2.5) * kff, fss, dt));
            const T ss = T(0.000035) * (mexp(MB_OVER(-(v + T(5.0)), 4.0)) + mexp(MB_OVER(v + T(5.0), 6.0)));
            io.put(26, rl_slow<T, RULE>(fs, mrcp(T(1000.0) + mrcp(ss)), fss, dt));
            const T sa = T(0.04) * (mexp(MB_OVER(-(v - T(4.0)), 7.0)) + mexp(MB_OVER(v - T(4.0), 7.0)));
            const T kfa = mrcp(T(7.0) + mrcp(sa));
            io.put(27, rl_slow<T, RULE>(fcaf, kfa, fss, dt));
            io.put(31, rl_slow<T, RULE>(fcafp, T(1.0 / 2.5) * kfa, fss, dt));
            const T sb = T(0.00012) * (mexp(MB_OVER(-v, 3.0)) + mexp(MB_OVER(v, 7.0)));
            io.put(28, rl_slow<T, RULE>(fcas, mrcp(T(100.0) + mrcp(sb)), fss, dt));
            io.put(29, rl_slow<T, RULE>(jca, T(1.0 / 75.0), sigm(MB_OVER(v + T(18.08), 2.7916)), dt));
        }
        io.fence();
        // driving forces with Davies activity coefficients
        const T gamma_cao = T(MB_TOR_GAMMA_CAO), gamma_o = T(MB_TOR_GAMMA_O);
        const T e1 = mexp(vfrt), e2 = mexp(T(2.0) * vfrt);
        // g1 = vffrt / (e1 - 1), g2 = vffrt / (e2 - 1)
        T g1, g2;
        if constexpr (sizeof(T) == 4) {
            g1 = F * ghk_b(vfrt);
            g2 = T(0.5) * F * ghk_b(T(2.0) * vfrt);
        } else {
            g1 = mdiv(vfrt * F, e1 - T(1.0));
            g2 = mdiv(vfrt * F, e2 - T(1.0));
        }
        const T fi = T(1) - T(0.8), fs = T(0.8);
        const T PNa = T(0.00125), PK = T(3.574e-4);
        {
            const T Ii = T(0.5) * (nass + kss + cli + T(4) * cass) * T(1.0 / 1000);
            T gamma_ca, gamma;
            davies(Ii, gamma_ca, gamma);
            Icass = fs * oss * (T(4.0) * g2 * (gamma_ca * cass * e2 - gamma_cao * cao));
            Inass = fs * PNa * oss * (g1 * (gamma * nass * e1 - gamma_o * nao));
            Ikss = fs * PK * oss * (g1 * (gamma * kss * e1 - gamma_o * ko));
        }
        const T Ii = T(0.5) * (nai + ki + cli + T(4) * cai) * T(1.0 / 1000);
        T gamma_ca, gamma;
        davies(Ii, gamma_ca, gamma);
        const T PhiCaL_i = T(4.0) * g2 * (gamma_ca * cai * e2 - gamma_cao * cao);
        Icai = fi * oi * PhiCaL_i;
        const T ICaNa_i = fi * PNa * oi * (g1 * (gamma * nai * e1 - gamma_o * nao));
        const T ICaK_i = fi * PK * oi * (g1 * (gamma * ki * e1 - gamma_o * ko));
        ICaL = Icass + Icai;
        const T INab = T(1.9239e-09) * g1 * (nai * e1 - nao);
        const T ICab = T(5.9194e-08) * PhiCaL_i;
        const T IpCa = T(5e-04) * mdiv(cai, T(0.0005) + cai);
        Iall += ICaL + (Inass + ICaNa_i) + (Ikss + ICaK_i) + INab + ICab + IpCa;
        Inai += ICaNa_i + INab;
        Iki += ICaK_i;
        Icai += IpCa + ICab;
    }
    // IKr, Lu-Vandenberg Markov model
    {
        const T c0 = io.get(34), c1 = io.get(35), c2 = io.get(36), I = io.get(37), o_ = io.get(38);
        T GKr = T(0.0321) * sc.IKr;                       // sqrt(ko / 5) = 1
        if (EPI) GKr = GKr * T(1.3);
        else if (MID) GKr = GKr * T(0.8);
        const T IKr = GKr * o_ * vek;
        Iki += IKr;
        Iall += IKr;
        const T alpha = T(0.1161) * mexp(T(0.2990) * vfrt);
        const T beta = T(0.2442) * mexp(T(-1.604) * vfrt);
        const T alpha1 = T(1.25) * T(0.1235), beta1 = T(0.1911);
        const T alpha2 = T(0.0578) * mexp(T(0.9710) * vfrt);
        const T beta2 = T(0.349e-3) * mexp(T(-1.062) * vfrt);
        const T alphai = T(0.2533) * mexp(T(0.5953) * vfrt);
        const T betai = T(1.25) * T(0.0522) * mexp(T(-0.8209) * vfrt);
        const T alphac2ToI = T(0.52e-4) * mexp(T(1.525) * vfrt);
        const T betaItoC2 = mdiv(beta2 * betai * alphac2ToI, alpha2 * alphai);
        io.euler(34, c0, c1 * beta - c0 * alpha);
        io.euler(35, c1, c0 * alpha + c2 * beta1 - c1 * (beta + alpha1));
        io.euler(36, c2, c1 * alpha1 + o_ * beta2 + I * betaItoC2 - c2 * (beta1 + alpha2 + alphac2ToI));
        io.euler(38, o_, c2 * alpha2 + I * betai - o_ * (beta2 + alphai));
        io.euler(37, I, c2 * alphac2ToI + o_ * alphai - I * (betaItoC2 + betai));
    }
    io.fence();
    // IKs, IK1, IKb
    {
        const T xs1 = io.get(39), xs2 = io.get(40);
        const T vks = v - RTF * mlog(mdiv(ko + T(0.01833) * nao, ki + T(0.01833) * nai));
        // 1 + 0.6 / (1 + (3.8e-5 / cai)^1.4) with u = (cai / 3.8e-5)^1.4 = w w^0.4
        const T w = cai * T(1.0 / 3.8e-5), u = w * mexp(T(0.4) * mlog(w));
        const T KsCa = T(1.0) + T(0.6) * mdiv(u, T(1) + u);
        const T IKs = (EPI ? T(0.0011) * T(1.4) : T(0.0011)) * sc.IKs * KsCa * xs1 * xs2 * vks;
        const T xss = sigm(MB_OVER(-(v + T(11.60)), 8.932));
        const T s1 = T(2.326e-4) * mexp(MB_OVER(v + T(48.28), 17.80)) + T(0.001292) * mexp(MB_OVER(-(v + T(210.0)), 230.0));
        io.put(39, rl_slow<T, RULE>(xs1, mrcp(T(817.3) + mrcp(s1)), xss, dt));
        const T k2 = T(0.01) * mexp(MB_OVER(v - T(50.0), 20.0)) + T(0.0193) * mexp(MB_OVER(-(v + T(66.54)), 31.0));
        io.put(40, rl_gate<T, RULE>(xs2, k2, xss, dt));
        const T aK1 = T(4.094) * sigm(T(0.1217) * (vek - T(49.934)));
        const T bK1 = mdiv(T(15.72) * mexp(T(0.0674) * (vek - T(3.257))) + mexp(T(0.0618) * (vek - T(594.31))),
                           T(1) + mexp(T(-0.1629) * (vek + T(14.207))));
        T GK1 = sc.IK1 * T(0.6992);
        if (EPI) GK1 = GK1 * T(1.2);
        else if (MID) GK1 = GK1 * T(1.3);
        const T IK1 = GK1 * mdiv(aK1, aK1 + bK1) * vek;
        const T IKb = (EPI ? T(0.0189) * T(0.6) : T(0.0189)) * sigm(MB_OVER(-(v - T(10.8968)), 23.9871)) * vek;
        Iki += IKs + IK1 + IKb;
        Iall += IKs + IK1 + IKb;
    }
    // INaCa (myoplasm and junctional subspace)
    {
        T Gncx = T(0.0034);
        if (EPI) Gncx = Gncx * T(1.1);
        else if (MID) Gncx = Gncx * T(1.4);
        const T hna = mexp(T(0.5224) * vfrt), ihna = mrcp(hna), ihca = mexp(T(-0.1670) * vfrt);
        const T INaCa_i = (T(1) - T(0.35)) * Gncx * torord_ncx(nai, cai, hna, ihna, ihca, nao, cao);
        const T INaCa_ss = T(0.35) * Gncx * torord_ncx(nass, cass, hna, ihna, ihca, nao, cao);
        Iall += INaCa_i + INaCa_ss;
        Inai += T(3.0) * INaCa_i;
        Icai -= T(2.0) * INaCa_i;
        Inass += T(3.0) * INaCa_ss;
        Icass -= T(2.0) * INaCa_ss;
    }
    // INaK
    {
        const T k1p = T(949.5), k1m = T(182.4), k2p = T(687.2), k2m = T(39.4);
        const T k3p = T(1899.0), k3m = T(79300.0), k4p = T(639.0), k4m = T(40.0);
        const T delta = T(-0.1550), MgADP = T(0.05), H = T(1.0e-7), Kko = T(0.3582);
        const T MgK = T(9.8 / 1.698e-7);                  // MgATP / Kmgatp
        const T rn = nai * T(1.0 / 9.073) * mexp(-(delta / T(3.0)) * vfrt);                 // nai / Knai
        const T rno = nao * T(1.0 / 27.78) * mexp(-((T(1.0) - delta) / T(3.0)) * vfrt);     // nao / Knao
        const T rk = ki * T(1.0 / 0.5), rko = ko / Kko;
        const T P = mdiv(T(4.2), T(1.0 + 1.0e-7 / 1.698e-7) + nai * T(1.0 / 224.0) + ki * T(1.0 / 292.0));
        const T ii = mrcp((T(1.0) + rn) * (T(1.0) + rn) * (T(1.0) + rn) + sq(T(1.0) + rk) - T(1.0));
        const T io_ = mrcp((T(1.0) + rno) * (T(1.0) + rno) * (T(1.0) + rno) + sq(T(1.0) + rko) - T(1.0));
        const T a1 = k1p * (rn * rn * rn) * ii, b1 = k1m * MgADP;
        const T a2 = k2p, b2 = k2m * (rno * rno * rno) * io_;
        const T a3 = k3p * sq(rko) * io_, b3 = P * (k3m * H / (T(1.0) + MgK));
        const T a4 = k4p * MgK / (T(1.0) + MgK), b4 = k4m * sq(rk) * ii;
        const T x1 = a4 * a1 * a2 + b2 * b4 * b3 + a2 * b4 * b3 + b3 * a1 * a2;
        const T x2 = b2 * b1 * b4 + a1 * a2 * a3 + a3 * b1 * b4 + a2 * a3 * b4;
        const T x3 = a2 * a3 * a4 + b3 * b2 * b1 + b2 * b1 * a4 + a3 * a4 * b1;
        const T x4 = b4 * b3 * b2 + a3 * a4 * a1 + b2 * a4 * a1 + b3 * b2 * a1;
        const T INaK = (EPI ? T(15.4509) * T(0.9) : T(15.4509)) *
                       mdiv(T(3.0) * (x1 * a3 - x2 * b3) + T(2.0) * (x4 * b1 - x3 * a1), x1 + x2 + x3 + x4);
        Iall += INaK;
        Inai += T(3.0) * INaK;
        Iki -= T(2.0) * INaK;
    }
    // chloride currents, V
    {
        const T vcl = v - RTF * T(MB_TOR_LOG_CL);         // ECl = RTF log(cli / clo)
        Iall += T(0.2843) * mdiv(cass, cass + T(0.1)) * vcl + T(1.98e-3) * vcl;
    }
    io.euler(0, v, -(Iall + stim));

    // SR release, SERCA uptake, leak, translocation, concentrations
    io.fence();
    {
        const T cansr = io.get(7), cajsr = io.get(8), Jnp = io.get(41), Jp = io.get(42);
        const T bt = T(4.75), btp = T(1.25) * T(4.75);
        T c2 = sq(cajsr);
        if constexpr (sizeof(T) == 4) c2 = c2 > T(1e8) ? T(1e8) : c2;   // c2^4 fits; the quotient is 1 from far below
        const T c8 = sq(sq(c2)), r8 = sq(sq(sq(T(1.7))));
        T inf = T(0.5) * bt * (-ICaL) * mdiv(c8, c8 + r8);              // 1 / (1 + (1.7 / cajsr)^8)
        if (MID) inf = inf * T(1.7);
        const T r = mdiv(cajsr, cajsr + T(0.0123));
        T tau = bt * r, taup = btp * r;
        if (tau < T(0.001)) tau = T(0.001);
        if (taup < T(0.001)) taup = T(0.001);
        io.put(41, rl_gate<T, RULE>(Jnp, mrcp(tau), inf, dt));
        io.put(42, rl_gate<T, RULE>(Jp, mrcp(taup), T(1.25) * inf, dt));
        const T Jrel = T(1.5378) * (q * Jnp + p * Jp);
        T up = q * mdiv(T(0.005425) * cai, cai + T(0.00092)) +
               p * mdiv(T(2.75) * T(0.005425) * cai, cai + T(0.00092) - T(0.00017));
        if (EPI) up = up * T(1.3);
        const T Jup = up - T(0.0048825) * cansr * T(1.0 / 15.0);
        const T Jtr = (cansr - cajsr) * T(1.0 / 60);
        io.euler(7, cansr, Jup - Jtr * (vjsr / vnsr));
        const T sq1 = sq(T(0.8) + cajsr);
        io.euler(8, cajsr, mdiv(sq1, sq1 + T(10.0) * T(0.8)) * (Jtr - Jrel));
        const T JdiffNa = (nass - nai) * T(0.5), JdiffK = (kss - ki) * T(0.5), Jdiff = (cass - cai) * T(1.0 / 0.2);
        io.euler(3, nai, -Inai * (Acap / (F * vmyo)) + JdiffNa * (vss / vmyo));
        io.euler(4, nass, -Inass * (Acap / (F * vss)) - JdiffNa);
        io.euler(5, ki, -(Iki + stim) * (Acap / (F * vmyo)) + JdiffK * (vss / vmyo));
        io.euler(6, kss, -Ikss * (Acap / (F * vss)) - JdiffK);
        // 1 / (1 + A / a^2 + B / b^2) = a^2 b^2 / (a^2 b^2 + A b^2 + B a^2)
        const T am = sq(T(0.00238) + cai), bm = sq(T(0.0005) + cai);
        const T cm = (EPI ? T(0.05) * T(1.3) : T(0.05)) * T(0.00238);
        const T Bcai = mdiv(am * bm, am * bm + cm * bm + T(0.07) * T(0.0005) * am);
        io.euler(9, cai, Bcai * (-Icai * (Acap / (T(2.0) * F * vmyo)) - Jup * (vnsr / vmyo) + Jdiff * (vss / vmyo)));
        const T as = sq(T(0.00087) + cass), bs = sq(T(0.0087) + cass);
        const T Bcass = mdiv(as * bs, as * bs + T(0.047) * T(0.00087) * bs + T(1.124) * T(0.0087) * as);
        io.euler(2, cass, Bcass * (-Icass * (Acap / (T(2.0) * F * vss)) + Jrel * (vjsr / vss) - Jdiff));
    }
}

// Default initial states (steady state after 200 beats) for endo, mid, epi,
// as the reference tabulates them (ToRORd_fkatp_mixed_endo_mid_epi.c:110-154,
// extra_data_library/helper_functions.c:166-300).
__host__ __device__ inline double torord_default_state(int celltype, int s) {
    const double endo[TOR_NEQ] = {
        -8.890585e+01, 1.107642e-02, 6.504164e-05, 1.210818e+01, 1.210851e+01, 1.426206e+02,
        1.426205e+02, 1.530373e+00, 1.528032e+00, 7.455488e-05, 7.814592e-04, 8.313839e-01,
        8.311938e-01, 6.752873e-01, 8.308255e-01, 1.585610e-04, 5.294475e-01, 2.896996e-01,
        9.419166e-04, 9.996194e-01, 5.938602e-01, 4.799180e-04, 9.996194e-01, 6.543754e-01,
        -2.898677e-33, 1.000000e+00, 9.389659e-01, 1.000000e+00, 9.999003e-01, 9.999773e-01,
        1.000000e+00, 1.000000e+00, 4.920606e-04, 8.337021e-04, 6.962775e-04, 8.425453e-04,
        9.980807e-01, 1.289824e-05, 3.675442e-04, 2.471690e-01, 1.742987e-04, 5.421027e-24,
        6.407933e-23};
    const double mid[TOR_NEQ] = {
        -8.924177e+01, 1.922391e-02, 6.585066e-05, 1.503347e+01, 1.503401e+01, 1.434407e+02,
        1.434406e+02, 1.959747e+00, 1.963459e+00, 8.177438e-05, 7.269124e-04, 8.379059e-01,
        8.377164e-01, 6.860578e-01, 8.372100e-01, 1.487602e-04, 5.350003e-01, 2.851164e-01,
        9.208259e-04, 9.996411e-01, 5.673539e-01, 4.691672e-04, 9.996412e-01, 6.265825e-01,
        -4.922960e-40, 1.000000e+00, 9.200354e-01, 1.000000e+00, 9.997888e-01, 9.999665e-01,
        1.000000e+00, 1.000000e+00, 5.161178e-04, 1.189422e-03, 6.917041e-04, 8.225453e-04,
        9.979358e-01, 1.835276e-05, 5.316232e-04, 2.650323e-01, 1.678628e-04, 2.091039e-25,
        2.438403e-23};
    const double epi[TOR_NEQ] = {
        -8.917755e+01, 1.288116e-02, 5.767956e-05, 1.284260e+01, 1.284291e+01, 1.429114e+02,
        1.429113e+02, 1.812268e+00, 1.810520e+00, 6.631866e-05, 7.370422e-04, 8.366816e-01,
        8.366012e-01, 6.840260e-01, 8.363958e-01, 1.505860e-04, 5.412669e-01, 3.043382e-01,
        9.248184e-04, 9.996371e-01, 9.996342e-01, 4.712023e-04, 9.996371e-01, 9.996366e-01,
        4.333129e-43, 1.000000e+00, 9.485160e-01, 1.000000e+00, 9.999339e-01, 9.999822e-01,
        1.000000e+00, 1.000000e+00, 3.086885e-04, 5.303737e-04, 6.775197e-04, 8.264829e-04,
        9.982135e-01, 9.433146e-06, 2.730221e-04, 2.308784e-01, 1.690386e-04, -1.103286e-23,
        -6.177055e-22};
    if (celltype == 1) return mid[s];
    if (celltype == 2) return epi[s];
    return endo[s];
}

MB_NS_END
