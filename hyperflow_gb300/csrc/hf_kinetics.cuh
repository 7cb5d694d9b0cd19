// Device code shared by the chemistry kernels (hf_chem.cu) and the discrete adjoint
// (hf_adjoint.cu): NASA7 species thermo, mass-action rates of the generated H2_Li table as
// the tagging kernel and the objectives' derivatives use them, and the Rodas4 tableau
// (Hairer & Wanner, Solving ODEs II, Sec. VI.7, KPP coefficient ordering).  The integrators
// are in hf_cell.cuh (one cell per lane) and hf_group.cuh (one per group of 8 lanes).
//
// Pre-exponential factors live in __constant__ memory, one copy per translation
// unit (static); each unit that includes this header uploads them with
// upload_rate_constants() (hf::chem_set_rate_scale and hf::adjoint_set_rate_scale).
#pragma once
#include <utility>
#include "hf_device.cuh"
#include "hf_fastmath.cuh"
#include "hf_internal.h"

namespace hf {

static __constant__ double c_A[NR];
static __constant__ double c_A0[NR];

// A_r and A0_r of the table times scale[r] (1 when scale is null): a rate
// multiplier on reaction r (forward and reverse, both falloff limits).
static inline cudaError_t upload_rate_constants(const double* scale) {
    double a[NR], a0[NR];
    for (int r = 0; r < NR; ++r) {
        const double s = scale ? scale[r] : 1.0;
        a[r] = RXN[r].A * s;
        a0[r] = RXN[r].A0 * s;
    }
    cudaError_t e = cudaMemcpyToSymbol(c_A, a, sizeof(a));
    if (e != cudaSuccess) return e;
    return cudaMemcpyToSymbol(c_A0, a0, sizeof(a0));
}

// ---------------------------------------------------------------- species thermo
// g/RT = h/RT - s/R with NASA7: h/RT = a0 + a1/2 T + a2/3 T^2 + a3/4 T^3 + a4/5 T^4 + a5/T,
// s/R = a0 lnT + a1 T + a2/2 T^2 + a3/3 T^3 + a4/4 T^4 + a6.  Every species of the
// table switches range at T_mid = 1000 K, so one branch selects the range.
template <int NS, int RG>
__device__ __forceinline__ void species_g_h_r(double T, double lnT, double invT, double* g, double* hRT) {
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const double* a = D_NASA.c[RG][k];
        hRT[k] = fma(T, fma(T, fma(T, fma(T, a[4] * 0.2, a[3] * 0.25), a[2] * (1.0 / 3.0)), a[1] * 0.5), a[0]) +
                 a[5] * invT;
        const double sR = fma(a[0], lnT, fma(T, fma(T, fma(T, fma(T, a[4] * 0.25, a[3] * (1.0 / 3.0)), a[2] * 0.5), a[1]), a[6]));
        g[k] = hRT[k] - sR;
    }
}
template <int NS>
__device__ __forceinline__ void species_g_h(double T, double lnT, double invT, double* g, double* hRT) {
    if (T <= TMID) species_g_h_r<NS, 0>(T, lnT, invT, g, hRT);
    else species_g_h_r<NS, 1>(T, lnT, invT, g, hRT);
}

// ---------------------------------------------------------------- kinetics
template <int R, int NS>
__device__ __forceinline__ double third_body(const double* C, double Csum) {
    constexpr Reaction rx = RXN[R];
    double M = Csum;
#pragma unroll
    for (int k = 0; k < NS; ++k)
        if (rx.eff[k] != 1.0) M = fma(rx.eff[k] - 1.0, C[k], M);
    return M;
}
// log10 of a constant in [0.5, 2] at compile time: 2 atanh((x-1)/(x+1)) / ln 10 by
// its odd power series (|z| <= 1/3: 40 terms reach the last bit; within 1 ulp of the
// correctly rounded value for the Troe constants 0.8 and 0.5 of the table).
constexpr double const_log10(double x) {
    const double z = (x - 1.0) / (x + 1.0), z2 = z * z;
    double term = z, sum = 0.0;
    for (int k = 0; k < 40; ++k) {
        sum += term / (2 * k + 1);
        term *= z2;
    }
    return 2.0 * sum / 2.302585092994045684;
}

// Troe: log10 F and its partial derivatives (d log10F/d log10Pr, d log10F/dT).
template <int R>
__device__ __forceinline__ double troe_log10F(double T, double Pr, double* dPr, double* dT) {
    constexpr Reaction rx = RXN[R];
    constexpr bool noT3 = rx.troeT3 < 1e-20, noT1 = rx.troeT1 > 1e20;
    constexpr bool constFcent = noT3 && noT1 && !rx.hasT2;
    double Fcent, dFcent;
    if constexpr (constFcent) {
        Fcent = rx.troeA;
        dFcent = 0.0;
    } else {
        const double e3 = fexp(-T / rx.troeT3), e1 = fexp(-T / rx.troeT1);
        Fcent = (1 - rx.troeA) * e3 + rx.troeA * e1;
        dFcent = -(1 - rx.troeA) / rx.troeT3 * e3 - rx.troeA / rx.troeT1 * e1;
        if (rx.hasT2) {
            const double e2 = fexp(-rx.troeT2 / T);
            Fcent += e2;
            dFcent += rx.troeT2 / (T * T) * e2;
        }
    }
    const bool prc = !(Pr > 1e-300);
    double lFc;
    if constexpr (constFcent && rx.troeA >= 0.5 && rx.troeA <= 2.0) {
        constexpr double c = const_log10(rx.troeA);  // F_cent is a constant of the table
        lFc = c;
    } else {
        lFc = flog(fmax(Fcent, 1e-300)) * fm::INV_LN10;
    }
    const double lPr = flog(fmax(Pr, 1e-300)) * fm::INV_LN10;
    const double c = -0.4 - 0.67 * lFc, nn = 0.75 - 1.27 * lFc;
    const double x = lPr + c, den = nn - 0.14 * x;
    const double f1 = x / den;
    const double g = 1.0 / (1.0 + f1 * f1);
    if (dPr) *dPr = prc ? 0.0 : lFc * (-2.0 * f1 * g * g) * (nn / (den * den));
    if (dT) {
        const double df1 = (-0.67 * den - x * (-1.27 + 0.14 * 0.67)) / (den * den);
        const double dlF_dlFc = g + lFc * (-2.0 * f1 * g * g) * df1;
        *dT = (Fcent > 1e-300) ? dlF_dlFc * dFcent / (Fcent * 2.302585092994046) : 0.0;
    }
    return lFc * g;
}

// Temperature factors T^b exp(-E/T) of the rate constants, evaluated in one rolled
// loop (one exp body for all reactions): k_inf of every reaction, then k_0 of the
// falloff reactions in reaction order.  Kinds by (b, E): 1 (b = E = 0), 1/T and
// 1/T^2 (E = 0, b = -1, -2), exp(-E/T) (b = 0), T*T*exp(-E/T) (b = 2), otherwise
// exp(b lnT - E/T).
enum : int { ARR_ONE = 0, ARR_INVT = 1, ARR_INVT2 = 2, ARR_EXP = 3, ARR_T2EXP = 4, ARR_EXPB = 5 };
struct ArrTerm {
    int kind;
    double b, E;
};
constexpr int fall_index(int R) {
    int n = 0;
    for (int r = 0; r < R; ++r) n += RXN[r].type == RXN_FALLOFF ? 1 : 0;
    return n;
}
constexpr int NFALL = fall_index(NR);
struct ArrTable {
    ArrTerm t[NR + NFALL];
};
constexpr ArrTable make_arr() {
    ArrTable a{};
    for (int r = 0; r < NR; ++r) {
        const double b = RXN[r].b, E = RXN[r].EaR;
        const int kind = (b == 0.0 && E == 0.0)   ? ARR_ONE
                         : (E == 0.0 && b == -1.0) ? ARR_INVT
                         : (E == 0.0 && b == -2.0) ? ARR_INVT2
                         : (b == 0.0)              ? ARR_EXP
                         : (b == 2.0)              ? ARR_T2EXP
                                                   : ARR_EXPB;
        a.t[r] = ArrTerm{kind, b, E};
        if (RXN[r].type == RXN_FALLOFF) {
            const double b0 = RXN[r].b0, E0 = RXN[r].Ea0R;
            const int k0 = (b0 == 0.0 && E0 == 0.0) ? ARR_ONE : (b0 == 0.0) ? ARR_EXP : ARR_EXPB;
            a.t[NR + fall_index(r)] = ArrTerm{k0, b0, E0};
        }
    }
    return a;
}
__device__ constexpr ArrTable D_ARR = make_arr();

// Per-evaluation shared quantities.
template <int NS>
struct KinCtx {
    double T, lnT, invT, Csum;
    double eg[NS], ieg[NS];   // exp(g_k), exp(-g_k), g = g0/RT
    double hRT[NS];
    double rt_p0;             // R T / p0
    double ar[NR + NFALL];    // temperature factors of k_inf (reactions) and k_0 (falloff)
};
// ARR: also the rate constants' temperature factors (the kinetics of the forward
// chemistry; the adjoint evaluates its own).
template <int NS, bool ARR = true>
__device__ __forceinline__ void kin_setup(double T, const double* C, KinCtx<NS>& k) {
    k.T = T;
    k.lnT = flog(T);
    k.invT = 1.0 / T;
    double g[NS];
    species_g_h<NS>(T, k.lnT, k.invT, g, k.hRT);
#pragma unroll 1
    for (int s = 0; s < NS; ++s) {
        fexp_pair(g[s], k.eg[s], k.ieg[s]);
    }
    if constexpr (ARR) {
#pragma unroll 1
        for (int r = 0; r < NR + NFALL; ++r) {
            const ArrTerm a = D_ARR.t[r];
            double v;
            if (a.kind == ARR_ONE) {
                v = 1.0;
            } else if (a.kind == ARR_INVT) {
                v = k.invT;
            } else if (a.kind == ARR_INVT2) {
                v = k.invT * k.invT;
            } else {
                const double x = a.kind == ARR_EXPB ? fma(a.b, k.lnT, -a.E * k.invT) : -a.E * k.invT;
                const double ex = fexp(x);
                v = a.kind == ARR_T2EXP ? k.T * k.T * ex : ex;
            }
            k.ar[r] = v;
        }
    }
    double cs = 0.0;
#pragma unroll
    for (int s = 0; s < NS; ++s) cs += C[s];
    k.Csum = cs;
    k.rt_p0 = RU * T * (1.0 / ONE_ATM);
}
template <int R, int NS>
__device__ __forceinline__ double kinf_T(const KinCtx<NS>& kc) {
    return kc.ar[R];
}
template <int R, int NS>
__device__ __forceinline__ double k0_T(const KinCtx<NS>& kc) {
    return kc.ar[NR + fall_index(R)];
}

// Rate constant k (third-body factor included) of reaction R.
template <int R, int NS>
__device__ __forceinline__ double rate_k(const KinCtx<NS>& kc, const double* C, double& M) {
    constexpr Reaction rx = RXN[R];
    const double kinf = c_A[R] * kinf_T<R, NS>(kc);
    if constexpr (rx.type == RXN_ELEMENTARY) {
        M = 0.0;
        return kinf;
    } else if constexpr (rx.type == RXN_THREE_BODY) {
        M = third_body<R, NS>(C, kc.Csum);
        return kinf * M;
    } else {
        M = third_body<R, NS>(C, kc.Csum);
        const double k0 = c_A0[R] * k0_T<R, NS>(kc);
        const double Pr = k0 * M / kinf;
        const double lF = troe_log10F<R>(kc.T, Pr, nullptr, nullptr);
        return kinf * (Pr / (1.0 + Pr)) * fexp(lF * fm::LN10);
    }
}

// 1/Kc = prod_reac exp(-g) prod_prod exp(g) (RT/p0)^dn
template <int R, int NS>
__device__ __forceinline__ double inv_kc(const KinCtx<NS>& kc) {
    constexpr Reaction rx = RXN[R];
    double v = 1.0;
#pragma unroll
    for (int i = 0; i < rx.nreac; ++i) v *= kc.ieg[rx.reac[i]];
#pragma unroll
    for (int i = 0; i < rx.nprod; ++i) v *= kc.eg[rx.prod[i]];
    constexpr int dn = rx.nprod - rx.nreac;
    if constexpr (dn == 1) v *= kc.rt_p0;
    else if constexpr (dn == -1) v /= kc.rt_p0;
    else if constexpr (dn != 0) v *= pow(kc.rt_p0, (double)dn);
    return v;
}

template <int R, int NS>
__device__ __forceinline__ void add_rate(const KinCtx<NS>& kc, const double* C, double* w) {
    constexpr Reaction rx = RXN[R];
    double M;
    const double k = rate_k<R, NS>(kc, C, M);
    double pf = k, pr = k * inv_kc<R, NS>(kc);
#pragma unroll
    for (int i = 0; i < rx.nreac; ++i) pf *= C[rx.reac[i]];
#pragma unroll
    for (int i = 0; i < rx.nprod; ++i) pr *= C[rx.prod[i]];
    const double q = pf - pr;
#pragma unroll
    for (int i = 0; i < rx.nreac; ++i) w[rx.reac[i]] -= q;
#pragma unroll
    for (int i = 0; i < rx.nprod; ++i) w[rx.prod[i]] += q;
}
template <int NS, size_t... Rs>
__device__ __forceinline__ void all_rates(const KinCtx<NS>& kc, const double* C, double* w, std::index_sequence<Rs...>) {
    (add_rate<(int)Rs, NS>(kc, C, w), ...);
}

// ---------------------------------------------------------------- ODE pieces
// composition of y (Y_0..Y_{N-1}; last species closes) -> z = Y/W, C = rho Y/W
template <int NS>
__device__ __forceinline__ void comp(const double* y, double rho, double* z, double* C) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < NS - 1; ++k) {
        s += y[k];
        z[k] = y[k] * INVW.v[k];
        C[k] = rho * z[k];
    }
    z[NS - 1] = (1.0 - s) * INVW.v[NS - 1];
    C[NS - 1] = rho * z[NS - 1];
}

// ---------------------------------------------------------------- Rodas4
__device__ constexpr double RA[15] = {
    1.544, 0.9466785280815826, 0.2557011698983284, 3.314825187068521, 2.896124015972201,
    0.9986419139977817, 1.221224509226641, 6.019134481288629, 12.53708332932087,
    -0.687886036105895, 1.221224509226641, 6.019134481288629, 12.53708332932087,
    -0.687886036105895, 1.0};
__device__ constexpr double RC[15] = {
    -5.6688, -2.430093356833875, -0.2063599157091915, -0.1073529058151375, -9.594562251023355,
    -20.47028614809616, 7.496443313967647, -10.24680431464352, -33.99990352819905,
    11.7089089320616, 8.083246795921522, -7.981132988064893, -31.52159432874371,
    16.31930543123136, -6.058818238834054};
__device__ constexpr double RM[6] = {1.221224509226641, 6.019134481288629, 12.53708332932087, -0.687886036105895, 1.0, 1.0};
constexpr double RGAMMA = 0.25;
constexpr long MAX_STEPS = 5000;

enum : int { CELL_CONTINUE = 0, CELL_DONE = 1, CELL_FAIL = 2, CELL_MAXSTEPS = 3 };

}  // namespace hf
