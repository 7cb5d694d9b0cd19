// The per-lane cell integrator of the forward chemistry (one cell per lane): the
// constant-(rho, e) ODE of HyperFlow_V3/src/chemistry.cpp:36-53 integrated with Rodas4
// (Hairer & Wanner, Solving ODEs II, Sec. VI.7, KPP coefficient ordering and step
// controller), WRMS errors with weights atol + rtol max(|y_old|, |y_new|).
//
// What bounds it: the FP64 pipe (hf_fp64.cuh: 64 cycles of a sub-partition per warp
// instruction) and instruction fetch (an attempt is tens of thousands of instructions).
// So the formulation counts FP64 instructions:
//  * Unknowns inside an attempt are the concentrations C_k = rho y_k / W_k of the 8 reacting
//    species: dC/dt is the production rate itself and J = dw/dC, without scaling by W and
//    rho.  N2 and AR never react, so their rows are left out; mass is a linear invariant
//    of the stages, so the closing species' concentration is a constant of the interval.
//    The state carried between attempts stays the mass fractions y.
//  * Reverse rates by activities X_k = C_k exp(g_k): with 1/Kc = prod_reac exp(-g)
//    prod_prod exp(g), q = k (prod_reac C - prod_reac exp(-g) prod_prod X).
//  * Reactions that differ only in k (the duplicate pairs) are evaluated once.
//  * g = h/RT - s/R by one polynomial; exponentials and logarithms from larger tables
//    (below); one second-order FP64 Newton step for T (newton_T).
//  * Jacobian, LU factorisation and the frozen-cell screen are one function, so J never
//    leaves the registers; every attempt starts with it.  A rejected step evaluates J
//    again, which costs nothing: the lanes of its warp that accepted theirs, or hold a new
//    cell, need it anyway.
//  * Species' g relative to the elements as H2 and O2, and the inert species' share of the
//    mixture polynomial kept with the cell.
// About 5,100 FP64 instructions an attempt against 13,900 with mass-fraction unknowns, J
// kept beside its factors, 11-instruction exponentials and two FP64 Newton steps; 206 us an
// attempt with the sub-partition to itself, 377 beside a second warp (then the pipe is full).
#pragma once
#include "hf_exptab.h"
#include "hf_kinetics.cuh"

namespace hf {
namespace cell {

constexpr int NQ = 8;  // reacting species: H2, O2, H2O, H, O, OH, HO2, H2O2

// exp(x), |x| < 340: x = k ln2/2048 + r, k from the FP32 product of x cut to FP32, so |r| <=
// 0.65 ln2/2048 (0.55 for |x| < 100); 2^(k/2048) from a table, exp(r) - 1 = r + C2 r^2 + r^3/6
// with C2 the 1/2 economised for 0.51.  6 FP64 instructions.  Table and result round to half a
// unit of the last place each, the polynomial adds 0.34 at most (1.06 in all was seen on the
// device).  The r^4 term would leave 1.01 and costs 1 to 2% of an integration, whose results it
// does not move (3,000 igniting cells against 64 bits: 3.4e-13 with and without).  After P. T. P.
// Tang's table-driven exponential (ACM TOMS 15 (1989) 144-157).  Other arguments: the library
// function.
__device__ __forceinline__ bool small_arg(double x) { return fp_abs_hi(x) < 0x40754000u; }
__device__ __forceinline__ double reduce(double x, int& k) {
    k = __float2int_rn(fp_to_f32(x) * et::INV_STEP);
    const double kd = fp_from_f32((float)k);
    return fma(-kd, et::STEP_LO, fma(-kd, et::STEP_HI, x));
}
__device__ __forceinline__ double fexp(double x) {
    if (!small_arg(x)) return fm_exp_lib(x);
    int k;
    const double r = reduce(x, k);
    const double p = fma(r * r, fma(r, 1.0 / 6.0, et::C2), r);
    const double t = et::EXP[k & 2047];
    return fm_scale(fma(t, p, t), k >> 11);
}
// exp(x) and exp(-x): 9 FP64 instructions
__device__ __forceinline__ void fexp_pair(double x, double& ep, double& em) {
    if (!small_arg(x)) {
        ep = fm_exp_lib(x);
        em = fm_exp_lib(-x);
        return;
    }
    int k;
    const double r = reduce(x, k);
    const double r2 = r * r, o = fma(r, r2 * (1.0 / 6.0), r);
    const double tp = et::EXP[k & 2047], tm = et::EXP[-k & 2047];
    ep = fm_scale(fma(tp, fma(et::C2, r2, o), tp), k >> 11);
    em = fm_scale(fma(tm, fma(et::C2, r2, -o), tm), -k >> 11);
}
// log(x) of a positive normal number: x = 2^m y, F = 1 + (j + 1/2)/256, u = (y - F)/F,
// |u| <= 1/513; log1p(u) = u - u^2/2 + u^3 (1/3 - u/4 + u^2/5), the bracket in FP32 (an
// error of 2e-16 at most: a quarter unit of the last place of ln T).  8 FP64 instructions; after
// Tang, ACM TOMS 16 (1990) 378-400.
__device__ __forceinline__ double flog(double x) {
    const int hi = __double2hiint(x);
    if ((unsigned)hi - 0x00200000u >= 0x7fc00000u) return fm_log_lib(x);
    const int j = (hi >> 12) & 255;
    const int yh = (hi & 0x000fffff) | 0x3ff00000;
    const double y = __hiloint2double(yh, __double2loint(x));
    const double F = __hiloint2double((yh & (int)0xfffff000) | 0x800, 0);
    const double u = (y - F) * et::LOG_IF[j];
    const float f = fp_to_f32(u);
    const double q = fp_from_f32(fmaf(f, fmaf(f, 0.2f, -0.25f), 1.0f / 3.0f));
    const double l = fma(u * u, fma(u, q, -0.5), u);
    const double m = fp_from_f32((float)((hi >> 20) - 1023));
    return fma(m, et::LN2_HI, et::LOG_F[j]) + fma(m, et::LN2_LO, l);
}

// ---------------------------------------------------------------- rate data
// Exponentials the rate constants need, one slot per distinct (b, E): T^b exp(-E/T), with b
// = 2 as T^2 times the slot of b = 0 (fewer exponentials).
struct ArrSlots {
    int n;
    int hasb[NR + NFALL];
    double b[NR + NFALL], E[NR + NFALL];
    int slot[NR + NFALL];  // of k_inf (reactions), then k_0 (falloff reactions); -1: none
};
constexpr ArrSlots make_slots() {
    ArrSlots a{};
    const ArrTable t = make_arr();
    for (int r = 0; r < NR + NFALL; ++r) {
        a.slot[r] = -1;
        if (t.t[r].kind < ARR_EXP) continue;
        const double b = t.t[r].kind == ARR_EXPB ? t.t[r].b : 0.0, E = t.t[r].E;
        for (int i = 0; i < a.n; ++i)
            if (a.b[i] == b && a.E[i] == E) a.slot[r] = i;
        if (a.slot[r] < 0) {
            a.b[a.n] = b;
            a.E[a.n] = E;
            a.hasb[a.n] = b != 0.0;
            a.slot[r] = a.n++;
        }
    }
    return a;
}
__device__ constexpr ArrSlots D_SLOTS = make_slots();
constexpr int NEXP = make_slots().n;
constexpr int slot_of(int i) { return make_slots().slot[i]; }

constexpr bool same_reaction(int a, int b) {
    if (RXN[a].type != RXN_ELEMENTARY || RXN[b].type != RXN_ELEMENTARY || RXN[a].nreac != RXN[b].nreac ||
        RXN[a].nprod != RXN[b].nprod)
        return false;
    for (int i = 0; i < RXN[a].nreac; ++i)
        if (RXN[a].reac[i] != RXN[b].reac[i]) return false;
    for (int i = 0; i < RXN[a].nprod; ++i)
        if (RXN[a].prod[i] != RXN[b].prod[i]) return false;
    return true;
}
constexpr int dup_of(int r) {  // an earlier reaction with the same species, or -1
    for (int q = 0; q < r; ++q)
        if (same_reaction(q, r)) return q;
    return -1;
}
constexpr int dup_next(int r) {
    for (int q = r + 1; q < NR; ++q)
        if (same_reaction(q, r)) return q;
    return -1;
}
constexpr bool at_most_pairs() {
    for (int r = 0; r < NR; ++r)
        if (dup_of(r) >= 0 && dup_next(r) >= 0) return false;
    return true;
}
constexpr bool reacting_only() {  // species >= NQ take part as third bodies only
    for (int r = 0; r < NR; ++r) {
        for (int i = 0; i < RXN[r].nreac; ++i)
            if (RXN[r].reac[i] >= NQ) return false;
        for (int i = 0; i < RXN[r].nprod; ++i)
            if (RXN[r].prod[i] >= NQ) return false;
        if (RXN[r].nreac < 1 || RXN[r].nreac > 2 || RXN[r].nprod < 1 || RXN[r].nprod > 2) return false;
        for (int s = NQ; s < NS_MAX; ++s)
            if (RXN[r].eff[s] != 1.0) return false;
    }
    return true;
}
static_assert(at_most_pairs() && reacting_only(), "the kinetics below assume this of the table");

struct NetNu { int v[NR][NQ]; };
constexpr NetNu make_nu() {
    NetNu t{};
    for (int r = 0; r < NR; ++r) {
        for (int i = 0; i < RXN[r].nreac; ++i) --t.v[r][RXN[r].reac[i]];
        for (int i = 0; i < RXN[r].nprod; ++i) ++t.v[r][RXN[r].prod[i]];
    }
    return t;
}
__device__ constexpr NetNu D_NU = make_nu();
// g_k = a0 (1 - lnT) + a5/T - a6 + c1 T + c2 T^2 + c3 T^3 + c4 T^4
struct GCoef { double c[2][NQ][7]; };  // -a6, c1..c4, a0, a5
constexpr GCoef make_gcoef() {
    GCoef g{};
    for (int r = 0; r < 2; ++r)
        for (int k = 0; k < NQ; ++k) {
            const double* a = r == 0 ? NASA_LOW[k] : NASA_HIGH[k];
            g.c[r][k][0] = -a[6];
            g.c[r][k][1] = -a[1] / 2.0;
            g.c[r][k][2] = -a[2] / 6.0;
            g.c[r][k][3] = -a[3] / 12.0;
            g.c[r][k][4] = -a[4] / 20.0;
            g.c[r][k][5] = a[0];
            g.c[r][k][6] = a[5];
        }
    return g;
}
__device__ constexpr GCoef D_GCOEF = make_gcoef();
// The same relative to the elements as H2 and O2: g_k - n_H/2 g_H2 - n_O/2 g_O2.  Reactions
// conserve both elements, so equilibrium constants are unchanged, and H2 and O2 need no
// exponential (six pairs instead of eight).
constexpr int ATOMS_H[NQ] = {2, 0, 2, 1, 0, 1, 1, 2}, ATOMS_O[NQ] = {0, 2, 1, 0, 1, 1, 2, 2};
constexpr int NREF = 2;  // species 0 and 1
constexpr bool conserves() {
    for (int r = 0; r < NR; ++r) {
        int h = 0, o = 0;
        for (int i = 0; i < RXN[r].nreac; ++i) { h -= ATOMS_H[RXN[r].reac[i]]; o -= ATOMS_O[RXN[r].reac[i]]; }
        for (int i = 0; i < RXN[r].nprod; ++i) { h += ATOMS_H[RXN[r].prod[i]]; o += ATOMS_O[RXN[r].prod[i]]; }
        if (h != 0 || o != 0) return false;
    }
    return true;
}
static_assert(conserves(), "species 0 and 1 as element references");
constexpr GCoef make_gref() {
    const GCoef g = make_gcoef();
    GCoef d{};
    for (int r = 0; r < 2; ++r)
        for (int k = 0; k < NQ; ++k)
            for (int j = 0; j < 7; ++j)
                d.c[r][k][j] = g.c[r][k][j] - 0.5 * ATOMS_H[k] * g.c[r][0][j] - 0.5 * ATOMS_O[k] * g.c[r][1][j];
    return d;
}
__device__ constexpr GCoef D_GREF = make_gref();

// T-dependent quantities of one evaluation.
struct Kin {
    double T, invT, lnT, rt, irt;  // rt = R T / p0, irt = 1 / rt
    double eg[NQ], ieg[NQ];        // exp(g_k), exp(-g_k), g relative to H2 and O2 (theirs: 1, unused)
    double ar[NEXP];
};
template <int RG>
__device__ __forceinline__ void g_of_T(double T, double lnT, double invT, double* g) {
    const double om = 1.0 - lnT;
#pragma unroll
    for (int k = NREF; k < NQ; ++k) {
        const double* c = D_GREF.c[RG][k];
        const double p = fma(T, fma(T, fma(T, fma(T, c[4], c[3]), c[2]), c[1]), c[0]);
        g[k] = fma(c[5], om, fma(c[6], invT, p));
    }
}
template <int RG>
__device__ __forceinline__ void h_of_T(double T, double invT, double* h) {
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
        const double* a = D_NASA.c[RG][k];
        double p = a[0];
        if (a[1] != 0.0 || a[4] != 0.0)
            p = fma(T, fma(T, fma(T, fma(T, a[4] * 0.2, a[3] * 0.25), a[2] * (1.0 / 3.0)), a[1] * 0.5), a[0]);
        h[k] = fma(a[5], invT, p);
    }
}
__device__ __forceinline__ void kin_at(double T, Kin& k) {
    k.T = T;
    k.lnT = flog(T);
    k.invT = fp_rcp(T);
    k.rt = T * (RU / ONE_ATM);
    k.irt = k.invT * (ONE_ATM / RU);
    double g[NQ];
    if (!fp_lt(TMID, T)) g_of_T<0>(T, k.lnT, k.invT, g);
    else g_of_T<1>(T, k.lnT, k.invT, g);
    // rolled: one body of each exponential, for the instruction cache
#pragma unroll 1
    for (int s = NREF; s < NQ; ++s) fexp_pair(g[s], k.eg[s], k.ieg[s]);
#pragma unroll 1
    for (int i = 0; i < NEXP; ++i) {
        double x = -D_SLOTS.E[i] * k.invT;
        if (D_SLOTS.hasb[i]) x = fma(D_SLOTS.b[i], k.lnT, x);
        k.ar[i] = fexp(x);
    }
}
template <int R>
__device__ __forceinline__ double k_inf(const Kin& k) {
    constexpr ArrTerm t = make_arr().t[R];
    if constexpr (t.kind == ARR_ONE) return c_A[R];
    else if constexpr (t.kind == ARR_INVT) return c_A[R] * k.invT;
    else if constexpr (t.kind == ARR_INVT2) return c_A[R] * k.invT * k.invT;
    else {
        constexpr int sl = slot_of(R);
        if constexpr (t.kind == ARR_T2EXP) return c_A[R] * k.ar[sl] * (k.T * k.T);
        else return c_A[R] * k.ar[sl];
    }
}
template <int R>
__device__ __forceinline__ double k_zero(const Kin& k) {
    constexpr int i = NR + fall_index(R);
    constexpr ArrTerm t = make_arr().t[i];
    if constexpr (t.kind == ARR_ONE) return c_A0[R];
    else {
        constexpr int sl = slot_of(i);
        return c_A0[R] * k.ar[sl];
    }
}
template <int R, int NS>
__device__ __forceinline__ double third(const double* C, double Csum) {
    constexpr Reaction rx = RXN[R];
    double M = Csum;
#pragma unroll
    for (int k = 0; k < NQ; ++k)
        if (rx.eff[k] != 1.0) M = fma(rx.eff[k] - 1.0, C[k], M);
    return M;
}
// Falloff rate constant: k0 M F / (1 + Pr), Pr = k0 M / kinf, F by Troe's formula with the
// table's constant F_cent.  JAC: also T dk/dT and dk/dM.
template <int R, bool JAC>
__device__ __forceinline__ double falloff(const Kin& kc, double M, double& Tdk, double& dkM) {
    constexpr Reaction rx = RXN[R];
    static_assert(rx.type != RXN_FALLOFF || (rx.troeT3 < 1e-20 && rx.troeT1 > 1e20 && !rx.hasT2 && rx.troeA >= 0.5 &&
                                             rx.troeA <= 2.0),
                  "constant F_cent");
    constexpr double lFc = const_log10(rx.troeA), c = -0.4 - 0.67 * lFc, nn = 0.75 - 1.27 * lFc;
    const double kinf = k_inf<R>(kc), k0 = k_zero<R>(kc), k0M = k0 * M;
    const double Pr = fp_div(k0M, kinf);
    const bool tiny = !(__double2hiint(Pr) >= 0x01a56e1f);  // about 1e-300; also 0, negative
    const double x = fma(flog(tiny ? 1e-300 : Pr), fm::INV_LN10, c);
    const double den = fma(-0.14, x, nn), iden = fp_rcp(den);
    const double f1 = x * iden;
    const double g = fp_rcp(fma(f1, f1, 1.0));
    const double F = fexp(g * (lFc * fm::LN10));
    const double i1 = fp_rcp(1.0 + Pr);
    const double Fi = F * i1, k = k0M * Fi;
    if constexpr (JAC) {
        const double dPr = tiny ? 0.0 : (-2.0 * lFc * nn) * (f1 * g * g) * (iden * iden);
        const double d = i1 + dPr;  // d ln k / d ln Pr
        // T dk/dT = k (s_inf + d (s_0 - s_inf)), s = b + E/T
        const double si = fma(rx.EaR, kc.invT, rx.b), s0 = fma(rx.Ea0R, kc.invT, rx.b0);
        Tdk = k * fma(d, s0 - si, si);
        dkM = k0 * Fi * d;
    }
    return k;
}

// prod_reac exp(-g) (RT/p0)^dn: the factor of prod_prod X in the reverse rate.
template <int R>
__device__ __forceinline__ double ieg_factor(const Kin& kc) {
    constexpr Reaction rx = RXN[R];
    constexpr int dn = rx.nprod - rx.nreac;
    double b = 1.0;
    bool set = false;
    auto mul = [&](double v) {
        b = set ? b * v : v;
        set = true;
    };
    if constexpr (rx.reac[0] >= NREF) mul(kc.ieg[rx.reac[0]]);
    if constexpr (rx.nreac == 2) {
        if constexpr (rx.reac[1] >= NREF) mul(kc.ieg[rx.reac[1]]);
    }
    if constexpr (dn == 1) mul(kc.rt);
    if constexpr (dn == -1) mul(kc.irt);
    return b;
}
// ... and with prod_prod exp(g): 1 / Kc
template <int R>
__device__ __forceinline__ double inv_kc_factor(const Kin& kc) {
    constexpr Reaction rx = RXN[R];
    double b = ieg_factor<R>(kc);
    if constexpr (rx.prod[0] >= NREF) b *= kc.eg[rx.prod[0]];
    if constexpr (rx.nprod == 2) {
        if constexpr (rx.prod[1] >= NREF) b *= kc.eg[rx.prod[1]];
    }
    return b;
}

// ---------------------------------------------------------------- right-hand side
template <int R, int NS>
__device__ __forceinline__ void rate(const Kin& kc, const double* C, const double* X, double Csum, double* w) {
    constexpr Reaction rx = RXN[R];
    if constexpr (dup_of(R) < 0) {
        double k;
        if constexpr (rx.type == RXN_FALLOFF) {
            double a, b;
            k = falloff<R, false>(kc, third<R, NS>(C, Csum), a, b);
        } else {
            k = k_inf<R>(kc);
            if constexpr (dup_next(R) >= 0) k += k_inf<dup_next(R)>(kc);
            if constexpr (rx.type == RXN_THREE_BODY) k *= third<R, NS>(C, Csum);
        }
        constexpr int dn = rx.nprod - rx.nreac;
        double f = C[rx.reac[0]];
        if constexpr (rx.nreac == 2) f *= C[rx.reac[1]];
        double b = X[rx.prod[0]];
        if constexpr (rx.nprod == 2) b *= X[rx.prod[1]];
        const double q = k * fma(-ieg_factor<R>(kc), b, f);
#pragma unroll
        for (int s = 0; s < NQ; ++s) {
            if (D_NU.v[R][s] == 1) w[s] += q;
            else if (D_NU.v[R][s] == -1) w[s] -= q;
            else if (D_NU.v[R][s] != 0) w[s] = fma((double)D_NU.v[R][s], q, w[s]);
        }
    }
}
template <int NS, size_t... Rs>
__device__ __forceinline__ void rates(const Kin& kc, const double* C, const double* X, double Csum, double* w,
                                      std::index_sequence<Rs...>) {
    (rate<(int)Rs, NS>(kc, C, X, Csum, w), ...);
}

// A cell between attempts.
template <int NS>
struct Cell {
    static constexpr int N = NS - 1, NI = NS - NQ;
    double y[N];     // mass fractions (the last species closes)
    double Cin[NI];  // concentrations of the inert species (constant over the interval)
    double mi[2][6], Ci;  // their mixture coefficients in both NASA ranges, and total
    double h, t, tend, rho, ir, e, et, T;  // et = rho e / R; T: of y, or near it
    double mom[3];   // rho*u, rho*v, rho*E: chemistry leaves them unchanged
    int steps, attempts;
    bool rejectLast, rejectMore, fresh;  // fresh: no attempt made yet
};

template <int NS>
__device__ __forceinline__ bool weights_T(const Cell<NS>& c, const double* C, double& T, double& cv, double& Csum) {
    Csum = c.Ci;
#pragma unroll
    for (int k = 0; k < NQ; ++k) Csum += C[k];
    const float t = fp_to_f32(T);
    const bool low = t <= (float)TMID;
    double m[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) m[j] = low ? c.mi[0][j] : c.mi[1][j];
    if (low) mix_add_r<NQ, 0>(C, m);
    else mix_add_r<NQ, 1>(C, m);
    if (newton_T(m, c.et, low, t, T, cv)) return true;
    double w[NS], Ts = T, cvs = 0.0;
#pragma unroll
    for (int k = 0; k < NQ; ++k) w[k] = C[k];
#pragma unroll
    for (int k = NQ; k < NS; ++k) w[k] = c.Cin[k - NQ];
    const bool ok = solve_T_slow<NS, false>(w, c.et, Ts, m, cvs);
    T = Ts;
    cv = cvs;
    return ok;
}

// w = dC/dt at concentrations C; T: guess in, temperature out.
template <int NS>
__device__ __noinline__ bool rhs(const Cell<NS>& c, const double* Cin, double& T_io, double* w_out) {
    double C[NQ], X[NQ], w[NQ], Csum, cv, T = T_io;
#pragma unroll
    for (int k = 0; k < NQ; ++k) C[k] = Cin[k];
    if (!weights_T<NS>(c, C, T, cv, Csum)) return false;
    T_io = T;
    Kin kc;
    kin_at(T, kc);
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
        X[k] = k < NREF ? C[k] : C[k] * kc.eg[k];
        w[k] = 0.0;
    }
    rates<NS>(kc, C, X, Csum, w, std::make_index_sequence<NR>{});
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
        ok = ok && fp_finite(w[k]);
        w_out[k] = w[k];
    }
    return ok;
}

// ---------------------------------------------------------------- Jacobian and LU
// -dw/dC (without the temperature and total-concentration terms) into A, those terms'
// row factors into Tn (-T dw/dT) and Dn (-dw/dM summed over third bodies of efficiency 1).
template <int R, int NS>
__device__ __forceinline__ void jac(const Kin& kc, const double* C, const double* h, double Csum, double* w, double* A,
                                    double* Tn, double* Dn) {
    constexpr Reaction rx = RXN[R];
    if constexpr (dup_of(R) < 0) {
        constexpr int dn = rx.nprod - rx.nreac, r0 = rx.reac[0], r1 = rx.nreac == 2 ? rx.reac[1] : -1,
                      p0 = rx.prod[0], p1 = rx.nprod == 2 ? rx.prod[1] : -1;
        double k, Tdk = 0.0, dkM = 0.0, s = 0.0;  // T dk/dT = Tdk, or k s where s is set
        constexpr bool bySum = dup_next(R) >= 0 || rx.type == RXN_FALLOFF;
        if constexpr (rx.type == RXN_FALLOFF) {
            k = falloff<R, true>(kc, third<R, NS>(C, Csum), Tdk, dkM);
        } else {
            k = k_inf<R>(kc);
            s = fma(rx.EaR, kc.invT, rx.b);
            if constexpr (dup_next(R) >= 0) {
                constexpr int q = dup_next(R);
                const double k2 = k_inf<q>(kc);
                Tdk = fma(k, s, k2 * fma(RXN[q].EaR, kc.invT, RXN[q].b));
                k += k2;
            }
            if constexpr (rx.type == RXN_THREE_BODY) {
                dkM = k;
                k *= third<R, NS>(C, Csum);
            }
        }
        double dr0, dr1 = 0.0, fwd;
        if constexpr (rx.nreac == 1) {
            dr0 = k;
            fwd = k * C[r0];
        } else if constexpr (r0 == r1) {
            dr0 = k * C[r0];
            fwd = dr0 * C[r0];
            dr0 += dr0;
        } else {
            dr0 = k * C[r1];
            dr1 = k * C[r0];
            fwd = dr0 * C[r0];
        }
        const double ikc = inv_kc_factor<R>(kc);
        double dp0, dp1 = 0.0, rev;
        const double b = k * ikc;  // reverse rate constant
        if constexpr (rx.nprod == 1) {
            dp0 = b;
            rev = b * C[p0];
        } else if constexpr (p0 == p1) {
            dp0 = b * C[p0];
            rev = dp0 * C[p0];
            dp0 += dp0;
        } else {
            dp0 = b * C[p1];
            dp1 = b * C[p0];
            rev = dp0 * C[p0];
        }
        const double q = fwd - rev;
        // T dq/dT = T dk/dT (q / k) + rev (T dlnKc/dT),  T dlnKc/dT = sum nu h/RT - dn
        double hh = h[p0];
        if constexpr (p1 >= 0) hh += h[p1 < 0 ? 0 : p1];
        hh -= h[r0];
        if constexpr (r1 >= 0) hh -= h[r1 < 0 ? 0 : r1];
        if constexpr (dn != 0) hh -= (double)dn;
        double net = 0.0, qT;
        if constexpr (bySum || rx.type != RXN_ELEMENTARY) {
            // q / k from the products, so that k = 0 needs no case of its own
            double f = C[r0], g = C[p0];
            if constexpr (rx.nreac == 2) f *= C[r1 < 0 ? 0 : r1];
            if constexpr (rx.nprod == 2) g *= C[p1 < 0 ? 0 : p1];
            net = fma(-ikc, g, f);
        }
        if constexpr (bySum) qT = fma(rev, hh, Tdk * net);
        else qT = fma(rev, hh, q * s);
        double t = 0.0;
        if constexpr (rx.type != RXN_ELEMENTARY) t = dkM * net;
        // columns: participants, and third bodies of another efficiency
#pragma unroll
        for (int m = 0; m < NQ; ++m) {
            const bool part = m == r0 || m == r1 || m == p0 || m == p1;
            const bool eff = rx.type != RXN_ELEMENTARY && rx.eff[m] != 1.0;
            if (!part && !eff) continue;
            double d = 0.0;
            bool set = false;
            if (m == r0) { d = dr0; set = true; }
            if (m == r1 && r0 != r1) { d = set ? d + dr1 : dr1; set = true; }
            if (m == p0) { d = set ? d - dp0 : -dp0; set = true; }
            if (m == p1 && p0 != p1) { d = set ? d - dp1 : -dp1; set = true; }
            if (eff) d = set ? fma(rx.eff[m] - 1.0, t, d) : (rx.eff[m] - 1.0) * t;
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                if (D_NU.v[R][i] == 1) A[i * NQ + m] -= d;
                else if (D_NU.v[R][i] == -1) A[i * NQ + m] += d;
                else if (D_NU.v[R][i] != 0) A[i * NQ + m] = fma(-(double)D_NU.v[R][i], d, A[i * NQ + m]);
            }
        }
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            const int nu = D_NU.v[R][i];
            if (nu == 0) continue;
            if (nu == 1) { w[i] += q; Tn[i] -= qT; }
            else if (nu == -1) { w[i] -= q; Tn[i] += qT; }
            else { w[i] = fma((double)nu, q, w[i]); Tn[i] = fma(-(double)nu, qT, Tn[i]); }
            if constexpr (rx.type != RXN_ELEMENTARY) {
                if (nu == 1) Dn[i] -= t;
                else if (nu == -1) Dn[i] += t;
                else Dn[i] = fma(-(double)nu, t, Dn[i]);
            }
        }
    }
}
template <int NS, size_t... Rs>
__device__ __forceinline__ void jacs(const Kin& kc, const double* C, const double* h, double Csum, double* w, double* A,
                                     double* Tn, double* Dn, std::index_sequence<Rs...>) {
    (jac<(int)Rs, NS>(kc, C, h, Csum, w, A, Tn, Dn), ...);
}

// LU with partial pivoting in registers: row interchanges as compare-and-swap of row k with
// every later row (28 possible, recorded in a mask; rare, as I/(h gamma) - J is dominated by
// its diagonal), so every index is static.  The diagonal holds 1/U_kk.
__device__ __forceinline__ bool lu8(double* A, unsigned& swaps) {
    swaps = 0;
    int bit = 0;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
#pragma unroll
        for (int i = k + 1; i < NQ; ++i, ++bit) {
            if (fp_abs_bits(A[i * NQ + k]) > fp_abs_bits(A[k * NQ + k])) {
                swaps |= 1u << bit;
#pragma unroll
                for (int j = 0; j < NQ; ++j) {
                    const double t = A[k * NQ + j];
                    A[k * NQ + j] = A[i * NQ + j];
                    A[i * NQ + j] = t;
                }
            }
        }
        if (fp_zero(A[k * NQ + k]) || !fp_finite(A[k * NQ + k])) return false;
        const double inv = fp_rcp(A[k * NQ + k]);
        A[k * NQ + k] = inv;
#pragma unroll
        for (int i = k + 1; i < NQ; ++i) {
            const double l = A[i * NQ + k] * inv;
            A[i * NQ + k] = l;
#pragma unroll
            for (int j = k + 1; j < NQ; ++j) A[i * NQ + j] = fma(-l, A[k * NQ + j], A[i * NQ + j]);
        }
    }
    return true;
}
static __device__ __noinline__ void swap_rows8(unsigned swaps, double* b) {
    int bit = 0;
#pragma unroll 1
    for (int k = 0; k < NQ; ++k)
#pragma unroll 1
        for (int i = k + 1; i < NQ; ++i, ++bit)
            if (swaps >> bit & 1u) {
                const double t = b[k];
                b[k] = b[i];
                b[i] = t;
            }
}
__device__ __forceinline__ void solve8(const double* Lu, unsigned swaps, double* b) {
    if (swaps) {
        double t[NQ];
#pragma unroll
        for (int i = 0; i < NQ; ++i) t[i] = b[i];
        swap_rows8(swaps, t);
#pragma unroll
        for (int i = 0; i < NQ; ++i) b[i] = t[i];
    }
#pragma unroll
    for (int i = 1; i < NQ; ++i)
#pragma unroll
        for (int j = 0; j < i; ++j) b[i] = fma(-Lu[(i * NQ + j)], b[j], b[i]);
#pragma unroll
    for (int i = NQ - 1; i >= 0; --i) {
#pragma unroll
        for (int j = i + 1; j < NQ; ++j) b[i] = fma(-Lu[(i * NQ + j)], b[j], b[i]);
        b[i] *= Lu[(i * NQ + i)];
    }
}

enum : int { LU_OK = 0, LU_RHS_FAILED, LU_SINGULAR, LU_SCREENED, LU_COLD };

// f0 = dC/dt, J and the factors of inv I - J at concentrations C (T: guess in, temperature
// out).  SCREEN, on a cell's first attempt: the frozen-cell screen (below), and LU_COLD
// when the cell has no step size yet.
//
// The screen: in the scaled variables z_i = y_i / sc_i (sc_i = atol + rtol |y_i|), with
// a = ||J_z||_inf dt, if a <= 20, ||f0_z||_inf dt e^a <= 1 and ||f0_z||_inf dt a^2 e^a / 6 <=
// 1e-5, the interval is taken as one second-order Taylor step y1 = y0 + dt f0 + dt^2/2 J f0:
// for the linearised system its remainder sum_{k>=3} dt^k/k! J^(k-1) f0 is bounded by the
// last expression, i.e. below 1e-5 tolerance units.
template <int NS, bool SCREEN>
__device__ __noinline__ int jac_lu(Cell<NS>& c, const double* Cm, double* f0, double* Lu, unsigned& swaps, double inv,
                                   double rtol, double atol) {
    double C[NQ], w[NQ], A[NQ * NQ], Tn[NQ], Dn[NQ], h[NQ], Csum, cv, T = c.T;
#pragma unroll
    for (int k = 0; k < NQ; ++k) C[k] = Cm[k];
    if (!weights_T<NS>(c, C, T, cv, Csum)) return LU_RHS_FAILED;
    c.T = T;
    Kin kc;
    kin_at(T, kc);
    if (!fp_lt(TMID, T)) h_of_T<0>(T, kc.invT, h);
    else h_of_T<1>(T, kc.invT, h);
#pragma unroll
    for (int i = 0; i < NQ * NQ; ++i) A[i] = 0.0;
#pragma unroll
    for (int k = 0; k < NQ; ++k) w[k] = Tn[k] = Dn[k] = 0.0;
    jacs<NS>(kc, C, h, Csum, w, A, Tn, Dn, std::make_index_sequence<NR>{});
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
        ok = ok && fp_finite(w[k]);
        f0[k] = w[k];
    }
    if (!ok) return LU_RHS_FAILED;
    // (1/T) dT/dC_j = -(h_j/RT - 1) / sum C cv; closing-species terms vanish on vectors
    // that conserve mass, as f0 and every stage do
    const double icv = -fp_rcp(cv);
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
        const double tj = (h[j] - 1.0) * icv;
#pragma unroll
        for (int i = 0; i < NQ; ++i) A[i * NQ + j] += fma(Tn[i], tj, Dn[i]);
    }
    if constexpr (SCREEN) {
        if (c.fresh) {
            const double dt = c.tend;
            double sc[NQ], fz = 0.0, jz = 0.0;
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                sc[i] = fma(rtol, fabs(c.y[i]), atol) * INVW.v[i];
                fz = fp_abs_max(fz, fp_div(w[i] * c.ir, sc[i]));
            }
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                double r = 0.0;
#pragma unroll
                for (int j = 0; j < NQ; ++j) r = fma(fabs(A[i * NQ + j]), sc[j], r);
                jz = fp_abs_max(jz, fp_div(r, sc[i]));
            }
            const double a = jz * dt;
            if (fp_lt(a, 20.0)) {
                const double fe = fz * dt * fexp(a);
                if (fp_ge0(1.0 - fe) && fp_ge0(6e-5 - fe * a * a)) {
#pragma unroll
                    for (int i = 0; i < NQ; ++i) {
                        double v = 0.0;
#pragma unroll
                        for (int j = 0; j < NQ; ++j) v = fma(A[i * NQ + j], w[j], v);
                        c.y[i] = fma(dt * fma(-0.5 * dt, v, w[i]), D_MW.v[i] * c.ir, c.y[i]);
                    }
                    return LU_SCREENED;
                }
            }
            if (!fp_pos(c.h)) return LU_COLD;
        }
    }
#pragma unroll
    for (int i = 0; i < NQ; ++i) A[i * NQ + i] += inv;
    if (!lu8(A, swaps)) return LU_SINGULAR;
#pragma unroll
    for (int i = 0; i < NQ * NQ; ++i) Lu[i] = A[i];
    return LU_OK;
}

// WRMS norm over the NS - 1 unknowns of the reference (N2's component, when N2 is one of
// them, is tail)
template <int NS>
__device__ __forceinline__ double wrms(const double* v, const double* y0, const double* y1, double rtol, double atol,
                                       double tail = 0.0) {
    double s = tail;
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
        const double sc = fma(rtol, fp_abs_max(y0[i], y1[i]), atol);
        const double r = fp_div(v[i], sc);
        s = fma(r, r, s);
    }
    return fp_max(fp_sqrt(s * (1.0 / (NS - 1))), 1e-10);
}

// Takes the state u into c (chemistry.cpp:55-62) and checks it; h = 0 (no step size yet).
template <int NS>
__device__ __forceinline__ bool load(Cell<NS>& c, const double* u, double dt) {
    constexpr int N = NS - 1;
    if (!(dt > 0.0) || !isfinite(dt)) return false;
    if (!admissible_state<NS>(u, 0.0)) return false;
    double rho = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k) rho += u[k];
    const double ir = 1.0 / rho;
    const double uu = u[NS] * ir, vv = u[NS + 1] * ir;
    c.rho = rho;
    c.ir = ir;
    c.e = u[NS + 2] * ir - 0.5 * (uu * uu + vv * vv);
    c.et = rho * c.e * (1.0 / RU);
    c.mom[0] = u[NS];
    c.mom[1] = u[NS + 1];
    c.mom[2] = u[NS + 2];
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        c.y[k] = u[k] * ir;
        s += c.y[k];
    }
    if constexpr (NS == 10) c.Cin[0] = u[8] * INVW.v[8];
    c.Cin[NS - 1 - NQ] = rho * (1.0 - s) * INVW.v[NS - 1];
    c.Ci = 0.0;
#pragma unroll
    for (int j = 0; j < 6; ++j) c.mi[0][j] = c.mi[1][j] = 0.0;
#pragma unroll
    for (int k = NQ; k < NS; ++k) {
        c.Ci += c.Cin[k - NQ];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            c.mi[0][j] = fma(c.Cin[k - NQ], D_ECOEF.c[0][k][j], c.mi[0][j]);
            c.mi[1][j] = fma(c.Cin[k - NQ], D_ECOEF.c[1][k][j], c.mi[1][j]);
        }
    }
    c.T = estimate_T<NS>(u, c.et);
    c.h = 0.0;
    c.t = 0.0;
    c.tend = dt;
    c.steps = 0;
    c.attempts = 0;
    c.rejectLast = c.rejectMore = false;
    c.fresh = true;
    return true;
}

// Starting step: Hairer's estimate in time scaled by the interval.
template <int NS>
__device__ __noinline__ bool first_step(Cell<NS>& c, double rtol, double atol) {
    double C[NQ], f0[NQ], f1[NQ], v[NQ], yn[NQ];
    const double dt = c.tend;
#pragma unroll
    for (int i = 0; i < NQ; ++i) C[i] = c.rho * c.y[i] * INVW.v[i];
    if (!rhs<NS>(c, C, c.T, f0)) return false;
    double tail = 0.0;
    if constexpr (NS == 10) {
        const double r = c.y[8] / (atol + rtol * fabs(c.y[8]));
        tail = r * r;
    }
    const double d0 = wrms<NS>(c.y, c.y, c.y, rtol, atol, tail);
#pragma unroll
    for (int i = 0; i < NQ; ++i) v[i] = f0[i] * (D_MW.v[i] * c.ir);
    const double d1 = wrms<NS>(v, c.y, c.y, rtol, atol) * dt;
    const double hh = d1 < 1e-5 ? 1.0 : fmin(1.0, 0.01 * d0 / d1);
#pragma unroll
    for (int i = 0; i < NQ; ++i) yn[i] = fma(hh * dt, f0[i], C[i]);
    double d2 = 1e30, T = c.T;
    if (rhs<NS>(c, yn, T, f1)) {
#pragma unroll
        for (int i = 0; i < NQ; ++i) v[i] = (f1[i] - f0[i]) / hh * (D_MW.v[i] * c.ir);
        d2 = wrms<NS>(v, c.y, c.y, rtol, atol);
    }
    const double mx = fmax(d1, d2);
    const double h1 = mx <= 1e-15 ? 1.0 : pow(0.01 / mx, 0.2);
    c.h = fmin(fmin(100.0 * hh, h1), 1.0) * dt;
    return true;
}

// Loads a cell and prepares the integration.  Returns CELL_CONTINUE or CELL_FAIL.
template <int NS>
__device__ __forceinline__ int begin(Cell<NS>& c, const double* u, double dt, double rtol, double atol) {
    if (!load<NS>(c, u, dt) || !first_step<NS>(c, rtol, atol)) return CELL_FAIL;
    return CELL_CONTINUE;
}
// The batched form's start (extension to the reference's per-call CVODE restart): the first
// step size is the cell's proposed step from the previous call (h_prev > 0), and the first
// attempt screens frozen cells (jac_lu).
template <int NS>
__device__ __forceinline__ int begin_warm(Cell<NS>& c, const double* u, double dt, double h_prev) {
    if (!load<NS>(c, u, dt)) return CELL_FAIL;
    if (h_prev > 0.0 && isfinite(h_prev)) c.h = fmin(h_prev, dt);
    return CELL_CONTINUE;
}

// One step attempt (the body of the KPP accept loop).  Lu: 64 doubles of scratch;
// screened is set when a frozen cell was finished by the screen.
template <int NS, bool SCREEN>
__device__ __forceinline__ int attempt(Cell<NS>& c, double rtol, double atol, double* Lu, bool* screened = nullptr) {
    double C0[NQ], K[6][NQ], Ys[NQ];
    unsigned swaps = 0;
    bool last = false;
    double h = c.h;
    if (fp_ge0(fma(1.01, h, c.t) - c.tend)) {
        h = c.tend - c.t;
        last = true;
    }
    if (!SCREEN || fp_pos(c.h)) c.h = h;
    const double ih = fp_pos(h) ? fp_rcp(h) : 0.0;
#pragma unroll
    for (int i = 0; i < NQ; ++i) Ys[i] = C0[i] = c.rho * c.y[i] * INVW.v[i];
    const int r = jac_lu<NS, SCREEN>(c, C0, K[0], Lu, swaps, ih * (1.0 / RGAMMA), rtol, atol);
    if (r == LU_RHS_FAILED) return CELL_FAIL;
    if (SCREEN) {
        if (r == LU_SCREENED) {
            c.t = c.tend;
            *screened = true;
            return CELL_DONE;
        }
        if (r == LU_COLD) return first_step<NS>(c, rtol, atol) && fp_pos(c.h) ? CELL_CONTINUE : CELL_FAIL;
        c.fresh = false;
    }
    if (++c.attempts > 4 * MAX_STEPS) return CELL_MAXSTEPS;
    bool ok = r == LU_OK;
    double T = c.T;
    if (ok) {
        double b[NQ];
#pragma unroll
        for (int i = 0; i < NQ; ++i) b[i] = K[0][i];
        solve8(Lu, swaps, b);
#pragma unroll
        for (int i = 0; i < NQ; ++i) K[0][i] = b[i];
    }
#pragma unroll 1
    for (int s = 1; ok && s < 6; ++s) {
        const int base = s * (s - 1) / 2;
        double b[NQ], f[NQ];
#pragma unroll
        for (int i = 0; i < NQ; ++i) b[i] = 0.0;
        // the last two stages and the result share y + sum a_j K_j term by term (RA rows 4, 5
        // and RM): each adds one K to the one before
        if (s < 5) {
#pragma unroll
            for (int i = 0; i < NQ; ++i) Ys[i] = C0[i];
        }
#pragma unroll 1
        for (int j = 0; j < s; ++j) {
            const double a = RA[base + j], g = RC[base + j];
            const bool add = s < 5 || j == 4;
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                const double kj = K[j][i];
                b[i] = fma(g, kj, b[i]);
                if (add) Ys[i] = fma(a, kj, Ys[i]);
            }
        }
        ok = rhs<NS>(c, Ys, T, f);
        if (!ok) break;
#pragma unroll
        for (int i = 0; i < NQ; ++i) b[i] = fma(ih, b[i], f[i]);
        solve8(Lu, swaps, b);
#pragma unroll
        for (int i = 0; i < NQ; ++i) K[s][i] = b[i];
    }
    double err = __longlong_as_double(0x7ff0000000000000ll), yn[NQ];  // +inf
    if (ok) {
        double ev[NQ];
        bool fin = true;
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            const double wr = D_MW.v[i] * c.ir;
            // the increments first: a cell that hardly moves keeps its y to the last bit
            yn[i] = fma((Ys[i] - C0[i]) + K[5][i], wr, c.y[i]);
            ev[i] = K[5][i] * wr;
            fin = fin && fp_finite(yn[i]);
        }
        if (fin) err = wrms<NS>(ev, c.y, yn, rtol, atol);
    }
    if (!fp_finite(err)) {
        c.h *= 0.25;
        c.rejectLast = true;
        if (!(c.h > 1e-300) || c.t + c.h == c.t) return CELL_FAIL;
        return CELL_CONTINUE;
    }
    const double fac = fp_div(0.9, fp_sqrt(fp_sqrt(err)));
    double hnew = c.h * fp_min(6.0, fp_max(0.2, fac));
    if (fp_ge0(1.0 - err)) {
        c.t = last ? c.tend : c.t + c.h;
        c.T = T;
#pragma unroll
        for (int i = 0; i < NQ; ++i) c.y[i] = yn[i];
        if (c.rejectLast) hnew = fp_min(hnew, c.h);
        c.rejectLast = c.rejectMore = false;
        ++c.steps;
        c.h = hnew;
        if (last || !fp_lt(c.t, c.tend)) return CELL_DONE;
        if (c.steps >= MAX_STEPS) return CELL_MAXSTEPS;
        return CELL_CONTINUE;
    }
    if (c.rejectMore) hnew = c.h * 0.1;
    c.rejectMore = c.rejectLast;
    c.rejectLast = true;
    c.h = hnew;
    if (!(c.h > 1e-300) || c.t + c.h == c.t) return CELL_FAIL;
    return CELL_CONTINUE;
}

// chemistry.cpp:63-70: clip, close the mass with the last species, final check.
// Writes the whole state u (momentum and energy as they came in).
template <int NS>
__device__ __forceinline__ bool finish(const Cell<NS>& c, double* u) {
    constexpr int N = NS - 1;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const double v = c.y[k];
        if (!fp_finite(v) || fp_lt(v, -1e-13)) return false;
        u[k] = c.rho * (fp_neg(v) ? 0.0 : v);
        s += u[k];
    }
    u[N] = c.rho - s;
    u[NS] = c.mom[0];
    u[NS + 1] = c.mom[1];
    u[NS + 2] = c.mom[2];
    return admissible_state<NS>(u, c.T);
}

}  // namespace cell
}  // namespace hf
