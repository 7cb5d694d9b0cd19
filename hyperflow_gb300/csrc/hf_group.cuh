// One cell per group of 8 lanes (4 cells per warp): the Rodas4 integration of hf_cell.cuh
// with the 8 reacting species (H2, O2, H2O, H, O, OH, HO2, H2O2) spread over a group's lanes.
//
// Why: a warp's FP64 instruction holds its sub-partition for 64 cycles whatever the number
// of active lanes, so one cell's step chain (about 5,100 FP64 instructions an attempt on one
// lane) is what a batch waits for once its expensive cells no longer fill the 608
// sub-partitions.  Here lane t holds species t, row t of the matrix and of its LU factors
// and evaluates reactions t, t + 8, t + 16: about 1,600 FP64 instructions an attempt:
// 73 us alone on its sub-partition against 206 on a lane, at about 3 times the pipe's time per
// cell once the chip is full (rates measured at k_order_scan, hf_chem.cu).  All four groups of a warp run the same
// instructions; groups without a cell, or whose step already failed, compute along on valid
// numbers and write nothing, so no shuffle is ever divergent.
//
// The same ODE, unknowns, tableau, error norm, controller and cell semantics as
// hf_cell.cuh; results agree to rounding (sums are taken in another order).
#pragma once
#include "hf_cell.cuh"

namespace hf {
namespace grp8 {

using cell::NQ;
constexpr int G = 8;
constexpr int NROUND = (NR + G - 1) / G, NSLOT = NROUND * G;
constexpr unsigned FULL = 0xffffffffu;

// ---------------------------------------------------------------- tables
struct Slot {
    double b, E, b0, E0, lfc;
    int r0, r1, p0, p1;  // species, -1 none
    int dn, type, third; // third: 1 + efficiency set, 0 none
    int low;             // falloff: the lane whose last slot is its k0; extra slots: the reaction
    int dup;             // 1: add the next slot's rate constant (same species); -1: added there
};
// Slots NR, NR + 1, ... (idle otherwise) evaluate the low-pressure rate constants of the
// falloff reactions, in one round with the others' exponentials.
constexpr int fall_reaction(int f) {
    for (int r = 0; r < NR; ++r)
        if (RXN[r].type == RXN_FALLOFF && fall_index(r) == f) return r;
    return -1;
}
constexpr int NEFF = 2, NVAL = 5;  // per slot: dq/dC of the four participants, dq/dM
constexpr int MAXLIST = 20;
struct Tables {
    Slot s[NSLOT];
    double eff[NEFF][NS_MAX];
    int neff;
    // w_t = sum_e wn[t][e] q[wr[t][e]]
    int nw;
    int wr[NQ][MAXLIST];
    double wn[NQ][MAXLIST];
    // J_tj = sum_e jn[t][e] v[jr[t][e]], e in [j0[j], j0[j + 1]); v[slot * NVAL + which]
    int j0[NQ + 1];
    int jr[NQ][NQ * MAXLIST];
    double jn[NQ][NQ * MAXLIST];
    bool ok;
};
constexpr Tables make_tables() {
    Tables t{};
    t.ok = NR + NFALL <= NSLOT && NR / G == NROUND - 1;  // the extra slots are in the last round
    const cell::NetNu nu = cell::make_nu();
    for (int r = 0; r < NSLOT; ++r) {
        Slot& s = t.s[r];
        s.r0 = s.r1 = s.p0 = s.p1 = -1;
        if (r >= NR) {
            if (r < NR + NFALL) {
                s.b = RXN[fall_reaction(r - NR)].b0;
                s.E = RXN[fall_reaction(r - NR)].Ea0R;
                s.low = fall_reaction(r - NR);
            }
            continue;
        }
        const Reaction& x = RXN[r];
        s.low = x.type == RXN_FALLOFF ? (NR + fall_index(r)) % G : 0;
        s.b = x.b; s.E = x.EaR; s.b0 = x.b0; s.E0 = x.Ea0R;
        s.type = x.type;
        s.lfc = x.type == RXN_FALLOFF ? const_log10(x.troeA) : 0.0;
        s.r0 = x.reac[0];
        if (x.nreac == 2) s.r1 = x.reac[1];
        s.p0 = x.prod[0];
        if (x.nprod == 2) s.p1 = x.prod[1];
        s.dn = x.nprod - x.nreac;
        if (cell::dup_next(r) >= 0) {
            s.dup = 1;
            if (cell::dup_next(r) != r + 1 || (r + 1) / G != r / G) t.ok = false;
        }
        if (cell::dup_of(r) >= 0) s.dup = -1;
        if (x.type != RXN_ELEMENTARY) {
            int q = -1;
            for (int e = 0; e < t.neff; ++e) {
                bool same = true;
                for (int k = 0; k < NS_MAX; ++k) same = same && t.eff[e][k] == x.eff[k];
                if (same) q = e;
            }
            if (q < 0) {
                if (t.neff == NEFF) { t.ok = false; continue; }
                q = t.neff++;
                for (int k = 0; k < NS_MAX; ++k) t.eff[q][k] = x.eff[k];
            }
            s.third = 1 + q;
        }
    }
    for (int k = 0; k < NQ; ++k) {
        int n = 0;
        for (int r = 0; r < NR; ++r)
            if (nu.v[r][k] != 0 && cell::dup_of(r) < 0) {
                if (n == MAXLIST) { t.ok = false; break; }
                t.wr[k][n] = r;
                t.wn[k][n] = nu.v[r][k];
                ++n;
            }
        t.nw = n > t.nw ? n : t.nw;
    }
    // columns padded to the longest row (index 0, weight 0)
    for (int j = 0; j < NQ; ++j) {
        int mx = 0;
        for (int k = 0; k < NQ; ++k) {
            int n = t.j0[j];
            auto add = [&](int r, int which, double w) {
                if (n >= NQ * MAXLIST) { t.ok = false; return; }
                t.jr[k][n] = r * NVAL + which;
                t.jn[k][n] = w;
                ++n;
            };
            for (int r = 0; r < NR; ++r) {
                const double v = nu.v[r][k];
                if (v == 0.0 || cell::dup_of(r) >= 0) continue;
                const Slot& s = t.s[r];
                if (s.r0 == j) add(r, 0, v);
                if (s.r1 == j) add(r, 1, v);
                if (s.p0 == j) add(r, 2, -v);
                if (s.p1 == j) add(r, 3, -v);
                if (s.third && RXN[r].eff[j] != 1.0) add(r, 4, v * (RXN[r].eff[j] - 1.0));
            }
            mx = n - t.j0[j] > mx ? n - t.j0[j] : mx;
        }
        t.j0[j + 1] = t.j0[j] + mx;
    }
    return t;
}
constexpr Tables H_TAB = make_tables();
static_assert(H_TAB.ok, "the group integrator's tables do not fit this mechanism");
__device__ constexpr Tables D_TAB = make_tables();
constexpr int NW = H_TAB.nw;
constexpr bool round_has_dn(int rnd) {
    for (int r = rnd * G; r < rnd * G + G && r < NR; ++r)
        if (RXN[r].nprod != RXN[r].nreac) return true;
    return false;
}
constexpr bool round_has_third(int rnd) {
    for (int r = rnd * G; r < rnd * G + G && r < NR; ++r)
        if (RXN[r].type != RXN_ELEMENTARY) return true;
    return false;
}
constexpr bool round_has_dup(int rnd) {
    for (int r = rnd * G; r < rnd * G + G && r < NR; ++r)
        if (cell::dup_next(r) >= 0) return true;
    return false;
}
// what inert species add to the values of a solve (mixture coefficients, then third bodies)
struct InertCoef { double v[2][2][G]; };  // [inert][range][value]
constexpr InertCoef make_inert() {
    InertCoef c{};
    const ECoef e = make_ecoef();
    for (int s = 0; s < 2; ++s)
        for (int r = 0; r < 2; ++r)
            for (int j = 0; j < G; ++j) c.v[s][r][j] = j < 6 ? e.c[r][NQ + s][j] : H_TAB.eff[j - 6][NQ + s];
    return c;
}
__device__ constexpr InertCoef D_INERT = make_inert();

// ---------------------------------------------------------------- group primitives
__device__ __forceinline__ int lane8() { return threadIdx.x & 7; }
__device__ __forceinline__ double get(double v, int src) { return __shfl_sync(FULL, v, src, 8); }
__device__ __forceinline__ double xsum(double v) {
    v += __shfl_xor_sync(FULL, v, 1);
    v += __shfl_xor_sync(FULL, v, 2);
    v += __shfl_xor_sync(FULL, v, 4);
    return v;
}
__device__ __forceinline__ double xmax_abs(double v) {
    v = fp_abs_max(v, __shfl_xor_sync(FULL, v, 1));
    v = fp_abs_max(v, __shfl_xor_sync(FULL, v, 2));
    return fp_abs_max(v, __shfl_xor_sync(FULL, v, 4));
}
// whether p holds on every lane of the caller's group
__device__ __forceinline__ bool all8(bool p) {
    return ((__ballot_sync(FULL, !p) >> (threadIdx.x & 24)) & 0xffu) == 0;
}
// Eight sums over the group's lanes, one per lane: lane t returns sum over lanes of v[t].
// 7 additions (each step halves the values a lane keeps).
__device__ __forceinline__ double reduce_scatter(const double (&v)[G]) {
    const int t = lane8();
    double a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double keep = t & 4 ? v[i + 4] : v[i], send = t & 4 ? v[i] : v[i + 4];
        a[i] = keep + __shfl_xor_sync(FULL, send, 4);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const double keep = t & 2 ? a[i + 2] : a[i], send = t & 2 ? a[i] : a[i + 2];
        b[i] = keep + __shfl_xor_sync(FULL, send, 2);
    }
    const double keep = t & 1 ? b[1] : b[0], send = t & 1 ? b[0] : b[1];
    return keep + __shfl_xor_sync(FULL, send, 1);
}

struct Partials {  // of one group's reactions: T dq/dT, and per reaction the NVAL partials
    double qT[NR], v[NR * NVAL];
};
struct Shared {  // of one group
    double q[NR];
    Partials p;
};

// A group's cell; every lane holds the same values but for y (mass fraction of its species).
template <int NS>
struct Cell {
    static constexpr int NI = NS - NQ;
    double y, yN2, Cin[NI];
    double h, t, tend, rho, ir, et, T;
    double hu;  // step size of the last attempt
    double mom[3];
    int steps, attempts;
    bool active, rejectLast, rejectMore, fresh;
};

// Temperature, heat capacity and third-body concentrations at the group's concentrations.
template <int NS>
__device__ __forceinline__ bool temperature(const double* Cin, double et, double C, bool active, double& T, double& cv,
                                            double& M1, double& M2) {
    const int t = lane8();
    const float tf = fp_to_f32(T);
    const bool low = tf <= (float)TMID;
    const int rg = low ? 0 : 1;
    double v[G];
#pragma unroll
    for (int j = 0; j < 6; ++j) v[j] = C * D_ECOEF.c[rg][t][j];
    v[6] = C * D_TAB.eff[0][t];
    v[7] = C * D_TAB.eff[1][t];
    double s = reduce_scatter(v);
    s = fma(Cin[0], D_INERT.v[0][rg][t], s);
    if constexpr (NS == 10) s = fma(Cin[1], D_INERT.v[1][rg][t], s);
    double m[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) m[j] = get(s, j);
    M1 = get(s, 6);
    M2 = get(s, 7);
    bool ok = newton_T(m, et, low, tf, T, cv);
    if (__any_sync(FULL, active && !ok)) {
        double w[NS], Ts = T, cvs;
#pragma unroll
        for (int k = 0; k < NQ; ++k) w[k] = get(C, k);
#pragma unroll
        for (int k = NQ; k < NS; ++k) w[k] = Cin[k - NQ];
        if (!ok) {
            ok = solve_T_slow<NS, false>(w, et, Ts, m, cvs);
            T = Ts;
            cv = cvs;
        }
    }
    return ok;
}

// T-dependent quantities of the lane's species and of the group.
struct Kin {
    double T, invT, lnT, rt, irt, eg, ieg, h;
};
template <bool H>
__device__ __forceinline__ void kin_at(double T, Kin& k) {
    const int t = lane8(), rg = fp_lt(TMID, T) ? 1 : 0;
    k.T = T;
    k.lnT = cell::flog(T);
    k.invT = fp_rcp(T);
    k.rt = T * (RU / ONE_ATM);
    k.irt = k.invT * (ONE_ATM / RU);
    const double* a = D_NASA.c[rg][t];
    const double* c = cell::D_GCOEF.c[rg][t];
    const double ai = a[5] * k.invT;
    const double p = fma(T, fma(T, fma(T, fma(T, c[4], c[3]), c[2]), c[1]), c[0]);
    cell::fexp_pair(fma(a[0], 1.0 - k.lnT, ai + p), k.eg, k.ieg);
    if constexpr (H)
        k.h = fma(T, fma(T, fma(T, fma(T, a[4] * 0.2, a[3] * 0.25), a[2] * (1.0 / 3.0)), a[1] * 0.5), a[0]) + ai;
}

// Falloff factor of the lanes whose slot is one (hf_cell.cuh falloff, data-driven).
template <bool JAC>
__device__ __forceinline__ double falloff(const Slot& s, const Kin& kc, double kinf, double k0, double M, double& Tdk,
                                          double& dkM) {
    const double lFc = s.lfc, c = fma(-0.67, lFc, -0.4), nn = fma(-1.27, lFc, 0.75), k0M = k0 * M;
    const double Pr = fp_div(k0M, kinf);
    const bool tiny = !(__double2hiint(Pr) >= 0x01a56e1f);
    const double x = fma(cell::flog(tiny ? 1e-300 : Pr), fm::INV_LN10, c);
    const double iden = fp_rcp(fma(-0.14, x, nn));
    const double f1 = x * iden;
    const double g = fp_rcp(fma(f1, f1, 1.0));
    const double F = cell::fexp(g * (lFc * fm::LN10));
    const double i1 = fp_rcp(1.0 + Pr);
    const double Fi = F * i1, k = k0M * Fi;
    if constexpr (JAC) {
        const double dPr = tiny ? 0.0 : (-2.0 * lFc * nn) * (f1 * g * g) * (iden * iden);
        const double d = i1 + dPr;
        const double si = fma(s.E, kc.invT, s.b), s0 = fma(s.E0, kc.invT, s.b0);
        Tdk = k * fma(d, s0 - si, si);
        dkM = k0 * Fi * d;
    }
    return k;
}

// The lane's reactions into shared memory: q, and with JAC also T dq/dT, the partials (p) and
// (where qo is given) the rates of progress with the slots' own rate constants.
// klast: in and out, the rate constant of the lane's slot of the last round (taken first).
template <int rnd, bool JAC>
__device__ __forceinline__ void reaction_round(const Kin& kc, double C, double X, double M1, double M2, double* q,
                                               Partials* p, double* qo, double& klast) {
    const int t = lane8();
    {
        const int r = rnd * G + t;
        const bool in = rnd < NROUND - 1 || r < NR;  // the slots past the reactions write nothing
        const Slot& s = D_TAB.s[r];
        double A = r < NR ? c_A[r] : 0.0;
        if constexpr (rnd == NROUND - 1) A = r >= NR && r < NR + NFALL ? c_A0[s.low] : A;
        double k = A * cell::fexp(fma(s.b, kc.lnT, -s.E * kc.invT));
        double Tdk = 0.0, dkM = 0.0;
        if constexpr (rnd == NROUND - 1) klast = k;
        if constexpr (JAC) Tdk = k * fma(s.E, kc.invT, s.b);
        if constexpr (round_has_third(rnd)) {
            const double M = s.third == 2 ? M2 : M1;
            const double k0 = get(klast, s.low & 7);
            if (s.type == RXN_FALLOFF) {
                k = falloff<JAC>(s, kc, k, k0, M, Tdk, dkM);
            } else if (s.type == RXN_THREE_BODY) {
                dkM = k;
                k *= M;
                if constexpr (JAC) Tdk *= M;
            }
        }
        const double own = k;
        if constexpr (round_has_dup(rnd)) {
            const double kn = __shfl_down_sync(FULL, k, 1, 8);
            if (s.dup == 1) k += kn;
            if constexpr (JAC) {
                const double Tn = __shfl_down_sync(FULL, Tdk, 1, 8);
                if (s.dup == 1) Tdk += Tn;
            }
        }
        const int i0 = s.r0 < 0 ? 0 : s.r0, i1 = s.r1 < 0 ? 0 : s.r1, i2 = s.p0 < 0 ? 0 : s.p0, i3 = s.p1 < 0 ? 0 : s.p1;
        const double Ca = get(C, i0), ia = get(kc.ieg, i0);
        double Cb = get(C, i1), ib = get(kc.ieg, i1);
        Cb = s.r1 < 0 ? 1.0 : Cb;
        ib = s.r1 < 0 ? 1.0 : ib;
        double b = ia * ib;
        if constexpr (round_has_dn(rnd)) b *= s.dn == 1 ? kc.rt : s.dn == -1 ? kc.irt : 1.0;
        if constexpr (!JAC) {
            const double Xc = get(X, i2);
            double Xd = get(X, i3);
            Xd = s.p1 < 0 ? 1.0 : Xd;
            if (in) q[r] = k * fma(-(b * Xc), Xd, Ca * Cb);
        } else {
            const double Cc = get(C, i2), ec = get(kc.eg, i2);
            double Cd = get(C, i3), ed = get(kc.eg, i3);
            Cd = s.p1 < 0 ? 1.0 : Cd;
            ed = s.p1 < 0 ? 1.0 : ed;
            b *= ec * ed;
            const double cc = Cc * Cd, net = fma(-b, cc, Ca * Cb), kr = k * b;
            const double ha = get(kc.h, i0), hc = get(kc.h, i2);
            double hb = get(kc.h, i1), hd = get(kc.h, i3);
            hb = s.r1 < 0 ? 0.0 : hb;
            hd = s.p1 < 0 ? 0.0 : hd;
            double hh = (hc + hd) - (ha + hb);
            if constexpr (round_has_dn(rnd)) hh -= s.dn == 1 ? 1.0 : s.dn == -1 ? -1.0 : 0.0;
            const double own_q = own * net;
            if (in) {
                q[r] = k * net;
                if (qo) qo[r] = own_q;
                p->qT[r] = fma(kr * cc, hh, Tdk * net);
                double* v = p->v + r * NVAL;
                v[0] = k * Cb;
                v[1] = k * Ca;
                v[2] = kr * Cd;
                v[3] = kr * Cc;
                v[4] = 0.0;
                if constexpr (round_has_third(rnd)) v[4] = dkM * net;
            }
        }
    }
}
template <bool JAC>
__device__ __forceinline__ void reactions(const Kin& kc, double C, double M1, double M2, double* q,
                                          Partials* p, double* qo = nullptr) {
    static_assert(NROUND == 3, "three rounds of reactions");
    const double X = C * kc.eg;
    double klast = 0.0;
    reaction_round<2, JAC>(kc, C, X, M1, M2, q, p, qo, klast);
    reaction_round<0, JAC>(kc, C, X, M1, M2, q, p, qo, klast);
    reaction_round<1, JAC>(kc, C, X, M1, M2, q, p, qo, klast);
}

struct RhsOut {
    double w, T;
    bool ok;
};
// dC/dt of the lane's species at C; T: guess in, temperature out; ok the same in the group.
template <int NS>
__device__ __noinline__ RhsOut rhs(double C, double T, double et, double Ci0, double Ci1, bool active, Shared* sh) {
    const double Cin[2] = {Ci0, Ci1};
    double cv, M1, M2;
    RhsOut o;
    o.ok = temperature<NS>(Cin, et, C, active, T, cv, M1, M2);
    o.T = T;
    Kin kc;
    kin_at<false>(T, kc);
    reactions<false>(kc, C, M1, M2, sh->q, &sh->p);
    __syncwarp();
    const int t = lane8();
    double w = 0.0;
#pragma unroll
    for (int e = 0; e < NW; ++e) w = fma(D_TAB.wn[t][e], sh->q[D_TAB.wr[t][e]], w);
    __syncwarp();
    o.w = w;
    o.ok = all8(o.ok && fp_finite(w));
    return o;
}

// f0 and row t of J = dw/dC (a[], the closing-species terms left out as in hf_cell.cuh).
template <int NS>
__device__ __noinline__ RhsOut rhs_jac(double C, double T, double et, double Ci0, double Ci1, bool active, Shared* sh,
                                       double* row) {
    const double Cin[2] = {Ci0, Ci1};
    double cv, M1, M2;
    RhsOut o;
    o.ok = temperature<NS>(Cin, et, C, active, T, cv, M1, M2);
    o.T = T;
    Kin kc;
    kin_at<true>(T, kc);
    reactions<true>(kc, C, M1, M2, sh->q, &sh->p);
    __syncwarp();
    const int t = lane8();
    double w = 0.0, wT = 0.0, wM = 0.0;
#pragma unroll
    for (int e = 0; e < NW; ++e) {
        const int r = D_TAB.wr[t][e];
        const double n = D_TAB.wn[t][e];
        w = fma(n, sh->q[r], w);
        wT = fma(n, sh->p.qT[r], wT);
        wM = fma(n, sh->p.v[r * NVAL + 4], wM);
    }
    const double tau = (1.0 - kc.h) * fp_rcp(cv);
    double a[NQ];
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
        double s = fma(wT, get(tau, j), wM);
#pragma unroll
        for (int e = D_TAB.j0[j]; e < D_TAB.j0[j + 1]; ++e) s = fma(D_TAB.jn[t][e], sh->p.v[D_TAB.jr[t][e]], s);
        a[j] = s;
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < NQ; ++j) row[j] = a[j];
    o.w = w;
    o.ok = all8(o.ok && fp_finite(w));
    return o;
}

// LU with partial pivoting of the row-distributed matrix (lane t: row t), the diagonal
// holding 1/U_kk; pivot rows (4 bits each) in piv.  False on a zero or non-finite pivot.
constexpr unsigned NO_PIVOT = 0x76543210u;
__device__ __forceinline__ bool lu(double (&a)[NQ], unsigned& piv) {
    const int t = lane8();
    bool ok = true;
    piv = 0;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
        unsigned long long best = t >= k ? fp_abs_bits(a[k]) : 0;
        int idx = t;
#pragma unroll
        for (int off = 1; off < G; off <<= 1) {
            const unsigned long long ob = __shfl_xor_sync(FULL, best, off);
            const int oi = __shfl_xor_sync(FULL, idx, off);
            if (ob > best || (ob == best && oi < idx)) { best = ob; idx = oi; }
        }
        ok = ok && best != 0 && best < 0x7ff0000000000000ull;
        idx = idx < k ? k : idx;
        piv |= (unsigned)idx << (4 * k);
        if (__any_sync(FULL, idx != k)) {
            const int from = t == k ? idx : t == idx ? k : t;
#pragma unroll
            for (int j = 0; j < NQ; ++j) a[j] = get(a[j], from);
        }
        double rk[NQ];
#pragma unroll
        for (int j = k; j < NQ; ++j) rk[j] = get(a[j], k);
        const double inv = fp_rcp(ok ? rk[k] : 1.0);
        const double l = a[k] * inv;
#pragma unroll
        for (int j = k + 1; j < NQ; ++j) {
            const double u = fma(-l, rk[j], a[j]);
            a[j] = t > k ? u : a[j];
        }
        a[k] = t == k ? inv : t > k ? l : a[k];
    }
    return ok;
}
__device__ __forceinline__ double solve(const double (&a)[NQ], unsigned piv, double b) {
    const int t = lane8();
    if (__any_sync(FULL, piv != NO_PIVOT)) {
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            const int p = piv >> (4 * k) & 7;
            b = get(b, t == k ? p : t == p ? k : t);
        }
    }
#pragma unroll
    for (int j = 0; j < NQ - 1; ++j) {
        const double u = fma(-a[j], get(b, j), b);
        b = t > j ? u : b;
    }
#pragma unroll
    for (int j = NQ - 1; j >= 0; --j) {
        const double x = get(b * a[j], j);  // lane j: its component times the reciprocal pivot
        const double u = fma(-a[j], x, b);
        b = t < j ? u : t == j ? x : b;
    }
    return b;
}

template <int NS>
__device__ __forceinline__ double wrms(double v, double y0, double y1, double rtol, double atol, double tail = 0.0) {
    const double r = fp_div(v, fma(rtol, fp_abs_max(y0, y1), atol));
    return fp_max(fp_sqrt((xsum(r * r) + tail) * (1.0 / (NS - 1))), 1e-10);
}

// The group takes the state u (all its lanes hold it) into c; false if inadmissible.
template <int NS>
__device__ __forceinline__ bool load(Cell<NS>& c, const double* u, double dt, double h_prev) {
    const int t = lane8();
    const bool ok = dt > 0.0 && isfinite(dt) && admissible_state<NS>(u, 0.0);
    double rho = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k) rho += u[k];
    const double ir = 1.0 / rho;
    const double uu = u[NS] * ir, vv = u[NS + 1] * ir;
    c.rho = rho;
    c.ir = ir;
    c.et = rho * (u[NS + 2] * ir - 0.5 * (uu * uu + vv * vv)) * (1.0 / RU);
    double s = 0.0, mine = 0.0;
#pragma unroll
    for (int k = 0; k < NS - 1; ++k) {
        const double y = u[k] * ir;
        s += y;
        mine = k == t ? y : mine;
    }
    c.y = mine;
    c.yN2 = NS == 10 ? u[8] * ir : 0.0;
    if constexpr (NS == 10) c.Cin[0] = u[8] * INVW.v[8];
    c.Cin[NS - 1 - NQ] = rho * (1.0 - s) * INVW.v[NS - 1];
    c.mom[0] = u[NS];
    c.mom[1] = u[NS + 1];
    c.mom[2] = u[NS + 2];
    c.T = estimate_T<NS>(u, c.et);
    c.h = h_prev > 0.0 && isfinite(h_prev) ? fmin(h_prev, dt) : 0.0;
    c.t = 0.0;
    c.tend = dt;
    c.steps = c.attempts = 0;
    c.rejectLast = c.rejectMore = false;
    c.fresh = true;
    return ok;
}

// One step attempt of the warp's four cells.  SCREEN: the frozen-cell screen on a cell's
// first attempt.  Returns CELL_*; screened is set when the screen finished the cell.
template <int NS, bool SCREEN>
__device__ __forceinline__ int attempt(Cell<NS>& c, double rtol, double atol, Shared* sh, bool& screened) {
    const int t = lane8();
    const double W = D_MW.v[t], iW = INVW.v[t];
    const double Ci0 = c.Cin[0], Ci1 = NS == 10 ? c.Cin[NS - 1 - NQ] : 0.0;
    const double C0 = c.rho * c.y * iW, wr = W * c.ir;
    double a[NQ];
    screened = false;
    const RhsOut f = rhs_jac<NS>(C0, c.T, c.et, Ci0, Ci1, c.active, sh, a);
    bool go = c.active && f.ok;  // still stepping
    int res = c.active && !f.ok ? CELL_FAIL : CELL_CONTINUE;
    c.T = f.ok ? f.T : c.T;
    if (SCREEN && __any_sync(FULL, go && c.fresh)) {
        const double dt = c.tend, sc = fma(rtol, fabs(c.y), atol) * iW;
        const double isc = fp_rcp(sc);
        const double fz = xmax_abs(f.w * c.ir * isc);
        double r = 0.0;
#pragma unroll
        for (int j = 0; j < NQ; ++j) r = fma(fabs(a[j]), get(sc, j), r);
        const double jz = xmax_abs(r * isc), A = jz * dt;
        const double ft = fz * dt * cell::fexp(fp_lt(A, 20.0) ? A : 20.0);
        double v = 0.0;
#pragma unroll
        for (int j = 0; j < NQ; ++j) v = fma(a[j], get(f.w, j), v);
        if (go && c.fresh && fp_lt(A, 20.0) && fp_ge0(1.0 - ft) && fp_ge0(6e-5 - ft * A * A)) {
            c.y = fma(dt * fma(0.5 * dt, v, f.w), wr, c.y);
            c.t = dt;
            screened = true;
            go = false;
            res = CELL_DONE;
        }
    }
    const bool cold = go && !fp_pos(c.h);
    if (__any_sync(FULL, cold)) {
        // starting step: Hairer's estimate in time scaled by the interval
        const double dt = c.tend;
        double tail = 0.0;
        if constexpr (NS == 10) {
            const double r = c.yN2 / (atol + rtol * fabs(c.yN2));
            tail = r * r;
        }
        const double d0 = wrms<NS>(c.y, c.y, c.y, rtol, atol, tail), d1 = wrms<NS>(f.w * wr, c.y, c.y, rtol, atol) * dt;
        const double hh = d1 < 1e-5 ? 1.0 : fmin(1.0, 0.01 * d0 / d1);
        const RhsOut g = rhs<NS>(fma(hh * dt, f.w, C0), c.T, c.et, Ci0, Ci1, cold, sh);
        const double dn = wrms<NS>((g.w - f.w) / hh * wr, c.y, c.y, rtol, atol);
        const double mx = fmax(d1, g.ok ? dn : 1e30);
        const double h1 = mx <= 1e-15 ? 1.0 : pow(0.01 / mx, 0.2);
        if (cold) c.h = fmin(fmin(100.0 * hh, h1), 1.0) * dt;
        if (cold && !fp_pos(c.h)) {
            go = false;
            res = CELL_FAIL;
        }
    }
    if (!__any_sync(FULL, go)) {
        if (c.active) c.fresh = false;
        return res;
    }
    bool last = false;
    if (go) {
        c.fresh = false;
        if (fp_ge0(fma(1.01, c.h, c.t) - c.tend)) {
            c.h = c.tend - c.t;
            last = true;
        }
        c.hu = c.h;
        if (++c.attempts > 4 * MAX_STEPS) {
            go = false;
            res = CELL_MAXSTEPS;
        }
    }
    const double ih = fp_rcp(go ? c.h : 1.0), inv = ih * (1.0 / RGAMMA);
#pragma unroll
    for (int j = 0; j < NQ; ++j) a[j] = (j == t ? inv : 0.0) - a[j];
    unsigned piv;
    bool ok = lu(a, piv);
    double K[6], Ys = C0, T = c.T;
    K[0] = solve(a, piv, f.w);
#pragma unroll
    for (int s = 1; s < 6; ++s) {
        const int base = s * (s - 1) / 2;
        if (s < 5) Ys = C0;
        double b = 0.0;
#pragma unroll
        for (int j = 0; j < s; ++j) {
            b = fma(RC[base + j], K[j], b);
            if (s < 5 || j == 4) Ys = fma(RA[base + j], K[j], Ys);
        }
        const RhsOut g = rhs<NS>(Ys, T, c.et, Ci0, Ci1, go && ok, sh);
        ok = ok && g.ok;
        T = ok ? g.T : T;
        K[s] = solve(a, piv, fma(ih, b, g.w));
    }
    const double yn = fma((Ys - C0) + K[5], wr, c.y);
    double err = wrms<NS>(K[5] * wr, c.y, yn, rtol, atol);
    ok = all8(ok && fp_finite(yn) && fp_finite(err));
    if (!go) return res;
    if (!ok) {
        c.h *= 0.25;
        c.rejectLast = true;
        return !(c.h > 1e-300) || c.t + c.h == c.t ? CELL_FAIL : CELL_CONTINUE;
    }
    double hnew = c.h * fp_min(6.0, fp_max(0.2, fp_div(0.9, fp_sqrt(fp_sqrt(err)))));
    if (fp_ge0(1.0 - err)) {
        c.t = last ? c.tend : c.t + c.h;
        c.T = T;
        c.y = yn;
        if (c.rejectLast) hnew = fp_min(hnew, c.h);
        c.rejectLast = c.rejectMore = false;
        ++c.steps;
        c.h = hnew;
        if (last || !fp_lt(c.t, c.tend)) return CELL_DONE;
        return c.steps >= MAX_STEPS ? CELL_MAXSTEPS : CELL_CONTINUE;
    }
    if (c.rejectMore) hnew = c.h * 0.1;
    c.rejectMore = c.rejectLast;
    c.rejectLast = true;
    c.h = hnew;
    return !(c.h > 1e-300) || c.t + c.h == c.t ? CELL_FAIL : CELL_CONTINUE;
}

// chemistry.cpp:63-70 for the warp's cells (called by all lanes): the state into every
// lane's u[], and whether it may be kept.
template <int NS>
__device__ __forceinline__ bool finish(const Cell<NS>& c, double* u) {
    const bool bad = !fp_finite(c.y) || fp_lt(c.y, -1e-13);
    const bool ok = all8(!bad);
    const double mine = c.rho * (fp_neg(c.y) ? 0.0 : c.y);
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
        u[k] = get(mine, k);
        s += u[k];
    }
    if constexpr (NS == 10) {
        u[8] = c.rho * (fp_neg(c.yN2) ? 0.0 : c.yN2);
        s += u[8];
    }
    u[NS - 1] = c.rho - s;
    u[NS] = c.mom[0];
    u[NS + 1] = c.mom[1];
    u[NS + 2] = c.mom[2];
    return ok && admissible_state<NS>(u, c.T);
}

}  // namespace grp8
}  // namespace hf
