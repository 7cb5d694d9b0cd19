// Reverse sweep of an accepted Rodas4 step, one cell per group of 8 lanes (the layout and
// primitives of hf_group.cuh): lane t holds component t of every vector, row t of the
// factors and reactions t, t + 8, t + 16.
//
// The differentiated step in concentrations C of the reacting species, with the inert
// species' concentrations Cin and et = rho e / R as inputs held fixed over it:
//     C+ = C + sum_s m_s K_s,  (inv I - J(C)) K_s = w(C_s) + sum_j c_sj/h K_j,
//     C_s = C + sum_j a_sj K_j,
// from lam = dJ/dC+:  Kb_s = m_s lam (+ later stages), R_s = M^-T Kb_s,
//     Yb_s = (dw/dC)(C_s)^T R_s, pb += (dw/dp)(C_s)^T R_s, Gm = sum_s R_s K_s^T,
//     dJ/dC += Yb_s and grad <J(C), Gm>, likewise for Cin, et and p = ln(multiplier).
// With w_i = sum_r nu_ir q_r, <J, Gm> = sum_r D_{beta_r} q_r, beta_rj = sum_i nu_ir Gm_ij, so
// its gradient is the tangent, along (beta_r, d lnT = tau . beta_r), of reaction r's own
// partial derivatives, plus the curvature of T(C, Cin, et).
//
// What bounds it: the step chain of a cell, about 250 us a reverse step with the forward attempt
// it follows (73 us).  The stages' partial derivatives are kept in shared memory from the forward
// recomputation (8 KB a cell), so the transposed products cost a sixth of an evaluation each:
// about 3,000 FP64 instructions a step for four cells, against 130,000 FP64 instruction times
// for 32 cells on one lane each.  Those 3,000 hold the pipe for 93 us; what the rest of the
// step waits for (table and weight loads ahead of dependent shared loads, the tape's strided
// loads, shuffles) was not separated.
#pragma once
#include "hf_group.cuh"

namespace hf {
namespace grp8 {

// The partials of all six stages stay from the forward recomputation to the reverse sweep;
// the rates of progress are those of the stage in hand.  7,800 bytes: with four cells to a block
// seven blocks fit an SM (9,792 bytes and five blocks with whole 8-lane rounds and the rates kept
// for every stage), so 4,096 cells run at once: ignition delay, 2,000 calls, 15.3 -> 11.3 s.
struct AdjShared {  // of one group
    Shared f;          // the forward attempts' too; f.p: the first stage's partials
    Partials p[5];     // the other stages'
    double qo[6][NR];  // rate of progress with the slot's own rate constant (duplicates apart)
    double m[NQ][NQ + 1];  // LU factors, then Gm
    __device__ __forceinline__ Partials* stage(int s) { return s ? &p[s - 1] : &f.p; }
};

// gC_m = sum_e cn[m][e] v[cr[m][e]] over per-slot partials (sign of the products included)
struct ColTables {
    int n;
    int cr[NQ][MAXLIST];
    double cn[NQ][MAXLIST];
    bool ok;
};
constexpr ColTables make_cols() {
    ColTables t{};
    t.ok = true;
    for (int m = 0; m < NQ; ++m) {
        int n = 0;
        for (int r = 0; r < NR; ++r) {
            if (cell::dup_of(r) >= 0) continue;
            const Slot& s = H_TAB.s[r];
            const int sp[4] = {s.r0, s.r1, s.p0, s.p1};
            for (int w = 0; w < 4; ++w)
                if (sp[w] == m) {
                    if (n == MAXLIST) { t.ok = false; continue; }
                    t.cr[m][n] = r * NVAL + w;
                    t.cn[m][n] = w < 2 ? 1.0 : -1.0;
                    ++n;
                }
            if (s.third && RXN[r].eff[m] != 1.0) {
                if (n == MAXLIST) { t.ok = false; continue; }
                t.cr[m][n] = r * NVAL + 4;
                t.cn[m][n] = RXN[r].eff[m] - 1.0;
                ++n;
            }
        }
        t.n = n > t.n ? n : t.n;
    }
    return t;
}
constexpr ColTables H_COL = make_cols();
static_assert(H_COL.ok, "a species' partial list is longer than its table");
__device__ constexpr ColTables D_COL = make_cols();
constexpr int NC = H_COL.n;

// One stage's temperature quantities that its transpose needs.
struct StageT {
    double T, tau, tin, dle;  // tau: (1/T) dT/dC_t; tin: of the inert species t; dle: (1/T) dT/d et
};

// Rates and partials at C into sh; w_t, and with ROW row t of J.
template <int NS, bool ROW>
__device__ __noinline__ RhsOut eval(double C, double T, double et, double Ci0, double Ci1, bool active, double* q,
                                    Partials* p, double* qo, StageT& out, double* row) {
    const double Cin[2] = {Ci0, Ci1};
    const int t = lane8();
    double cv, M1, M2;
    RhsOut o;
    o.ok = temperature<NS>(Cin, et, C, active, T, cv, M1, M2);
    o.T = T;
    Kin kc;
    kin_at<true>(T, kc);
    reactions<true>(kc, C, M1, M2, q, p, qo);
    __syncwarp();
    double w = 0.0, wT = 0.0, wM = 0.0;
#pragma unroll
    for (int e = 0; e < NW; ++e) {
        const int r = D_TAB.wr[t][e];
        const double n = D_TAB.wn[t][e];
        w = fma(n, q[r], w);
        if constexpr (ROW) {
            wT = fma(n, p->qT[r], wT);
            wM = fma(n, p->v[r * NVAL + 4], wM);
        }
    }
    const double icv = fp_rcp(cv);
    const double* a = D_NASA.c[fp_lt(TMID, T) ? 1 : 0][NQ + (t < NS - NQ ? t : 0)];
    const double hin = fma(T, fma(T, fma(T, fma(T, a[4] * 0.2, a[3] * 0.25), a[2] * (1.0 / 3.0)), a[1] * 0.5), a[0]) +
                       a[5] * kc.invT;
    out.T = T;
    out.tau = (1.0 - kc.h) * icv;
    out.tin = (1.0 - hin) * icv;
    out.dle = kc.invT * icv;
    if constexpr (ROW) {
#pragma unroll
        for (int j = 0; j < NQ; ++j) {
            double s = fma(wT, get(out.tau, j), wM);
#pragma unroll
            for (int e = D_TAB.j0[j]; e < D_TAB.j0[j + 1]; ++e) s = fma(D_TAB.jn[t][e], p->v[D_TAB.jr[t][e]], s);
            row[j] = s;
        }
    }
    __syncwarp();
    o.w = w;
    o.ok = all8(o.ok && fp_finite(w));
    return o;
}

// x = M^-T b from column t of the factors (at[j] = LU[j][t]) and the pivots.
__device__ __forceinline__ double solve_T8(const double (&at)[NQ], unsigned piv, double b) {
    const int t = lane8();
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
        const double x = get(b * at[j], j);
        const double u = fma(-at[j], x, b);
        b = t > j ? u : t == j ? x : b;
    }
#pragma unroll
    for (int j = NQ - 1; j > 0; --j) {
        const double u = fma(-at[j], get(b, j), b);
        b = t < j ? u : b;
    }
    if (__any_sync(FULL, piv != NO_PIVOT)) {
#pragma unroll
        for (int k = NQ - 1; k >= 0; --k) {
            const int p = piv >> (4 * k) & 7;
            b = get(b, t == k ? p : t == p ? k : t);
        }
    }
    return b;
}

// What a cell's reverse sweep accumulates besides lam.
struct Acc {
    double pb[NROUND];  // dJ/dp of the lane's reactions
    double gin;         // dJ/dCin of inert species t (lanes 0..NI-1)
    double get;         // dJ/d et (every lane)
};

// (dw/dC)^T R of a stage (its partials are consumed), into acc for p, Cin, et.
__device__ __forceinline__ double vjp(Partials* p, const double* qo, const StageT& st, double R, Acc& acc) {
    const int t = lane8();
    double gT = 0.0, gM = 0.0;
#pragma unroll
    for (int rnd = 0; rnd < NROUND; ++rnd) {
        const int r = rnd * G + t;
        const Slot& s = D_TAB.s[r];
        const double a0 = get(R, s.r0 < 0 ? 0 : s.r0), a2 = get(R, s.p0 < 0 ? 0 : s.p0);
        double a1 = get(R, s.r1 < 0 ? 0 : s.r1), a3 = get(R, s.p1 < 0 ? 0 : s.p1);
        a1 = s.r1 < 0 ? 0.0 : a1;
        a3 = s.p1 < 0 ? 0.0 : a3;
        if (r < NR) {
            const double al = (a2 + a3) - (a0 + a1);
            acc.pb[rnd] = fma(al, qo[r], acc.pb[rnd]);
            const double ax = s.dup < 0 ? 0.0 : al;
            gT = fma(ax, p->qT[r], gT);
            double* v = p->v + r * NVAL;
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] *= ax;
            v[4] *= ax;
            gM += v[4];
        }
    }
    __syncwarp();
    gT = xsum(gT);
    gM = xsum(gM);
    double y = 0.0;
#pragma unroll
    for (int e = 0; e < NC; ++e) y = fma(D_COL.cn[t][e], p->v[D_COL.cr[t][e]], y);
    // inside the small jump of e(T) at T_mid the inversion returns T_mid, which does not move
    const double g = st.T == TMID ? 0.0 : gT;
    acc.gin += fma(g, st.tin, gM);
    acc.get = fma(g, st.dle, acc.get);
    return fma(g, st.tau, y + gM);
}

// ---------------------------------------------------------------- second derivatives
struct Dual {
    double v, d;
};
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return {a.v + b.v, a.d + b.d}; }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return {a.v - b.v, a.d - b.d}; }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) { return {a.v * b.v, fma(a.d, b.v, a.v * b.d)}; }
__device__ __forceinline__ Dual operator*(double a, Dual b) { return {a * b.v, a * b.d}; }
__device__ __forceinline__ Dual operator+(double a, Dual b) { return {a + b.v, b.d}; }
__device__ __forceinline__ Dual rcp(Dual a) {
    const double r = fp_rcp(a.v);
    return {r, -(r * r) * a.d};
}
__device__ __forceinline__ Dual fexp(Dual a) {
    const double e = cell::fexp(a.v);
    return {e, e * a.d};
}

// falloff() of hf_group.cuh with tangents: k, T dk/dT and dk/dM along d lnT = th, dM.
__device__ __forceinline__ void falloff_dual(const Slot& s, const Kin& kc, Dual kinf, double A0, Dual M, double th,
                                             Dual& k, Dual& Tdk, Dual& dkM) {
    const double lFc = s.lfc, c = fma(-0.67, lFc, -0.4), nn = fma(-1.27, lFc, 0.75);
    const Dual lnT{kc.lnT, th}, invT{kc.invT, -kc.invT * th};
    const Dual k0 = A0 * fexp(s.b0 * lnT + (-s.E0) * invT), k0M = k0 * M;
    const Dual Pr = k0M * rcp(kinf);
    const bool tiny = !(__double2hiint(Pr.v) >= 0x01a56e1f);
    const double pv = tiny ? 1e-300 : Pr.v;
    const Dual lPr{cell::flog(pv) * fm::INV_LN10, tiny ? 0.0 : fp_div(Pr.d, pv) * fm::INV_LN10};
    const Dual x = c + lPr;
    const Dual iden = rcp(nn + (-0.14) * x);
    const Dual f1 = x * iden;
    const Dual g = rcp(1.0 + f1 * f1);
    const Dual F = fexp((lFc * fm::LN10) * g);
    const Dual i1 = rcp(1.0 + Pr);
    const Dual Fi = F * i1;
    k = k0M * Fi;
    const Dual dPr = tiny ? Dual{0.0, 0.0} : (-2.0 * lFc * nn) * (f1 * (g * g) * (iden * iden));
    const Dual d = i1 + dPr;
    const Dual si = s.b + s.E * invT, s0 = s.b0 + s.E0 * invT;
    Tdk = k * (si + d * (s0 - si));
    dkM = k0 * Fi * d;
}

template <int rnd>
__device__ __forceinline__ void hess_round(const Kin& kc, double z, double C, double M1, double M2,
                                           const double (&tj)[NQ], AdjShared* sh, double (&B)[NQ], double& hT, double& gM,
                                           Acc& acc) {
    const int t = lane8(), r = rnd * G + t;
    const Slot& s = D_TAB.s[r];
    const int i0 = s.r0 < 0 ? 0 : s.r0, i1 = s.r1 < 0 ? 0 : s.r1, i2 = s.p0 < 0 ? 0 : s.p0, i3 = s.p1 < 0 ? 0 : s.p1;
    const bool h1 = s.r1 >= 0, h3 = s.p1 >= 0, live = r < NR;
    // tangent along beta
    double th = 0.0, dM = 0.0, ba = 0.0, bb = 0.0, bc = 0.0, bd = 0.0, be[NQ];
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
        const double a = h1 ? sh->m[i1][j] : 0.0, b = h3 ? sh->m[i3][j] : 0.0;
        const double v = live ? (sh->m[i2][j] + b) - (sh->m[i0][j] + a) : 0.0;
        be[j] = v;
        th = fma(tj[j], v, th);
        if constexpr (round_has_third(rnd)) dM = fma(D_TAB.eff[s.third == 2 ? 1 : 0][j], v, dM);
        ba = i0 == j ? v : ba;
        bb = h1 && i1 == j ? v : bb;
        bc = i2 == j ? v : bc;
        bd = h3 && i3 == j ? v : bd;
    }
    const double A = live ? c_A[r] : 0.0;
    const double sv = fma(s.E, kc.invT, s.b), sd = -s.E * kc.invT * th;  // T dlnk/dT and its tangent
    Dual k;
    k.v = A * cell::fexp(fma(s.b, kc.lnT, -s.E * kc.invT));
    k.d = k.v * sv * th;
    Dual Tdk = k * Dual{sv, sd}, dkM{0.0, 0.0};
    if constexpr (round_has_third(rnd)) {
        const Dual M{s.third == 2 ? M2 : M1, dM};
        if (s.type == RXN_FALLOFF) {
            falloff_dual(s, kc, k, c_A0[live ? r : 0], M, th, k, Tdk, dkM);
        } else if (s.type == RXN_THREE_BODY) {
            dkM = k;
            k = k * M;
            Tdk = Tdk * M;
        }
    }
    const Dual own = k;
    if constexpr (round_has_dup(rnd)) {
        const double kv = __shfl_down_sync(FULL, k.v, 1, 8), kd = __shfl_down_sync(FULL, k.d, 1, 8);
        const double Tv = __shfl_down_sync(FULL, Tdk.v, 1, 8), Td = __shfl_down_sync(FULL, Tdk.d, 1, 8);
        if (s.dup == 1) {
            k.v += kv;
            k.d += kd;
            Tdk.v += Tv;
            Tdk.d += Td;
        }
    }
    const Dual Ca{get(C, i0), ba}, Cc{get(C, i2), bc};
    Dual Cb{get(C, i1), bb}, Cd{get(C, i3), bd};
    const double ia = get(kc.ieg, i0), ec = get(kc.eg, i2), ha = get(kc.h, i0), hc = get(kc.h, i2), za = get(z, i0),
                 zc = get(z, i2);
    double ib = get(kc.ieg, i1), ed = get(kc.eg, i3), hb = get(kc.h, i1), hd = get(kc.h, i3), zb = get(z, i1),
           zd = get(z, i3);
    Cb.v = h1 ? Cb.v : 1.0;
    Cd.v = h3 ? Cd.v : 1.0;
    ib = h1 ? ib : 1.0;
    ed = h3 ? ed : 1.0;
    hb = h1 ? hb : 0.0;
    hd = h3 ? hd : 0.0;
    zb = h1 ? zb : 0.0;
    zd = h3 ? zd : 0.0;
    double b = ia * ib;
    if constexpr (round_has_dn(rnd)) b *= s.dn == 1 ? kc.rt : s.dn == -1 ? kc.irt : 1.0;
    b *= ec * ed;
    double hh = (hc + hd) - (ha + hb);
    if constexpr (round_has_dn(rnd)) hh -= s.dn == 1 ? 1.0 : s.dn == -1 ? -1.0 : 0.0;
    const Dual H{hh, ((zc + zd) - (za + zb)) * th}, bD{b, -hh * b * th};
    const Dual f = Ca * Cb, cc = Cc * Cd, net = f - bD * cc, kr = k * bD;
    acc.pb[rnd] += fma(own.d, net.v, own.v * net.d);
    const bool on = live && s.dup >= 0;
    const Dual qT = kr * cc * H + Tdk * net;
    hT += on ? qT.d : 0.0;
#pragma unroll
    for (int j = 0; j < NQ; ++j) B[j] = fma(on ? qT.v : 0.0, be[j], B[j]);
    double v4 = 0.0;
    if constexpr (round_has_third(rnd)) {
        v4 = (dkM * net).d;
        gM += on ? v4 : 0.0;
    }
    if (rnd < NROUND - 1 || r < NR) {
        double* v = sh->f.p.v + r * NVAL;
        v[0] = (k * Cb).d;
        v[1] = (k * Ca).d;
        v[2] = (kr * Cd).d;
        v[3] = (kr * Cc).d;
        v[4] = v4;
    }
}

// grad <J(C), Gm> (Gm in sh->m): the lane's component of the C gradient; p, Cin, et into acc.
template <int NS>
__device__ __noinline__ double hess(double C, double T, double et, double Ci0, double Ci1, bool active, AdjShared* sh,
                                    const StageT& st, Acc& acc) {
    const double Cin[2] = {Ci0, Ci1};
    const int t = lane8();
    double cv, M1, M2;
    temperature<NS>(Cin, et, C, active, T, cv, M1, M2);
    Kin kc;
    kin_at<true>(T, kc);
    const int rg = fp_lt(TMID, T) ? 1 : 0;
    const double* a = D_NASA.c[rg][t];
    const double* ai = D_NASA.c[rg][NQ + (t < NS - NQ ? t : 0)];
    const double cp = fma(T, fma(T, fma(T, fma(T, a[4], a[3]), a[2]), a[1]), a[0]);
    const double cpi = fma(T, fma(T, fma(T, fma(T, ai[4], ai[3]), ai[2]), ai[1]), ai[0]);
    // T dcp/dT, weighted by the concentrations: T dCV/dT
    const double dc = T * fma(T, fma(T, fma(T, 4.0 * a[4], 3.0 * a[3]), 2.0 * a[2]), a[1]);
    const double dci = T * fma(T, fma(T, fma(T, 4.0 * ai[4], 3.0 * ai[3]), 2.0 * ai[2]), ai[1]);
    const double ci = t < NS - NQ ? (t == 0 ? Ci0 : Ci1) : 0.0;
    const double cvT = xsum(fma(ci, dci, C * dc));
    double tj[NQ], B[NQ], hT = 0.0, gM = 0.0;
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
        tj[j] = get(st.tau, j);
        B[j] = 0.0;
    }
    const double z = cp - kc.h;
    hess_round<0>(kc, z, C, M1, M2, tj, sh, B, hT, gM, acc);
    hess_round<1>(kc, z, C, M1, M2, tj, sh, B, hT, gM, acc);
    hess_round<2>(kc, z, C, M1, M2, tj, sh, B, hT, gM, acc);
    __syncwarp();
    const double Bt = reduce_scatter(B);
    hT = xsum(hT);
    gM = xsum(gM);
    const double tw = xsum(Bt * st.tau), zw = xsum(Bt * z), icv = fp_rcp(cv);
    double y = 0.0;
#pragma unroll
    for (int e = 0; e < NC; ++e) y = fma(D_COL.cn[t][e], sh->f.p.v[D_COL.cr[t][e]], y);
    // tau_j = -(h_j/RT - 1)/CV:  T dtau_j/dT = -(z_j + tau_j T dCV/dT)/CV,  dtau_j/dC_m =
    // -tau_j cv_m/CV.  At the T_mid jump T does not move: only the latter is left.
    const double g = T == TMID ? 0.0 : hT - fma(tw, cvT, zw) * icv;
    const double q = tw * icv;
    acc.gin += fma(g, st.tin, gM - (cpi - 1.0) * q);
    acc.get = fma(g, st.dle, acc.get);
    return fma(g, st.tau, y + gM - (cp - 1.0) * q);
}

// Reverse sweep of one accepted step from y (the lane's mass fraction) with step h: lam =
// dJ/dC+ in, dJ/dC out.  False when an evaluation failed.
template <int NS>
__device__ __forceinline__ bool step_adjoint(double rho, double et, double Ci0, double Ci1, double y, double h,
                                             double T, bool active, double& lam, Acc& acc, AdjShared* sh) {
    const int t = lane8();
    const double C0 = rho * y * INVW.v[t];
    const double ih = fp_rcp(active ? h : 1.0), inv = ih * (1.0 / RGAMMA);
    double a[NQ], K[6];
    StageT st[6];
    RhsOut f = eval<NS, true>(C0, T, et, Ci0, Ci1, active, sh->f.q, &sh->f.p, sh->qo[0],
                             st[0], a);
    bool ok = f.ok;
    T = f.T;
#pragma unroll
    for (int j = 0; j < NQ; ++j) a[j] = (j == t ? inv : 0.0) - a[j];
    unsigned piv;
    ok = lu(a, piv) && ok;
    K[0] = solve(a, piv, f.w);
    double Ys = C0;
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
        f = eval<NS, false>(Ys, T, et, Ci0, Ci1, active && ok, sh->f.q, sh->stage(s), sh->qo[s], st[s],
                             nullptr);
        ok = ok && f.ok;
        T = ok ? f.T : T;
        K[s] = solve(a, piv, fma(ih, b, f.w));
    }
    double at[NQ];
#pragma unroll
    for (int j = 0; j < NQ; ++j) sh->m[t][j] = a[j];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < NQ; ++j) at[j] = sh->m[j][t];
    __syncwarp();
    double Kb[6], cb = lam, g[NQ];
#pragma unroll
    for (int s = 0; s < 6; ++s) Kb[s] = RM[s] * lam;
#pragma unroll
    for (int j = 0; j < NQ; ++j) g[j] = 0.0;
#pragma unroll
    for (int s = 5; s >= 0; --s) {
        const int base = s * (s - 1) / 2;
        const double R = solve_T8(at, piv, Kb[s]);
#pragma unroll
        for (int j = 0; j < NQ; ++j) g[j] = fma(R, get(K[s], j), g[j]);
        const double Y = vjp(sh->stage(s), sh->qo[s], st[s], R, acc);
        cb += Y;
#pragma unroll
        for (int j = 0; j < s; ++j) Kb[j] = fma(RC[base + j] * ih, R, fma(RA[base + j], Y, Kb[j]));
    }
#pragma unroll
    for (int j = 0; j < NQ; ++j) sh->m[t][j] = g[j];
    __syncwarp();
    cb += hess<NS>(C0, st[0].T, et, Ci0, Ci1, active && ok, sh, st[0], acc);
    __syncwarp();
    if (active) lam = cb;
    return ok;
}

}  // namespace grp8
}  // namespace hf
