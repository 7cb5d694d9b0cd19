// Device-side thermodynamics, equation of state and HLLC flux for the H2_Li
// mechanism (NS = 9 species of the file, or 10 with the inert AR extension).
//
// Layout: a cell state is NV = NS + 3 doubles in the reference's order
// (rhoY_0..rhoY_{NS-1}, rho*u, rho*v, rho*E), HyperFlow_V3/src/solver.hpp:17-25.
//
// The EOS closure restates what physics.cpp:4-15 gets from Cantera's ideal-gas
// phase: NASA7 polynomials (T <= T_mid uses the low range), e = sum Y_k e_k(T),
// p = rho R T / W, frozen sound speed a = sqrt(cp/cv R T / W).  The UV inversion
// is a Newton solve on T.  It first iterates in FP32 (cheap on this part), then
// finishes in FP64, which leaves T converged to rounding: the FP64 answer does not
// depend on the guess or on the FP32 phase.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "hf_fp64.cuh"
#include "mech_h2li.h"

namespace hf {
using namespace hfmech;

constexpr double RU = GAS_CONSTANT;

// Per-species coefficients of e_k(T)*W_k/R = c0 T + c1 T^2 + c2 T^3 + c3 T^4 + c4 T^5 + c5
// with c0 = a0 - 1, c1 = a1/2, c2 = a2/3, c3 = a3/4, c4 = a4/5, c5 = a5.
struct ECoef { double c[2][NS_MAX][6]; };
constexpr ECoef make_ecoef() {
    ECoef e{};
    for (int r = 0; r < 2; ++r)
        for (int k = 0; k < NS_MAX; ++k) {
            const double* a = r == 0 ? NASA_LOW[k] : NASA_HIGH[k];
            e.c[r][k][0] = a[0] - 1.0;
            e.c[r][k][1] = a[1] / 2.0;
            e.c[r][k][2] = a[2] / 3.0;
            e.c[r][k][3] = a[3] / 4.0;
            e.c[r][k][4] = a[4] / 5.0;
            e.c[r][k][5] = a[5];
        }
    return e;
}
__device__ constexpr ECoef D_ECOEF = make_ecoef();
struct InvW { double v[NS_MAX]; };
constexpr InvW make_invw() {
    InvW w{};
    for (int k = 0; k < NS_MAX; ++k) w.v[k] = 1.0 / MW[k];
    return w;
}
__device__ constexpr InvW INVW = make_invw();
struct MolW { double v[NS_MAX]; };
constexpr MolW make_mw() {
    MolW w{};
    for (int k = 0; k < NS_MAX; ++k) w.v[k] = MW[k];
    return w;
}
__device__ constexpr MolW D_MW = make_mw();
struct Nasa { double c[2][NS_MAX][7]; };
constexpr Nasa make_nasa() {
    Nasa n{};
    for (int k = 0; k < NS_MAX; ++k)
        for (int j = 0; j < 7; ++j) { n.c[0][k][j] = NASA_LOW[k][j]; n.c[1][k][j] = NASA_HIGH[k][j]; }
    return n;
}
__device__ constexpr Nasa D_NASA = make_nasa();
constexpr double TMID = 1000.0;  // T_MID is 1000 K for every species of the table

// Coefficients per unit mass density in J (c_kj R / W_k), for weights q_k = rho Y_k, and R / W_k:
// the doubles nearest to the quotients (products and remainders exact by Dekker's splitting).
// With R in the tables the energy equation and the pressure take one rounding and one product
// less each than with 1 / W_k.
constexpr double prod_lo(double a, double b) {  // a b - fl(a b)
    const double s = 134217729.0, p = a * b;
    const double ah = s * a - (s * a - a), bh = s * b - (s * b - b), al = a - ah, bl = b - bh;
    return ((ah * bh - p) + ah * bl + al * bh) + al * bl;
}
constexpr double times_RU_over(double a, double w) {
    const double p = a * RU, q = p / w;
    return q + (((p - q * w) - prod_lo(q, w)) + prod_lo(a, RU)) / w;
}
constexpr ECoef make_ecoef_mass() {
    ECoef e = make_ecoef();
    for (int r = 0; r < 2; ++r)
        for (int k = 0; k < NS_MAX; ++k)
            for (int j = 0; j < 6; ++j) e.c[r][k][j] = times_RU_over(e.c[r][k][j], MW[k]);
    return e;
}
__device__ constexpr ECoef D_ECOEF_MASS = make_ecoef_mass();
constexpr InvW make_rinvw() {
    InvW w{};
    for (int k = 0; k < NS_MAX; ++k) w.v[k] = times_RU_over(1.0, MW[k]);
    return w;
}
__device__ constexpr InvW RINVW = make_rinvw();
// e_k(T) at the temperatures that bracket the solve
constexpr double T_LO = 250.0, T_HI = 5000.0;
struct EAt { double lo[NS_MAX], mid[NS_MAX], hi[NS_MAX]; };
constexpr double ecoef_at(const double (&c)[6], double T) {
    return ((((c[4] * T + c[3]) * T + c[2]) * T + c[1]) * T + c[0]) * T + c[5];
}
constexpr EAt make_eat(const ECoef& e) {
    EAt a{};
    for (int k = 0; k < NS_MAX; ++k) {
        a.lo[k] = ecoef_at(e.c[0][k], T_LO);
        a.mid[k] = ecoef_at(e.c[0][k], TMID);
        a.hi[k] = ecoef_at(e.c[1][k], T_HI);
    }
    return a;
}
__device__ constexpr EAt D_EAT_MASS = make_eat(make_ecoef_mass());
// the same over R, for the chemistry, whose energies are rho e / R
constexpr ECoef make_ecoef_mass_R() {
    ECoef e = make_ecoef();
    for (int r = 0; r < 2; ++r)
        for (int k = 0; k < NS_MAX; ++k)
            for (int j = 0; j < 6; ++j) e.c[r][k][j] /= MW[k];
    return e;
}
__device__ constexpr EAt D_EAT_R = make_eat(make_ecoef_mass_R());

// Mixture polynomial of one NASA range: e(T)/R = sum_j m[j] T^(j+1) + m[5], with
// m[j] = sum_k w_k c_kj for weights w_k: moles (z_k = Y_k / W_k, or concentrations) or,
// with MASS, partial densities.  Coefficients that are zero in the table (the atoms H and
// AR have constant heat capacity) take no instruction.
template <int NS, int RG, bool MASS = false>
__device__ __forceinline__ void mix_coef_r(const double* w, double* m) {
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        double s = 0.0;
        bool first = true;
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            const double c = MASS ? D_ECOEF_MASS.c[RG][k][j] : D_ECOEF.c[RG][k][j];
            if (c != 0.0) {
                s = first ? w[k] * c : fma(w[k], c, s);
                first = false;
            }
        }
        m[j] = s;
    }
}
// m[j] += the same sum over the first N species (moles)
template <int N, int RG>
__device__ __forceinline__ void mix_add_r(const double* w, double* m) {
#pragma unroll
    for (int j = 0; j < 6; ++j)
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (D_ECOEF.c[RG][k][j] != 0.0) m[j] = fma(w[k], D_ECOEF.c[RG][k][j], m[j]);
}
template <int NS, bool MASS = false>
__device__ __forceinline__ void mix_coef(const double* w, int range, double* m) {
    if (range == 0) mix_coef_r<NS, 0, MASS>(w, m);
    else mix_coef_r<NS, 1, MASS>(w, m);
}
// e/R and cv/R from mixture coefficients
__device__ __forceinline__ double poly_e(const double* m, double T) {
    return fma(T, fma(T, fma(T, fma(T, fma(T, m[4], m[3]), m[2]), m[1]), m[0]), m[5]);
}
__device__ __forceinline__ double poly_cv(const double* m, double T) {
    return fma(T, fma(T, fma(T, fma(T, 5.0 * m[4], 4.0 * m[3]), 3.0 * m[2]), 2.0 * m[1]), m[0]);
}
__device__ __forceinline__ float poly_e_f(const float* m, float T) {
    return fmaf(T, fmaf(T, fmaf(T, fmaf(T, fmaf(T, m[4], m[3]), m[2]), m[1]), m[0]), m[5]);
}
__device__ __forceinline__ float poly_cv_f(const float* m, float T) {
    return fmaf(T, fmaf(T, fmaf(T, fmaf(T, 5.0f * m[4], 4.0f * m[3]), 3.0f * m[2]), 2.0f * m[1]), m[0]);
}

// The UV inversion for any state: FP64 Newton from T until the applied correction is below
// 1e-10 T (quadratic convergence leaves T at rounding level).  Inside the small jump of
// e(T) at T_mid (no root), two consecutive sub-kelvin flips across T_mid return T_mid.
// Returns false when the iteration does not converge to a finite positive T.
template <int NS, bool MASS>
__device__ __forceinline__ bool solve_T_any(const double* w, double et, double& T, double* m) {
    if (!(T > 0.0) || !(T < 1e5)) T = 1000.0;
    int range = T <= TMID ? 0 : 1;
    mix_coef<NS, MASS>(w, range, m);
    int flips = 0;
    for (int it = 0; it < 60; ++it) {
        const int r = T <= TMID ? 0 : 1;
        if (r != range) {
            range = r;
            mix_coef<NS, MASS>(w, range, m);
        }
        double dT = (et - poly_e(m, T)) / poly_cv(m, T);
        if (!isfinite(dT)) return false;
        dT = fmin(1000.0, fmax(-1000.0, dT));
        double Tn = T + dT;
        if (!(Tn > 0.0)) Tn = 0.5 * T;
        const double step = fabs(Tn - T);
        if (step <= 1e-10 * Tn) {
            T = Tn;
            const int rf = T <= TMID ? 0 : 1;
            if (rf != range) mix_coef<NS, MASS>(w, rf, m);
            return true;
        }
        flips = ((T <= TMID) != (Tn <= TMID) && step < 0.5) ? flips + 1 : 0;
        if (flips >= 2) {
            T = TMID;
            mix_coef<NS, MASS>(w, 0, m);
            return true;
        }
        T = Tn;
    }
    return false;
}

template <int NS, bool MASS>
__device__ __noinline__ bool solve_T_slow(const double* w, double et, double& T, double* m, double& cv) {
    if (!solve_T_any<NS, MASS>(w, et, T, m)) return false;
    cv = poly_cv(m, T);
    return true;
}

// The fast solve of e(T) = R et: newton_T from the FP64 mixture coefficients m of the range
// that holds T, giving T and the heat capacity cv = poly_cv(m, T).  FP64 instructions are
// what a solve costs, so one FP64 Newton step of second order replaces the iteration to
// 1e-10: secant_T compares et with e at T_LO, T_MID and T_HI in FP32 for the range and a
// guess t (the chemistry has both from the step before), FP32 Newton steps converge to FP32
// accuracy (T within about 1e-6), and with r = et - e(T0) the FP64 step
//     T = T0 + d - (cv'/2cv) d^2,  d = r / cv
// leaves an error of order (d/T)^3, below rounding for d <= 4e-6 T.  The mixture
// coefficients (a sum over species for each power of T) are most of what is left.  States near T_mid, outside [T_LO, T_HI], or whose FP32 phase does
// not settle take solve_T_any.
//
// newton_T: the Newton steps from mixture coefficients m of the range `low` names; false
// (T the FP32 phase's result, or as it came) when the state needs solve_T_any.
__device__ __forceinline__ bool newton_T(const double* m, double et, bool low, float t, double& T, double& cv) {
    const float etf = fp_to_f32(et);
    float mf[6], dt = 0.0f;
#pragma unroll
    for (int j = 0; j < 6; ++j) mf[j] = fp_to_f32(m[j]);
    bool fine = false;
    for (int it = 0; it < 12; ++it) {
        dt = (etf - poly_e_f(mf, t)) * fp_rcp_seed(poly_cv_f(mf, t));
        t += dt;
        fine = fabsf(dt) <= 1e-5f * t;
        if (fine || !(fabsf(dt) < 1e4f)) break;
    }
    if (fine && t > 1.0f && t < 1e5f) T = fp_from_f32(t);  // where the iteration of any state starts
    const float edge = 0.02f;
    fine = fine && (low ? t > (float)T_LO && t < (float)TMID - edge : t > (float)TMID + edge && t < (float)T_HI);
    if (fine) {
        const double T0 = fp_from_f32(t);
        double p = m[4];  // Horner: e, and by synthetic division its first two derivatives
        double d1 = p;
        p = fma(p, T0, m[3]);
        double d2 = d1;
        d1 = fma(d1, T0, p);
        p = fma(p, T0, m[2]);
        d2 = fma(d2, T0, d1);
        d1 = fma(d1, T0, p);
        p = fma(p, T0, m[1]);
        d2 = fma(d2, T0, d1);
        d1 = fma(d1, T0, p);
        p = fma(p, T0, m[0]);
        d2 = fma(d2, T0, d1);
        d1 = fma(d1, T0, p);
        p = fma(p, T0, m[5]);
        const double r = et - p;
        const double r0 = fp_from_f32(fp_rcp_seed(fp_to_f32(d1)));
        const double d = r * fma(r0, fma(-d1, r0, 1.0), r0);
        const float df = fp_to_f32(d), h = fp_to_f32(d2) * fp_to_f32(r0);  // d2 = cv'/2
        if (fabsf(df) <= 4e-6f * t) {
            const double dT = fma(d, fp_from_f32(-h * df), d);
            T = T0 + dT;
            // cv(T0 + dT) = cv + cv' dT + cv''/2 dT^2, the last term in FP32
            const float d3 = fmaf(t, fmaf(t, 10.0f * mf[4], 4.0f * mf[3]), mf[2]);  // cv''/6
            cv = fma(dT, fma(2.0, d2, fp_from_f32(3.0f * d3 * df)), d1);
            return true;
        }
    }
    return false;
}
template <int NS, bool PER_R = false>
__device__ __forceinline__ void secant_T(const double* w, float et, bool& low, float& t) {
    float lo = 0.0f, mid = 0.0f, hi = 0.0f;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const float f = fp_to_f32(w[k]);
        lo = fmaf(f, (float)(PER_R ? D_EAT_R.lo[k] : D_EAT_MASS.lo[k]), lo);
        mid = fmaf(f, (float)(PER_R ? D_EAT_R.mid[k] : D_EAT_MASS.mid[k]), mid);
        hi = fmaf(f, (float)(PER_R ? D_EAT_R.hi[k] : D_EAT_MASS.hi[k]), hi);
    }
    low = et <= mid;
    t = low ? (float)T_LO + (et - lo) * ((float)(TMID - T_LO) * fp_rcp_seed(mid - lo))
            : (float)TMID + (et - mid) * ((float)(T_HI - TMID) * fp_rcp_seed(hi - mid));
}

// The same for a specific energy e (J/kg) and weights z_k = Y_k / W_k, from a warm guess:
// FP32 Newton with both ranges' coefficients, then solve_T_any (two FP64 iterations).  Kept for
// the arithmetic of recorded runs (hf_record.cuh) and the derivatives of an objective
// (hf_adjoint.cu).
template <int NS, int RG>
__device__ __forceinline__ void mix_coef_f(const double* z, float* m) {
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        float s = 0.0f;
#pragma unroll
        for (int k = 0; k < NS; ++k) s = fmaf((float)z[k], (float)D_ECOEF.c[RG][k][j], s);
        m[j] = s;
    }
}
template <int NS>
__device__ __forceinline__ bool solve_T_iter(const double* z, double e_target, double& T, double* m) {
    if (!(T > 0.0) || !(T < 1e5)) T = 1000.0;
    {
        float mlo[6], mhi[6];
        mix_coef_f<NS, 0>(z, mlo);
        mix_coef_f<NS, 1>(z, mhi);
        const float et = (float)(e_target * (1.0 / RU));
        float t = (float)T;
        for (int it = 0; it < 40; ++it) {
            const float* mm = t <= 1000.0f ? mlo : mhi;
            float dt = (et - poly_e_f(mm, t)) / poly_cv_f(mm, t);
            dt = fminf(1000.0f, fmaxf(-1000.0f, dt));
            float tn = t + dt;
            if (!(tn > 0.0f)) tn = 0.5f * t;
            t = tn;
            if (!(fabsf(dt) > 1e-5f * t)) break;
        }
        if (t > 0.0f && t < 1e5f) T = (double)t;
    }
    return solve_T_any<NS, false>(z, e_target * (1.0 / RU), T, m);
}

struct Props { double p, a, T; };

// The terms of the EOS that the face fluxes use as well.
struct Prim { double rho, ir; };

// The conditions of an admissible state that need no temperature: finite, rho > 0, no
// negative partial density.  On bit patterns: with no negative q_k, rho = sum q_k is a
// NaN or infinite if and only if some q_k is.
template <int NS>
__device__ __forceinline__ bool state_ok(const double* q, double rho) {
    bool neg = false;
    unsigned top = fp_abs_hi(rho);
#pragma unroll
    for (int k = 0; k < NS; ++k) neg = neg || fp_neg_or_nan(q[k]);
#pragma unroll
    for (int n = NS; n < NS + 3; ++n) top = max(top, fp_abs_hi(q[n]));
    return !neg && top < 0x7ff00000u && !fp_zero(rho) && __double2hiint(rho) >= 0;
}

// physics.cpp:4-15 for a state held in registers.  Returns false when the state
// is inadmissible (non-finite, rho <= 0, a negative partial density, or an EOS
// solve that fails).  T_guess seeds the UV inversion.  In units of volume: with
// M_j = sum_k q_k c_kj R / W_k the energy equation is sum_j M_j T^(j+1) + M_5 =
// E - |m|^2 / 2 rho, so no mass fractions are formed.  Rounding errors (rms over the
// measured fields' states, against 80 bits) of p, a and T: 1.1 to 1.6, 0.9 to 1.1 and 0.9 to
// 1.4 e-16; with the operators, mass fractions and two FP64 Newton steps 1.4 to 2.5, 0.9 to 1.4
// and 1.2 to 1.3.
// Species whose partial density is below 2^-110 of the largest are left out of the sums by a
// warp in which all lanes agree on it.  Together they change the density, the heat capacity,
// sum q_k / W_k and, through the energy, T by less than 2^-94 of each (trace_bound): far below a
// rounding.  (A single coefficient of the mixture may lose all it has: H and AR have zeros in
// four.)  In unburnt gas that is 7 of 10, and a solve takes 58 FP64 instructions instead of 114.
constexpr double TRACE_RATIO = 65536.0;  // 2^16: times 2^-110
constexpr double abs_of(double x) { return x < 0 ? -x : x; }
constexpr bool trace_bound() {
    const ECoef e = make_ecoef_mass();
    const InvW w = make_rinvw();
    double w_lo = 1e300, w_hi = 0.0;
    for (int k = 0; k < NS_MAX; ++k) {
        w_lo = w.v[k] < w_lo ? w.v[k] : w_lo;
        w_hi = w.v[k] > w_hi ? w.v[k] : w_hi;
    }
    if (!(NS_MAX * w_hi < TRACE_RATIO * w_lo)) return false;
    for (double T = T_LO; T <= T_HI; T += 25.0) {
        double cv_lo = 1e300, cv_hi = 0.0, e_hi = 0.0;
        for (int k = 0; k < NS_MAX; ++k) {
            const double(&c)[6] = e.c[T <= TMID ? 0 : 1][k];
            const double cv = (((5.0 * c[4] * T + 4.0 * c[3]) * T + 3.0 * c[2]) * T + 2.0 * c[1]) * T + c[0];
            const double en = abs_of(ecoef_at(c, T));
            cv_lo = cv < cv_lo ? cv : cv_lo;
            cv_hi = cv > cv_hi ? cv : cv_hi;
            e_hi = en > e_hi ? en : e_hi;
        }
        // of the energy against cv T of the largest species: what it moves T by
        if (!(cv_lo > 0.0 && NS_MAX * cv_hi < TRACE_RATIO * cv_lo && NS_MAX * e_hi < TRACE_RATIO * cv_lo * T)) return false;
    }
    return true;
}
static_assert(trace_bound(), "a trace species can matter: the cut of live_species is too high for this mechanism");
template <int NS>
__device__ __forceinline__ unsigned live_species(const double* q) {
    unsigned top = 0, live = 0;
#pragma unroll
    for (int k = 0; k < NS; ++k) top = max(top, fp_abs_hi(q[k]));
#pragma unroll
    for (int k = 0; k < NS; ++k) live |= (fp_abs_hi(q[k]) + 0x06e00000u >= top ? 1u : 0u) << k;
    return __reduce_or_sync(__activemask(), live);
}
template <int NS, int RG>
__device__ __forceinline__ void mix_live(const double* q, unsigned live, double* m) {
#pragma unroll
    for (int j = 0; j < 6; ++j) m[j] = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k)
        if (live >> k & 1u) {
#pragma unroll
            for (int j = 0; j < 6; ++j)
                if (D_ECOEF_MASS.c[RG][k][j] != 0.0) m[j] = fma(q[k], D_ECOEF_MASS.c[RG][k][j], m[j]);
        }
}
template <int NS>
__device__ __forceinline__ bool properties(const double* q, Props& s, double T_guess, Prim& pr) {
    const unsigned live = live_species<NS>(q);
    double rho = 0.0, zs = 0.0;  // zs = sum_k q_k R / W_k
#pragma unroll
    for (int k = 0; k < NS; ++k)
        if (live >> k & 1u) {
            rho += q[k];
            zs = fma(q[k], RINVW.v[k], zs);
        }
    if (!state_ok<NS>(q, rho)) return false;
    const double ir = fp_rcp(rho);
    const double ke = fma(q[NS], q[NS], q[NS + 1] * q[NS + 1]) * ir;
    const double et = fma(-0.5, ke, q[NS + 2]);
    double T = T_guess, m[6], cv;
    {
        float t;
        bool low;
        secant_T<NS>(q, fp_to_f32(et), low, t);
        if (low) mix_live<NS, 0>(q, live, m);
        else mix_live<NS, 1>(q, live, m);
        if (!newton_T(m, et, low, t, T, cv)) {
            // through copies, so that the arrays of the fast path stay in registers
            double ws[NS], Ts = T, cvs = 0.0;
#pragma unroll
            for (int k = 0; k < NS; ++k) ws[k] = q[k];
            if (!solve_T_slow<NS, true>(ws, et, Ts, m, cvs)) return false;
            T = Ts;
            cv = cvs;
        }
    }
    pr.rho = rho;
    pr.ir = ir;
    s.T = T;
    s.p = T * zs;
    // a^2 = (1 + zs / cv) p / rho: zs / cv, rounded twice, is 0.2 to 0.7 of the sum
    const double P = s.p * ir;
    s.a = fp_sqrt_near(fma(P, zs * fp_rcp(cv), P));
    return fp_pos(s.T) && fp_pos(s.p) && fp_pos(s.a) && fp_finite(s.a);
}
template <int NS>
__device__ __forceinline__ bool properties(const double* q, Props& s, double T_guess) {
    Prim pr;
    return properties<NS>(q, s, T_guess, pr);
}

// A temperature of the state q near its own (secants of e(T) in FP32), to start a solve; et =
// rho e / R.
template <int NS>
__device__ __forceinline__ double estimate_T(const double* q, double et) {
    float t;
    bool low;
    secant_T<NS, true>(q, fp_to_f32(et), low, t);
    return t > 50.0f && t < 9000.0f ? fp_from_f32(t) : 1000.0;
}

// properties<NS>(q, ...) as a yes or no, without FP64 instructions where the answer is
// clear.  The energy equation e(T) = et has cv > 0 on [T_LO, T_HI] for every species (and
// cv within a factor of two of its value at T_mid on either side, so that Newton's steps
// contract): when et lies between the energies at T_LO and T_HI by more than FP32's
// rounding, there is a root between them, the solve finds it and p and a are positive.
// Anything else is left to properties().
template <int NS>
__device__ __forceinline__ bool admissible_state(const double* q, double T_guess) {
    bool neg = false, mass = false;
    unsigned top = 0;
    float lo = 0.0f, hi = 0.0f, mag = 0.0f, rho = 0.0f;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        neg = neg || fp_neg_or_nan(q[k]);
        top = max(top, fp_abs_hi(q[k]));
        const float f = fp_to_f32(q[k]);
        rho += f;
        lo = fmaf(f, (float)D_EAT_MASS.lo[k], lo);
        hi = fmaf(f, (float)D_EAT_MASS.hi[k], hi);
        mag = fmaf(f, fmaxf(fabsf((float)D_EAT_MASS.lo[k]), fabsf((float)D_EAT_MASS.hi[k])), mag);
    }
#pragma unroll
    for (int n = NS; n < NS + 3; ++n) top = max(top, fp_abs_hi(q[n]));
    mass = rho > 1e-12f && rho < 1e12f;
    if (!neg && mass && top < 0x7ff00000u) {
        const float mu = fp_to_f32(q[NS]), mv = fp_to_f32(q[NS + 1]), E = fp_to_f32(q[NS + 2]);
        const float ke = 0.5f * fmaf(mu, mu, mv * mv) * fp_rcp_seed(rho);
        const float et = E - ke, err = 1e-5f * (mag + fabsf(E) + ke);
        if (et - err > lo && et + err < hi) return true;
    }
    Props p;
    return properties<NS>(q, p, T_guess);
}

// physics.cpp:40-44, one component: x y > 0 ? copysign(min(|x|, |y|), x) : 0, from the bit
// patterns.  The product of two numbers of one sign is positive unless it underflows or
// one is a NaN; those cases are decided by the product itself (as is any denormal operand,
// whose exponent field says too little).
__device__ __forceinline__ double minmod(double x, double y) {
    const unsigned hx = fp_abs_hi(x), hy = fp_abs_hi(y);
    const unsigned long long ax = fp_abs_bits(x), ay = fp_abs_bits(y);
    const unsigned long long lo = ax < ay ? ax : ay;
    bool pos = (__double2hiint(x) ^ __double2hiint(y)) >= 0;
    if (hx + hy < 0x3cf00000u || min(hx, hy) < 0x00100000u ? lo != 0 : max(hx, hy) >= 0x7ff00000u)
        pos = fp_prod_pos_lib(x, y);
    pos = pos && lo != 0;
    return __hiloint2double(pos ? (int)((unsigned)(lo >> 32) | ((unsigned)__double2hiint(x) & 0x80000000u)) : 0,
                            pos ? (int)(unsigned)lo : 0);
}

// physics.cpp:17-38: multispecies HLLC with Davis speeds in direction n (NS or NS+1).  In
// the star region every advected component's flux is q (v + s (scale - 1)).  dl, dr:
// density and its reciprocal on each side.
template <int NS, int N>
__device__ __forceinline__ void hllc(const double* l, const double* r, const Props& pl, const Props& pr,
                                     const Prim& dl_, const Prim& dr_, double* f) {
    constexpr int E = NS + 2;
    const double rl = dl_.rho, rr = dr_.rho;
    const double ul = l[N] * dl_.ir, ur = r[N] * dr_.ir;
    const double sl = fp_min(ul - pl.a, ur - pr.a), sr = fp_max(ul + pl.a, ur + pr.a);
    const bool allL = fp_ge0(sl), allR = !allL && !fp_pos(sr);
    const double wl = sl - ul, wr = sr - ur;
    const double dl = rl * wl, dr = rr * wr;
    double sm = 0.0;
    bool left = allL;
    if (!allL && !allR) {
        sm = fp_div((pr.p - pl.p) + fma(dl, ul, -dr * ur), dl - dr);
        left = fp_ge0(sm);
    }
    const double v = left ? ul : ur, p = left ? pl.p : pr.p;
    double qn = left ? l[N] : r[N], qe = left ? l[E] : r[E];
    double wgt = v, fn = fma(v, qn, p), fe = v * (qe + p);
    if (!allL && !allR) {
        const double s = left ? sl : sr, w = left ? wl : wr, d = left ? dl : dr, rq = left ? rl : rr;
        const double scale = fp_div(w, s - sm);
        const double rs = rq * scale;
        const double estar = fma(qe, scale, rs * (sm - v) * (sm + fp_div(p, d)));
        wgt = fma(s, scale - 1.0, v);
        fn = fma(s, fma(rs, sm, -qn), fn);
        fe = fma(s, estar - qe, fe);
    }
#pragma unroll
    for (int m = 0; m < NS + 3; ++m) {
        const double q = left ? l[m] : r[m];
        f[m] = m == N ? fn : m == E ? fe : q * wgt;
    }
}

}  // namespace hf
