// The EOS and HLLC of recorded runs (hf_flow_record) and of their reverse sweep.  In gas at
// rest with a uniform pressure the contact speed is a difference of rounding errors, and
// its sign picks the side that the reverse sweep of the flux differentiates.  So the
// derivative is that of this arithmetic: the recorded stages and the reverse sweep's
// recomputation of them (hf_flux_adjoint.cu) evaluate these forms bit for bit, and no other
// path uses them (properties() and hllc() of hf_device.cuh agree to rounding with a third of
// the FP64 instructions).
#pragma once
#include "hf_device.cuh"

namespace hf {
namespace rec {

// physics.cpp:4-15 for a state held in registers.  Returns false when the state
// is inadmissible (non-finite, rho <= 0, a negative partial density, or an EOS
// solve that fails).  T_guess seeds the UV inversion.
template <int NS>
__device__ __forceinline__ bool properties(const double* q, Props& s, double T_guess) {
    bool ok = true;
    double rho = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        rho += q[k];
        ok = ok && (q[k] >= 0.0);
    }
#pragma unroll
    for (int n = NS; n < NS + 3; ++n) ok = ok && isfinite(q[n]);
    ok = ok && isfinite(rho) && (rho > 0.0);
    if (!ok) return false;
    const double ir = 1.0 / rho;
    double z[NS];
    double zs = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        z[k] = q[k] * ir * INVW.v[k];
        zs += z[k];
    }
    const double u = q[NS] * ir, v = q[NS + 1] * ir;
    const double e = q[NS + 2] * ir - 0.5 * (u * u + v * v);
    double T = T_guess, m[6];
    if (!solve_T_iter<NS>(z, e, T, m)) return false;
    const double cvR = poly_cv(m, T);  // cv/R per unit mass (times W units)
    const double cpR = cvR + zs;
    s.T = T;
    s.p = rho * RU * T * zs;
    s.a = sqrt(cpR / cvR * RU * T * zs);
    return s.T > 0.0 && s.p > 0.0 && s.a > 0.0 && isfinite(s.a);
}

// physics.cpp:17-38: multispecies HLLC with Davis speeds in direction n (NS or NS+1).
template <int NS, int N>
__device__ __forceinline__ void hllc(const double* l, const double* r, const Props& pl, const Props& pr,
                                     double* f) {
    constexpr int E = NS + 2;
    double rl = 0.0, rr = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k) { rl += l[k]; rr += r[k]; }
    const double ul = l[N] / rl, ur = r[N] / rr;
    const double sl = fmin(ul - pl.a, ur - pr.a), sr = fmax(ul + pl.a, ur + pr.a);
    if (sl >= 0.0 || sr <= 0.0) {
        const bool useL = sl >= 0.0;
        const double* q = useL ? l : r;
        const double v = useL ? ul : ur, p = useL ? pl.p : pr.p;
#pragma unroll
        for (int m = 0; m < NS + 3; ++m) f[m] = v * q[m];
        f[N] += p;
        f[E] += p * v;
        return;
    }
    const double dl = rl * (sl - ul), dr = rr * (sr - ur);
    const double sm = (pr.p - pl.p + dl * ul - dr * ur) / (dl - dr);
    const bool left = sm >= 0.0;
    const double* q = left ? l : r;
    const double v = left ? ul : ur, s = left ? sl : sr, p = left ? pl.p : pr.p, rq = left ? rl : rr;
    const double scale = (s - v) / (s - sm);
    double rs = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k) rs += q[k] * scale;
    const double estar = q[E] * scale + rs * (sm - v) * (sm + p / (rq * (s - v)));
#pragma unroll
    for (int m = 0; m < NS + 3; ++m) {
        double st = q[m] * scale;
        if (m == N) st = rs * sm;
        if (m == E) st = estar;
        double fl = v * q[m];
        if (m == N) fl += p;
        if (m == E) fl += p * v;
        f[m] = fl + s * (st - q[m]);
    }
}

}  // namespace rec
}  // namespace hf
