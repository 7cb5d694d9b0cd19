// Discrete adjoint of the chemistry calls (a build-defined extension: the
// reference has no sensitivity code).  A 0D cell at constant (rho, e) is advanced
// by ncalls chemistry calls of dt each, every call exactly as Chemistry::advance
// (HyperFlow_V3/src/chemistry.cpp:55-76, here the Rodas4 integration of
// hf_group.cuh: adaptive steps, clip y >= -1e-13 to 0, last species closes the
// mass).  An objective J of the temperatures / pressures at the call boundaries
// is differentiated with respect to p_r = ln(multiplier_r) of every reaction
// (the multiplier scales the forward and reverse rate constants; for falloff
// reactions both limits) and to the initial mass fractions.
//
// Differentiated map: the accepted step sequence of the run is frozen (the step
// sizes are constants), so the map is a composition of Rodas4 steps
//     y+ = y + sum_s m_s K_s,   (I/(h g) - J(y)) K_s = f(Y_s) + sum_j c_sj/h K_j,
//     Y_s = y + sum_j a_sj K_j,
// and of the clips at call ends; hf_group_adjoint.cuh has its reverse sweep per step, one
// cell per group of 8 lanes.
//
// Memory: checkpoints of the state every K calls; in the reverse sweep a segment
// of K calls is recomputed from its checkpoint, storing the state at every call
// boundary and the tape of accepted steps (y, h, T); a segment whose tape exceeds
// its capacity recomputes each call again from the stored boundary states.
#include <type_traits>
#include "hf_group_adjoint.cuh"

namespace hf {

cudaError_t adjoint_set_rate_scale(const double* scale) { return upload_rate_constants(scale); }

// cp/R of every species
template <int NS>
__device__ __forceinline__ void species_cp(double T, double* cpR) {
    const int rg = T <= TMID ? 0 : 1;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const double* a = D_NASA.c[rg][k];
        cpR[k] = fma(T, fma(T, fma(T, fma(T, a[4], a[3]), a[2]), a[1]), a[0]);
    }
}

// Constant-(rho, e) temperature derivatives at y (R units: e_k/R = T (h_k/RT - 1)/W_k,
// cv_k/R = (cp_k/R - 1)/W_k):  dT/dy_j = -(e_j - e_L)/cv.
template <int NS>
__device__ __forceinline__ void temp_grad(const KinCtx<NS>& kc, const double* cpR, const double* y, double* dTdy) {
    constexpr int N = NS - 1, L = NS - 1;
    double YL = 1.0;
#pragma unroll
    for (int k = 0; k < N; ++k) YL -= y[k];
    double cv = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const double Yk = k < N ? y[k] : YL;
        cv = fma(Yk, (cpR[k] - 1.0) * INVW.v[k], cv);
    }
    const double eL = kc.T * (kc.hRT[L] - 1.0) * INVW.v[L];
#pragma unroll
    for (int j = 0; j < N; ++j) dTdy[j] = -(kc.T * (kc.hRT[j] - 1.0) * INVW.v[j] - eL) / cv;
}

// dT/dy and dp/dy of the state u (y = u/rho at fixed rho, e).
template <int NS>
__device__ bool state_grads(const double* u, double* dT, double* dp, double& T) {
    constexpr int N = NS - 1;
    double rho = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k) rho += u[k];
    const double ir = 1.0 / rho;
    const double uu = u[NS] * ir, vv = u[NS + 1] * ir;
    const double e = u[NS + 2] * ir - 0.5 * (uu * uu + vv * vv);
    double y[N], z[NS], C[NS], m[6];
#pragma unroll
    for (int k = 0; k < N; ++k) y[k] = u[k] * ir;
    comp<NS>(y, rho, z, C);
    if (!solve_T_iter<NS>(z, e, T, m)) return false;
    KinCtx<NS> kc;
    kin_setup<NS, false>(T, C, kc);
    double cpR[NS];
    species_cp<NS>(T, cpR);
    temp_grad<NS>(kc, cpR, y, dT);
    double zs = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k) zs += z[k];
    // p = rho R T sum_k Y_k/W_k
#pragma unroll
    for (int j = 0; j < N; ++j) dp[j] = rho * RU * (zs * dT[j] + T * (INVW.v[j] - INVW.v[NS - 1]));
    return true;
}

namespace {

using grp8::AdjShared;
using grp8::Acc;
using grp8::NQ;

// One chemistry call on the conserved state u (every lane of the group holds it) of each of
// the warp's cells with act set, optionally appending every accepted step (y, h, T) to the
// tape at slot nrec (stored while nrec < cap).  clip receives bit k when y_k was clipped, y
// the lane's component of the result before the clip.
template <int NS>
__device__ int run_call(double* u, double dt, double rtol, double atol, double* tape, int64_t tstride, int& nrec, int cap,
                        uint32_t& clip, double& y, bool act, grp8::Shared* sh) {
    constexpr int N = NS - 1;
    const int t = grp8::lane8();
    grp8::Cell<NS> c;
    const bool ok = grp8::load<NS>(c, u, dt, 0.0);
    c.active = act && ok;
    int res = act && !ok ? CELL_FAIL : CELL_DONE;
    while (__any_sync(grp8::FULL, c.active)) {
        const double yp = c.y, Tp = c.T;
        const int s0 = c.steps;
        bool screened;
        const int r = grp8::attempt<NS, false>(c, rtol, atol, sh, screened);
        if (c.active && c.steps > s0) {
            if (tape && nrec < cap) {
                double* p = tape + (int64_t)nrec * (N + 2) * tstride;
                p[t * tstride] = yp;
                if (t == 0) {
                    if (NS == 10) p[8 * tstride] = c.yN2;
                    p[N * tstride] = c.hu;
                    p[(N + 1) * tstride] = Tp;
                }
            }
            ++nrec;
        }
        if (c.active && r != CELL_CONTINUE) {
            res = r;
            c.active = false;
        }
    }
    double uo[NS + 3];
    const bool keep = grp8::finish<NS>(c, uo);
    const unsigned neg = __ballot_sync(grp8::FULL, fp_neg(c.y));
    if (act) {
        clip = neg >> (threadIdx.x & 24) & 0xffu;
        y = c.y;
        if (res == CELL_DONE && !keep) res = CELL_FAIL;
        if (res == CELL_DONE) {
#pragma unroll
            for (int n = 0; n < NS + 3; ++n) u[n] = uo[n];
        }
    }
    __syncwarp();
    return res;
}

// Constants of a cell's interval from its state u.
template <int NS>
struct Interval {
    double rho, ir, e, et, Ci0, Ci1;
};
template <int NS>
__device__ __forceinline__ Interval<NS> interval(const double* u) {
    Interval<NS> v;
    double rho = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k) rho += u[k];
    v.rho = rho;
    v.ir = 1.0 / rho;
    const double uu = u[NS] * v.ir, vv = u[NS + 1] * v.ir;
    v.e = u[NS + 2] * v.ir - 0.5 * (uu * uu + vv * vv);
    v.et = rho * v.e * (1.0 / RU);
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < NS - 1; ++k) s += u[k] * v.ir;
    const double last = rho * (1.0 - s) * INVW.v[NS - 1];
    v.Ci0 = NS == 10 ? u[8] * INVW.v[8] : last;
    v.Ci1 = NS == 10 ? last : 0.0;
    return v;
}

// Reverse sweep of the cnt tape steps of one call (recorded from slot base on): lamC =
// dJ/dC at its end in, at its start out; acc as in step_adjoint.
template <int NS>
__device__ __forceinline__ bool call_adjoint(const Interval<NS>& v, const double* tape, int64_t tstride, int base, int cnt,
                                             bool act, double& lamC, Acc& acc, AdjShared* sh) {
    constexpr int N = NS - 1;
    const int t = grp8::lane8();
    bool ok = true;
    int mx = act ? cnt : 0;
    for (int o = 16; o >= 8; o >>= 1) mx = max(mx, __shfl_xor_sync(grp8::FULL, mx, o));
    double y = 0.1, h = 1e-9, T = 1500.0;  // groups without a step left compute along
    for (int s = mx - 1; s >= 0; --s) {
        const bool on = act && ok && s < cnt;
        if (on) {
            const double* p = tape + (int64_t)(base + s) * (N + 2) * tstride;
            y = p[t * tstride];
            h = p[N * tstride];
            T = p[(N + 1) * tstride];
        }
        Acc a = acc;
        const bool good = grp8::step_adjoint<NS>(v.rho, v.et, v.Ci0, v.Ci1, y, h, T, on, lamC, a, sh);
        if (on) {
            acc = a;
            ok = good;
        }
    }
    return ok;
}

enum { OBJ_IGNITION = HF_OBJ_IGNITION_DELAY, OBJ_PEAK_PRESSURE = HF_OBJ_PEAK_PRESSURE, OBJ_FINAL_T = HF_OBJ_FINAL_T };

// Forward pass: ncalls calls with checkpoints (ckpt may be null), objective
// bookkeeping; then (BACKWARD) the reverse sweep.  One cell per group of 8 lanes, four per
// warp and block: the cells' step chains are what a run waits for (1,024 cells, 8 calls and
// their reverse: 155 ms, 1,236 with one cell per lane).  The forward-only instantiation carries
// none of the reverse sweep's registers.
#pragma nv_diag_suppress 128  // the forward-only instantiation ends before the reverse sweep's loops
template <int NS, bool BACKWARD>
__global__ void __launch_bounds__(32) k_chem_adjoint(AdjointArgs a) {
    constexpr int N = NS - 1, NV = NS + 3;
    using Sh = std::conditional_t<BACKWARD, AdjShared, grp8::Shared>;
    __shared__ Sh shm[4];
    Sh* const sh = &shm[threadIdx.x >> 3];
    grp8::Shared* fs;
    if constexpr (BACKWARD) fs = &sh->f;
    else fs = sh;
    const int t = grp8::lane8();
    const int64_t want = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 3);
    bool live = want < a.chunk;
    const int64_t i = live ? want : a.chunk - 1;  // groups past the end compute along
    const int64_t gi = a.i0 + i;
    const int64_t cst = a.chunk;  // stride of the scratch arrays
    double u[NV];
#pragma unroll
    for (int n = 0; n < NV; ++n) u[n] = a.U0[gi + n * a.cs];
    auto put = [&](double* p, const double* q) {  // a state into a scratch slot
#pragma unroll
        for (int n = 0; n < NV; ++n)
            if ((n & 7) == t) p[n * cst + i] = q[n];
    };
    auto fail_cell = [&](int code) {
        if (t == 0) {
            a.fail[gi] = code;
            atomicOr(&a.st->flags, code == CELL_MAXSTEPS ? ST_MAXSTEPS : ST_CHEM_FAIL);
            atomicMin(&a.st->bad_cell, (unsigned long long)gi);
            a.J[gi] = __longlong_as_double(0x7ff8000000000000ll);
        }
    };
    Props pr{};
    if (live && !properties<NS>(u, pr, 1000.0)) {
        fail_cell(CELL_FAIL);
        live = false;
    }
    const double T0 = pr.T, Ts = T0 + a.dT;
    int n_ign = -1, n_pmax = 0;
    double Ta = 0.0, Tb = 0.0, pmax = pr.p, Tprev = T0, yend = 0.0;
    unsigned long long steps = 0;
    // BACKWARD: the last segment (from call nlast on) is recorded here already
    const int nlast = (a.ncalls - 1) / a.K * a.K;
    int nrec_last = 0;
    for (int n = 0; n < a.ncalls && __any_sync(grp8::FULL, live); ++n) {
        if (a.ckpt && n % a.K == 0 && live) put(a.ckpt + (int64_t)(n / a.K) * NV * cst, u);
        const bool record = BACKWARD && n >= nlast;
        if (record && n == nlast && live) put(a.seg, u);
        const int before = nrec_last;
        int none = 0;
        uint32_t clip = 0;
        const int r = run_call<NS>(u, a.dt, a.rtol, a.atol, record ? a.tape + i : nullptr, cst,
                                   record ? nrec_last : none, a.cap, clip, yend, live, fs);
        if (record && live && r == CELL_DONE) {
            if (t == 0) {
                a.nstep[(int64_t)(n - nlast) * cst + i] = nrec_last - before;
                a.clipm[(int64_t)(n - nlast) * cst + i] = clip;
            }
            put(a.seg + (int64_t)(n - nlast + 1) * NV * cst, u);
        }
        if (live && r != CELL_DONE) {
            fail_cell(r == CELL_MAXSTEPS ? CELL_MAXSTEPS : CELL_FAIL);
            live = false;
        }
        if (live && !properties<NS>(u, pr, Tprev)) {
            fail_cell(CELL_FAIL);
            live = false;
        }
        if (live) {
            if (n_ign < 0 && pr.T >= Ts) { n_ign = n; Ta = Tprev; Tb = pr.T; }
            if (pr.p > pmax) { pmax = pr.p; n_pmax = n + 1; }
            Tprev = pr.T;
        }
    }
    if (live && t == 0) {
        double Jv;
        if (a.objective == OBJ_FINAL_T) Jv = Tprev;
        else if (a.objective == OBJ_PEAK_PRESSURE) Jv = pmax;
        else Jv = n_ign < 0 ? __longlong_as_double(0x7ff8000000000000ll)
                            : n_ign * a.dt + a.dt * (Ts - Ta) / (Tb - Ta);
        a.J[gi] = Jv;
        a.fail[gi] = 0;
    }
    if constexpr (!BACKWARD) {
        return;
    } else {
        Acc acc{};
        double lam = 0.0, lamN2 = 0.0;  // dJ/dy of the lane's species, of N2 (NS = 10)
        const bool active = live && !(a.objective == OBJ_IGNITION && n_ign < 0);
        // seed dJ/dy_n at call boundary n (state un)
        auto seed = [&](int n, const double* un) -> bool {
            double w = 0.0;
            bool useT = true;
            if (a.objective == OBJ_FINAL_T) {
                if (n == a.ncalls) w = 1.0;
            } else if (a.objective == OBJ_PEAK_PRESSURE) {
                if (n == n_pmax) { w = 1.0; useT = false; }
            } else {
                const double d = Tb - Ta;
                if (n == n_ign) w = a.dt * (Ts - Tb) / (d * d);
                else if (n == n_ign + 1) w = -a.dt * (Ts - Ta) / (d * d);
                if (n == 0) w += a.dt / d;  // through the threshold T_0 + dT
            }
            if (w == 0.0) return true;
            double gT[N], gp[N], T = 1000.0;
            if (!state_grads<NS>(un, gT, gp, T)) return false;
#pragma unroll
            for (int k = 0; k < NQ; ++k)
                if (k == t) lam = fma(w, useT ? gT[k] : gp[k], lam);
            if (NS == 10) lamN2 = fma(w, useT ? gT[N - 1] : gp[N - 1], lamN2);
            return true;
        };
        bool ok = active;
        const int nseg = (a.ncalls + a.K - 1) / a.K;
        for (int sg = nseg - 1; sg >= 0 && __any_sync(grp8::FULL, ok); --sg) {
            const int n0 = sg * a.K, n1 = min(n0 + a.K, a.ncalls);
            // recompute the segment: boundary states and the tape of accepted steps
            const double* c = a.ckpt + (int64_t)sg * NV * cst;
            const bool have = sg == nseg - 1;  // by the forward pass
            __syncwarp();
            if (ok && !have) {
#pragma unroll
                for (int v = 0; v < NV; ++v) u[v] = c[v * cst + i];
                put(a.seg, u);
            }
            int nrec = have ? nrec_last : 0;
            for (int n = n0; n < n1 && !have && __any_sync(grp8::FULL, ok); ++n) {
                uint32_t clip = 0;
                const int before = nrec;
                const int r = run_call<NS>(u, a.dt, a.rtol, a.atol, a.tape + i, cst, nrec, a.cap, clip, yend, ok, fs);
                if (ok) {
                    ok = r == CELL_DONE;
                    if (t == 0) {
                        a.nstep[(int64_t)(n - n0) * cst + i] = nrec - before;
                        a.clipm[(int64_t)(n - n0) * cst + i] = clip;
                    }
                    put(a.seg + (int64_t)(n - n0 + 1) * NV * cst, u);
                }
            }
            __syncwarp();
            const bool overflow = nrec > a.cap;
            if (ok && sg == nseg - 1) {
                double ue[NV];
                const double* sb = a.seg + (int64_t)(n1 - n0) * NV * cst;
#pragma unroll
                for (int v = 0; v < NV; ++v) ue[v] = sb[v * cst + i];
                ok = seed(n1, ue);
            }
            int end = nrec;
            for (int n = n1 - 1; n >= n0 && __any_sync(grp8::FULL, ok); --n) {
                const uint32_t clip = ok ? a.clipm[(int64_t)(n - n0) * cst + i] : 0;
                if (clip >> t & 1u) lam = 0.0;
                const int cnt = ok ? a.nstep[(int64_t)(n - n0) * cst + i] : 0;
                double un[NV];
                const double* sb = a.seg + (int64_t)(n - n0) * NV * cst;
#pragma unroll
                for (int v = 0; v < NV; ++v) un[v] = ok ? sb[v * cst + i] : u[v];
                int base = end - cnt;
                end = base;
                if (__any_sync(grp8::FULL, ok && overflow)) {
                    // recompute this call alone into the start of the tape
                    double uc[NV];
#pragma unroll
                    for (int v = 0; v < NV; ++v) uc[v] = un[v];
                    int nr = 0;
                    uint32_t cl = 0;
                    const bool redo = ok && overflow;
                    const int r = run_call<NS>(uc, a.dt, a.rtol, a.atol, a.tape + i, cst, nr, a.cap, cl, yend, redo, fs);
                    if (redo) {
                        ok = r == CELL_DONE && nr == cnt;
                        base = 0;
                    }
                    __syncwarp();
                }
                // y = C W / rho at the end of the call; y_k = u_k / rho, the last species closing
                // the mass, at its start
                const Interval<NS> v = interval<NS>(un);
                const double W = D_MW.v[t];
                double lamC = lam * W * v.ir;
                acc.gin = NS == 10 && t == 0 ? lamN2 * D_MW.v[8] * v.ir : 0.0;
                const bool good = call_adjoint<NS>(v, a.tape + i, cst, base, cnt, ok, lamC, acc, sh);
                if (ok) {
                    ok = good;
                    steps += t == 0 ? cnt : 0;
                }
                const double gL = grp8::get(acc.gin, NS - 1 - NQ) * INVW.v[NS - 1];
                const double g2 = grp8::get(acc.gin, 0) * INVW.v[8];
                if (ok) {
                    lam = v.rho * (lamC * INVW.v[t] - gL);
                    if (NS == 10) lamN2 = v.rho * (g2 - gL);
                    ok = seed(n, un);
                }
            }
        }
        if (active && !ok) {
            fail_cell(CELL_FAIL);
            return;
        }
        if (!live) return;
        if (t == 0) atomicAdd(&a.st->steps, steps);
#pragma unroll
        for (int rnd = 0; rnd < grp8::NROUND; ++rnd) {
            const int r = rnd * grp8::G + t;
            if (r < NR) a.dJdp[(int64_t)r * a.count + gi] = acc.pb[rnd];
        }
        if (a.dJdy0) {
            a.dJdy0[(int64_t)t * a.count + gi] = lam;
            if (NS == 10 && t == 0) a.dJdy0[(int64_t)(N - 1) * a.count + gi] = lamN2;
        }
    }
}
#pragma nv_diag_default 128

// Adjoint of the react phase of a Strang step on the cells of a ghosted patch: one
// chemistry call (as recorded, its accepted steps recomputed into the tape)
// per cell.  ubar_in = (du_out/du_in)^T ubar_out through
//   u_in -> (y = u_k/rho, rho = sum u_k, e = E/rho - |m|^2/(2 rho^2)) -> C, Cin, et -> Rodas4
//   steps -> y = C W/rho -> clip -> u_out_k = rho max(0, y_k), u_out_L = rho - sum u_out_k, m
//   and E unchanged,
// and pcell[r][cell] += dJ/d ln A_r of the cell.  One cell of [i0, i0+chunk) per group.
template <int NS>
__global__ void __launch_bounds__(32) k_chem_call_adjoint(hf_patch P, const double* __restrict__ U,
                                                          const double* __restrict__ ubar_out,
                                                          double* __restrict__ ubar_in, double dt, double rtol,
                                                          double atol, double* __restrict__ tape, int cap, int64_t i0,
                                                          int64_t chunk, double* __restrict__ pcell, DevStatus* st) {
    constexpr int N = NS - 1, NV = NS + 3;
    __shared__ AdjShared shm[4];
    AdjShared* const sh = &shm[threadIdx.x >> 3];
    const int t = grp8::lane8();
    const int64_t nc = (int64_t)P.nx * P.ny, top = min(chunk, nc - i0);
    const int64_t want = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 3);
    const bool live = want < top;
    const int64_t li = live ? want : top - 1, i = i0 + li;
    const int ci = (int)(i % P.nx), cj = (int)(i / P.nx);
    const int64_t g = P.offset + (int64_t)(cj + P.ng) * P.pitch + (ci + P.ng);
    double u[NV], ub[NV], uc[NV];
#pragma unroll
    for (int n = 0; n < NV; ++n) {
        u[n] = U[g + n * P.comp_stride];
        ub[n] = ubar_out[g + n * P.comp_stride];
        uc[n] = u[n];
    }
    int nrec = 0;
    uint32_t clip = 0;
    double yend = 0.0;
    const int r = run_call<NS>(uc, dt, rtol, atol, tape + li, chunk, nrec, cap, clip, yend, live, &sh->f);
    bool ok = live && r == CELL_DONE && nrec <= cap;
    const Interval<NS> v = interval<NS>(u);
    const double mx = u[NS], my = u[NS + 1], ir = v.ir;
    // output side: u_out_k = rho Y'_k (k < N), u_out_L = rho (1 - sum Y'_k)
    double lam = 0.0, lamN2 = 0.0, rhob = ub[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const double d = ub[k] - ub[N];
        if (k == t) lam = (clip >> k & 1u) ? 0.0 : v.rho * d;
        if (k == 8) lamN2 = v.rho * d;
        rhob = fma(uc[k] * ir, d, rhob);
    }
    // y' = C W / rho
    double lamC = lam * D_MW.v[t] * ir;
    Acc acc{};
    acc.gin = NS == 10 && t == 0 ? lamN2 * D_MW.v[8] * ir : 0.0;
    double own = -lam * yend;  // through y' = C W / rho
    if (NS == 10 && t == 0) own = fma(-lamN2, u[8] * ir, own);
    rhob = fma(grp8::xsum(ok ? own : 0.0), ir, rhob);
    __syncwarp();
    ok = call_adjoint<NS>(v, tape + li, chunk, 0, nrec, ok, lamC, acc, sh) && ok;
    // input side: C_k = u_k / W_k, Cin likewise (the closing species' too), et = (E - |m|^2 /
    // 2 rho) / R with rho = sum u_k
    double out[NV];
    const double mine = lamC * INVW.v[t];
#pragma unroll
    for (int k = 0; k < NQ; ++k) out[k] = grp8::get(mine, k);
#pragma unroll
    for (int k = NQ; k < NS; ++k) out[k] = grp8::get(acc.gin, k - NQ) * INVW.v[k];
    const double eb = acc.get * (1.0 / RU);
    rhob = fma(eb, 0.5 * (mx * mx + my * my) * ir * ir, rhob);
#pragma unroll
    for (int k = 0; k < NS; ++k) out[k] += rhob;
    out[NS] = ub[NS] - eb * mx * ir;
    out[NS + 1] = ub[NS + 1] - eb * my * ir;
    out[NS + 2] = ub[NS + 2] + eb;
    if (!live) return;
    if (ok) {
#pragma unroll
        for (int rnd = 0; rnd < grp8::NROUND; ++rnd) {
            const int q = rnd * grp8::G + t;
            if (q < NR) pcell[(int64_t)q * nc + i] += acc.pb[rnd];
        }
    } else if (t == 0) {
        atomicOr(&st->flags, ST_CHEM_FAIL);
        atomicMin(&st->bad_cell, (unsigned long long)i);
    }
#pragma unroll
    for (int n = 0; n < NV; ++n)
        if ((n & 7) == t) ubar_in[g + n * P.comp_stride] = ok ? out[n] : 0.0;
}

}  // namespace

cudaError_t launch_chem_call_adjoint(int ns, const hf_patch& P, const double* U, const double* ubar_out,
                                     double* ubar_in, double dt, double rtol, double atol, double* tape, int cap,
                                     int64_t i0, int64_t chunk, double* pcell, DevStatus* st, cudaStream_t s,
                                     int64_t* launches) {
    if (chunk <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)((chunk + 3) / 4);
    if (ns == 9)
        k_chem_call_adjoint<9><<<grid, 32, 0, s>>>(P, U, ubar_out, ubar_in, dt, rtol, atol, tape, cap, i0, chunk, pcell,
                                                   st);
    else
        k_chem_call_adjoint<10><<<grid, 32, 0, s>>>(P, U, ubar_out, ubar_in, dt, rtol, atol, tape, cap, i0, chunk,
                                                    pcell, st);
    if (launches) ++*launches;
    return cudaGetLastError();
}

size_t adjoint_bytes_per_cell(int ns, int ncalls, int K, int cap) {
    const int nv = ns + 3, n = ns - 1;
    const int nck = (ncalls + K - 1) / K;
    return sizeof(double) * ((size_t)nck * nv + (size_t)(K + 1) * nv + (size_t)cap * (n + 2)) +
           sizeof(int32_t) * 2 * (size_t)K;
}

cudaError_t launch_chem_adjoint(int ns, const AdjointArgs& a, cudaStream_t s, int64_t* launches) {
    if (a.chunk <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)((a.chunk + 3) / 4);
    if (a.backward) {
        if (ns == 9) k_chem_adjoint<9, true><<<grid, 32, 0, s>>>(a);
        else k_chem_adjoint<10, true><<<grid, 32, 0, s>>>(a);
    } else {
        if (ns == 9) k_chem_adjoint<9, false><<<grid, 32, 0, s>>>(a);
        else k_chem_adjoint<10, false><<<grid, 32, 0, s>>>(a);
    }
    if (launches) ++*launches;
    return cudaGetLastError();
}

}  // namespace hf
