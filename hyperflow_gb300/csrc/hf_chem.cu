// Stiff per-cell chemistry: the reference's constant-(rho, e) ODE
// (HyperFlow_V3/src/chemistry.cpp:36-53: unknowns Y_0..Y_{NS-2}, last species
// dependent, T from the UV inversion at every evaluation) integrated over dt with
// Rodas4 (Hairer & Wanner, Solving ODEs II, Sec. VI.7; KPP coefficient ordering),
// WRMS errors with weights atol + rtol*max(|y_old|, |y_new|), an analytic Jacobian,
// and the KPP step controller.  Cell semantics follow Chemistry::advance
// (chemistry.cpp:55-76): properties() check, clip y >= -1e-13 to 0, dependent
// species closes the mass, final properties() check.  Batch semantics follow
// ChemistryBatch::advance (chemistry_batch.cpp:21-50): all-or-nothing with the
// lowest failing index.
//
// The integrators are in hf_cell.cuh (one cell per lane) and hf_group.cuh (one per group of
// 8 lanes); this file holds the chemistry kernels (plain, persistent, batched with its
// cost-ordered queues, small batches in groups), the ErrorEst tagging kernel and the
// allocation-free entry point.  Rate data: pre-exponential factors sit in
// __constant__ memory (c_A, c_A0) so they can be scaled for sensitivity checks;
// reaction structure, temperature exponents and activation temperatures are
// compile-time constants of the generated mechanism table, so every species index
// is a register index.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include "hf_cell.cuh"
#include "hf_group.cuh"

namespace hf {

cudaError_t chem_set_rate_scale(const double* scale) { return upload_rate_constants(scale); }

// ---------------------------------------------------------------- kernels
template <int NS>
__device__ __forceinline__ void load_cell(const double* U, int64_t cs, int64_t base, double* u) {
#pragma unroll
    for (int n = 0; n < NS + 3; ++n) u[n] = U[base + n * cs];
}
__device__ __forceinline__ void report(DevStatus* st, int* fail, int64_t i, int code) {
    fail[i] = code;
    atomicOr(&st->flags, code == CELL_MAXSTEPS ? ST_MAXSTEPS : ST_CHEM_FAIL);
    atomicMin(&st->bad_cell, (unsigned long long)i);
}

// Plain form: one thread runs one cell to completion.
template <int NS>
__global__ void __launch_bounds__(64) k_chem_plain(const double* __restrict__ U, int64_t cs,
                                                   const int64_t* __restrict__ cell_index, int64_t count, double dt,
                                                   const double* __restrict__ dt_dev,
                                                   const double* __restrict__ dt_cell, double rtol, double atol,
                                                   double* __restrict__ trial, int* __restrict__ fail, DevStatus* st) {
    if (st->abort_run) return;  // an earlier step of this device-resident run failed
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    if (dt_dev) dt = *dt_dev;  // interval from device memory (graph-captured steps)
    double u[NS + 3];
    load_cell<NS>(U, cs, cell_index ? cell_index[i] : i, u);
    cell::Cell<NS> c;
    double Lu[cell::NQ * cell::NQ];
    c.attempts = 0;
    int r = cell::begin<NS>(c, u, dt_cell ? dt_cell[i] : dt, rtol, atol);
    while (r == CELL_CONTINUE) r = cell::attempt<NS, false>(c, rtol, atol, Lu);
    atomicAdd(&st->steps, (unsigned long long)c.attempts);
    if (r == CELL_DONE && cell::finish<NS>(c, u)) {
#pragma unroll
        for (int n = 0; n < NS + 3; ++n) trial[n * count + i] = u[n];
        fail[i] = 0;
    } else {
        report(st, fail, i, r == CELL_MAXSTEPS ? CELL_MAXSTEPS : CELL_FAIL);
    }
}

// Persistent form: each lane holds one cell and the warp advances all its lanes by
// one step attempt per iteration (the same instruction stream for every lane).
// A lane whose cell finishes writes it and takes the next cell index from the
// device work queue (one atomic per warp refill round).  The number of step
// attempts per lane varies freely; lanes stay busy until the queue is empty.
template <int NS>
__global__ void __launch_bounds__(64) k_chem_persistent(const double* __restrict__ U, int64_t cs,
                                                        const int64_t* __restrict__ cell_index, int64_t count,
                                                        double dt, const double* __restrict__ dt_cell, double rtol,
                                                        double atol, double* __restrict__ trial,
                                                        int* __restrict__ fail, DevStatus* st) {
    const unsigned lane = threadIdx.x & 31;
    cell::Cell<NS> c;
    double Lu[cell::NQ * cell::NQ];
    int64_t cell = -1;
    bool active = false, drained = false;
    unsigned long long my_attempts = 0;
    for (;;) {
        // refill lanes without a cell: one atomic per warp and round
        if (!drained) {
            const unsigned need = __ballot_sync(0xffffffffu, !active);
            bool none = false;
            if (need) {
                const int leader = __ffs(need) - 1;
                unsigned long long base = 0;
                if ((int)lane == leader) base = atomicAdd(&st->counter, (unsigned long long)__popc(need));
                base = __shfl_sync(0xffffffffu, base, leader);
                if (!active) {
                    const int64_t k = (int64_t)(base + __popc(need & ((1u << lane) - 1u)));
                    if (k < count) {
                        cell = k;
                        double u[NS + 3];
                        load_cell<NS>(U, cs, cell_index ? cell_index[k] : k, u);
                        const int r = cell::begin<NS>(c, u, dt_cell ? dt_cell[k] : dt, rtol, atol);
                        if (r == CELL_CONTINUE) active = true;
                        else report(st, fail, k, CELL_FAIL);
                    } else {
                        none = true;
                    }
                }
            }
            drained = __any_sync(0xffffffffu, none);
        }
        if (!__any_sync(0xffffffffu, active)) {
            if (drained) break;
            continue;
        }
        if (active) {
            const int r = cell::attempt<NS, false>(c, rtol, atol, Lu);
            if (r != CELL_CONTINUE) {
                my_attempts += c.attempts;
                double u[NS + 3];
                if (r == CELL_DONE && cell::finish<NS>(c, u)) {
#pragma unroll
                    for (int n = 0; n < NS + 3; ++n) trial[n * count + cell] = u[n];
                    fail[cell] = 0;
                } else {
                    report(st, fail, cell, r == CELL_MAXSTEPS ? CELL_MAXSTEPS : CELL_FAIL);
                }
                active = false;
            }
        }
    }
    if (my_attempts) atomicAdd(&st->steps, my_attempts);
}

template <int NS>
__global__ void k_chem_commit(double* __restrict__ U, int64_t cs, const int64_t* __restrict__ cell_index, int64_t count,
                              const double* __restrict__ trial) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const int64_t b = cell_index ? cell_index[i] : i;
#pragma unroll
    for (int n = 0; n < NS + 3; ++n) U[b + n * cs] = trial[n * count + i];
}

// Cells of a queue (positions [0, n) of order, or cells 0..n-1), one per group of 8 lanes
// (hf_group.cuh): the refill scheme of the per-lane loop with groups in place of lanes.
// Returns the step attempts of the caller's cells (on the first lane of each group).
template <int NS, bool SCREEN>
__device__ __forceinline__ unsigned long long group_phase(const double* __restrict__ U, int64_t cs,
                                                          const int64_t* __restrict__ cell_index,
                                                          const int32_t* __restrict__ order, int64_t n, int64_t count,
                                                          double dt, const double* __restrict__ dt_cell, double rtol,
                                                          double atol, double* __restrict__ trial,
                                                          int* __restrict__ fail, double* __restrict__ h_hist,
                                                          int32_t* __restrict__ cost, DevStatus* st,
                                                          grp8::Shared* sh) {
    const unsigned lane = threadIdx.x & 31;
    const int t = grp8::lane8();
    grp8::Cell<NS> c;
    c.active = false;
    int64_t cell = -1;
    bool drained = false, loaded = false;
    unsigned long long attempts = 0;
    for (;;) {
        if (!drained) {
            const unsigned need = __ballot_sync(0xffffffffu, !c.active) & 0x01010101u;  // first lane of each group
            bool none = false;
            if (need) {
                const int leader = __ffs(need) - 1;
                unsigned long long base = 0;
                if ((int)lane == leader) base = atomicAdd(&st->coop_counter, (unsigned long long)__popc(need));
                base = __shfl_sync(0xffffffffu, base, leader);
                if (!c.active) {
                    const int64_t q = (int64_t)(base + __popc(need & ((1u << (lane & 24)) - 1u)));
                    const bool got = q < n;
                    none = !got;
                    // a group that never held a cell computes along on the queue's first one
                    if (got || !loaded) {
                        const int64_t p = got ? q : 0, k = order ? (int64_t)order[p] : p;
                        double u[NS + 3];
                        load_cell<NS>(U, cs, cell_index ? cell_index[k] : k, u);
                        const bool ok = grp8::load<NS>(c, u, dt_cell ? dt_cell[k] : dt, h_hist ? h_hist[k] : 0.0);
                        loaded = true;
                        if (got) {
                            cell = k;
                            c.active = ok;
                            if (t == 0 && SCREEN) atomicAdd(&st->coop_cells, 1ull);
                            if (t == 0 && !ok) report(st, fail, k, CELL_FAIL);
                        }
                    }
                }
            }
            drained = __any_sync(0xffffffffu, none);
        }
        if (!__any_sync(0xffffffffu, c.active)) {
            if (drained) break;
            continue;
        }
        bool screened = false;
        const int r = grp8::attempt<NS, SCREEN>(c, rtol, atol, sh, screened);
        const bool done = c.active && r != CELL_CONTINUE;
        if (__any_sync(0xffffffffu, done)) {
            double u[NS + 3];
            const bool keep = grp8::finish<NS>(c, u);
            if (done) {
                if (t == 0) attempts += c.attempts;
                if (r == CELL_DONE && keep) {
#pragma unroll
                    for (int m = 0; m < NS + 3; ++m)
                        if ((m & 7) == t) trial[m * count + cell] = u[m];
                    if (t == 0) {
                        fail[cell] = 0;
                        if (h_hist && !screened) h_hist[cell] = c.h;
                        if (cost) cost[cell] = c.attempts;
                    }
                } else if (t == 0) {
                    report(st, fail, cell, r == CELL_MAXSTEPS ? CELL_MAXSTEPS : CELL_FAIL);
                }
                c.active = false;
            }
        }
    }
    return attempts;
}

// The plain and persistent forms of a small batch: every cell in a group.
template <int NS>
__global__ void __launch_bounds__(64) k_chem_group(const double* __restrict__ U, int64_t cs,
                                                   const int64_t* __restrict__ cell_index, int64_t count, double dt,
                                                   const double* __restrict__ dt_dev,
                                                   const double* __restrict__ dt_cell, double rtol, double atol,
                                                   double* __restrict__ trial, int* __restrict__ fail, DevStatus* st) {
    __shared__ grp8::Shared sh[8];
    if (st->abort_run) return;
    if (dt_dev) dt = *dt_dev;
    const unsigned long long a =
        group_phase<NS, false>(U, cs, cell_index, nullptr, count, count, dt, dt_cell, rtol, atol, trial, fail, nullptr,
                               nullptr, st, &sh[threadIdx.x >> 3]);
    if (a) atomicAdd(&st->steps, a);
}

// Measured on the batched form (warm history): 65,536 cells of very uneven stiffness 351 ms
// without groups, 133 with them (4,639 cells of 255 to 1,340 attempts); 512 x 128 cells with
// 19,400 burning ones 80 ms in order of arrival, 37 to 50 with one warp of them to a
// sub-partition; 1D detonation of 4,000 cells 149 ms (8 steps) on lanes, 40 with groups.
//
// Batched form: the persistent lane-refill loop of k_chem_persistent over a work
// queue ordered most-expensive-first (order[]), starting each cell with
// cell::begin_warm, and recording per cell the attempts taken (cost[]) and the
// controller's proposed next step (h_hist[]) for the next call.
template <int NS, int MINB, bool COOP>
__global__ void __launch_bounds__(64, MINB) k_chem_batched(const double* __restrict__ U, int64_t cs,
                                                     const int64_t* __restrict__ cell_index,
                                                     const int32_t* __restrict__ order, int64_t count, double dt,
                                                     const double* __restrict__ dt_dev,
                                                     const double* __restrict__ dt_cell, double rtol, double atol,
                                                     double* __restrict__ trial, int* __restrict__ fail,
                                                     double* __restrict__ h_hist, int32_t* __restrict__ cost,
                                                     const unsigned long long* __restrict__ coop_n, int64_t lanes_first,
                                                     DevStatus* st) {
    if (st->abort_run) return;  // an earlier step of this device-resident run failed
    const unsigned lane = threadIdx.x & 31;
    if (dt_dev) dt = *dt_dev;  // interval from device memory (graph-captured steps)
    unsigned slot;
    asm volatile("mov.u32 %0, %%warpid;" : "=r"(slot));
    unsigned long long my_attempts = 0;
    // Two queues: the costly cells after the cooperative ones, then the rest.  Warps in the
    // first slot of their SM sub-partition start with the costly ones and the others with the
    // rest, so that every sub-partition gets one warp of long step chains before any gets
    // two (a second one beside it slows both: 377 against 230 us an attempt); when there are
    // more costly cells than those warps have lanes, all warps start with them.
    int64_t ncoop = 0;
    if constexpr (COOP) ncoop = (order && coop_n) ? (int64_t)*coop_n : 0;
    const int64_t nhi = (order && coop_n) ? (int64_t)coop_n[1] : 0;
    bool costly = nhi > 0 && (slot < 4 || nhi > lanes_first);
    int dry = 0;  // queues found empty
    // COOP: the costliest cells one per group of 8 lanes.  Warps in the first slots take them
    // before anything else, the others after their lane cells, unless there are more than
    // those warps have groups.  Without COOP the kernel holds no shared memory (the L1 keeps
    // the lanes' stacks).
    const bool groups_first = slot < 4 || 8 * ncoop > lanes_first;
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
        if ((part == 0) == groups_first) {
            if constexpr (COOP) {
                __shared__ grp8::Shared sh[8];
                if (ncoop > 0)
                    my_attempts += group_phase<NS, true>(U, cs, cell_index, order, ncoop, count, dt, dt_cell, rtol, atol,
                                                         trial, fail, h_hist, cost, st, &sh[threadIdx.x >> 3]);
            }
            continue;
        }
        cell::Cell<NS> c;
        double Lu[cell::NQ * cell::NQ];
        int64_t cell = -1;
        bool active = false, drained = false;
        for (;;) {
            if (!drained) {
                const unsigned need = __ballot_sync(0xffffffffu, !active);
                bool none = false;
                if (need) {
                    const int leader = __ffs(need) - 1;
                    unsigned long long base = 0;
                    if ((int)lane == leader)
                        base = atomicAdd(costly ? &st->costly_counter : &st->counter, (unsigned long long)__popc(need));
                    base = __shfl_sync(0xffffffffu, base, leader);
                    if (!active) {
                        const int64_t q = ncoop + (costly ? 0 : nhi) + (int64_t)(base + __popc(need & ((1u << lane) - 1u)));
                        if (q < (costly ? ncoop + nhi : count)) {
                            const int64_t k = order ? (int64_t)order[q] : q;
                            cell = k;
                            double u[NS + 3];
                            load_cell<NS>(U, cs, cell_index ? cell_index[k] : k, u);
                            if (cell::begin_warm<NS>(c, u, dt_cell ? dt_cell[k] : dt, h_hist ? h_hist[k] : 0.0) ==
                                CELL_CONTINUE)
                                active = true;
                            else
                                report(st, fail, k, CELL_FAIL);
                        } else {
                            none = true;
                        }
                    }
                }
                if (__any_sync(0xffffffffu, none)) {  // this queue is empty: the other one next
                    costly = !costly;
                    drained = ++dry == 2 || (nhi == 0 && dry == 1);
                }
            }
            if (!__any_sync(0xffffffffu, active)) {
                if (drained) break;
                continue;
            }
            if (active) {
                bool screened = false;
                const int r = cell::attempt<NS, true>(c, rtol, atol, Lu, &screened);
                if (r != CELL_CONTINUE) {
                    my_attempts += c.attempts;
                    double u[NS + 3];
                    if (r == CELL_DONE && cell::finish<NS>(c, u)) {
#pragma unroll
                        for (int n = 0; n < NS + 3; ++n) trial[n * count + cell] = u[n];
                        fail[cell] = 0;
                        if (h_hist && !screened) h_hist[cell] = c.h;
                        if (cost) cost[cell] = c.attempts;
                    } else {
                        report(st, fail, cell, r == CELL_MAXSTEPS ? CELL_MAXSTEPS : CELL_FAIL);
                    }
                    active = false;
                }
            }
        }
    }
    if (my_attempts) atomicAdd(&st->steps, my_attempts);
}

// Launch settings of the batched form, process-wide (hf_set_chem_tuning; the first use
// reads HF_CHEM_MINB and HF_COOP_MIN_BUCKET / HF_COOP=0):
//  * blocks of 64 lanes per SM the queue kernel's register budget is built for: 4 (255
//    registers) or 5, 6, 8 (fewer registers, more resident lanes); the same per-cell code;
//  * the cooperative queue takes cells that used at least 2^coop_min - 1 attempts in the
//    previous call (coop_min = NBUCKET: no cooperative phase, and the kernel
//    instance without it).
//    COOP_AUTO, the default: k_order_scan decides.
constexpr int COOP_AUTO = 17;
std::atomic<int> g_tune_minb{0}, g_tune_coop{0};
void chem_tuning(int* minb, int* coop_min) {
    if (g_tune_minb.load() == 0) {
        const char* e = getenv("HF_CHEM_MINB");
        const int v = e ? atoi(e) : 4;
        int expect = 0;
        g_tune_minb.compare_exchange_strong(expect, (v == 5 || v == 6 || v == 8) ? v : 4);
    }
    if (g_tune_coop.load() == 0) {
        const char* off = getenv("HF_COOP");
        const char* e = getenv("HF_COOP_MIN_BUCKET");
        int v = e ? atoi(e) : COOP_AUTO;
        if (e) v = v < 1 ? 1 : (v > COOP_AUTO ? 16 : v);
        if (off && atoi(off) == 0) v = 16;
        int expect = 0;
        g_tune_coop.compare_exchange_strong(expect, v);
    }
    *minb = g_tune_minb.load();
    *coop_min = g_tune_coop.load();
}

// Work-queue order: counting sort of the cells by cost bin, most expensive bin first: SUB bins
// to a factor of two of cost + 1, 128 in all, so that the cells of a warp have about the same
// cost.  Cells of one bin keep no particular order; a cell's result does not depend on its place
// in the queue, only (to rounding) on whether its bin goes to groups.
constexpr int NBUCKET = 16, SUB = 8, NBIN = NBUCKET * SUB;
constexpr int COSTLY_BUCKET = 4;  // at least 15 attempts
static_assert(NBIN + 2 <= CHEM_BINS, "bins");
__device__ __forceinline__ int cost_bin(int32_t c) {
    const unsigned m = (unsigned)c + 1u;
    const int b = 31 - __clz(m);
    return min(b * SUB + (int)(((unsigned long long)m * SUB >> b) - SUB), NBIN - 1);
}
__global__ void k_order_hist(const int32_t* __restrict__ cost, int64_t count, unsigned long long* __restrict__ bins) {
    __shared__ unsigned int sb[NBIN];
    if (threadIdx.x < NBIN) sb[threadIdx.x] = 0;
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&sb[cost_bin(max(cost[i], 0))], 1u);
    __syncthreads();
    if (threadIdx.x < NBIN && sb[threadIdx.x]) atomicAdd(&bins[threadIdx.x], (unsigned long long)sb[threadIdx.x]);
}
// bins[b] -> start offset of bin b, descending bins first; bins[NBIN] = the cells of the
// cooperative queue: whole bins from the costliest down to bucket min_bucket while they fit
// in cap cells (whole bins, so the choice does not depend on the order within one);
// bins[NBIN + 1] = the cells after them in buckets from COSTLY_BUCKET up.
// min_bucket < 0: the line with the least estimated time, the root of the sum of squares
// (they run side by side, but slow each other) of
//   the FP64 pipe's:  attempts of the groups / 33.8 + attempts of the lanes / 103 per us,
//   the longest chain in a group:  73 us an attempt alone, 113 beside a second warp,
//   the longest chain on a lane:   230 us an attempt with one warp of costly cells to a
//                                  sub-partition and no groups, 377 beside another warp
// (measured, 10 species, cells of 398 attempts, 152 SMs).  A group's chain is three times
// as fast and costs the pipe three times as much: it pays for cells far above the mean.
constexpr float GROUP_RATE = 33.8f, LANE_RATE = 103.0f, GROUP_ALONE = 73.0f, GROUP_PAIR = 113.0f, LANE_ALONE = 230.0f,
                LANE_PAIR = 377.0f;
__device__ __forceinline__ float bin_cost(int b) {  // attempts at the bin's lower edge
    return (float)(1u << (b / SUB)) * (1.0f + (float)(b % SUB) / SUB) - 1.0f;
}
// One block of NBIN threads: the bins and their costs in shared memory, suffix sums by
// doubling, the line by one thread per candidate bin (45 us in one thread over global memory).
__global__ void __launch_bounds__(NBIN) k_order_scan(unsigned long long* bins, unsigned long long cap, int min_bucket,
                                                     int subparts) {
    __shared__ unsigned long long cum[NBIN];  // cells of bins >= b
    __shared__ float work[NBIN];              // their attempts
    __shared__ float best_t[NBIN];
    __shared__ int top, line;
    const int b = threadIdx.x;
    const unsigned long long n = bins[b];
    cum[b] = n;
    work[b] = (float)n * bin_cost(b);
    if (b == 0) {
        top = 0;
        line = NBIN;
    }
    __syncthreads();
    if (n) atomicMax(&top, b + 1);
    for (int o = 1; o < NBIN; o <<= 1) {
        const unsigned long long c = b + o < NBIN ? cum[b + o] : 0;
        const float w = b + o < NBIN ? work[b + o] : 0.0f;
        __syncthreads();
        cum[b] += c;
        work[b] += w;
        __syncthreads();
    }
    int min_bin = min_bucket * SUB;
    if (min_bucket < 0) {
        const float r = 608.0f / (float)subparts, total = work[0], most = bin_cost(top);
        const float p0 = total / LANE_RATE * r;
        const float l0 = most * (cum[COSTLY_BUCKET * SUB] <= 32ull * subparts ? LANE_ALONE : LANE_PAIR);
        const float p = (work[b] / GROUP_RATE + (total - work[b]) / LANE_RATE) * r;
        const float g = most * (cum[b] <= 4ull * subparts ? GROUP_ALONE : GROUP_PAIR), l = bin_cost(b) * LANE_PAIR;
        const float t = p * p + g * g + l * l;
        best_t[b] = b >= SUB && n && cum[b] <= cap && t < p0 * p0 + l0 * l0 ? t : 3e38f;
        __syncthreads();
        for (int o = NBIN / 2; o > 0; o >>= 1) {
            if (b < o) best_t[b] = fminf(best_t[b], best_t[b + o]);
            __syncthreads();
        }
        if (best_t[0] < 3e38f && b >= SUB && n && cum[b] <= cap && t == best_t[0]) atomicMin(&line, b);
        __syncthreads();
        min_bin = line;
    }
    // whole bins from the top down to min_bin while they fit
    const bool coop = b >= min_bin && cum[b] <= cap;
    __syncthreads();
    const unsigned long long above = b + 1 < NBIN ? cum[b + 1] : 0;
    bins[b] = above;
    __shared__ unsigned long long ncoop;
    if (b == 0) ncoop = 0;
    __syncthreads();
    if (coop) atomicMax(&ncoop, cum[b]);
    __syncthreads();
    if (b == 0) {
        bins[NBIN] = ncoop;
        const unsigned long long hi = cum[COSTLY_BUCKET * SUB];
        bins[NBIN + 1] = hi > ncoop ? hi - ncoop : 0;
    }
}
// Bound by atomics on one address: most cells of a developed flow share a bin.  One atomic
// per warp and bin, the warp's cells of a bin in order: 25 us for 2048 x 512 cells, 653 with
// one per cell.
__global__ void k_order_scatter(const int32_t* __restrict__ cost, int64_t count, unsigned long long* __restrict__ bins,
                                int32_t* __restrict__ order) {
    const unsigned lane = threadIdx.x & 31;
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x; b < count; b += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = b + threadIdx.x;
        const int bin = i < count ? cost_bin(max(cost[i], 0)) : NBIN;
        const unsigned same = __match_any_sync(0xffffffffu, bin);
        const int leader = __ffs(same) - 1;
        unsigned long long pos = 0;
        if ((int)lane == leader && i < count) pos = atomicAdd(&bins[bin], (unsigned long long)__popc(same));
        pos = __shfl_sync(0xffffffffu, pos, leader);
        if (i < count) order[pos + __popc(same & ((1u << lane) - 1u))] = (int32_t)i;
    }
}

template <int NS>
static cudaError_t chem_batched_impl(double* U, int64_t cs, const int64_t* idx, int64_t count, double dt,
                                     const double* dt_dev, const double* dtc, double rtol, double atol,
                                     double* h_hist, int32_t* cost, int32_t* order, unsigned long long* bins,
                                     double* trial, int* fail, DevStatus* st, int sm_count, cudaStream_t s,
                                     int64_t* launches) {
    int minb, coop_min;
    chem_tuning(&minb, &coop_min);
    const bool coop = coop_min != NBUCKET;
    auto kern = coop ? (minb == 8   ? k_chem_batched<NS, 8, true>
                        : minb == 6 ? k_chem_batched<NS, 6, true>
                        : minb == 5 ? k_chem_batched<NS, 5, true>
                                    : k_chem_batched<NS, 4, true>)
                     : (minb == 8   ? k_chem_batched<NS, 8, false>
                        : minb == 6 ? k_chem_batched<NS, 6, false>
                        : minb == 5 ? k_chem_batched<NS, 5, false>
                                    : k_chem_batched<NS, 4, false>);
    const int bs = 64;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, bs, 0);
    if (per_sm < 1) per_sm = 1;
    const int64_t most = (int64_t)sm_count * per_sm;
    int64_t blocks = std::min(most, std::max<int64_t>(1, (count + bs - 1) / bs));
    // cells the cooperative queue may take: one per group of 8 lanes of the launch; under the
    // automatic rule the launch has a group for every cell of a small batch
    unsigned long long cap = (unsigned long long)blocks * (bs / 8);
    if (coop_min == COOP_AUTO) {
        blocks = std::min(most, std::max<int64_t>(1, (count + bs / 8 - 1) / (bs / 8)));
        cap = (unsigned long long)blocks * (bs / 8);
    }
    const unsigned long long* coop_n = nullptr;
    if (cost && order) {
        cudaError_t e = cudaMemsetAsync(bins, 0, sizeof(unsigned long long) * (NBIN + 2), s);
        if (e != cudaSuccess) return e;
        const int g = sm_count * 4;
        k_order_hist<<<g, 256, 0, s>>>(cost, count, bins);
        k_order_scan<<<1, NBIN, 0, s>>>(bins, cap, coop_min == COOP_AUTO ? -1 : coop_min, 4 * sm_count);
        k_order_scatter<<<g, 256, 0, s>>>(cost, count, bins, order);
        *launches += 3;
        coop_n = bins + NBIN;
    } else {
        order = nullptr;
    }
    kern<<<(unsigned)blocks, bs, 0, s>>>(U, cs, idx, order, count, dt, dt_dev, dtc, rtol, atol, trial, fail, h_hist,
                                         cost, coop_n, 128 * (int64_t)sm_count, st);
    ++*launches;
    return cudaGetLastError();
}
// The batched kernel instances without the cooperative phase use no shared memory: the
// unified L1 / shared storage goes to L1, which caches the lanes' stack frames.
cudaError_t chem_prefer_l1() {
    const void* kernels[] = {(const void*)k_chem_batched<9, 4, false>,  (const void*)k_chem_batched<9, 5, false>,
                             (const void*)k_chem_batched<9, 6, false>,  (const void*)k_chem_batched<9, 8, false>,
                             (const void*)k_chem_batched<10, 4, false>, (const void*)k_chem_batched<10, 5, false>,
                             (const void*)k_chem_batched<10, 6, false>, (const void*)k_chem_batched<10, 8, false>};
    for (const void* k : kernels) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                                   (int)cudaSharedmemCarveoutMaxL1);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
cudaError_t launch_chem_batched(int ns, double* U, int64_t cs, const int64_t* idx, int64_t count, double dt,
                                const double* dt_dev, const double* dtc, double rtol, double atol, double* h_hist,
                                int32_t* cost, int32_t* order, unsigned long long* bins, double* trial, int* fail,
                                DevStatus* st, int sm_count, cudaStream_t s, int64_t* launches) {
    return ns == 9 ? chem_batched_impl<9>(U, cs, idx, count, dt, dt_dev, dtc, rtol, atol, h_hist, cost, order, bins,
                                          trial, fail, st, sm_count, s, launches)
                   : chem_batched_impl<10>(U, cs, idx, count, dt, dt_dev, dtc, rtol, atol, h_hist, cost, order, bins,
                                           trial, fail, st, sm_count, s, launches);
}

// Batches of the plain and persistent forms up to this many cells per SM go to
// k_chem_group: at 64 (9,728 cells) a group for each cell costs the FP64 pipe what the lanes'
// step chains take (29,000 pipe cycles of a sub-partition an attempt against 450,000 for 32
// lanes).  3,000 igniting cells: 5.8 ms in groups, 16.6 on lanes.
constexpr int GROUP_CELLS_PER_SM = 64;
template <int NS>
static cudaError_t chem_impl(int form, double* U, int64_t cs, const int64_t* idx, int64_t count, double dt,
                             const double* dtc, double rtol, double atol, double* trial, int* fail, DevStatus* st,
                             int sm_count, cudaStream_t s, int64_t* launches, const double* dt_dev) {
    const int bs = 64;
    if (form == CHEM_GROUPS || count <= (int64_t)sm_count * GROUP_CELLS_PER_SM) {
        // every cell in a group of 8 lanes; both forms, so that they stay bit-identical
        const int64_t blocks = std::min<int64_t>((count + 7) / 8, (int64_t)sm_count * 4);
        k_chem_group<NS><<<(unsigned)blocks, bs, 0, s>>>(U, cs, idx, count, dt, dt_dev, dtc, rtol, atol, trial, fail, st);
    } else if (form == HF_CHEM_PLAIN) {
        k_chem_plain<NS><<<(unsigned)((count + bs - 1) / bs), bs, 0, s>>>(U, cs, idx, count, dt, dt_dev, dtc, rtol, atol,
                                                                          trial, fail, st);
    } else {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_chem_persistent<NS>, bs, 0);
        if (per_sm < 1) per_sm = 1;
        int64_t blocks = (int64_t)sm_count * per_sm;
        const int64_t need = (count + bs - 1) / bs;
        if (blocks > need) blocks = need;
        if (blocks < 1) blocks = 1;
        k_chem_persistent<NS><<<(unsigned)blocks, bs, 0, s>>>(U, cs, idx, count, dt, dtc, rtol, atol, trial, fail, st);
    }
    ++*launches;
    return cudaGetLastError();
}
cudaError_t launch_chem(int ns, int form, double* U, int64_t cs, const int64_t* idx, int64_t count, double dt,
                        const double* dtc, double rtol, double atol, double* trial, int* fail, DevStatus* st,
                        int sm_count, cudaStream_t s, int64_t* launches, const double* dt_dev) {
    return ns == 9 ? chem_impl<9>(form, U, cs, idx, count, dt, dtc, rtol, atol, trial, fail, st, sm_count, s, launches,
                                  dt_dev)
                   : chem_impl<10>(form, U, cs, idx, count, dt, dtc, rtol, atol, trial, fail, st, sm_count, s, launches,
                                   dt_dev);
}
cudaError_t launch_chem_commit(int ns, double* U, int64_t cs, const int64_t* idx, int64_t count, const double* trial,
                               cudaStream_t s, int64_t* launches) {
    const int bs = 128;
    if (ns == 9) k_chem_commit<9><<<(unsigned)((count + bs - 1) / bs), bs, 0, s>>>(U, cs, idx, count, trial);
    else k_chem_commit<10><<<(unsigned)((count + bs - 1) / bs), bs, 0, s>>>(U, cs, idx, count, trial);
    ++*launches;
    return cudaGetLastError();
}

// ---------------------------------------------------------------- tagging
// BlockAMR::ErrorEst (BlockAMR.cpp:170-200) per valid cell: tag box (optionally moving),
// relative pressure and temperature jumps to the face neighbours, fuel consumption
// rate -w_H2 W_H2 / rho, plus the relative density jump (extension, density_tag > 0).
template <int NS>
__global__ void k_tag(Level L, const hf_patch* __restrict__ patches, const double* __restrict__ U, double t,
                      hf_tag_criteria c, uint8_t* __restrict__ tags, const int64_t* __restrict__ tag_off,
                      DevStatus* st) {
    constexpr int NV = NS + 3;
    const hf_patch P = patches[blockIdx.y];
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= (int64_t)P.nx * P.ny) return;
    const int li = (int)(k % P.nx), lj = (int)(k / P.nx);
    const int i = P.ilo + li, j = P.jlo + lj;
    const double x = L.xlo + (i + 0.5) * L.dx - c.velocity[0] * t;
    const double y = L.ylo + (j + 0.5) * L.dy - c.velocity[1] * t;
    bool marked = c.has_box && x >= c.box[0] && x <= c.box[1] && y >= c.box[2] && y <= c.box[3];
    if (!c.box_only) {
        auto load = [&](int a, int b, double* q) {
#pragma unroll
            for (int n = 0; n < NV; ++n)
                q[n] = U[P.offset + (int64_t)n * P.comp_stride + (int64_t)(b + P.ng) * P.pitch + (a + P.ng)];
        };
        double q[NV];
        load(li, lj, q);
        Props p;
        bool ok = properties<NS>(q, p, 1000.0);
        double rho = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s) rho += q[s];
        for (int d = 0; d < 2 && ok; ++d) {
            const int di = d == 0, dj = d == 1;
            double ql[NV], qr[NV];
            load(li - di, lj - dj, ql);
            load(li + di, lj + dj, qr);
            Props pl, pr;
            ok = properties<NS>(ql, pl, p.T) && properties<NS>(qr, pr, p.T);
            if (!ok) break;
            const double jump = fmax(fabs(pl.p - p.p) / fmin(pl.p, p.p), fabs(pr.p - p.p) / fmin(pr.p, p.p));
            const double temp = fmax(fabs(pl.T - p.T) / fmin(pl.T, p.T), fabs(pr.T - p.T) / fmin(pr.T, p.T));
            marked = marked || jump > c.pressure_tag || temp > c.temperature_tag;
            if (c.density_tag > 0.0) {
                double rl = 0.0, rr = 0.0;
#pragma unroll
                for (int s = 0; s < NS; ++s) { rl += ql[s]; rr += qr[s]; }
                const double rj = fmax(fabs(rl - rho) / fmin(rl, rho), fabs(rr - rho) / fmin(rr, rho));
                marked = marked || rj > c.density_tag;
            }
        }
        if (!ok) {
            atomicOr(&st->flags, ST_STAGE_BAD);
            atomicMin(&st->bad_cell, (unsigned long long)(tag_off[blockIdx.y] + k));
        } else if (c.chemistry) {
            double C[NS], w[NS];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                C[s] = q[s] * INVW.v[s];
                w[s] = 0.0;
            }
            KinCtx<NS> kc;
            kin_setup<NS>(p.T, C, kc);
            all_rates<NS>(kc, C, w, std::make_index_sequence<NR>{});
            marked = marked || -w[0] * D_MW.v[0] / rho > c.fuel_rate_tag;
        }
    }
    tags[tag_off[blockIdx.y] + k] = marked ? 1 : 0;
}
cudaError_t launch_tag(int ns, const Level& L, const hf_patch* patches_dev, const hf_patch* patches_host, int npatch,
                       const double* U, double time, const hf_tag_criteria& c, uint8_t* tags, const int64_t* tag_off,
                       DevStatus* st, cudaStream_t s, int64_t* launches) {
    int64_t mx = 1;
    for (int p = 0; p < npatch; ++p) mx = max(mx, (int64_t)patches_host[p].nx * patches_host[p].ny);
    dim3 grid((unsigned)((mx + 127) / 128), (unsigned)npatch);
    if (ns == 9) k_tag<9><<<grid, 128, 0, s>>>(L, patches_dev, U, time, c, tags, tag_off, st);
    else k_tag<10><<<grid, 128, 0, s>>>(L, patches_dev, U, time, c, tags, tag_off, st);
    ++*launches;
    return cudaGetLastError();
}

// ---------------------------------------------------------------- allocation-free entry
// Scratch of hf_chem_advance_noalloc: a file-scope device array of fixed size, so the
// entry point allocates nothing.  Host code reaches it only through the device address
// that cudaGetSymbolAddress returns (the symbol itself is a host-side stand-in).
struct NoAllocScratch {
    DevStatus st;
    int fail[HF_NOALLOC_MAX_CELLS];
    double trial[(NS_MAX + 3) * HF_NOALLOC_MAX_CELLS];
};
static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

}  // namespace hf

namespace hf {
__global__ void k_fastmath(const double* __restrict__ x, int64_t n, double* __restrict__ e, double* __restrict__ ep,
                           double* __restrict__ em, double* __restrict__ l) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    e[i] = fexp(v);
    fexp_pair(v, ep[i], em[i]);
    l[i] = flog(v);
}
__global__ void k_cellmath(const double* __restrict__ x, int64_t n, double* __restrict__ e, double* __restrict__ ep,
                           double* __restrict__ em, double* __restrict__ l) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    e[i] = cell::fexp(v);
    cell::fexp_pair(v, ep[i], em[i]);
    l[i] = cell::flog(v);
}
}  // namespace hf
extern "C" hf_status hf_cellmath_eval(const double* x, int64_t n, double* exp_out, double* pair_pos, double* pair_neg,
                                      double* log_out, void* stream) {
    if (n < 0 || !x || !exp_out || !pair_pos || !pair_neg || !log_out) return HF_ERR_ARG;
    if (n == 0) return HF_OK;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    hf::k_cellmath<<<blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(x, n, exp_out, pair_pos, pair_neg,
                                                                              log_out);
    return cudaGetLastError() == cudaSuccess ? HF_OK : HF_ERR_CUDA;
}
extern "C" hf_status hf_fastmath_eval(const double* x, int64_t n, double* exp_out, double* pair_pos, double* pair_neg,
                                      double* log_out, void* stream) {
    if (n < 0 || !x || !exp_out || !pair_pos || !pair_neg || !log_out) return HF_ERR_ARG;
    if (n == 0) return HF_OK;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    hf::k_fastmath<<<blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(x, n, exp_out, pair_pos, pair_neg,
                                                                              log_out);
    return cudaGetLastError() == cudaSuccess ? HF_OK : HF_ERR_CUDA;
}
extern "C" hf_status hf_set_chem_tuning(int32_t blocks_per_sm, int32_t coop_min_bucket) {
    if (blocks_per_sm < 0 || coop_min_bucket < 0 || coop_min_bucket > hf::COOP_AUTO ||
        (blocks_per_sm && blocks_per_sm != 4 && blocks_per_sm != 5 && blocks_per_sm != 6 && blocks_per_sm != 8))
        return HF_ERR_ARG;
    int m = 0, c = 0;
    hf::chem_tuning(&m, &c);  // settle the defaults first
    if (blocks_per_sm) hf::g_tune_minb.store(blocks_per_sm);
    if (coop_min_bucket) hf::g_tune_coop.store(coop_min_bucket);
    return HF_OK;
}
extern "C" void hf_get_chem_tuning(int32_t* blocks_per_sm, int32_t* coop_min_bucket) {
    int m = 0, c = 0;
    hf::chem_tuning(&m, &c);
    if (blocks_per_sm) *blocks_per_sm = m;
    if (coop_min_bucket) *coop_min_bucket = c;
}

#include <mutex>

namespace {
constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mutex;
hf::NoAllocScratch* g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {};

// Once per device, with that device current: the array's device address, and the
// rate constants if no context has loaded them on this device yet.
cudaError_t noalloc_setup(int dev, hf::NoAllocScratch** out) {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        hf::NoAllocScratch* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress((void**)&p, hf::g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        double a0 = 0.0;
        e = cudaMemcpyFromSymbol(&a0, hf::c_A, sizeof(double));
        if (e != cudaSuccess) return e;
        if (a0 == 0.0) {
            e = hf::chem_set_rate_scale(nullptr);
            if (e != cudaSuccess) return e;
        }
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return cudaSuccess;
}
}  // namespace

extern "C" hf_status hf_chem_advance_noalloc(int nspecies, double* U, int64_t comp_stride, const int64_t* cell_index,
                                             int64_t count, double dt, const double* dt_cell, double rtol, double atol,
                                             int64_t* first_failed, void* stream) {
    using namespace hf;
    if (first_failed) *first_failed = -1;
    if ((nspecies != 9 && nspecies != 10) || !U || count < 0 || count > HF_NOALLOC_MAX_CELLS ||
        (!cell_index && comp_stride < count) || (!dt_cell && (!(dt > 0) || !isfinite(dt))) || !(rtol > 0) ||
        !(atol > 0))
        return HF_ERR_ARG;
    if (count == 0) return HF_OK;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return HF_ERR_CUDA;
    NoAllocScratch* S = nullptr;
    if (noalloc_setup(dev, &S) != cudaSuccess) return HF_ERR_CUDA;
    const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(&S->st, 0, sizeof(DevStatus), s) != cudaSuccess ||
        cudaMemsetAsync(&S->st.bad_cell, 0xff, sizeof(unsigned long long), s) != cudaSuccess)
        return HF_ERR_CUDA;
    int64_t launches = 0;
    int sms = 1;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        launch_chem(nspecies, HF_CHEM_PLAIN, U, comp_stride, cell_index, count, dt, dt_cell, rtol, atol, S->trial,
                    S->fail, &S->st, sms, s, &launches) != cudaSuccess)
        return HF_ERR_CUDA;
    DevStatus h;
    if (cudaMemcpyAsync(&h, &S->st, sizeof h, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return HF_ERR_CUDA;
    if (h.flags & (ST_CHEM_FAIL | ST_MAXSTEPS)) {
        if (first_failed) *first_failed = (int64_t)h.bad_cell;
        return (h.flags & ST_CHEM_FAIL) ? HF_ERR_CHEM_FAIL : HF_ERR_MAXSTEPS;
    }
    if (launch_chem_commit(nspecies, U, comp_stride, cell_index, count, S->trial, s, &launches) != cudaSuccess)
        return HF_ERR_CUDA;
    return HF_OK;
}
