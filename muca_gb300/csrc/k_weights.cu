// k_weights.cu -- histogram statistics and weight updates on the device, FP64.
//
// Replaces the host code that runs after every sweep of the reference weight
// program (muca_delta_multigpu.cu:422-476): hist_range (:573-596), the
// Kullback-Leibler divergence against a uniform distribution over visited
// bins (:598-618), the trivial update lnW -= ln H for H > 1 followed by
// lnW -= lnW[0] (:466-476), and weight_recursion (:833-859).  One cluster,
// a few launches or one block serve one histogram of N+1 <= 16385 bins (see
// launch_weight_update and the batch's update).  Element-wise steps use the
// reference's operation order with explicitly rounded FP64 operations, so
// the updated weights equal the host's up to the last-bit differences of the
// device and host log(); the divergence is a tree sum and agrees to ~1e-15.
#include "muca_device.cuh"
#include "muca_internal.h"

#include <algorithm>

#include <cfloat>

namespace muca {

constexpr int kUpdThreads = 1024;

// Reduction over a block of whole warps; lanes beyond the number of warps
// enter the second stage with the operation's identity.
template <typename T, typename Op>
__device__ T block_reduce(T v, Op op, T *sh)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    if (wid == 0) {
        v = lane < nw ? sh[lane] : Op::id();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) sh[0] = v;
    }
    __syncthreads();
    const T r = sh[0];
    __syncthreads();
    return r;
}

// The integer statistics of a histogram: first and last bin with more than one
// entry, visited bins, entries, smallest count.
struct HistSum {
    int lo, hi;
    unsigned long long vis, ev, mn;
    __device__ __forceinline__ void add(int i, unsigned long long h)
    {
        if (h > 1) {
            lo = min(lo, i);
            hi = max(hi, i);
        }
        if (h > 0) {
            ++vis;
            ev += h;
        }
        mn = h < mn ? h : mn;
    }
    __device__ __forceinline__ void join(const HistSum &o)
    {
        lo = min(lo, o.lo);
        hi = max(hi, o.hi);
        vis += o.vis;
        ev += o.ev;
        mn = o.mn < mn ? o.mn : mn;
    }
    __device__ __forceinline__ void warp_join()
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            HistSum x;
            x.lo = __shfl_xor_sync(0xffffffffu, lo, o);
            x.hi = __shfl_xor_sync(0xffffffffu, hi, o);
            x.vis = __shfl_xor_sync(0xffffffffu, vis, o);
            x.ev = __shfl_xor_sync(0xffffffffu, ev, o);
            x.mn = __shfl_xor_sync(0xffffffffu, mn, o);
            join(x);
        }
    }
};
// over the block, to every thread
__device__ HistSum block_join(HistSum v, HistSum *sh, uint32_t N)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v.warp_join();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    v = lane < nw ? sh[lane] : HistSum{(int)N + 1, -1, 0ull, 0ull, ~0ull};
    v.warp_join();
    return v;
}

struct AddD {
    __device__ double operator()(double a, double b) const { return a + b; }
    __device__ static double id() { return 0.0; }
};

// The prefix of weight_recursion (muca_delta_multigpu.cu:848-858) over the
// pairs i in [start, end):  x_start = lnW[start],
//   x_{i+1} = x_i + dS_i  if pair i is connected (valid[i]),  else lnW[i+1]
// (a pair with an empty bin leaves lnW[i+1] as it was).  The reference runs
// it as one dependent chain of FP64 additions; here the block of (whole
// warps of) threads splits [start, end) into contiguous chunks, each thread
// composes its chunk's maps x -> x + d / x -> c into one, the block scans
// those compositions (warp shuffles, then the warp totals), and every thread
// replays its chunk from its prefix.  Inside a chunk the additions keep the
// reference's order; across chunks they are grouped by the tree, which moves
// the result by a few units in the last place of the partial sums.
// `inc` holds dS_i and `cval` lnW[i+1] of the pairs; out[i] gets x_{i+1}.
// Must be called by every thread of the block.
struct SegMap {
    double t;  // valid: the added sum; not valid: the constant
    int v;     // 1: x -> x + t, 0: x -> t
};
__device__ __forceinline__ SegMap seg_then(SegMap first, SegMap then)
{
    SegMap r;
    r.v = first.v & then.v;
    r.t = then.v ? __dadd_rn(first.t, then.t) : then.t;
    return r;
}

__device__ void block_segmented_prefix(int start, int end, double x0, const double *__restrict__ inc,
                                       const unsigned char *__restrict__ valid,
                                       const double *__restrict__ cval, double *__restrict__ out)
{
    __shared__ double s_t[32];
    __shared__ int s_v[32];
    const int n = end - start;
    if (n <= 0) return;
    const int nt = (int)blockDim.x, tid = (int)threadIdx.x;
    const int chunk = (n + nt - 1) / nt;
    const int lo = start + tid * chunk, hi = min(lo + chunk, end);
    SegMap a{0.0, 1};
    for (int i = lo; i < hi; ++i) {
        const SegMap e{valid[i] ? inc[i] : cval[i], valid[i] ? 1 : 0};
        a = seg_then(a, e);
    }
    // inclusive scan of the thread maps within the warp
    const int lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
    SegMap sc = a;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        SegMap pr;
        pr.t = __shfl_up_sync(0xffffffffu, sc.t, o);
        pr.v = __shfl_up_sync(0xffffffffu, sc.v, o);
        if (lane >= o) sc = seg_then(pr, sc);
    }
    if (lane == 31) { s_t[wid] = sc.t; s_v[wid] = sc.v; }
    __syncthreads();
    if (wid == 0) {
        SegMap w{lane < nw ? s_t[lane] : 0.0, lane < nw ? s_v[lane] : 1};
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            SegMap pr;
            pr.t = __shfl_up_sync(0xffffffffu, w.t, o);
            pr.v = __shfl_up_sync(0xffffffffu, w.v, o);
            if (lane >= o) w = seg_then(pr, w);
        }
        s_t[lane] = w.t;
        s_v[lane] = w.v;
    }
    __syncthreads();
    // exclusive prefix of this thread: the warps before it, then the lanes before it
    SegMap ex{0.0, 1};
    if (wid > 0) ex = SegMap{s_t[wid - 1], s_v[wid - 1]};
    SegMap lp;
    lp.t = __shfl_up_sync(0xffffffffu, sc.t, 1);
    lp.v = __shfl_up_sync(0xffffffffu, sc.v, 1);
    if (lane > 0) ex = seg_then(ex, lp);
    double x = ex.v ? __dadd_rn(x0, ex.t) : ex.t;
    for (int i = lo; i < hi; ++i) {
        x = valid[i] ? __dadd_rn(x, inc[i]) : cval[i];
        out[i] = x;
    }
    __syncthreads();
}

// Statistics of hist[0..N], then (if the update is due) the weight update.
// ctl == nullptr: standalone call, update iff rule >= 0.
// ctl != nullptr: one iteration of a device-driven run (see RunCtl).
// NUPDATES of the next iteration.  sched 0: the reference's (NUP+1)*1.01
// once the width is full (muca_delta_multigpu.cu:379-382); 1: doubling once
// the width is full; 2: doubling every iteration; 3: the reference's growth
// once the width is full and doubling once, in addition, every bin of this
// iteration's histogram holds at least 5 % of the mean count (`covered`);
// 4: NUP * 1.05 every iteration, truncated (the CPU program,
// muca_mag.cpp:131); 5: NUP held until the width is full (as the reference
// GPU program holds it, :379-382), then NUP * 1.05 per iteration (the CPU
// program's growth).  The result is capped at `cap` (0: no cap for sched 0,
// 2^30 otherwise) but never falls below nup.
__host__ __device__ __forceinline__ uint32_t next_nupdates(uint32_t nup, bool full, bool covered, uint32_t sched,
                                                           uint32_t cap)
{
    unsigned long long nx = nup;
    if (sched == 2 || (sched == 1 && full) || (sched == 3 && full && covered)) {
        nx = 2ull * nup;
        if (cap == 0) cap = 1u << 30;
    } else if ((sched == 0 || sched == 3) && full) {
        const unsigned nu = nup + 1u;
        nx = (unsigned)(nu * 1.01);
    } else if (sched == 4 || (sched == 5 && full)) {
        nx = (unsigned long long)((double)nup * 1.05);
        if (cap == 0) cap = 1u << 30;
    }
    if (cap != 0 && nx > cap) nx = cap > nup ? cap : nup;
    return (uint32_t)nx;
}

// Whether an update clears the histogram for the run's next iteration.
__device__ __forceinline__ bool clears_hist(const RunCtl *ctl) { return ctl && !ctl->st.stop && !ctl->keep_hist; }

// The statistics' consumers, one thread: the stats record, and in a
// device-driven run the running width, convergence, record and NUPDATES of
// the next iteration (muca_delta_multigpu.cu:431-447,464-466).  Returns
// whether the weights are to be updated.
__device__ __forceinline__ int bookkeep(int start, int end, unsigned long long vis, unsigned long long ev,
                                        unsigned long long mn, double kl, uint32_t N, int rule,
                                        HistStatsDev *__restrict__ stats, RunCtl *__restrict__ ctl)
{
    const double mean = __ddiv_rn((double)ev, (double)(N + 1));
    const double mom = mean > 0 ? __ddiv_rn((double)mn, mean) : 0.0;
    if (stats) {
        stats->start = start;
        stats->end = end;
        stats->width = (uint32_t)(end - start);
        stats->visited = (uint32_t)vis;
        stats->events = ev;
        stats->min_count = mn;
        stats->d_kl = kl;
        stats->min_over_mean = mom;
    }
    int upd = rule >= 0;
    if (ctl) {
        IterState &st = ctl->st;
        const uint32_t wt = (uint32_t)(end - start);
        st.width_temp = wt;
        if (wt > st.width) st.width = wt;
        if (st.width == N && !st.reach) { st.reach = 1; st.reach_k = st.k; st.nwidth_step = st.total_run; }
        const bool conv = ctl->flat_minmean ? (mom >= ctl->mom_thr) : (st.width == N && kl < ctl->dkl_max);
        const uint32_t ri = ctl->rec_ring ? (ctl->rec_cap ? st.k % ctl->rec_cap : 0u) : st.k;
        if (ri < ctl->rec_cap && ctl->recs) {
            IterRecordDev &r = ctl->recs[ri];
            r.k = st.k; r.width_temp = wt; r.width = st.width; r.nupdates = st.nup;
            r.total_run = st.total_run; r.d_kl = kl; r.min_over_mean = mom;
        }
        upd = !conv && (!ctl->hold || st.width == N);
        if (conv) {
            st.converged = 1;
            st.stop = 1;
        } else {
            st.k += 1;
            if (st.k >= ctl->max_iter) {
                st.stop = 1;
            } else {
                st.nup = next_nupdates(st.nup, st.width == N, mom >= 0.05, ctl->sched, ctl->nup_max);
                st.total_run += (unsigned long long)st.nup * ctl->nchains_total;
            }
        }
    }
    return upd;
}

// Pair i of weight_recursion (muca_delta_multigpu.cu:850-856): for i in
// [start, end) with H_i, H_{i+1} both nonzero,
//   p = H_i H_{i+1} / (H_i + H_{i+1}),  k = p / (p + p_acc[i]),
//   dS_i = (lnW[i+1] - lnW[i]) + k ln(H_i / H_{i+1}),  p_acc[i] += p;
// returns whether the pair is connected (ds[i] written).
__device__ __forceinline__ unsigned char recursion_increment(const unsigned long long *__restrict__ hist,
                                                             const double *__restrict__ lnw,
                                                             double *__restrict__ p_acc, uint32_t i, int start,
                                                             int end, double *__restrict__ ds)
{
    if ((int)i < start || (int)i >= end) return 0;
    const unsigned long long a = hist[i], b = hist[i + 1];
    if ((a == 0) | (b == 0)) return 0;
    const double p = __ddiv_rn((double)(a * b), (double)(a + b));
    const double k = __ddiv_rn(p, __dadd_rn(p, p_acc[i]));
    const double lg = log(__ddiv_rn((double)a, (double)b));
    ds[i] = __dadd_rn(__dadd_rn(-lnw[i], lnw[i + 1]), __dmul_rn(k, lg));
    p_acc[i] = __dadd_rn(p_acc[i], p);
    return 1;
}

// One block's statistics and update of an instance of a batch.  `dyn`: dynamic
// shared memory of update_smem(N, rule) bytes.
__device__ __forceinline__ void weight_update_body(const unsigned long long *__restrict__ hist, uint32_t N,
                                                   double *__restrict__ lnw, float *__restrict__ w32,
                                                   double *__restrict__ p_acc, int rule, RunCtl *__restrict__ ctl,
                                                   unsigned char *dyn)
{
    __shared__ HistSum shs[32];
    __shared__ double shd[32];
    __shared__ int do_update;
    const uint32_t tid = threadIdx.x, bs = blockDim.x;
    if (ctl->st.stop) return;

    // values needed before anything is written (normalisation constant)
    const unsigned long long h0 = hist[0];
    const double lnw0 = lnw[0];

    HistSum hs{(int)N + 1, -1, 0ull, 0ull, ~0ull};
    for (uint32_t i = tid; i <= N; i += bs) hs.add((int)i, hist[i]);
    hs = block_join(hs, shs, N);
    const unsigned long long vis = hs.vis, ev = hs.ev, mn = hs.mn;
    const int lo = hs.lo, hi = hs.hi;
    int start = lo, end = hi < 0 ? 0 : hi;
    if (start > end) { start = 0; end = 0; }

    // Kullback-Leibler divergence: sum over H>0 of P ln(P/Q), P = H/events, Q = 1/visited
    const double num_event = (double)ev, Q = __ddiv_rn(1.0, (double)vis);
    double kl = 0.0;
    for (uint32_t i = tid; i <= N; i += bs) {
        const unsigned long long h = hist[i];
        if (h > 0) {
            const double P = __ddiv_rn((double)h, num_event);
            kl = __dadd_rn(kl, __dmul_rn(P, log(__ddiv_rn(P, Q))));
        }
    }
    kl = block_reduce(kl, AddD(), shd);
    if (tid == 0) do_update = bookkeep(start, end, vis, ev, mn, kl, N, rule, nullptr, ctl);
    __syncthreads();
    if (!do_update) return;

    if (rule == 0 || rule == 1) {
        // tmp = lnW[0] after the ln H subtraction (:469), computed from the
        // values read before any write
        const unsigned long long thr = rule == 0 ? 1ull : 0ull;
        const double tmp = h0 > thr ? __dsub_rn(lnw0, log((double)h0)) : lnw0;
        for (uint32_t i = tid; i <= N; i += bs) {
            const unsigned long long h = hist[i];
            double v = lnw[i];
            if (h > thr) v = __dsub_rn(v, log((double)h));
            if (rule == 0 || h > 0) v = __dsub_rn(v, tmp);
            lnw[i] = v;
            w32[i] = (float)v;
        }
        return;
    }

    // rule 2: weight_recursion (:848-858) then lnW -= lnW[0].
    // (a) the increments dS_i of all connected pairs, in parallel;
    double *ds = reinterpret_cast<double *>(dyn);
    unsigned char *valid = dyn + sizeof(double) * (size_t)N;
    for (uint32_t i = tid; i < N; i += bs) valid[i] = recursion_increment(hist, lnw, p_acc, i, start, end, ds);
    __syncthreads();
    // (b) the prefix lnW[i+1] = lnW[i] + dS_i, in place over ds (a pair
    //     with an empty bin leaves lnW[i+1] at its old value);
    block_segmented_prefix(start, end, lnw[start], ds, valid, lnw + 1, ds);
    // (c) write back and normalise by lnW[0] (bin 0 is never rewritten)
    for (uint32_t i = tid; i <= N; i += bs) {
        double v = ((int)i > start && (int)i <= end) ? ds[i - 1] : lnw[i];
        v = __dsub_rn(v, lnw0);
        lnw[i] = v;
        w32[i] = (float)v;
    }
}

// ---- the same statistics and update over kUpdBlocks blocks ---------------
// The divergence terms and the ln H of the update are FP64 per bin, and FP64
// issues slowly on this GPU: one block leaves all of them to one SM (ncu:
// 67 % of that SM's FP64 pipe, 28 us at L=72).  Here pass 1 forms the integer
// statistics per block; pass 2 the divergence terms per block, after every
// block has summed the partial event and visited counts in block order; the
// last block of pass 2 sums all partials in block order, keeps the books as
// the one-block update does (bookkeep) and decides the update; pass 3
// applies it.  Integer statistics and the updated weights equal the one-block
// update's; the divergence sum runs in another order.
constexpr int kUpdMultiThreads = 256;

__global__ void __launch_bounds__(kUpdMultiThreads) k_upd_stats(const unsigned long long *__restrict__ hist,
                                                                uint32_t N, const RunCtl *__restrict__ ctl,
                                                                UpdScratch *__restrict__ sc)
{
    __shared__ HistSum shs[32];
    if (ctl && ctl->st.stop) return;
    HistSum v{(int)N + 1, -1, 0ull, 0ull, ~0ull};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= N; i += gridDim.x * blockDim.x)
        v.add((int)i, hist[i]);
    v = block_join(v, shs, N);
    if (threadIdx.x == 0) {
        UpdPart &p = sc->part[blockIdx.x];
        p.lo = v.lo; p.hi = v.hi; p.vis = v.vis; p.ev = v.ev; p.mn = v.mn;
    }
}

__global__ void __launch_bounds__(kUpdMultiThreads) k_upd_kl(const unsigned long long *__restrict__ hist, uint32_t N,
                                                             const double *__restrict__ lnw, int rule,
                                                             HistStatsDev *__restrict__ stats,
                                                             RunCtl *__restrict__ ctl, UpdScratch *__restrict__ sc)
{
    __shared__ double shd[32];
    __shared__ unsigned long long s_ev, s_vis;
    __shared__ int s_last;
    if (ctl && ctl->st.stop) {
        // an iteration after the stop: no update either
        if (blockIdx.x == 0 && threadIdx.x == 0) sc->upd = sc->clear = 0;
        return;
    }
    if (threadIdx.x < 32) {
        // the partial counts, two per lane, then a warp sum (fixed order)
        unsigned long long e = 0, v = 0;
        for (uint32_t b = threadIdx.x; b < gridDim.x; b += 32) { e += sc->part[b].ev; v += sc->part[b].vis; }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            e += __shfl_xor_sync(0xffffffffu, e, o);
            v += __shfl_xor_sync(0xffffffffu, v, o);
        }
        if (threadIdx.x == 0) {
            s_ev = e;
            s_vis = v;
        }
    }
    __syncthreads();
    // sum over H>0 of P ln(P/Q), P = H/events, Q = 1/visited (as the one-block update)
    const double num_event = (double)s_ev, Q = __ddiv_rn(1.0, (double)s_vis);
    double kl = 0.0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= N; i += gridDim.x * blockDim.x) {
        const unsigned long long h = hist[i];
        if (h > 0) {
            const double P = __ddiv_rn((double)h, num_event);
            kl = __dadd_rn(kl, __dmul_rn(P, log(__ddiv_rn(P, Q))));
        }
    }
    kl = block_reduce(kl, AddD(), shd);
    if (threadIdx.x == 0) {
        sc->part[blockIdx.x].kl = kl;
        __threadfence();
        s_last = atomicAdd(&sc->done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last || threadIdx.x >= 32) return;
    __threadfence();
    // all partials, two per lane, then warp reductions (fixed order)
    int lo = (int)N + 1, hi = -1;
    unsigned long long vis = 0, ev = 0, mn = ~0ull;
    double klt = 0.0;
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += 32) {
        const UpdPart &p = sc->part[b];
        lo = min(lo, p.lo);
        hi = max(hi, p.hi);
        vis += p.vis;
        ev += p.ev;
        mn = p.mn < mn ? p.mn : mn;
        klt = __dadd_rn(klt, __ldcg(&p.kl));  // written by other blocks of this launch
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        vis += __shfl_xor_sync(0xffffffffu, vis, o);
        ev += __shfl_xor_sync(0xffffffffu, ev, o);
        const unsigned long long m2 = __shfl_xor_sync(0xffffffffu, mn, o);
        mn = m2 < mn ? m2 : mn;
        klt = __dadd_rn(klt, __shfl_xor_sync(0xffffffffu, klt, o));
    }
    if (threadIdx.x != 0) return;
    int start = lo, end = hi < 0 ? 0 : hi;
    if (start > end) { start = 0; end = 0; }
    sc->upd = bookkeep(start, end, vis, ev, mn, klt, N, rule, stats, ctl);
    sc->clear = clears_hist(ctl);
    sc->start = start;
    sc->end = end;
    // lnW[0] after its ln H subtraction (:469), from the weights before any write
    const unsigned long long h0 = hist[0], thr = rule == 0 ? 1ull : 0ull;
    sc->tmp = h0 > thr ? __dsub_rn(lnw[0], log((double)h0)) : lnw[0];
    sc->done = 0;
}

__global__ void __launch_bounds__(kUpdMultiThreads) k_upd_apply(unsigned long long *__restrict__ hist, uint32_t N,
                                                                double *__restrict__ lnw,
                                                                float *__restrict__ w32, int rule,
                                                                const UpdScratch *__restrict__ sc)
{
    const bool upd = sc->upd != 0, clear = sc->clear != 0;
    if (!upd && !clear) return;
    const unsigned long long thr = rule == 0 ? 1ull : 0ull;
    const double tmp = sc->tmp;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= N; i += gridDim.x * blockDim.x) {
        if (upd) {
            const unsigned long long h = hist[i];
            double v = lnw[i];
            if (h > thr) v = __dsub_rn(v, log((double)h));
            if (rule == 0 || h > 0) v = __dsub_rn(v, tmp);
            lnw[i] = v;
            w32[i] = (float)v;
        }
        if (clear) hist[i] = 0ull;
    }
}

// ---- the trivial updates and the statistics in one launch -----------------
// A cluster of sixteen blocks does the three passes with cluster barriers
// between them, the partial results read from the other blocks' shared memory
// and the bins held in registers, and forms the updated weights while one
// thread keeps the books.  What bounds it is the latency of its FP64 divisions
// and logarithms (FP64 issues slowly on this GPU) and of the barriers.  Whole
// iterations of 4096 chains with few attempts, against the three launches (a
// third of the bins visited): host-buffer calls 90 us for 102 at N = 4096, 103
// for 113 at 5184, 124 for 129 at 8100; runs in a graph 55.7 for 58.4, 66.2 for
// 68.4 and 88.7 for 89.0 an iteration.  The update alone back to back, every bin
// visited: 16.4 for 22.5 us at N = 256, 17.4 at 3969, 23.0 at 5184, 23.5 at 8100
// (and in a graph 21.1 for 15.9 from two bins per thread on, where nothing lies
// between the updates).  Above 8191 bins the three launches with their 64 SMs
// stay.
constexpr uint32_t kClusterBlocks = 16, kClusterThreads = 256;
constexpr int kClusterPer = 2;  // bins per thread at most
constexpr uint32_t kClusterBins = kClusterBlocks * kClusterThreads * kClusterPer;

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// a 64-bit word of block `rank`'s shared memory at the place of this block's `p`
__device__ __forceinline__ unsigned long long cluster_load(const void *p, uint32_t rank)
{
    unsigned long long v;
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    return v;
}

// The update by this block's cluster (kClusterBlocks successive blocks), PER
// bins per thread at most.  CLEAR: in a device-driven run, zero the histogram
// for the next iteration (clears_hist).  Returns whether this
// thread (one of the cluster) has seen the run go on.
template <int PER, bool CLEAR>
__device__ __forceinline__ bool cluster_update(unsigned long long *__restrict__ hist, uint32_t N,
                                               double *__restrict__ lnw, float *__restrict__ w32, int rule,
                                               HistStatsDev *__restrict__ stats, RunCtl *__restrict__ ctl)
{
    const uint32_t rank = blockIdx.x % kClusterBlocks;
    __shared__ HistSum shs[32];
    __shared__ double shd[32];
    __shared__ unsigned long long s_part[4], s_kl, s_do;
    __shared__ RunCtl s_ctl;
    // (read by every block before the first barrier, written after the second)
    if (ctl && ctl->st.stop) return false;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, i0 = rank * kClusterThreads + tid;
    constexpr uint32_t st = kClusterBlocks * kClusterThreads;
    // the run state, near for the one thread that keeps the books
    if (ctl && rank == 0 && tid < sizeof(RunCtl) / 4)
        reinterpret_cast<uint32_t *>(&s_ctl)[tid] = reinterpret_cast<const uint32_t *>(ctl)[tid];
    const unsigned long long h0 = hist[0], thr = rule == 0 ? 1ull : 0ull;
    const double lnw0 = lnw[0];
    unsigned long long h[PER];
    double x[PER];
    HistSum v{(int)N + 1, -1, 0ull, 0ull, ~0ull};
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const uint32_t i = i0 + k * st;
        h[k] = 0ull;
        x[k] = 0.0;
        if (i <= N) {
            h[k] = hist[i];
            x[k] = lnw[i];
            v.add((int)i, h[k]);
        }
    }
    v = block_join(v, shs, N);
    if (tid == 0) {
        s_part[0] = (unsigned long long)(uint32_t)v.lo << 32 | (uint32_t)v.hi;
        s_part[1] = v.vis;
        s_part[2] = v.ev;
        s_part[3] = v.mn;
    }
    cluster_sync();
    {
        // every warp joins all blocks' parts; the upper 16 lanes repeat the extremes
        const uint32_t r = lane % kClusterBlocks;
        const bool once = lane < kClusterBlocks;
        const unsigned long long range = cluster_load(&s_part[0], r), vis = cluster_load(&s_part[1], r),
                                 ev = cluster_load(&s_part[2], r), mn = cluster_load(&s_part[3], r);
        v = HistSum{(int)(uint32_t)(range >> 32), (int)(uint32_t)range, once ? vis : 0ull, once ? ev : 0ull, mn};
        v.warp_join();
    }
    // sum over H>0 of P ln(P/Q), P = H/events, Q = 1/visited (as the one-block update)
    const double num_event = (double)v.ev, Q = __ddiv_rn(1.0, (double)v.vis);
    double kl = 0.0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        if (h[k] > 0) {
            const double P = __ddiv_rn((double)h[k], num_event);
            kl = __dadd_rn(kl, __dmul_rn(P, log(__ddiv_rn(P, Q))));
        }
    }
    kl = block_reduce(kl, AddD(), shd);
    if (tid == 0) s_kl = (unsigned long long)__double_as_longlong(kl);
    cluster_sync();
    if (rank == 0 && tid < 32) {
        // the blocks' sums joined as a tree
        double klt = lane < kClusterBlocks ? __longlong_as_double((long long)cluster_load(&s_kl, lane)) : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) klt = __dadd_rn(klt, __shfl_xor_sync(0xffffffffu, klt, o));
        if (tid == 0) {
            int start = v.lo, end = v.hi < 0 ? 0 : v.hi;
            if (start > end) { start = 0; end = 0; }
            const int upd = bookkeep(start, end, v.vis, v.ev, v.mn, klt, N, rule, stats, ctl ? &s_ctl : nullptr);
            s_do = (upd ? 1u : 0u) | (ctl && !s_ctl.st.stop ? 2u : 0u) | (ctl && clears_hist(&s_ctl) ? 4u : 0u);
            if (ctl) ctl->st = s_ctl.st;
        }
    }
    // meanwhile the updated weights: lnW[0] after its ln H subtraction (:469),
    // from the values before any write
    if (rule >= 0) {
        const double tmp = h0 > thr ? __dsub_rn(lnw0, log((double)h0)) : lnw0;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            if (h[k] > thr) x[k] = __dsub_rn(x[k], log((double)h[k]));
            if (rule == 0 || h[k] > 0) x[k] = __dsub_rn(x[k], tmp);
        }
    }
    cluster_sync();
    const uint32_t todo = (uint32_t)cluster_load(&s_do, 0);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const uint32_t i = i0 + k * st;
        if (i <= N) {
            if (todo & 1u) {
                lnw[i] = x[k];
                w32[i] = (float)x[k];
            }
            if (CLEAR && (todo & 4u)) hist[i] = 0ull;
        }
    }
    cluster_sync();  // no block leaves while another may read its shared memory
    return rank == 0 && tid == 0 && (todo & 2u);
}
__global__ void __launch_bounds__(kClusterThreads) k_upd_cluster(unsigned long long *__restrict__ hist, uint32_t N,
                                                                 double *__restrict__ lnw, float *__restrict__ w32,
                                                                 int rule, HistStatsDev *__restrict__ stats,
                                                                 RunCtl *__restrict__ ctl)
{
    cluster_update<kClusterPer, true>(hist, N, lnw, w32, rule, stats, ctl);
}

// One iteration's tail for every instance of a batch without the recursion, a
// cluster per instance (up to 16385 bins), and the count of the instances still
// running: the form of few and large instances (batch_update_by_cluster).
constexpr int kBatchPer = 5;
static_assert(kClusterBlocks * kClusterThreads * kBatchPer >= 16385, "bins of the largest instance");
__global__ void __launch_bounds__(kClusterThreads) k_batch_update(const BatchInst *__restrict__ insts,
                                                                  uint32_t *__restrict__ running)
{
    const BatchInst &I = insts[blockIdx.x / kClusterBlocks];
    if (cluster_update<kBatchPer, false>(I.a.hist, I.a.N, I.lnw, I.w32, (int)I.rule, nullptr, I.ctl))
        atomicAdd(running, 1u);
}

static cudaLaunchConfig_t cluster_config(cudaLaunchAttribute *at, uint32_t updates, cudaStream_t s)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kClusterBlocks * updates);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.stream = s;
    *at = cudaLaunchAttribute{};
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = kClusterBlocks;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}


static cudaError_t launch_update_cluster(unsigned long long *hist, uint32_t N, double *lnw, float *w32, int rule,
                                         HistStatsDev *stats, RunCtl *ctl, cudaStream_t s)
{
    const cudaError_t e = cudaFuncSetAttribute(k_upd_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = cluster_config(&at, 1, s);
    return cudaLaunchKernelEx(&cfg, k_upd_cluster, hist, N, lnw, w32, rule, stats, ctl);
}

// Rule 2 over kUpdBlocks blocks: the increments of every connected pair
// (FP64 divisions and a logarithm each) ...
__global__ void __launch_bounds__(kUpdMultiThreads) k_upd_rec_inc(const unsigned long long *__restrict__ hist,
                                                                  uint32_t N, const double *__restrict__ lnw,
                                                                  double *__restrict__ p_acc,
                                                                  const UpdScratch *__restrict__ sc, RecScratch rs)
{
    if (!sc->upd) return;
    const int start = sc->start, end = sc->end;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
        rs.valid[i] = recursion_increment(hist, lnw, p_acc, i, start, end, rs.ds);
}

// ... then the prefix as one block's segmented scan, the write-back and the
// normalisation by lnW[0] (bin 0 is never rewritten by the recursion).
__global__ void __launch_bounds__(kUpdThreads) k_upd_rec_scan(unsigned long long *__restrict__ hist, uint32_t N,
                                                               double *__restrict__ lnw, float *__restrict__ w32,
                                                               const UpdScratch *__restrict__ sc, RecScratch rs)
{
    if (sc->clear)
        for (uint32_t i = threadIdx.x; i <= N; i += blockDim.x) hist[i] = 0ull;
    if (!sc->upd) return;
    const int start = sc->start, end = sc->end;
    const double lnw0 = lnw[0];
    block_segmented_prefix(start, end, lnw[start], rs.ds, rs.valid, lnw + 1, rs.ds);
    for (uint32_t i = threadIdx.x; i <= N; i += blockDim.x) {
        double v = ((int)i > start && (int)i <= end) ? rs.ds[i - 1] : lnw[i];
        v = __dsub_rn(v, lnw0);
        lnw[i] = v;
        w32[i] = (float)v;
    }
}

static cudaError_t launch_update_multi(unsigned long long *hist, uint32_t N, double *lnw, float *w32,
                                       double *p_acc, int rule, HistStatsDev *stats, RunCtl *ctl, UpdScratch *sc,
                                       const RecScratch *rs, cudaStream_t s)
{
    k_upd_stats<<<kUpdBlocks, kUpdMultiThreads, 0, s>>>(hist, N, ctl, sc);
    k_upd_kl<<<kUpdBlocks, kUpdMultiThreads, 0, s>>>(hist, N, lnw, rule, stats, ctl, sc);
    if (rule == 2) {
        k_upd_rec_inc<<<kUpdBlocks, kUpdMultiThreads, 0, s>>>(hist, N, lnw, p_acc, sc, *rs);
        k_upd_rec_scan<<<1, kUpdThreads, 0, s>>>(hist, N, lnw, w32, sc, *rs);
    } else if (rule >= 0) {
        k_upd_apply<<<kUpdBlocks, kUpdMultiThreads, 0, s>>>(hist, N, lnw, w32, rule, sc);
    }
    return cudaGetLastError();
}

// The tail of a batch's iteration by a block per instance: the recursion, and
// the trivial updates of many or small instances.
__global__ void __launch_bounds__(kUpdThreads) k_batch_update_block(const BatchInst *__restrict__ insts,
                                                                   uint32_t *__restrict__ running)
{
    extern __shared__ __align__(16) unsigned char dyn[];
    const BatchInst &I = insts[blockIdx.x];
    weight_update_body(I.a.hist, I.a.N, I.lnw, I.w32, I.p_acc, (int)I.rule, I.ctl, dyn);
    if (threadIdx.x == 0 && !I.ctl->st.stop) atomicAdd(running, 1u);
}

// What follows the arrival of FP64 weights: their FP32 shadow, the
// reweighting copy, and the cleared histogram of the sweep to come (n_hist
// bins, 0: none).
__global__ void k_weights_in(const double *__restrict__ lnw, float *__restrict__ w32, double *__restrict__ obs,
                             uint32_t n, unsigned long long *__restrict__ hist, uint32_t n_hist)
{
    const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x, st = gridDim.x * blockDim.x;
    for (uint32_t i = i0; i < n; i += st) {
        const double v = lnw[i];
        w32[i] = (float)v;
        if (obs) obs[i] = v;
    }
    for (uint32_t i = i0; i < n_hist; i += st) hist[i] = 0ull;
}

static size_t update_smem(uint32_t N, int rule) { return rule == 2 ? (size_t)N * (sizeof(double) + 1) : 0; }

// Sixteen blocks of a cluster need SMs of one GPC: a partition of the device (or
// an SM-restricted context) may have none to place them on.
bool update_cluster_fits(cudaStream_t s, bool batch)
{
    const void *kern = batch ? (const void *)k_batch_update : (const void *)k_upd_cluster;
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = cluster_config(&at, 1, s);
    int clusters = 0;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess && clusters > 0;
}

cudaError_t launch_weight_update(unsigned long long *hist, uint32_t N, double *lnw, float *w32, double *p_acc,
                                 int rule, HistStatsDev *stats, cudaStream_t s, bool cluster, UpdScratch *sc,
                                 const RecScratch *rs)
{
    if (cluster && rule != 2 && N < kClusterBins)
        return launch_update_cluster(hist, N, lnw, w32, rule, stats, nullptr, s);
    return launch_update_multi(hist, N, lnw, w32, p_acc, rule, stats, nullptr, sc, rs, s);
}

cudaError_t launch_run_update(unsigned long long *hist, double *lnw, float *w32, double *p_acc, RunCtl *ctl,
                              cudaStream_t s, uint32_t N, int rule, bool cluster, UpdScratch *sc,
                              const RecScratch *rs)
{
    if (cluster && rule != 2 && N < kClusterBins)
        return launch_update_cluster(hist, N, lnw, w32, rule, nullptr, ctl, s);
    return launch_update_multi(hist, N, lnw, w32, p_acc, rule, nullptr, ctl, sc, rs, s);
}

cudaError_t prepare_batch_update(uint32_t max_N)
{
    // the limit of the largest size, whatever this batch's: another batch of the
    // process shares the kernel
    if (update_smem(max_N, 2) > 48 * 1024)
        return cudaFuncSetAttribute(k_batch_update_block, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)update_smem(16384, 2));
    return cudaSuccess;
}

// Clusters spread an instance's FP64 work over sixteen SMs but run some twenty at
// a time, blocks run one per SM, so which is faster follows from the sizes.
// Microseconds by cluster / by block, every bin visited:
//   instances      1          16          64          200         1000
//   L = 8       14.4/20.8   30.7/22.6   69.3/22.6  185.8/41.0   852/133
//   L = 32      18.5/45.2   40.1/47.2    104/47.1   278/90.1   1309/307
//   L = 64      20.5/116    42.5/117     117/117    314/229    1472/794
//   L = 128     38.0/395    94.0/396     282/396    793/788    3852/2788
//   L = 16..128             65.2/395     153/395    440/395    2130/1099
// The two estimates below are fitted to these.
bool batch_update_by_cluster(uint64_t sum_N, uint32_t max_N, uint32_t n_inst, int sms)
{
    const double cluster = 14.0 + 1.15 * n_inst + 0.00017 * (double)sum_N;
    const double block = std::max(20.0 + 0.023 * max_N, (20.0 * n_inst + 0.023 * (double)sum_N) / sms);
    return cluster < block;
}

cudaError_t launch_batch_update(const BatchInst *insts, uint32_t n_inst, uint32_t max_N, int recursion, bool cluster,
                                uint32_t *running, cudaStream_t s)
{
    if (!recursion && cluster) {
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t cfg = cluster_config(&at, n_inst, s);
        return cudaLaunchKernelEx(&cfg, k_batch_update, insts, running);
    }
    k_batch_update_block<<<n_inst, kUpdThreads, recursion ? update_smem(max_N, 2) : 0, s>>>(insts, running);
    return cudaGetLastError();
}

cudaError_t launch_weights_in(const double *lnw, float *w32, double *obs, uint32_t n, unsigned long long *hist,
                              uint32_t n_hist, cudaStream_t s)
{
    k_weights_in<<<(n + 255) / 256, 256, 0, s>>>(lnw, w32, obs, n, hist, n_hist);
    return cudaGetLastError();
}

}  // namespace muca
