// k_batch_sweep.cuh -- the sweep kernel of a batch (k_batch.cu).  Its instances
// take most of the build's time, so four files share them.
#pragma once
#include "window.cuh"

namespace muca {

using BatchKernel = void (*)(const BatchInst *, const BatchItem *, uint32_t, uint32_t *, uint32_t, uint32_t);

// The kernel of R Philox rounds and placement LAT; feed only with kLatWhereFits
// and hist_smem.
template <int R, int LAT>
BatchKernel batch_kernel_of(bool hist_smem, bool feed);

#ifdef MUCA_BATCH_INSTANCES
// FEED (shapes of one or two warps of chains per SM): as many warps more draw
// for those that walk, see window.cuh; their rings end the shared memory.
template <int R, int LAT, bool HS, bool FEED = false>
__global__ void __launch_bounds__(256, 1) k_batch_sweep(const BatchInst *__restrict__ insts,
                                                         const BatchItem *__restrict__ items, uint32_t n_items,
                                                         uint32_t *__restrict__ next_item, uint32_t cpb,
                                                         uint32_t smem_bytes)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_item;
    __shared__ float s_btab[kBetaTab];
    const uint32_t feed_off = smem_bytes - (FEED ? (cpb + 31u) / 32u * kFeedBytes : 0u);
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(next_item, 1u);
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= n_items) return;  // uniform: every thread read the same item
        const BatchItem item = items[it];
        const BatchInst *I = insts + item.inst;
        const SweepArgs a = I->a;
        uint32_t iter;
        unsigned long long nup;
        if (launch_params(a, iter, nup)) {  // the instance is still running
            // -beta dE by dE + 8, then beta times the neighbour spin sum by code sum
            if (threadIdx.x < kBetaTab)
                s_btab[threadIdx.x] = I->btab[threadIdx.x < 17 ? threadIdx.x : 29 - threadIdx.x];
            // s_btab is read only after the block barrier inside the sweep's prologue
            if (LAT == kLatShared) {
                win_sweep_block<kModeWeight, R, true, HS, true>(a, smem, cpb, item.blk, iter, nup, s_btab);
            } else {
                // uniform per item: the lattice joins the weights (and bins) in
                // shared memory when all fit in the launch's allocation
                // (kLatWhereFits); otherwise it stays in global memory, behind
                // a four-row ring per lane where that fits
                const size_t base = smem_weights_bytes(kModeWeight, a.N) + (HS ? smem_hist_bytes(kModeWeight, a.N) : 0);
                if (LAT == kLatWhereFits && base + (size_t)a.L * a.WPR * 4u * cpb <= feed_off)
                    win_sweep_block<kModeWeight, R, true, HS, true, false, true, false, FEED>(a, smem, cpb, item.blk, iter, nup,
                                                                                             s_btab, feed_off);
                else if (a.L % 4 == 0 && a.WPR <= 8 && base + ring_bytes(a.L, cpb) <= feed_off)
                    win_sweep_block<kModeWeight, R, false, HS, true, true, true, false, FEED>(a, smem, cpb, item.blk, iter, nup,
                                                                                             s_btab, feed_off);
                else
                    win_sweep_block<kModeWeight, R, false, HS, true, false, true, false, FEED>(a, smem, cpb, item.blk, iter, nup,
                                                                                              s_btab, feed_off);
            }
        }
        __syncthreads();
    }
}

template <int R, int LAT>
BatchKernel batch_kernel_of(bool hist_smem, bool feed)
{
    if constexpr (LAT == kLatWhereFits) {
        if (feed) return k_batch_sweep<R, LAT, true, true>;
    }
    return hist_smem ? k_batch_sweep<R, LAT, true> : k_batch_sweep<R, LAT, false>;
}
#endif

}  // namespace muca
