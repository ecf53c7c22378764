// k_batch.cu -- kernels of a batch of independent weight-estimation runs.
//
// Many (L, beta) instances of uneven size advance one weight iteration
// together: a prep kernel clears the histograms of the instances still
// running, one persistent sweep kernel works through the list of chain
// blocks of all instances, and a cluster or a block per instance applies the
// statistics, the schedule and the weight update (k_weights.cu).  The three
// launches of an iteration are captured into a CUDA graph by the host
// (muca_batch.cu) and replayed.
//
// The sweep of a chain block is the single-simulation windowed sweep
// (window.cuh) with two differences: the Metropolis term -beta*dE comes
// from the instance's table (exactly -2 dE for the reference's beta = 2), and
// the histogram may go straight to the u64 device histogram, which frees the
// shared memory of the u32 bins for more blocks per SM.  Work is fetched by
// an atomic counter over items sorted by decreasing cost, so the large
// lattices start first and the small ones fill the tail.  The kernel is in
// k_batch_sweep.cuh, its instances in k_batch_fits*.cu and k_batch_place*.cu.
#include "k_batch_sweep.cuh"

namespace muca {

__global__ void k_batch_prep(const BatchInst *__restrict__ insts, uint32_t *__restrict__ next_item,
                             uint32_t *__restrict__ running)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *next_item = 0u;
        *running = 0u;
    }
    const BatchInst &I = insts[blockIdx.x];
    if (I.ctl->st.stop) return;
    const uint32_t n = I.a.N + 1;
    unsigned long long *h = I.a.hist;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) h[i] = 0ull;
}

cudaError_t launch_batch_prep(const BatchInst *insts, uint32_t n_inst, uint32_t *next_item, uint32_t *running,
                              cudaStream_t s)
{
    k_batch_prep<<<n_inst, 256, 0, s>>>(insts, next_item, running);
    return cudaGetLastError();
}

size_t batch_sweep_smem(uint32_t L, uint32_t cpb, bool lat_smem, bool hist_smem, bool row_ring)
{
    const uint32_t N = L * L, WPR = (L + 15) / 16;
    return smem_weights_bytes(kModeWeight, N) + (hist_smem ? smem_hist_bytes(kModeWeight, N) : 0) +
           (lat_smem ? (size_t)L * WPR * 4 * cpb : (row_ring ? ring_bytes(L, cpb) : 0));
}

template <int R>
static BatchKernel batch_kernel_r(uint32_t lat, bool hist_smem, bool feed)
{
    return lat == kLatWhereFits ? batch_kernel_of<R, kLatWhereFits>(hist_smem, feed)
         : lat == kLatShared    ? batch_kernel_of<R, kLatShared>(hist_smem, false)
                                : batch_kernel_of<R, kLatGlobal>(hist_smem, false);
}

static BatchKernel batch_kernel(int rounds, uint32_t lat, bool hist_smem, bool feed)
{
    // where all lattices fit, "where it fits" is "in shared memory"
    if (feed) lat = kLatWhereFits;
    return rounds == 10 ? batch_kernel_r<10>(lat, hist_smem, feed) : batch_kernel_r<7>(lat, hist_smem, feed);
}

// Every launch raises the kernel's limit to all that a block may have: a limit
// set to one batch's own size would be the wrong one for another batch of the
// process that shares the kernel.
static cudaError_t raise_smem_limit(BatchKernel k, size_t smem_limit)
{
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_limit);
}

size_t batch_feed_smem(uint32_t cpb) { return (cpb + 31u) / 32u * kFeedBytes; }

static uint32_t batch_threads(uint32_t cpb, bool feed) { return (cpb + 31u) / 32u * 32u * (feed ? 2u : 1u); }
static bool feed_allowed(uint32_t cpb, uint32_t lat, bool hist_smem)
{
    return cpb <= 64 && lat != kLatGlobal && hist_smem;
}

cudaError_t batch_sweep_occupancy(uint32_t cpb, int rounds, uint32_t lat, bool hist_smem, bool feed, size_t smem,
                                  size_t smem_limit, int *blocks)
{
    if (lat > kLatWhereFits || (feed && !feed_allowed(cpb, lat, hist_smem))) return cudaErrorInvalidValue;
    const BatchKernel k = batch_kernel(rounds, lat, hist_smem, feed);
    const cudaError_t e = raise_smem_limit(k, smem_limit);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, k, (int)batch_threads(cpb, feed), smem);
}

cudaError_t launch_batch_sweep(const BatchInst *insts, const BatchItem *items, uint32_t n_items, uint32_t *next_item,
                               uint32_t cpb, int rounds, uint32_t lat, bool hist_smem, bool feed, uint32_t grid,
                               size_t smem, size_t smem_limit, cudaStream_t s)
{
    if (cpb == 0 || cpb > 256 || lat > kLatWhereFits || (feed && !feed_allowed(cpb, lat, hist_smem)))
        return cudaErrorInvalidValue;
    const BatchKernel k = batch_kernel(rounds, lat, hist_smem, feed);
    const cudaError_t e = raise_smem_limit(k, smem_limit);
    if (e != cudaSuccess) return e;
    k<<<grid, batch_threads(cpb, feed), smem, s>>>(insts, items, n_items, next_item, cpb, (uint32_t)smem);
    return cudaGetLastError();
}

}  // namespace muca
