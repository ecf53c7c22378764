// k_sweep_win.cuh -- the windowed sweep kernel (window.cuh) and its dispatch;
// k_win_weight.cu and k_win_produce.cu hold the kernels of the two modes.
#pragma once
#include "window.cuh"

namespace muca {

// One block per chain block, blockDim = cpb rounded up to a warp.
// RING: the lattice stays in global memory behind a four-row ring per lane.
// ALIGNED: L % 8 == 0.  MANY: up to 512 chains per block, four warps per SM
// sub-partition, so at most 128 registers per thread.
// FEED: behind the (one or two) walking warps as many that draw for them.
template <int MODE, int R, bool LAT_SMEM, bool RING, bool ALIGNED, bool MANY, bool FEED = false>
__global__ void __launch_bounds__(MANY ? 512 : 128, 1) k_sweep_win(const SweepArgs a, uint32_t cpb)
{
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t iter;
    unsigned long long nup;
    if (!launch_params(a, iter, nup)) return;
    win_sweep_block<MODE, R, LAT_SMEM, true, false, RING, ALIGNED, MANY, FEED>(
        a, smem, cpb, blockIdx.x, iter, nup, nullptr,
        FEED ? (uint32_t)(win_smem_base(MODE, a.N, true) + align16((size_t)a.L * a.WPR * 4u * cpb)) : 0u);
}

template <int MODE, int R>
cudaError_t launch_sweep_win(const SweepPlan &p, const SweepArgs &a, cudaStream_t s)
{
    void (*kern)(const SweepArgs, uint32_t);
    if (a.L % 8 == 0) {
        if (p.feed) kern = k_sweep_win<MODE, R, true, false, true, false, true>;
        else if (p.many) kern = p.lat_smem ? k_sweep_win<MODE, R, true, false, true, true> : k_sweep_win<MODE, R, false, true, true, true>;
        else if (p.lat_smem) kern = k_sweep_win<MODE, R, true, false, true, false>;
        else if (p.row_ring) kern = k_sweep_win<MODE, R, false, true, true, false>;
        else return cudaErrorInvalidValue;  // the planner's ring always fits
    } else {
        kern = p.feed ? k_sweep_win<MODE, R, true, false, false, false, true> : p.lat_smem ? k_sweep_win<MODE, R, true, false, false, false> : k_sweep_win<MODE, R, false, false, false, false>;
    }
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem_limit);
    if (e != cudaSuccess) return e;
    kern<<<p.blocks, p.threads, p.smem, s>>>(a, p.cpb);
    return cudaGetLastError();
}

}  // namespace muca
