// k_lattice.cu -- chain initialisation and lattice (un)packing on the device.
//
// The reference initialises every chain's lattice on the host, one Philox
// block per 4 sites, then copies it to the device and runs computeEnergies /
// computeDeltaE (/computeM) (muca_delta_multigpu.cu:340-359,
// produce2_multigpu.cu:126-140,272-274).  Here one thread builds one packed
// 16-site word of one chain directly in device memory (the Philox stream of
// a site is a pure function of (chain, site), so words are independent), and
// a second kernel forms E_J, E_Delta and M per chain.
#include "muca_device.cuh"
#include "muca_internal.h"

namespace muca {

template <int R>
__device__ __forceinline__ uint4 init_block(const InitArgs &ia, uint32_t W, uint32_t dev, uint32_t chain,
                                            uint32_t jack, uint32_t g)
{
    RoundKeys<R> k;
    uint32_t c[4];
    k.init(ia.key0_mul * W + ia.key0_jack_mul * jack + ia.key0_add, ia.key1 + ia.key1_jack_mul * jack);
    if (ia.chain_in_ctr) {
        c[0] = ia.chain_offset + chain; c[1] = g; c[2] = 0; c[3] = 0;
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) c[j] = ia.ctr0[j] + ia.ctr0_dev_mul[j] * dev;
        c[ia.ctr_word] += g + 1u;  // ++c[word] before every 4th site
    }
    return philox<R>(c[0], c[1], c[2], c[3], k);
}

// Word w of a chain's packed lattice.
template <int R>
__device__ __forceinline__ uint32_t init_word(const InitArgs &ia, uint32_t L, uint32_t WPR, uint32_t w, uint32_t chain,
                                              uint32_t nchains, uint32_t chains_per_dev, uint32_t jack)
{
    if (chain >= nchains) return kZeroWord;
    const uint32_t dev = chain / chains_per_dev, W = chain - dev * chains_per_dev;
    const uint32_t row = w / WPR, q = w - row * WPR;
    const uint32_t c_lo = 16u * q, c_hi = min(16u * q + 16u, L);
    uint32_t word = 0;
    uint32_t g_cur = 0xFFFFFFFFu;
    uint4 r = make_uint4(0, 0, 0, 0);
    for (uint32_t col = c_lo; col < c_hi; ++col) {
        int s;
        if (ia.ordered) {
            s = 1;
        } else {
            const uint32_t site = row * L + col, g = site >> 2;
            if (g != g_cur) {
                r = init_block<R>(ia, W, dev, chain, jack, g);
                g_cur = g;
            }
            const uint32_t rw = pick(r, (int)(site & 3u));
            s = ia.graded ? graded_spin(rw, W, chains_per_dev) : init_spin(rw);
        }
        word |= (uint32_t)(s + 1) << (2u * (col - c_lo));
    }
    return word;
}

template <int R>
__global__ void k_init(uint32_t *lat, uint32_t L, uint32_t WPR, uint32_t cpb, uint32_t nchains,
                       uint32_t chains_per_dev, uint32_t jack, InitArgs ia)
{
    const uint32_t words = L * WPR;
    const size_t total = (size_t)((nchains + cpb - 1) / cpb) * cpb * words;
    const bool narrow = total <= 0xFFFFFFFFull;  // 32-bit index arithmetic (uniform)
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        // t enumerates [block][word][lane] exactly like the packed layout
        uint32_t lane, w, blk;
        if (narrow) {
            const uint32_t t32 = (uint32_t)t, bw = t32 / cpb;
            lane = t32 - bw * cpb;
            blk = bw / words;
            w = bw - blk * words;
        } else {
            const size_t bw = t / cpb;
            lane = (uint32_t)(t - bw * cpb);
            blk = (uint32_t)(bw / words);
            w = (uint32_t)(bw - (size_t)blk * words);
        }
        lat[t] = init_word<R>(ia, L, WPR, w, blk * cpb + lane, nchains, chains_per_dev, jack);
    }
}

// The lattices of a batch's instances: blockIdx.x = work item, the words of
// its chain block spread over blockIdx.y; emulated device index = the
// instance's seed.
__global__ void k_batch_init(const BatchInst *__restrict__ insts, const BatchItem *__restrict__ items, uint32_t cpb,
                             InitArgs ia)
{
    const BatchItem it = items[blockIdx.x];
    const BatchInst &I = insts[it.inst];
    const uint32_t L = I.a.L, WPR = I.a.WPR, words = L * WPR, nch = I.a.nchains;
    ia.ctr0[0] += ia.ctr0_dev_mul[0] * I.seed;
    uint32_t *lat = I.a.lat + (size_t)it.blk * words * cpb;
    for (uint32_t t = blockIdx.y * blockDim.x + threadIdx.x; t < words * cpb; t += gridDim.y * blockDim.x) {
        const uint32_t w = t / cpb, lane = t - w * cpb;
        lat[t] = init_word<7>(ia, L, WPR, w, it.blk * cpb + lane, nch, nch, 0);
    }
}

__global__ void k_pack(uint32_t *lat, const int8_t *src, uint32_t L, uint32_t WPR, uint32_t cpb, uint32_t nchains)
{
    const uint32_t words = L * WPR;
    const size_t total = (size_t)((nchains + cpb - 1) / cpb) * cpb * words;
    const size_t N = (size_t)L * L;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const uint32_t lane = (uint32_t)(t % cpb);
        const size_t bw = t / cpb;
        const uint32_t w = (uint32_t)(bw % words);
        const uint32_t chain = (uint32_t)(bw / words) * cpb + lane;
        uint32_t word = kZeroWord;
        if (chain < nchains) {
            const uint32_t row = w / WPR, q = w - row * WPR;
            const uint32_t c_lo = 16u * q, c_hi = min(16u * q + 16u, L);
            const int8_t *p = src + chain * N + (size_t)row * L;
            word = 0;
            for (uint32_t col = c_lo; col < c_hi; ++col) word |= (uint32_t)(p[col] + 1) << (2u * (col - c_lo));
        }
        lat[t] = word;
    }
}

__global__ void k_unpack(const uint32_t *lat, int8_t *dst, uint32_t L, uint32_t WPR, uint32_t cpb, uint32_t nchains)
{
    const uint32_t words = L * WPR;
    const size_t total = (size_t)((nchains + cpb - 1) / cpb) * cpb * words;
    const size_t N = (size_t)L * L;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const uint32_t lane = (uint32_t)(t % cpb);
        const size_t bw = t / cpb;
        const uint32_t w = (uint32_t)(bw % words);
        const uint32_t chain = (uint32_t)(bw / words) * cpb + lane;
        if (chain >= nchains) continue;
        const uint32_t row = w / WPR, q = w - row * WPR;
        const uint32_t c_lo = 16u * q, c_hi = min(16u * q + 16u, L);
        const uint32_t word = lat[t];
        int8_t *p = dst + chain * N + (size_t)row * L;
        for (uint32_t col = c_lo; col < c_hi; ++col) p[col] = (int8_t)((int)spin_code(word, col) - 1);
    }
}

// E_J = -sum over bonds (right and up neighbour of every site), which equals
// total_energy of muca_delta_multigpu.cu:563-571 (the sum over all four
// neighbours, halved), E_Delta = sum s^2, M = sum s.
// A block of 32 x kEnergyRows threads takes 32 chains, thread (x, y) rows y,
// y + kEnergyRows, ... of chain x, whole words at a time: a code is nonzero
// where its low bit is clear, its high bit the sign, so a word's 16 bonds are
// two population counts.  (Site by site, one thread per chain, L = 128 took
// 300 us however few the chains.)
constexpr uint32_t kEnergyRows = 8;
__device__ __forceinline__ void chain_energies(const uint32_t *base, uint32_t L, uint32_t WPR, uint32_t cpb, bool on,
                                               int32_t *ej, int32_t *edel, int32_t *mag)
{
    __shared__ int sh[3][kEnergyRows][32];
    const uint32_t x = threadIdx.x & 31u, y = threadIdx.x >> 5;
    const uint32_t last = L - 16u * (WPR - 1u);  // sites of a row's last word
    int bonds = 0, d = 0, m = 0;
    auto pairs = [](uint32_t nz, uint32_t a, uint32_t b) -> int {
        const uint32_t both = nz & ~b;
        return __popc(both) - 2 * __popc(both & ((a ^ b) >> 1));
    };
    for (uint32_t r = y; on && r < L; r += kEnergyRows) {
        const uint32_t *row = base + (size_t)(r * WPR) * cpb;
        const uint32_t *up = base + (size_t)((r + 1 == L ? 0u : r + 1u) * WPR) * cpb;
        const uint32_t first = row[0];
        uint32_t C = first;
        for (uint32_t q = 0; q < WPR; ++q) {
            const bool end = q + 1 == WPR;
            const uint32_t next = end ? first : row[(size_t)(q + 1) * cpb], U = up[(size_t)q * cpb];
            const uint32_t valid = end && last < 16u ? (1u << (2u * last)) - 1u : ~0u;
            const uint32_t nz = ~C & valid & 0x55555555u;
            const uint32_t right = end ? ((C & valid) >> 2) | (first << (2u * last - 2u)) : (C >> 2) | (next << 30);
            bonds += pairs(nz, C, right) + pairs(nz, C, U);
            const int n = __popc(nz);
            d += n;
            m += 2 * __popc(nz & (C >> 1)) - n;
            C = next;
        }
    }
    sh[0][y][x] = bonds;
    sh[1][y][x] = d;
    sh[2][y][x] = m;
    __syncthreads();
    if (y < 3 && on) {
        int v = 0;
#pragma unroll
        for (uint32_t k = 0; k < kEnergyRows; ++k) v += sh[y][k][x];
        if (y == 0) *ej = -v;
        else if (y == 1) *edel = v;
        else if (mag) *mag = v;
    }
}
__global__ void __launch_bounds__(32 * kEnergyRows) k_energies(const uint32_t *lat, int32_t *ej, int32_t *edel,
                                                               int32_t *mag, uint32_t L, uint32_t WPR, uint32_t cpb,
                                                               uint32_t nchains)
{
    const uint32_t chain = blockIdx.x * 32u + (threadIdx.x & 31u);
    const bool on = chain < nchains;
    const uint32_t c = on ? chain : 0u;
    chain_energies(lat + (size_t)(c / cpb) * L * WPR * cpb + c % cpb, L, WPR, cpb, on, ej + c, edel + c,
                   mag ? mag + c : nullptr);
}
// blockIdx.x = work item of a batch, blockIdx.y = 32 of its chains
__global__ void __launch_bounds__(32 * kEnergyRows) k_batch_energies(const BatchInst *__restrict__ insts,
                                                                     const BatchItem *__restrict__ items, uint32_t cpb)
{
    const BatchItem it = items[blockIdx.x];
    const SweepArgs &a = insts[it.inst].a;
    const uint32_t lane = blockIdx.y * 32u + (threadIdx.x & 31u), chain = it.blk * cpb + lane;
    const bool on = lane < cpb && chain < a.nchains;
    const uint32_t c = on ? chain : 0u;
    chain_energies(a.lat + (size_t)it.blk * a.L * a.WPR * cpb + (on ? lane : 0u), a.L, a.WPR, cpb, on, a.ej + c,
                   a.edel + c, a.mag + c);
}

__global__ void k_validate(const int8_t *src, size_t n, unsigned long long *bad)
{
    unsigned long long cnt = 0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int v = src[i];
        cnt += (v < -1 || v > 1);
    }
    if (cnt) atomicAdd(bad, cnt);
}

static unsigned grid_for(size_t total)
{
    size_t g = (total + 255) / 256;
    return (unsigned)(g > 65535 * 8 ? 65535 * 8 : (g ? g : 1));
}

cudaError_t launch_init(uint32_t *lat, uint32_t L, uint32_t WPR, uint32_t cpb, uint32_t nchains,
                        uint32_t chains_per_dev, uint32_t jack, const InitArgs &ia, cudaStream_t s)
{
    const size_t total = (size_t)((nchains + cpb - 1) / cpb) * cpb * L * WPR;
    if (ia.rounds == 10)
        k_init<10><<<grid_for(total), 256, 0, s>>>(lat, L, WPR, cpb, nchains, chains_per_dev, jack, ia);
    else
        k_init<7><<<grid_for(total), 256, 0, s>>>(lat, L, WPR, cpb, nchains, chains_per_dev, jack, ia);
    return cudaGetLastError();
}

cudaError_t launch_pack(uint32_t *lat, const int8_t *src, uint32_t L, uint32_t WPR, uint32_t cpb, uint32_t nchains,
                        cudaStream_t s)
{
    const size_t total = (size_t)((nchains + cpb - 1) / cpb) * cpb * L * WPR;
    k_pack<<<grid_for(total), 256, 0, s>>>(lat, src, L, WPR, cpb, nchains);
    return cudaGetLastError();
}

cudaError_t launch_unpack(const uint32_t *lat, int8_t *dst, uint32_t L, uint32_t WPR, uint32_t cpb,
                          uint32_t nchains, cudaStream_t s)
{
    const size_t total = (size_t)((nchains + cpb - 1) / cpb) * cpb * L * WPR;
    k_unpack<<<grid_for(total), 256, 0, s>>>(lat, dst, L, WPR, cpb, nchains);
    return cudaGetLastError();
}

cudaError_t launch_energies(const uint32_t *lat, int32_t *ej, int32_t *edel, int32_t *mag, uint32_t L, uint32_t WPR,
                            uint32_t cpb, uint32_t nchains, cudaStream_t s)
{
    k_energies<<<(nchains + 31) / 32, 32 * kEnergyRows, 0, s>>>(lat, ej, edel, mag, L, WPR, cpb, nchains);
    return cudaGetLastError();
}

cudaError_t launch_batch_init(const BatchInst *insts, const BatchItem *items, uint32_t n_items, uint32_t cpb,
                              const InitArgs &ia, cudaStream_t s)
{
    k_batch_init<<<dim3(n_items, 16), 256, 0, s>>>(insts, items, cpb, ia);
    k_batch_energies<<<dim3(n_items, (cpb + 31) / 32), 32 * kEnergyRows, 0, s>>>(insts, items, cpb);
    return cudaGetLastError();
}

cudaError_t launch_validate(const int8_t *src, size_t n, unsigned long long *bad, cudaStream_t s)
{
    k_validate<<<grid_for(n), 256, 0, s>>>(src, n, bad);
    return cudaGetLastError();
}

}  // namespace muca
