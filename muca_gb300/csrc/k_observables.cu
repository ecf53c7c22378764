// k_observables.cu -- production reweighting on the device, FP64.
//
// Replaces the host code of the reference production program that runs per
// Delta point: weight_shift (produce2_multigpu.cu:391-400), the Boltzmann
// factors boltz_j = exp(-beta*delta*j - lnW_j) (:297), the reweighting sums
// over the triangular (E_Delta, M) histogram (observables, :498-518; the
// reference sums in x87 long double on the host) and the jackknife
// (:520-535).  The triangle's row i (E_Delta = i) holds the i+1 bins
// m = -i, -i+2, ..., i at (i^2 + 2i + m)/2 = i(i+1)/2 + (m+i)/2.
//
// The sums stream the u64 histogram once (HBM bound at 8 B per bin), one
// warp per row, with exact integer moments per row (see row_moments);
// the per-row FP64 terms are combined per block and then in a fixed-order
// second pass, so the result is deterministic and agrees with
// the long-double host sum to ~1e-15.
#include "muca_device.cuh"
#include "muca_internal.h"

#include <algorithm>
#include <mutex>

namespace muca {

constexpr int kObsThreads = 512;
// One block for each of the 152 SMs of GB300, 16 warps with 32 loads of 256 B
// each in flight.  L = 128: 169 us a pass; 24 warps with 16 loads each 174.
constexpr int kObsBlocks = 152;
constexpr int kObsRows = 8;  // rows of a warp at most
static_assert(kObsBlocks * (kObsThreads / 32) * kObsRows >= 16385, "rows of the largest lattice");

__global__ void k_weight_shift(double *lnw, uint32_t N, double beta, double delta)
{
    __shared__ double sh[32];
    const double bd = __dmul_rn(beta, delta);
    double mx = -1.0 / 0.0;
    for (uint32_t i = threadIdx.x; i <= N; i += blockDim.x) {
        const double v = __dsub_rn(-lnw[i], __dmul_rn(bd, (double)i));
        mx = v > mx ? v : mx;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { const double t = __shfl_xor_sync(0xffffffffu, mx, o); mx = t > mx ? t : mx; }
    if (lane == 0) sh[wid] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = sh[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = sh[w] > m ? sh[w] : m;
        sh[0] = m;
    }
    __syncthreads();
    const double m = sh[0];
    for (uint32_t i = threadIdx.x; i <= N; i += blockDim.x) lnw[i] = __dadd_rn(lnw[i], m);
}

// One warp per row of the triangle at a time (row i = E_Delta holds the i+1
// bins m = -i, -i+2, ..., i from b = i(i+1)/2).  Within a row boltz_i is a
// common factor, so H, |m| H, m^2 H and m^4 H are summed exactly in integers
// (row_moments), and one FP64 product per row and moment follows.
//
// HBM bounds it: the histogram is read once.  To stay there a bin may cost
// about 44 issue cycles of a warp (152 SMs, 6.7 TB/s); with 128-bit products
// per bin it took 96.  So the moments are formed without a product:
//   * the bins of m and -m are folded, since every moment is one of |m|;
//   * lane l takes |m| = b + 64 k, b = (i & 1) + 2 l, for k = K-1 ... 0 and runs
//     five nested sums, c0 += G, c1 += c0, ... c4 += c3, which end as
//     e_p = sum_k C(k+p, p) G_k: ten additions for two bins;
//   * the sums of k^p G and of |m|^p G follow from them once per row.
// They are 64-bit: G < 2^30 and K <= 257 keep e4 <= 2^30 C(261, 5) < 2^64.  A
// row with a bin of 2^29 or more is summed again in two parts (row_moments_wide),
// and so are a warp's next rows from the start while they have such bins; both
// give the exact sums.
// L = 128 (1.07 GB): 169 us a pass (6.4 TB/s), 351 with products for every bin;
// every bin 2^30: 229 us, 351 with products at once, 997 with them after a first
// reading.
constexpr int kObsUnroll = 8;

typedef unsigned __int128 u128;

__device__ __forceinline__ u128 shfl_xor_u128(u128 v, int o)
{
    const unsigned long long lo = __shfl_xor_sync(0xffffffffu, (unsigned long long)v, o);
    const unsigned long long hi = __shfl_xor_sync(0xffffffffu, (unsigned long long)(v >> 64), o);
    return ((u128)hi << 64) | lo;
}

__device__ __forceinline__ double u128_to_double(u128 v)
{
    return __dadd_rn(__dmul_rn((double)(unsigned long long)(v >> 64), 18446744073709551616.0),
                     (double)(unsigned long long)v);
}

// A sum of terms >= 0 with the error of its additions beside it (the larger
// operand first, so three operations give it): chi subtracts <m>^2 from <m^2>,
// which magnifies what the sums lose to rounding.
struct DoubleSum {
    double h = 0.0, l = 0.0;
    __device__ __forceinline__ void add(double x)
    {
        const bool swap = __double_as_longlong(h) < __double_as_longlong(x);
        const double a = swap ? x : h, b = swap ? h : x, t = __dadd_rn(a, b);
        l = __dadd_rn(l, __dsub_rn(b, __dsub_rn(t, a)));
        h = t;
    }
    __device__ __forceinline__ void join_xor(int o)
    {
        const double oh = __shfl_xor_sync(0xffffffffu, h, o), ol = __shfl_xor_sync(0xffffffffu, l, o);
        l = __dadd_rn(l, ol);
        add(oh);
    }
    // (of an overflowed sum the error is a NaN)
    __device__ __forceinline__ double value() const { return l == l ? __dadd_rn(h, l) : h; }
};

struct RowMoments {
    u128 a0, a1, a2, a4;  // sums of H, |m| H, m^2 H, m^4 H
};

// The moments from nested sums: s_p = sum_k k^p G_k from C(k+1,1) = k + 1,
// 2 C(k+2,2) = k^2 + 3k + 2, 6 C(k+3,3) = k^3 + 6k^2 + 11k + 6 and
// 24 C(k+4,4) = k^4 + 10k^3 + 35k^2 + 50k + 24, then (b + 64 k)^p term by term.
__device__ __noinline__ RowMoments moments_of_nested(u128 c0, u128 c1, u128 c2, u128 c3, u128 c4, uint32_t b)
{
    const u128 s1 = c1 - c0, s2 = 2 * c2 - 3 * s1 - 2 * c0, s3 = 6 * c3 - 6 * s2 - 11 * s1 - 6 * c0;
    const u128 s4 = 24 * c4 - 10 * s3 - 35 * s2 - 50 * s1 - 24 * c0;
    const uint32_t b2 = b * b;  // b <= 63
    RowMoments r;
    r.a0 = c0;
    r.a1 = c0 * b + s1 * 64u;
    r.a2 = c0 * b2 + s1 * (128u * b) + s2 * 4096u;
    r.a4 = c0 * (b2 * b2) + s1 * (256u * b2 * b) + s2 * (24576u * b2) + s3 * (1048576u * b) + (s4 << 24);
    return r;
}

// A lane's part of row i with bins of any size: the nested sums of their low 29
// bits and of the rest beside each other (the rest is below 2^35, so its fourth
// sum may reach 2^70 and takes 96 bits).  Twice the additions keep it near HBM's
// pace where a 128-bit product per bin did not; `big`: some bin needs it.
__device__ __forceinline__ RowMoments row_moments_wide(const unsigned long long *row, uint32_t i, uint32_t lane,
                                                       bool &big)
{
    typedef unsigned long long u64;
    const uint32_t half = i / 2 + 1;
    const u64 *up = row + (i + 1) / 2, *dn = row + i / 2;
    constexpr int U = kObsUnroll / 2;
    constexpr uint32_t low = (1u << 29) - 1u;
    int k = (int)((half + 32u * U - 1) / (32u * U)) * U - 1;
    u64 hu[U], hd[U], nu[U], ndn[U];
    auto load = [&](int k0, u64 (&a)[U], u64 (&b)[U]) {
#pragma unroll
        for (int t = 0; t < U; ++t) {
            const uint32_t n = lane + 32u * (uint32_t)(k0 - t);
            const bool in = k0 - t >= 0 && n < half;
            a[t] = in ? __ldcs(up + n) : 0ull;
            b[t] = in ? __ldcs(dn - (int)n) : 0ull;
        }
    };
    load(k, hu, hd);
    u64 c0 = 0, c1 = 0, c2 = 0, c3 = 0, c4 = 0, g0 = 0, g1 = 0, g2 = 0, g3 = 0, g4 = 0;
    uint32_t g5 = 0;
    for (; k >= 0; k -= U) {
        load(k - U, nu, ndn);
#pragma unroll
        for (int t = 0; t < U; ++t) {
            c0 += ((uint32_t)hu[t] & low) + ((uint32_t)hd[t] & low);
            c1 += c0;
            c2 += c1;
            c3 += c2;
            c4 += c3;
            g0 += (hu[t] >> 29) + (hd[t] >> 29);
            g1 += g0;
            g2 += g1;
            g3 += g2;
            g4 += g3;
            g5 += g4 < g3;
        }
#pragma unroll
        for (int t = 0; t < U; ++t) {
            hu[t] = nu[t];
            hd[t] = ndn[t];
        }
    }
    big = g0 != 0;
    u128 g4w = ((u128)g5 << 64) | g4;
    if ((i & 1u) == 0 && lane == 0) {
        // the bin m = 0 was folded with itself
        const u64 z = *dn & low, y = *dn >> 29;
        c0 -= z;
        c1 -= z;
        c2 -= z;
        c3 -= z;
        c4 -= z;
        g0 -= y;
        g1 -= y;
        g2 -= y;
        g3 -= y;
        g4w -= y;
    }
    const uint32_t b = (i & 1u) + 2u * lane;
    RowMoments r = moments_of_nested(c0, c1, c2, c3, c4, b);
    const RowMoments q = moments_of_nested(g0, g1, g2, g3, g4w, b);
    r.a0 += q.a0 << 29;
    r.a1 += q.a1 << 29;
    r.a2 += q.a2 << 29;
    r.a4 += q.a4 << 29;
    return r;
}

// A lane's part of row i by nested sums (above); bins from 2^29 are reported in
// `big` (the sums are then wrong).
__device__ __forceinline__ RowMoments row_moments(const unsigned long long *row, uint32_t i, uint32_t lane, bool &big)
{
    typedef unsigned long long u64;
    // |m| = (i & 1) + 2 n, n = 0 .. i/2: bins (i+1)/2 + n and i/2 - n
    const uint32_t half = i / 2 + 1;
    const u64 *up = row + (i + 1) / 2, *dn = row + i / 2;
    constexpr int U = kObsUnroll;
    int k = (int)((half + 32u * U - 1) / (32u * U)) * U - 1;  // K - 1, K a multiple of U
    u64 hu[U], hd[U], nu[U], ndn[U];
    auto load = [&](int k0, u64 (&a)[U], u64 (&b)[U]) {
#pragma unroll
        for (int t = 0; t < U; ++t) {
            const uint32_t n = lane + 32u * (uint32_t)(k0 - t);
            const bool in = k0 - t >= 0 && n < half;
            a[t] = in ? __ldcs(up + n) : 0ull;
            b[t] = in ? __ldcs(dn - (int)n) : 0ull;
        }
    };
    load(k, hu, hd);
    u64 c0 = 0, c1 = 0, c2 = 0, c3 = 0, c4 = 0;
    uint32_t any_hi = 0, any_lo = 0;
    for (; k >= 0; k -= U) {
        load(k - U, nu, ndn);
#pragma unroll
        for (int t = 0; t < U; ++t) {
            any_hi |= (uint32_t)(hu[t] >> 32) | (uint32_t)(hd[t] >> 32);
            any_lo |= (uint32_t)hu[t] | (uint32_t)hd[t];
            c0 += (uint32_t)hu[t] + (uint32_t)hd[t];
            c1 += c0;
            c2 += c1;
            c3 += c2;
            c4 += c3;
        }
#pragma unroll
        for (int t = 0; t < U; ++t) {
            hu[t] = nu[t];
            hd[t] = ndn[t];
        }
    }
    big = any_hi != 0 || (any_lo >> 29) != 0;
    if ((i & 1u) == 0 && lane == 0) {
        // the bin m = 0 was folded with itself
        const u64 z = *dn;
        c0 -= z;
        c1 -= z;
        c2 -= z;
        c3 -= z;
        c4 -= z;
    }
    // as moments_of_nested, in 64 bits where they suffice
    const u64 s1 = c1 - c0, s2 = 2 * c2 - 3 * s1 - 2 * c0, s3 = 6 * c3 - 6 * s2 - 11 * s1 - 6 * c0;
    const u128 s4 = (u128)c4 * 24u - (u128)s3 * 10u - (u128)s2 * 35u - (u128)s1 * 50u - (u128)c0 * 24u;
    const uint32_t b = (i & 1u) + 2u * lane, b2 = b * b;  // <= 63
    RowMoments r;
    r.a0 = c0;
    r.a1 = (u64)b * c0 + 64u * s1;  // < 2^52
    r.a2 = (u128)c0 * b2 + (u128)s1 * (128u * b) + (u128)s2 * 4096u;
    r.a4 = (u128)c0 * (b2 * b2) + (u128)s1 * (256u * b2 * b) + (u128)s2 * (24576u * b2) + (u128)s3 * (1048576u * b) +
           (s4 << 24);
    return r;
}

__global__ void __launch_bounds__(kObsThreads, 1) k_observables(const unsigned long long *__restrict__ hist,
                                                             const double *__restrict__ lnw, uint32_t N,
                                                             double beta, double delta,
                                                             double *__restrict__ partials)
{
    const double nbd = __dmul_rn(-beta, delta);
    const uint32_t ln = threadIdx.x & 31u;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5, w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    // Warp w takes the w-th longest row, then that many from the other end of
    // the next nwarps rows, and so on, so that all warps read about as much.
    // Lane s keeps the s-th row's sums: FP64 issues slowly on this GPU, so the
    // terms of all rows are formed at once.
    uint32_t first = 0, slot = 0, my_row = 0;
    RowMoments mine{0, 0, 0, 0};
    bool turn = false;
    bool wide = false;  // (uniform) the last row had bins of 2^29 or more
    while (first <= N) {
        const uint32_t at = first + (turn ? nwarps - 1u - w : w);
        if (at <= N) {
            const uint32_t i = N - at;
            const unsigned long long *row = hist + (unsigned long long)i * (i + 1) / 2;
            bool big = false;
            RowMoments r;
            if (!wide) {
                r = row_moments(row, i, ln, big);
                wide = __any_sync(0xffffffffu, big);
                if (wide) r = row_moments_wide(row, i, ln, big);
            } else {
                r = row_moments_wide(row, i, ln, big);
                wide = __any_sync(0xffffffffu, big);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                r.a0 += shfl_xor_u128(r.a0, o);
                r.a1 += shfl_xor_u128(r.a1, o);
                r.a2 += shfl_xor_u128(r.a2, o);
                r.a4 += shfl_xor_u128(r.a4, o);
            }
            if (ln == slot) {
                mine = r;
                my_row = i;
            }
            ++slot;
        }
        first += nwarps;
        turn = !turn;
    }
    __shared__ double terms[4][kObsThreads / 32][kObsRows];
    if (ln < (uint32_t)kObsRows) {
        double t0 = 0.0, t1 = 0.0, t2 = 0.0, t4 = 0.0;
        if (ln < slot && mine.a0 != 0) {
            const double bz = exp(__dsub_rn(__dmul_rn(nbd, (double)my_row), lnw[my_row]));
            t0 = __dmul_rn(u128_to_double(mine.a0), bz);
            t1 = __dmul_rn(u128_to_double(mine.a1), bz);
            t2 = __dmul_rn(u128_to_double(mine.a2), bz);
            t4 = __dmul_rn(u128_to_double(mine.a4), bz);
        }
        const uint32_t wid = threadIdx.x >> 5;
        terms[0][wid][ln] = t0;
        terms[1][wid][ln] = t1;
        terms[2][wid][ln] = t2;
        terms[3][wid][ln] = t4;
    }
    __syncthreads();
    if (threadIdx.x < 128) {
        const uint32_t q = threadIdx.x >> 5;
        const double *of_q = &terms[q][0][0];
        DoubleSum v;
#pragma unroll
        for (int k = 0; k < kObsThreads / 32 * kObsRows; k += 32) v.add(of_q[k + ln]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v.join_xor(o);
        if (ln == 0) partials[(size_t)blockIdx.x * 4 + q] = v.value();
    }
}

// Warp q sums the blocks' partials of moment q.  (An FP64 instruction takes a
// warp 64 cycles here, so the partials are few: one block per SM.)
__global__ void k_observables_final(const double *partials, int nblocks, double *out)
{
    const uint32_t q = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    DoubleSum v;
    for (int b = (int)lane; b < nblocks; b += 32) v.add(partials[(size_t)b * 4 + q]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v.join_xor(o);
    if (lane == 0) out[q] = v.value();
}

// jakknife (muca_delta_multigpu.cu:620-635), one thread, same order.
__global__ void k_jackknife(const double *x, uint32_t J, double *out)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double avg = 0;
    for (uint32_t i = 0; i < J; i++) avg += x[i];
    const double total = avg;
    avg = avg / (double)J;
    double dev = 0;
    for (uint32_t i = 0; i < J; i++) {
        const double mi = (total - x[i]) / (double)(J - 1);
        dev += (avg - mi) * (avg - mi);
    }
    dev = (double)(J - 1) * dev / (double)J;
    out[0] = avg;
    out[1] = sqrt(dev);
}

cudaError_t launch_weight_shift(double *lnw, uint32_t N, double beta, double delta, cudaStream_t s)
{
    k_weight_shift<<<1, 1024, 0, s>>>(lnw, N, beta, delta);
    return cudaGetLastError();
}

size_t observables_partials(uint32_t) { return (size_t)kObsBlocks * 4; }

cudaError_t launch_observables(const unsigned long long *hist2d, const double *lnw, uint32_t N, double beta,
                               double delta, double *partials, double *out, cudaStream_t s)
{
    // no more warps than rows
    const int blocks = std::min(kObsBlocks, (int)(N / (kObsThreads / 32)) + 1);
    k_observables<<<blocks, kObsThreads, 0, s>>>(hist2d, lnw, N, beta, delta, partials);
    k_observables_final<<<1, 128, 0, s>>>(partials, blocks, out);
    return cudaGetLastError();
}

cudaError_t launch_jackknife(const double *x, uint32_t n, double *out2, cudaStream_t s)
{
    k_jackknife<<<1, 32, 0, s>>>(x, n, out2);
    return cudaGetLastError();
}

// ---- the reweighting sums without any allocation ------------------------
//
// Some callers cannot let this library allocate device memory.  Example: a
// scheduler that packs many production instances into a fixed HBM budget
// through its own pool, where a hidden cudaMalloc would break the budget and
// also synchronise the device under the scheduler's other streams.  Another:
// a process that only reweights histograms it already holds on the device.
// It has no lattice and so no engine context, whose creation allocates.  For
// them, the two kernels above run with their block partials in the
// file-scope array below instead of context memory.
//
// The array holds the partials of the largest grid, kObsBlocks blocks:
// kObsBlocks x 4 doubles (4,864 bytes), whatever L is.  Each block
// overwrites its own four entries before the final pass reads them, so
// nothing in it has to start at zero, and no state carries from one call to
// the next.  There is one array per device, shared by every caller in the
// process: two calls in flight at once on the same device (two streams, or
// two host threads) write the same entries and race.
constexpr size_t kStaticPartials = (size_t)kObsBlocks * 4;
static __device__ __align__(256) double g_obs_partials[kStaticPartials];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_partials_mu;
double *g_partials_addr[kMaxDevices] = {};
}  // namespace

size_t observables_static_partials() { return kStaticPartials; }

cudaError_t launch_observables_static(int device, const unsigned long long *hist2d, const double *lnw, uint32_t N,
                                      double beta, double delta, double *out, cudaStream_t s)
{
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    if (observables_partials(N) > kStaticPartials) return cudaErrorInvalidValue;
    double *partials = nullptr;
    {
        // The address is resolved once per device, with that device current
        // (the caller has made it current).  The first resolution may load
        // this module onto the device.
        std::lock_guard<std::mutex> lock(g_partials_mu);
        if (!g_partials_addr[device]) {
            void *p = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&p, g_obs_partials);
            if (e != cudaSuccess) return e;
            g_partials_addr[device] = static_cast<double *>(p);
        }
        partials = g_partials_addr[device];
    }
    return launch_observables(hist2d, lnw, N, beta, delta, partials, out, s);
}

}  // namespace muca
