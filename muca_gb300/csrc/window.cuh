// window.cuh -- the lean window of the sweep: the draws, the proposals and
// the accept/reject scan of the (up to 8) same-parity sites of one 16-site
// word of one row, and the walk of a chain block over the reference's sweep
// order (k_sweep.cu, k_batch.cu).
//
// What bounds a window is the ALU pipe (16 lanes per SM sub-partition: a warp
// instruction every two cycles) at one warp per sub-partition, so the window
// is written for few ALU instructions:
//   * of a Philox block's rounds the first two keep only what varies.  The
//     counter is {cc, seed, iter, tag}: the product of cc and the one that
//     follows it depend on the launch alone, the other two on the chain
//     alone, so a block of R rounds costs 2 (R - 2) products;
//   * a site's code and direction form a 3-bit nibble, four of which are a
//     byte-permute selector: the byte tables below turn four attempts into
//     their proposed moves with one instruction;
//   * a byte becomes a float by a permute into the mantissa of 2^23 and one
//     subtraction (FMA pipe); -beta dE is formed inside the addition that
//     needs it, fma(s_new - s_old, beta * neighbour sum, w), whose product is
//     exact, so the sum is rounded once as the reference's is;
//   * E_J runs as a float on the FMA pipe (2 E_J is an integer below 2^24).
// Decisions are those of the reference: the scan decides on a fast logarithm
// and replays the window with logf (and in production with FP64 weights)
// where that could differ, see scan_weight and scan_produce.
#pragma once
#include "sweep_core.cuh"

#include <cmath>
#include <type_traits>

namespace muca {

// Dynamic shared memory in front of a windowed block's lattice: the FP32
// weights (production: their differences) and, in weight mode with the
// histogram in shared memory, its u32 bins.
__host__ __device__ inline size_t win_smem_base(int mode, uint32_t N, bool hist_smem)
{
    return align16((size_t)(N + 1) * 4) * (mode == kModeWeight && hist_smem ? 2 : 1);
}

// The uniform u01f(r) with its mantissa taken by one funnel shift:
// (0x7F : r) >> 9 is 0x3F800000 | (r >> 9).
__device__ __forceinline__ float u01s(uint32_t r)
{
    return __fsub_rn(__uint_as_float(__funnelshift_r(r, 0x7Fu, 9)), __uint_as_float(0x3F7FFFFFu));
}

template <uint32_t SEL>
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "n"(SEL));
    return d;
}
__device__ __forceinline__ uint32_t prmt_var(uint32_t a, uint32_t b, uint32_t sel)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
// byte I of x as a signed integer (permute with sign replication)
template <int I>
__device__ __forceinline__ int sbyte(uint32_t x)
{
    return (int)prmt<(uint32_t)I | (8u + I) << 4 | (8u + I) << 8 | (8u + I) << 12>(x, x);
}
// 2^23 + byte I of x, as a float
template <int I>
__device__ __forceinline__ float magic_byte(uint32_t x)
{
    return __uint_as_float(prmt<0x7540u + (uint32_t)I>(x, 0x4B000000u));
}

// ---------------------------------------------------------------------------
// The two Philox streams of a chain.  With x = {cc, seed, iter, tag} and key
// {k0, khi}, round 1 gives
//   x0' = hi(M1 iter) ^ seed ^ k0,  x1' = lo(M1 iter),
//   x2' = hi(M0 cc) ^ tag ^ khi,    x3' = lo(M0 cc),
// of which x0', x1' are constants of the chain, x2', x3' the same for every
// chain; so in round 2 the products M0 x0' (chain) and M1 x2' (all chains)
// are not formed per chain and group either.
template <int R>
struct Stream {
    uint32_t a2, h, l;      // (k0 + W0) ^ lo(M1 iter); hi(M0 x0') ^ (khi + W1); lo(M0 x0')
    uint32_t khi;           // key word 1 (the same for every chain)
    uint32_t ka[R - 2];     // key word 0 of rounds 3..R
    __device__ __forceinline__ void init(uint32_t k0, uint32_t k1, uint32_t seed, uint32_t iter)
    {
        const uint32_t x0 = __umulhi(kPhiloxM1, iter) ^ seed ^ k0;
        khi = k1;
        a2 = (k0 + kPhiloxW0) ^ (kPhiloxM1 * iter);
        h = __umulhi(kPhiloxM0, x0) ^ (k1 + kPhiloxW1);
        l = kPhiloxM0 * x0;
#pragma unroll
        for (int r = 2; r < R; ++r) ka[r - 2] = k0 + (uint32_t)r * kPhiloxW0;
    }
    // the block of counter word cc, given q = M0 cc
    __device__ __forceinline__ void block(unsigned long long q, uint32_t *out) const
    {
        const unsigned long long p = (unsigned long long)kPhiloxM1 * ((uint32_t)(q >> 32) ^ kCtrTag ^ khi);
        uint32_t x0 = (uint32_t)(p >> 32) ^ a2, x1 = (uint32_t)p, x2 = h ^ (uint32_t)q, x3 = l;
#pragma unroll
        for (int r = 2; r < R; ++r) {
            const unsigned long long p0 = (unsigned long long)kPhiloxM0 * x0;
            const unsigned long long p1 = (unsigned long long)kPhiloxM1 * x2;
            x0 = (uint32_t)(p1 >> 32) ^ x1 ^ ka[r - 2];
            x1 = (uint32_t)p1;
            x2 = (uint32_t)(p0 >> 32) ^ x3 ^ (khi + (uint32_t)r * kPhiloxW1);
            x3 = (uint32_t)p0;
        }
        out[0] = x0; out[1] = x1; out[2] = x2; out[3] = x3;
    }
};
template <int R>
struct Draws {
    Stream<R> s1, s3;  // acceptance, direction
    // ln 2, the factor of the binary logarithm of u; -infinity in lanes
    // without a chain: their logarithm is then +infinity (or, of 0, a NaN) and
    // they never accept, with no test of their own on the chain of decisions
    // (one cost 22 cycles per attempt)
    float ln2;
    __device__ __forceinline__ float log_u(uint32_t r) const { return __fmul_rn(lg2_ftz(u01s(r)), ln2); }
    __device__ __forceinline__ void group(uint32_t cc, uint32_t *r1, uint32_t *r3) const
    {
        const unsigned long long q = (unsigned long long)kPhiloxM0 * cc;
        s1.block(q, r1);
        s3.block(q, r3);
    }
};

// The acceptance logarithms and direction nibbles of eight attempts (two
// groups), drawn one window ahead of the scan.
struct Ahead {
    float l[8];
    uint32_t dn;
};
// nibble t of the result: the direction bit (top bit) of r3[t]
__device__ __forceinline__ uint32_t direction4(const uint32_t *r3)
{
    const uint32_t a = prmt<0x0073>(r3[0], r3[2]), b = prmt<0x0073>(r3[1], r3[3]);
    return ((a >> 7) & 0x0101u) | ((b >> 3) & 0x1010u);
}
__device__ __forceinline__ uint32_t direction8(const uint32_t *r3)
{
    const uint32_t a = prmt<0x5410>(prmt<0x0073>(r3[0], r3[2]), prmt<0x0073>(r3[4], r3[6]));
    const uint32_t b = prmt<0x5410>(prmt<0x0073>(r3[1], r3[3]), prmt<0x0073>(r3[5], r3[7]));
    return ((a >> 7) & 0x01010101u) | ((b >> 3) & 0x10101010u);
}
// groups c and c + 1
template <int R>
__device__ __forceinline__ void draw8(const Draws<R> &d, uint32_t c, Ahead &a)
{
    uint32_t r1[8], r3[8];
    d.group(c, r1, r3);
    d.group(c + 1, r1 + 4, r3 + 4);
    a.dn = direction8(r3);
#pragma unroll
    for (int t = 0; t < 8; ++t) a.l[t] = d.log_u(r1[t]);
}
// the second group moves up and group c follows it
template <int R>
__device__ __forceinline__ void draw4(const Draws<R> &d, uint32_t c, Ahead &a)
{
    uint32_t r1[4], r3[4];
    d.group(c, r1, r3);
    a.dn = (a.dn >> 16) | (direction4(r3) << 16);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        a.l[t] = a.l[t + 4];
        a.l[t + 4] = d.log_u(r1[t]);
    }
}

// The same for rows whose attempts do not come in whole groups: three groups
// c - 2 .. c, of whose attempts the first `off` (0..3) are used up.
struct AheadAny {
    float l[12];
    unsigned long long dn;
    uint32_t off;
};
// drops the first group, draws group c
template <int R>
__device__ __forceinline__ void shift_in(const Draws<R> &d, uint32_t c, AheadAny &a)
{
    uint32_t r1[4], r3[4];
    d.group(c, r1, r3);
#pragma unroll
    for (int t = 0; t < 8; ++t) a.l[t] = a.l[t + 4];
#pragma unroll
    for (int t = 0; t < 4; ++t) a.l[t + 8] = d.log_u(r1[t]);
    a.dn = (a.dn >> 16) | ((unsigned long long)direction4(r3) << 32);
}
// the next eight attempts
__device__ __forceinline__ Ahead next8(const AheadAny &a)
{
    Ahead x;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const float x0 = (a.off & 1u) ? a.l[t + 1] : a.l[t], x2 = (a.off & 1u) ? a.l[t + 3] : a.l[t + 2];
        x.l[t] = (a.off & 2u) ? x2 : x0;
    }
    x.dn = (uint32_t)(a.dn >> (4u * a.off)) & 0x11111111u;
    return x;
}

// ---------------------------------------------------------------------------
// Draws from another warp.  With no more chains than fill two of an SM's four
// sub-partitions the idle ones draw: a warp per 32 chains writes their groups
// into a ring in shared memory, and the warp that walks reads them.  Draws do
// not depend on the lattice, so the two meet only once per kFeedGroups groups,
// at a named barrier of the 64 threads that both sides pass equally often
// (feed_halves).  Cycles per attempt at L = 72, 4000 chains: 70.5 and 76.1
// (thermalising and recording) for 90.7 and 94.6 in one warp; production 80.5
// and 137 for 95.6 and 150.  Halves of 8 groups: 72.1; two drawing warps for
// one: no gain.
constexpr uint32_t kFeedGroups = 16, kFeedSlots = 2 * kFeedGroups;  // a half of the ring; the ring
constexpr uint32_t kFeedLogs = kFeedSlots * 32 * 16, kFeedBytes = kFeedLogs + kFeedSlots * 32 * 4;  // per warp
// halves drawn and read in a launch: the groups of both phases and two ahead
__device__ __forceinline__ unsigned long long feed_halves(unsigned long long therm, unsigned long long nup)
{
    return ((therm + 3ull) / 4ull + (nup + 3ull) / 4ull + 2ull + kFeedGroups - 1ull) / kFeedGroups;
}
__device__ __forceinline__ void named_sync(uint32_t id, uint32_t threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void named_arrive(uint32_t id, uint32_t threads)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// the drawing warp
template <int R>
__device__ __forceinline__ void feed_draw(const Draws<R> &d, unsigned char *ring, uint32_t lane, uint32_t bar,
                                          unsigned long long halves)
{
    for (unsigned long long t = 0; t < halves; ++t) {
        const uint32_t h = (uint32_t)t & 1u;
        if (t >= 2ull) named_sync(bar + 2u + h, 64u);
        float4 *logs = reinterpret_cast<float4 *>(ring) + h * kFeedGroups * 32u + lane;
        uint32_t *dirs = reinterpret_cast<uint32_t *>(ring + kFeedLogs) + h * kFeedGroups * 32u + lane;
        const uint32_t c = (uint32_t)t * kFeedGroups + 1u;
#pragma unroll 2
        for (uint32_t g = 0; g < kFeedGroups; ++g) {
            uint32_t r1[4], r3[4];
            d.group(c + g, r1, r3);
            logs[g * 32u] = make_float4(d.log_u(r1[0]), d.log_u(r1[1]), d.log_u(r1[2]), d.log_u(r1[3]));
            dirs[g * 32u] = direction4(r3);
        }
        named_arrive(bar + h, 64u);
    }
}
// the reader's side
struct Feed {
    const unsigned char *ring;  // this lane's
    uint32_t bar, b, off;       // first group of the coming window (from 0) and its attempts used up
    uint32_t ev, avail;         // the next event; groups that may be read
    unsigned long long t, halves;
    bool rel;                   // the next event gives a half back
    __device__ __forceinline__ void init(const unsigned char *r, uint32_t lane, uint32_t id, unsigned long long n)
    {
        ring = r + 16u * lane;
        bar = id;
        b = off = ev = avail = 0;
        t = 0;
        halves = n;
        rel = false;
    }
    // before the groups of the window at (b, off) are read: up to three from b
    template <bool ALIGNED>
    __device__ __forceinline__ void ready()
    {
        const uint32_t end = b + (ALIGNED || off == 0 ? 2u : 3u);
        if ((int32_t)(end - ev) > 0) {  // uniform
            __syncwarp();
            if (rel) {
                // every group before end - 3 has been read: half t - 2, which
                // the producer waits for if it has a half t to draw
                if (t < halves) named_arrive(bar + 2u + ((uint32_t)t & 1u), 64u);
                rel = false;
                ev = avail;
            } else {
                named_sync(bar + ((uint32_t)t & 1u), 64u);
                rel = t > 0;
                ev = rel ? avail + 2u : kFeedGroups;
                avail += kFeedGroups;
                ++t;
            }
        }
    }
    template <bool ALIGNED>
    __device__ __forceinline__ void read(Ahead &a) const
    {
        const uint32_t s0 = b % kFeedSlots, s1 = (b + 1u) % kFeedSlots;
        const unsigned char *dirs = ring + kFeedLogs - 12u * (threadIdx.x & 31u);
        auto dir = [&](uint32_t s) { return *reinterpret_cast<const uint32_t *>(dirs + s * 128u); };
        const uint32_t d = dir(s0) | dir(s1) << 16;
        if (ALIGNED) {
            const float4 x = *reinterpret_cast<const float4 *>(ring + s0 * 512u);
            const float4 y = *reinterpret_cast<const float4 *>(ring + s1 * 512u);
            a.l[0] = x.x; a.l[1] = x.y; a.l[2] = x.z; a.l[3] = x.w;
            a.l[4] = y.x; a.l[5] = y.y; a.l[6] = y.z; a.l[7] = y.w;
            a.dn = d;
        } else {
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const uint32_t k = (b % kFeedSlots) * 4u + off + i;
                a.l[i] = *reinterpret_cast<const float *>(ring + (k / 4u % kFeedSlots) * 512u + k % 4u * 4u);
            }
            // the third group only where it is used (and so drawn, see ready)
            a.dn = __funnelshift_r(d, off ? dir((b + 2u) % kFeedSlots) : 0u, 4u * off) & 0x11111111u;
        }
    }
};
// flush_hist by the block's first `threads` threads
__device__ __forceinline__ void flush_hist_of(uint32_t *histS, unsigned long long *histG, uint32_t N, uint32_t threads)
{
    named_sync(15u, threads);
    for (uint32_t b = threadIdx.x; b <= N; b += threads) {
        const uint32_t v = histS[b];
        if (v) {
            atomicAdd(&histG[b], (unsigned long long)v);
            histS[b] = 0;
        }
    }
    named_sync(15u, threads);
}

// Tables over the 3-bit code (s + 1) | direction << 2, direction 0: s + 1,
// 1: s - 1 (cyclic): codes 0, 1, 2 and 4, 5, 6 (3 and 7 do not occur).
//   code   s -> s_new   dDel   s_new - s_old
//   0     -1 ->  0       -1     +1
//   1      0 -> +1       +1     +1
//   2     +1 -> -1        0     -2
//   4     -1 -> +1        0     +2
//   5      0 -> -1       +1     -1
//   6     +1 ->  0       -1     -1
constexpr uint32_t kTabDD4_0 = 0x000004FCu, kTabDD4_1 = 0x00FC0400u;   // 4 dDel (signed bytes)
constexpr uint32_t kTabDV_0 = 0x00000303u, kTabDV_1 = 0x00010104u;     // s_new - s_old + 2
// production: byte offset of the weight difference an attempt needs,
// u[E] = w[E+1] - w[E] for dDel = +1, u[E-1] for dDel = -1 (any for 0)
constexpr uint32_t kTabUO_0 = 0x000000FCu, kTabUO_1 = 0x00FC0000u;
constexpr uint32_t kTabDD_0 = 0x00010200u, kTabDD_1 = 0x00000201u;     // dDel + 1
// (E_Delta, M) bin: b' - b = dDel E + k, in bytes of u64 bins 2 dDel (4 E) + 8 k
constexpr uint32_t kTabD2_0 = 0x000002FEu, kTabD2_1 = 0x00FE0200u;     // 2 dDel
constexpr uint32_t kTabK8_0 = 0x00F81000u, kTabK8_1 = 0x00F80808u;     // 8 k

// A window ready for its scan.  S slots; slot t's byte quantities are byte
// t % 4 of word t / 4 of the tables' results.
template <int S>
struct Win {
    uint32_t ctr, vnib;  // old and proposed codes (nibbles)
    uint32_t code[2];    // the 3-bit codes of slots 0..3 and 4..7 as permute selectors
    float ns2[S];        // beta * neighbour spin sum (2 ns for beta = 2; the table's value with BT)
    float dv[S];         // s_new - s_old
    float l[S];          // fast_logf(u)
};

constexpr uint32_t kBetaTab = 26;  // entries of a beta table (see win_sweep_block)

template <int S, int T = 0, typename F>
__device__ __forceinline__ void unrolled(const F &f)
{
    if constexpr (T < S) {
        f(std::integral_constant<int, T>{});
        unrolled<S, T + 1>(f);
    }
}

// HALF 0: the even sites of word C, `side` = the word to its left (site 15
// in the top bits); HALF 1: the odd sites, `side` = the word to its right.
// For a 4-slot window side's site lies where the row's next site would be
// (decode is given C with that site merged in).  BT: ns2 from the table
// btab[17 + neighbour code sum] instead of 2 ns.
template <int S, int HALF, bool BT>
__device__ __forceinline__ void decode(uint32_t C, uint32_t U, uint32_t D, uint32_t side, const Ahead &a,
                                       const float *btab, Win<S> &w)
{
    constexpr uint32_t M2 = 0x33333333u, N1 = 0x11111111u, B4 = 0x0F0F0F0Fu;
    uint32_t nbs;
    if (HALF == 0) {
        w.ctr = C & M2;
        nbs = ((C >> 2) & M2) + (__funnelshift_l(side, C, 2) & M2) + (U & M2) + (D & M2);
    } else {
        w.ctr = (C >> 2) & M2;
        nbs = (C & M2) + (__funnelshift_r(C, side, 4) & M2) + ((U >> 2) & M2) + ((D >> 2) & M2);
    }
    const uint32_t dn = a.dn;
    const uint32_t x = w.ctr + N1 + dn;            // 1..4
    const uint32_t ge3 = ((x + N1) >> 2) & N1;     // 1 where x >= 3
    w.vnib = x - 3u * ge3;
    const uint32_t code = w.ctr + 4u * dn;
    w.code[0] = code;
    w.code[1] = code >> 16;
    const uint32_t nb[2] = {nbs & B4, (nbs >> 4) & B4};  // even and odd slots
    uint32_t dvb[2];
    dvb[0] = prmt_var(kTabDV_0, kTabDV_1, w.code[0]);
    dvb[1] = S > 4 ? prmt_var(kTabDV_0, kTabDV_1, w.code[1]) : 0u;
    unrolled<S>([&](auto tc) {
        constexpr int t = decltype(tc)::value;
        w.dv[t] = __fsub_rn(magic_byte<(t & 3)>(dvb[t >> 2]), 8388610.0f);
        if (BT)
            w.ns2[t] = btab[17u + prmt<0x4440u + (t >> 1)>(nb[t & 1], 0u)];
        else
            w.ns2[t] = __fmaf_rn(magic_byte<(t >> 1)>(nb[t & 1]), 2.0f, -16777224.0f);
        w.l[t] = a.l[t];
    });
}

// A chain's running state in a weight-mode walk: the byte offset of its bin
// in the staged weights, that weight, and 2 E_J.
struct WState {
    uint32_t e4;
    float wE, ej2;
};

// x += c if p: a predicated addition costs one issue slot where a select costs
// two (it issues on the half-rate ALU pipe)
__device__ __forceinline__ void add_if(bool p, uint32_t &x, uint32_t c)
{
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p add.u32 %0, %0, %1;\n\t}"
        : "+r"(x)
        : "r"(c), "r"((uint32_t)p));
}

// The accept/reject scan of weight mode over E_Delta:
//   accept  <=>  diff >= 0 || logf(u) < diff,
//   diff = fl(fl(-beta dE + w[E + dDel]) - w[E])   (muca_delta_multigpu.cu:810-816),
// which is logf(u) < diff, since logf(u) < 0 for every u <= 1 - 2^-24.  The
// scan decides with fast_logf; where that lies within eps of diff in any lane
// the window is replayed with logf.
// At one warp per SM sub-partition the chain of one decision to the next is
// kept to a select and a compare: both values diff can take (the attempt
// before rejected or accepted) are formed from weights loaded one attempt
// ahead.  With several warps (MANY) the load waits for the decision: the other
// warps fill its latency, and an attempt takes eight instructions fewer (L=72,
// 311296 chains: 6.20 ms with both values formed ahead, 5.88 ms without; one
// warp: 0.62 and 0.68 ms).
// len: the attempts that take place (a masked window's other logarithms are
// infinite).  A lane without a chain has infinite logarithms and an infinite wE.
// Es[] gets the bin offset after every attempt.
template <int S, bool EJ, bool MANY, typename REDRAW>
__device__ __forceinline__ uint32_t scan_weight(uint32_t len, const Win<S> &w, const unsigned char *wS, float eps,
                                                WState &st, uint32_t (&Es)[S], REDRAW &&redraw)
{
    const uint32_t ddb[2] = {prmt_var(kTabDD4_0, kTabDD4_1, w.code[0]),
                             S > 4 ? prmt_var(kTabDD4_0, kTabDD4_1, w.code[1]) : 0u};
    int dd[S];
    unrolled<S>([&](auto tc) {
        constexpr int t = decltype(tc)::value;
        dd[t] = sbyte<(t & 3)>(ddb[t >> 2]);
    });
    auto W = [&](uint32_t e) -> float { return *reinterpret_cast<const float *>(wS + e); };
    const WState s0 = st;
    uint32_t accm = 0;
    bool near = false;
    if constexpr (MANY) {
#pragma unroll
        for (int t = 0; t < S; ++t) {
            const uint32_t e1 = st.e4 + dd[t];
            const float A = W(e1);
            const float diff = __fsub_rn(__fmaf_rn(w.dv[t], w.ns2[t], A), st.wE);
            const bool acc = w.l[t] < diff;
            add_if(acc, accm, 0xFu << (4 * t));
            near |= fabsf(__fsub_rn(w.l[t], diff)) <= eps;
            if (EJ && acc) st.ej2 = __fmaf_rn(-w.dv[t], w.ns2[t], st.ej2);
            add_if(acc, st.e4, (uint32_t)dd[t]);
            st.wE = acc ? A : st.wE;
            Es[t] = st.e4;
        }
    } else {
        uint32_t e1 = st.e4 + dd[0];  // the bin if this attempt is accepted
        float A = W(e1);              // its weight
        float diff = __fsub_rn(__fmaf_rn(w.dv[0], w.ns2[0], A), st.wE);
        float c0 = 0.0f, c1 = 0.0f;
        if (S > 1) {
            c0 = W(st.e4 + dd[1]);
            c1 = W(e1 + dd[1]);
        }
#pragma unroll
        for (int t = 0; t < S; ++t) {
            float d0 = 0.0f, d1 = 0.0f;
            if (t + 1 < S) {  // the next attempt's diff if this one is rejected / accepted
                d0 = __fsub_rn(__fmaf_rn(w.dv[t + 1], w.ns2[t + 1], c0), st.wE);
                d1 = __fsub_rn(__fmaf_rn(w.dv[t + 1], w.ns2[t + 1], c1), A);
            }
            const bool acc = w.l[t] < diff;
            add_if(acc, accm, 0xFu << (4 * t));
            near |= fabsf(__fsub_rn(w.l[t], diff)) <= eps;
            if (EJ && acc) st.ej2 = __fmaf_rn(-w.dv[t], w.ns2[t], st.ej2);
            add_if(acc, st.e4, (uint32_t)dd[t]);
            st.wE = acc ? A : st.wE;
            Es[t] = st.e4;
            if (t + 1 < S) {
                A = acc ? c1 : c0;
                diff = acc ? d1 : d0;
                e1 = st.e4 + dd[t + 1];
                if (t + 2 < S) {
                    c0 = W(st.e4 + dd[t + 2]);
                    c1 = W(e1 + dd[t + 2]);
                }
            }
        }
    }
    if (__any_sync(0xffffffffu, near)) {
        uint32_t r1[S];
        redraw(r1);
        st = s0;
        accm = 0;
#pragma unroll
        for (int t = 0; t < S; ++t) {
            const float wn = W(st.e4 + dd[t]);
            const float df = __fsub_rn(__fmaf_rn(w.dv[t], w.ns2[t], wn), st.wE);
            bool acc = df >= 0.0f;
            if (!acc) acc = logf(u01s(r1[t])) < df;
            acc = acc && (uint32_t)t < len;
            if (acc) {
                accm |= 0xFu << (4 * t);
                if (EJ) st.ej2 = __fmaf_rn(-w.dv[t], w.ns2[t], st.ej2);
                st.e4 += dd[t];
                st.wE = wn;
            }
            Es[t] = st.e4;
        }
    }
    return accm;
}

// A chain's running state in a production walk: the byte offset of its bin
// in the staged weight differences, 2 E_J, M, and while recording the byte
// offset of its (E_Delta, M) bin and minus the attempts spent there and not
// yet counted (relative to the end of the window being scanned).
struct PState {
    uint32_t e4;
    float ej2, mag;
    uint32_t bin;
    int since;
};
// Attempts a chain may spend in one bin before its count is sent (at a row's
// start): far below 2^32, and too seldom to cost anything.
constexpr uint32_t kRunAttempts = 1u << 30;

// An accepted attempt leaves the chain's bin of the 2D histogram: the attempts
// since it came there go to the bin as one reduction, and the chain moves on
// by `step` bytes.  `now` is the attempt's position against `since`'s origin.
__device__ __forceinline__ void leave_bin(bool acc, unsigned long long *hist, uint32_t &bin, uint32_t step, int &since,
                                          int now)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, v;\n\t.reg .b32 c;\n\t"
        "setp.ne.u32 p, %5, 0;\n\t"
        "cvt.u64.u32 a, %0;\n\tadd.u64 a, a, %2;\n\t"
        "sub.s32 c, %4, %1;\n\tcvt.u64.u32 v, c;\n\t"
        "@p red.global.add.u64 [a], v;\n\t"
        "@p add.u32 %0, %0, %3;\n\t"
        "@p mov.u32 %1, %4;\n\t}"
        : "+r"(bin), "+r"(since)
        : "l"(hist), "r"(step), "r"(now), "r"((uint32_t)acc)
        : "memory");
}

// *p += c if on, as a predicated reduction: with a branch around each a batch's
// iteration with its bins in global memory took 1.54 ms (64 instances of L = 72,
// 128 chains per block), without 1.04
__device__ __forceinline__ void add_global_if(bool on, unsigned long long *p, uint32_t c)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 v;\n\tsetp.ne.u32 p, %2, 0;\n\tcvt.u64.u32 v, %1;\n\t"
        "@p red.global.add.u64 [%0], v;\n\t}"
        :
        : "l"(p), "r"(c), "r"((uint32_t)on)
        : "memory");
}

// The scan of production.  len: the attempts of the window that count (S, or
// fewer in a masked window, whose other logarithms are infinite).  The reference forms
//   diff = ((double)(-2 dE) + w[E + dDel]) - w[E]   (produce2_multigpu.cu:474)
// with FP64 weights, and FP64 issues slowly on this GPU.  Here, on the FP32
// differences u[E] = w[E+1] - w[E],
//   g = h - dDel u[E or E-1],  h = fast_logf(u) + 2 dE,
// is within `band` of logf(u) - diff (stage_differences), so its sign
// decides unless |g| <= band in some lane: then the window is replayed with
// the FP64 weights in global memory and logf.  One band serves every dDel,
// since logf(u) < 0.  Both values g can take are formed one attempt ahead.
// REC: after every attempt the chain's (E_Delta, M) bin counts once; a run of
// attempts in one bin goes to the u64 histogram as one reduction when the
// chain leaves the bin (leave_bin; an accepted attempt always changes the bin).
template <int S, bool REC, typename REDRAW>
__device__ __forceinline__ uint32_t scan_produce(uint32_t len, const Win<S> &w, const unsigned char *uS,
                                                 const double *__restrict__ wG, unsigned long long *histG,
                                                 bool store, float band, PState &st, REDRAW &&redraw)
{
    const uint32_t lo = w.code[0], hi = w.code[1];
    const uint32_t ddb[2] = {prmt_var(kTabDD4_0, kTabDD4_1, lo), S > 4 ? prmt_var(kTabDD4_0, kTabDD4_1, hi) : 0u};
    const uint32_t uob[2] = {prmt_var(kTabUO_0, kTabUO_1, lo), S > 4 ? prmt_var(kTabUO_0, kTabUO_1, hi) : 0u};
    const uint32_t dfb[2] = {prmt_var(kTabDD_0, kTabDD_1, lo), S > 4 ? prmt_var(kTabDD_0, kTabDD_1, hi) : 0u};
    const uint32_t kb[2] = {prmt_var(kTabK8_0, kTabK8_1, lo), S > 4 ? prmt_var(kTabK8_0, kTabK8_1, hi) : 0u};
    const uint32_t d2b[2] = {prmt_var(kTabD2_0, kTabD2_1, lo), S > 4 ? prmt_var(kTabD2_0, kTabD2_1, hi) : 0u};
    int dd[S], uo[S];
    float nd[S], h[S];
    unrolled<S>([&](auto tc) {
        constexpr int t = decltype(tc)::value;
        dd[t] = sbyte<(t & 3)>(ddb[t >> 2]);
        uo[t] = sbyte<(t & 3)>(uob[t >> 2]);
        nd[t] = __fsub_rn(8388609.0f, magic_byte<(t & 3)>(dfb[t >> 2]));  // -dDel
        h[t] = __fmaf_rn(-w.dv[t], w.ns2[t], w.l[t]);
    });
    auto U = [&](uint32_t e) -> float { return *reinterpret_cast<const float *>(uS + e); };
    if (REC) st.since -= (int)len;
    const PState s0 = st;
    uint32_t accm = 0;
    bool near = false;
    uint32_t e1 = st.e4 + dd[0];
    float g = __fmaf_rn(nd[0], U(st.e4 + uo[0]), h[0]);
    float c0 = 0.0f, c1 = 0.0f;
    if (S > 1) {
        c0 = U(st.e4 + uo[1]);
        c1 = U(e1 + uo[1]);
    }
    uint32_t Eb[S];
    bool av[S];
#pragma unroll
    for (int t = 0; t < S; ++t) {
        float g0 = 0.0f, g1 = 0.0f;
        if (t + 1 < S) {
            g0 = __fmaf_rn(nd[t + 1], c0, h[t + 1]);
            g1 = __fmaf_rn(nd[t + 1], c1, h[t + 1]);
        }
        const bool acc = g < 0.0f;
        near |= !(fabsf(g) > band);  // a NaN (differences beyond FP32) is in doubt too
        av[t] = acc;
        Eb[t] = st.e4;
        add_if(acc, accm, 0xFu << (4 * t));
        if (acc) {
            st.ej2 = __fmaf_rn(-w.dv[t], w.ns2[t], st.ej2);
            st.mag = __fadd_rn(st.mag, w.dv[t]);
        }
        add_if(acc, st.e4, (uint32_t)dd[t]);
        if (t + 1 < S) {
            g = acc ? g1 : g0;
            e1 = st.e4 + dd[t + 1];
            if (t + 2 < S) {
                c0 = U(st.e4 + uo[t + 2]);
                c1 = U(e1 + uo[t + 2]);
            }
        }
    }
    if (__any_sync(0xffffffffu, near)) {
        uint32_t r1[S];
        redraw(r1);
        st = s0;
        accm = 0;
#pragma unroll
        for (int t = 0; t < S; ++t) {
            const int E = (int)(st.e4 >> 2);
            const double diff = __dsub_rn(__dadd_rn((double)__fmul_rn(w.dv[t], w.ns2[t]), wG[E + (dd[t] >> 2)]), wG[E]);
            bool acc = diff >= 0.0;
            if (!acc) acc = (double)logf(u01s(r1[t])) < diff;
            acc = acc && store && (uint32_t)t < len;
            av[t] = acc;
            Eb[t] = st.e4;
            if (acc) {
                accm |= 0xFu << (4 * t);
                st.ej2 = __fmaf_rn(-w.dv[t], w.ns2[t], st.ej2);
                st.mag = __fadd_rn(st.mag, w.dv[t]);
                st.e4 += dd[t];
            }
        }
    }
    if (REC) {
        unrolled<S>([&](auto tc) {
            constexpr int t = decltype(tc)::value;
            // bytes from this attempt's bin to the proposed one, 8 (dDel E + k)
            const uint32_t step = (uint32_t)(sbyte<(t & 3)>(d2b[t >> 2]) * (int)Eb[t] + sbyte<(t & 3)>(kb[t >> 2]));
            leave_bin(av[t], histG, st.bin, step, st.since, t - (int)len);
        });
    }
    return accm;
}

// Stages the FP32 differences u[E] = w[E+1] - w[E] (u[N] = 0) of the FP64
// weights w[0..N] in shared memory (every thread of the block calls it) and
// returns the bound of production's fast test on logf(u) - diff without the
// logarithm's own error.  With m = max |w[E+1] - w[E]|, |f2| <= 16 and
// |fast_logf(u)| < 17 the FP32 roundings of u, h and g move g by at most
// 2^-24 (m + 33 + (33 + m)), and the reference's two FP64 roundings move diff
// by at most 2^-53 (|w| + 16 + |diff|) with |diff| <= 16 + m; twice that.
__device__ __forceinline__ float stage_differences(const double *__restrict__ w64, uint32_t N, float *u)
{
    __shared__ float s_md[32];
    __shared__ double s_mw[32];
    const uint32_t nt = blockDim.x, tid = threadIdx.x;
    float md = 0.0f;
    double mw = 0.0;
    for (uint32_t i = tid; i <= N; i += nt) {
        const double w0 = w64[i];
        const float dp = i < N ? (float)__dsub_rn(w64[i + 1], w0) : 0.0f;
        u[i] = dp;
        md = fmaxf(md, fabsf(dp));
        mw = fmax(mw, fabs(w0));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        md = fmaxf(md, __shfl_xor_sync(0xffffffffu, md, o));
        mw = fmax(mw, __shfl_xor_sync(0xffffffffu, mw, o));
    }
    if ((tid & 31u) == 0) { s_md[tid >> 5] = md; s_mw[tid >> 5] = mw; }
    __syncthreads();
    md = s_md[0];
    mw = s_mw[0];
    for (uint32_t k = 1; k < (nt + 31) / 32; ++k) { md = fmaxf(md, s_md[k]); mw = fmax(mw, s_mw[k]); }
    __syncthreads();
    const double m = (double)md * 1.0001;
    return (float)((2.0 * 5.9604644775390625e-8 * (2.0 * m + 66.0) +
                    2.0 * 1.1102230246251565e-16 * (mw + 32.0 + 2.0 * m)) * 1.0001);
}

// Stages what a block's walk reads: the weights (production: their FP32
// differences, `band` gets the bound above), the cleared histogram, and with
// LAT_SMEM the block's lattice columns.  Only lanes < cpb copy.  Returns the
// lane's lattice base; gl gets its base in global memory.
template <int MODE, bool LAT_SMEM, bool HS>
__device__ __forceinline__ uint32_t *win_prologue(const SweepArgs &a, unsigned char *smem, size_t lat_offset,
                                                  uint32_t cpb, uint32_t lane, uint32_t blk, uint32_t *histS,
                                                  uint32_t *&gl, float &band)
{
    const uint32_t N = a.N, nt = blockDim.x, tid = threadIdx.x;
    uint32_t *latS = reinterpret_cast<uint32_t *>(smem + lat_offset);
    if (MODE == kModeProduce) {
        band = stage_differences(reinterpret_cast<const double *>(a.w), N, reinterpret_cast<float *>(smem));
    } else {
        const float *wg = reinterpret_cast<const float *>(a.w);
        for (uint32_t i = tid; i <= N; i += nt) reinterpret_cast<float *>(smem)[i] = wg[i];
        if (HS)
            for (uint32_t i = tid; i <= N; i += nt) histS[i] = 0u;
        band = 0.0f;
    }
    const uint32_t words = a.L * a.WPR;
    const uint32_t l = lane < cpb ? lane : 0u;  // padding lanes read lane 0's words, never write
    gl = a.lat + (size_t)blk * words * cpb + l;
    if (LAT_SMEM) {
        if (lane < cpb)
            for (uint32_t w = 0; w < words; ++w) latS[(size_t)w * cpb + lane] = gl[(size_t)w * cpb];
        return latS + l;
    }
    return gl;
}

// The windowed sweep of chain block `blk` (cpb chains, lanes >= cpb are
// padding): every lane draws its own Philox numbers one window ahead, so that
// this work fills the latency of the scan; with FEED another warp draws them
// (the block has twice as many threads, the rings of the draws lie at feed_off).
// Ends with the block synchronised
// and, with HS, the shared histogram drained.
// RING (with LAT_SMEM false): the lattice stays in global memory and each
// lane keeps a four-row ring of its chain in shared memory (RowRing), at the
// offset where the whole lattice would go.
// BT: any beta (batch).  btab holds (float)(-beta dE) at dE + 8 and, for the
// windows, (float)(beta ns) at 17 + ns + 4: with dv = +-1 or +-2 the product
// dv * (float)(beta ns) is exactly (float)(-beta dE).  E_J is not tracked (a
// batch has no way to read it).
// Lanes without a chain (padding lanes, and the last block's lanes past the
// chain count) never accept and hold E_Delta = 3, so that every speculative
// index stays inside the weights.
constexpr int kIdleE = 3;
template <int MODE, int R, bool LAT_SMEM, bool HS = true, bool BT = false, bool RING = false,
          bool ALIGNED = true, bool MANY = false, bool FEED = false>
__device__ __forceinline__ void win_sweep_block(const SweepArgs &a, unsigned char *smem, uint32_t cpb, uint32_t blk,
                                                uint32_t iter, unsigned long long nup,
                                                const float *__restrict__ btab = nullptr, uint32_t feed_off = 0)
{
    static_assert(!(RING && LAT_SMEM), "the ring serves lattices in global memory");
    static_assert(ALIGNED || !RING, "the ring serves L % 8 == 0");
    constexpr bool PROD = MODE == kModeProduce;
    const uint32_t lane = threadIdx.x;
    const size_t hist_off = align16((size_t)(a.N + 1) * 4);
    const size_t lat_off = win_smem_base(MODE, a.N, HS);
    uint32_t *histS = reinterpret_cast<uint32_t *>(smem + hist_off), *gl;
    float tol;
    uint32_t *lat = win_prologue<MODE, LAT_SMEM, HS && !PROD>(a, smem, lat_off, cpb, lane, blk, histS, gl, tol);
    RowRing ring;
    const bool own = lane < cpb;  // owns its lattice column
    if (RING) {
        ring.init(reinterpret_cast<uint32_t *>(smem + lat_off) + (own ? lane : 0u), gl);
        lat = ring.rs;
    }
    constexpr uint32_t rmask = RING ? 3u : ~0u;
    __syncthreads();
    const double *wG = reinterpret_cast<const double *>(a.w);
    // the warps that walk, and with FEED as many behind them that draw for them
    const uint32_t walkers = FEED ? blockDim.x / 2u : blockDim.x;
    const bool draws = FEED && threadIdx.x >= walkers;
    const uint32_t clane = draws ? threadIdx.x - walkers : lane, of_warp = clane / 32u;
    const uint32_t chain = blk * cpb + clane;
    const bool active = clane < cpb && chain < a.nchains;
    Draws<R> dr;
    {
        const uint32_t dev = chain / a.chains_per_dev, W = chain - dev * a.chains_per_dev;
        const uint32_t seed = a.seed_base + a.seed_dev_mul * dev;
        dr.s1.init(a.k1_mul * W + a.k1_add, a.k1_hi, seed, iter);
        dr.s3.init(a.k3_mul * W + a.k3_add, a.k3_hi, seed, iter);
        dr.ln2 = active ? kLn2 : -INFINITY;
    }
    Feed feed;
    if constexpr (FEED) {
        unsigned char *ring_of = smem + feed_off + of_warp * kFeedBytes;
        const unsigned long long halves = feed_halves(a.therm, nup);
        if (draws) {
            feed_draw(dr, ring_of, threadIdx.x & 31u, 1u + 4u * of_warp, halves);
            __syncthreads();
            if (HS && !PROD) drain_hist<MODE>(histS, a.hist, a.N);
            return;
        }
        feed.init(ring_of, threadIdx.x & 31u, 1u + 4u * of_warp, halves);
    }
    // lanes without a chain write their word and count their bin here, so that
    // the windows need no test for them
    __shared__ uint32_t s_scratch[2];
    uint32_t *const scratch = &s_scratch[0];
    unsigned char *const hist_lane =
        active ? smem + hist_off : reinterpret_cast<unsigned char *>(&s_scratch[1]) - 4 * kIdleE;
    const int E0 = active ? a.edel[chain] : kIdleE;
    const int EJ0 = active ? a.ej[chain] : 0;
    const int M0 = (active && PROD) ? a.mag[chain] : 0;
    WState ws{(uint32_t)E0 * 4u, 0.0f, (float)(2 * EJ0)};
    PState ps{(uint32_t)E0 * 4u, (float)(2 * EJ0), (float)M0, 0u, 0};
    // an infinite weight makes every difference of a lane without a chain -infinity
    if (!PROD) ws.wE = active ? reinterpret_cast<const float *>(smem)[E0] : INFINITY;
    const float eps = (float)a.log_eps, band = tol + eps;
    const uint32_t L = a.L, WPR = a.WPR;
    const uint32_t W8 = L >> 4, per_row = L >> 1, tail = per_row & 7u;
    const uint32_t last_sites = L - 16u * (WPR - 1u);  // sites of a row's last word
    // the draws ahead: groups cc - 1 and cc (not ALIGNED: cc - 2 .. cc)
    std::conditional_t<ALIGNED || FEED, Ahead, AheadAny> ah;
    uint32_t cc;
    if constexpr (FEED) {
        feed.ready<ALIGNED>();
        feed.read<ALIGNED>(ah);
        cc = 0;
    } else if constexpr (ALIGNED) {
        draw8(dr, 1u, ah);
        cc = 2;
    } else {
        ah.dn = 0;
        ah.off = 0;
#pragma unroll
        for (int t = 0; t < 12; ++t) ah.l[t] = 0.0f;
        for (cc = 0; cc < 3;) shift_in(dr, ++cc, ah);
    }

    // One window: its word at p (C, with the site right of the row's last one
    // merged in: Cm), its up / down / side words.  MASKED: only len of its
    // attempts take place; the others' logarithms become infinite.
    auto window = [&](auto sc, auto hc, auto rc, auto mc, uint32_t *p, uint32_t C, uint32_t Cm, uint32_t Uw,
                      uint32_t Dw, uint32_t side, uint32_t len) {
        constexpr int S = decltype(sc)::value, HALF = decltype(hc)::value;
        constexpr bool REC = decltype(rc)::value, MASKED = decltype(mc)::value;
        Win<S> w;
        uint32_t c0, off = 0;
        if constexpr (FEED) {
            c0 = feed.b + 1u;
            off = feed.off;
            if (ALIGNED) {
                feed.b += S == 4 || (MASKED && len <= 4u) ? 1u : 2u;
            } else {
                feed.b += (feed.off + len) >> 2;
                feed.off = (feed.off + len) & 3u;
            }
            feed.ready<ALIGNED>();
            decode<S, HALF, BT>(Cm, Uw, Dw, side, ah, btab, w);
            feed.read<ALIGNED>(ah);
        } else if constexpr (ALIGNED) {
            decode<S, HALF, BT>(Cm, Uw, Dw, side, ah, btab, w);
            c0 = cc - 1u;
            // the next window's draws, independent of the scan below
            if (S == 4 || (MASKED && len <= 4u)) {
                draw4(dr, cc + 1u, ah);
                cc += 1;
            } else {
                draw8(dr, cc + 1u, ah);
                cc += 2;
            }
        } else {
            const Ahead x = next8(ah);
            decode<S, HALF, BT>(Cm, Uw, Dw, side, x, btab, w);
            c0 = cc - 2u;
            off = ah.off;
            for (ah.off += len; ah.off >= 4u; ah.off -= 4u) shift_in(dr, ++cc, ah);
        }
        if (MASKED) {
            // slots past the last attempt: never accepted, and no move to look ahead for
#pragma unroll
            for (int t = 0; t < S; ++t)
                if ((uint32_t)t >= len) w.l[t] = INFINITY;
            const uint32_t keep = (1u << (4u * len)) - 1u;  // len < 8
            w.code[0] = (w.code[0] & keep) | (0x22222222u & ~keep);
            w.code[1] = w.code[0] >> 16;
        }
        auto redraw = [&](uint32_t(&r1)[S]) {
            if (ALIGNED) {
                dr.s1.block((unsigned long long)kPhiloxM0 * c0, r1);
                if (S > 4) dr.s1.block((unsigned long long)kPhiloxM0 * (c0 + 1u), r1 + (S > 4 ? 4 : 0));
            } else {
                uint32_t r[12];
#pragma unroll
                for (int g = 0; g < 3; ++g) dr.s1.block((unsigned long long)kPhiloxM0 * (c0 + g), r + 4 * g);
#pragma unroll
                for (int t = 0; t < S; ++t) {
                    const uint32_t x0 = (off & 1u) ? r[t + 1] : r[t], x2 = (off & 1u) ? r[t + 3] : r[t + 2];
                    r1[t] = (off & 2u) ? x2 : x0;
                }
            }
        };
        const uint32_t m = MASKED ? len : (uint32_t)S;
        uint32_t accm;
        if (PROD) {
            accm = scan_produce<S, REC>(m, w, smem, wG, a.hist, active, band, ps, redraw);
        } else {
            uint32_t Es[S];
            accm = scan_weight<S, !BT, MANY>(m, w, smem, eps, ws, Es, redraw);
            if (REC && HS) {
                // one fire-and-forget shared atomic per attempt
#pragma unroll
                for (int t = 0; t < S; ++t)
                    if (!MASKED || (uint32_t)t < len) atomicAdd(reinterpret_cast<uint32_t *>(hist_lane + Es[t]), 1u);
            } else if (REC && !HS) {
                // entries merged into runs of equal bins: fewer global atomics
                uint32_t cur = Es[0], cnt = 1;
#pragma unroll
                for (int t = 1; t < S; ++t) {
                    if (MASKED && (uint32_t)t >= len) break;
                    const bool same = Es[t] == cur;
                    add_global_if(active && !same, a.hist + (cur >> 2), cnt);
                    cnt = same ? cnt + 1u : 1u;
                    cur = Es[t];
                }
                add_global_if(active, a.hist + (cur >> 2), cnt);
            }
        }
        const uint32_t word = C ^ (((w.ctr ^ w.vnib) & accm) << (HALF ? 2 : 0));
        if (LAT_SMEM || RING) *(active ? p : scratch) = word;
        else if (active) *p = word;
    };
    using S8 = std::integral_constant<int, 8>;
    using S4 = std::integral_constant<int, 4>;
    using H0 = std::integral_constant<int, 0>;
    using H1 = std::integral_constant<int, 1>;
    // `left` attempts of row-half (row, HALF): PART false: all of them (full
    // windows of 8, then the row's last word), else a phase's last ones.
    auto row_half = [&](auto hc, auto rc, auto pc_, uint32_t row, uint32_t left) {
        constexpr int HALF = decltype(hc)::value;
        constexpr bool PART = decltype(pc_)::value;
        using Whole = std::false_type;
        using Masked = std::true_type;
        const uint32_t rup = (row + 1 == L) ? 0u : row + 1, rdn = (row == 0) ? L - 1 : row - 1;
        uint32_t *pc = lat + (size_t)((row & rmask) * WPR) * cpb;
        const uint32_t *pu = lat + (size_t)((rup & rmask) * WPR) * cpb;
        const uint32_t *pd = lat + (size_t)((rdn & rmask) * WPR) * cpb;
        const uint32_t n8 = PART ? left >> 3 : W8, rest = PART ? left & 7u : tail;
        uint32_t C = *pc;
        const uint32_t first = C;  // (HALF 1) its even sites do not change in this half
        // HALF 0: the word to the left, its last site at the top; its odd sites
        // do not change in this half
        uint32_t side = HALF == 0 ? pc[(size_t)(WPR - 1) * cpb] << (32u - 2u * last_sites) : 0u;
        uint32_t q = 0;
        for (; q < n8; ++q, pc += cpb, pu += cpb, pd += cpb) {
            const uint32_t next = q + 1 < WPR ? pc[cpb] : first;
            window(S8{}, hc, rc, Whole{}, pc, C, C, *pu, *pd, HALF == 0 ? side : next, 8u);
            side = C;
            C = next;
        }
        if (rest) {
            uint32_t Cm = C;
            if (HALF == 1) {
                side = q + 1 < WPR ? pc[cpb] : first;
                // the site right of the row's last one is its first
                if (q + 1 == WPR && last_sites != 16u)
                    Cm = (C & ((1u << (2u * last_sites)) - 1u)) | (first << (2u * last_sites));
            }
            if (ALIGNED && !PART) window(S4{}, hc, rc, Whole{}, pc, C, Cm, *pu, *pd, side, 4u);
            else                  window(S8{}, hc, rc, Masked{}, pc, C, Cm, *pu, *pd, side, rest);
        }
    };

    // The reference's sweep order: the even sites row by row, then the odd
    // ones (muca_delta_multigpu.cu:173).  A phase's last row-half is partial
    // when therm or nup is not a multiple of L/2.
    // Recorded attempts per lane since the shared u32 bins were last flushed:
    // no bin can reach 2^32 while cpb * since stays below it
    unsigned long long since = 0;
    // production: rows until the attempts in the chains' bins (PState::since) are sent
    const uint32_t run_rows = (a.hooks & kHookFlushRows) ? 0u : kRunAttempts / per_row;
    uint32_t rows_left = run_rows;
    auto send_run = [&]() {
        if (active && ps.since) atomicAdd(a.hist + (ps.bin >> 3), (unsigned long long)(uint32_t)-ps.since);
        ps.since = 0;
    };
    auto phase = [&](auto rc, unsigned long long n) {
        constexpr bool REC = decltype(rc)::value;
        uint32_t row = 0, half = 0;
        auto row_begin = [&]() {
            if (RING) ring.row_start(row, L, cpb, WPR, own);
            if (HS && !PROD && REC) {
                if ((since + per_row) * cpb > 0xFFFFFFFFull || (a.hooks & kHookFlushRows)) {  // uniform
                    if (FEED) flush_hist_of(histS, a.hist, a.N, walkers);
                    else      flush_hist<MODE>(histS, a.hist, a.N);
                    since = 0;
                }
                since += per_row;
            }
            // a chain that stays in its bin for 2^32 attempts would wrap its count
            if (PROD && REC) {
                if (rows_left-- == 0) {  // uniform
                    send_run();
                    rows_left = run_rows;
                }
            }
        };
        while (n >= per_row) {
            row_begin();
            if (half == 0) row_half(H0{}, rc, std::false_type{}, row, per_row);
            else           row_half(H1{}, rc, std::false_type{}, row, per_row);
            n -= per_row;
            if (++row == L) {
                row = 0;
                half ^= 1u;
            }
        }
        if (n) {
            row_begin();
            if (half == 0) row_half(H0{}, rc, std::true_type{}, row, (uint32_t)n);
            else           row_half(H1{}, rc, std::true_type{}, row, (uint32_t)n);
        }
        // a phase's draws start at a new group
        if constexpr (FEED && !ALIGNED) {
            if (feed.off) {
                feed.off = 0;
                ++feed.b;
                feed.ready<ALIGNED>();
                feed.read<ALIGNED>(ah);
            }
        } else if constexpr (!ALIGNED) {
            if (ah.off) {
                shift_in(dr, ++cc, ah);
                ah.off = 0;
            }
        }
    };
    phase(std::false_type{}, a.therm);
    if (PROD) {
        const uint32_t E = ps.e4 >> 2;
        ps.bin = ((uint32_t)((int)ps.mag + (int)(E * E + 2u * E)) >> 1) * 8u;
        if (a.hooks & kHookAgedRun) {
            ps.since = (int)(0u - kAgedRun);
            rows_left = 0;
        }
    }
    phase(std::true_type{}, nup);
    if (PROD) send_run();
    if (LAT_SMEM && own) {
        const uint32_t words = L * WPR;
        for (uint32_t w = 0; w < words; ++w) gl[(size_t)w * cpb] = lat[(size_t)w * cpb];
    }
    if (RING) ring.finish(cpb, WPR, own);
    if (active) {
        a.edel[chain] = (int)((PROD ? ps.e4 : ws.e4) >> 2);
        if (!BT) a.ej[chain] = (int)(PROD ? ps.ej2 : ws.ej2) / 2;
        if (PROD) a.mag[chain] = (int)ps.mag;
    }
    __syncthreads();
    if (HS && !PROD) drain_hist<MODE>(histS, a.hist, a.N);
}

}  // namespace muca
