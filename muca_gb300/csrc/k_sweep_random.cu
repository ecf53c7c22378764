// k_sweep_random.cu -- the random-site Metropolis sweep of the reference's
// CPU weight program (muca_mag.cpp:312-393, `mcs`) and of the GPU kernel
// mcs2 it was ported to (muca_delta_multigpu.cu:637-734), one chain per lane.
//
// Per chain (the reference's MPI rank WORKER, `seed` = jack index mm):
//   keys  k1 = {10 W + 1000 seed, 0xdecafbad}    (acceptance)
//         k2 = {100 W + 4000 seed, 0x20202041}   (site)
//         k3 = {1000 W + 10000 seed, 0x11cafead} (direction)
//   ctr   {c0, 0xbadbad11, 2 iter, 0xBADC0DED}, ++c0 before every 4th attempt,
//         continuing from the thermalisation into the production loop;
//   site  idx = (unsigned)(u01fixedpt<float>(r2) * N), truncated;
//   step  the same proposal and energy change as the sweep kernels, with
//         FP64 weights: diff = (double)(-2 dE) + w[E + dDel] - w[E];
//   test  diff >= 0 || log(u01fixedpt<float>(r1)) < diff, where log is the
//         host libm's logf (the CPU program) when a table of its values is
//         given, else CUDA's logf (mcs2).
// The lattice uses the packed layout of the other sweeps (2-bit codes, rows
// of 16-site words, [block][word][lane]); the FP32 differences of the FP64
// weights (stage_differences) and a u32 histogram are staged in shared memory,
// the lattice too when it fits.
//
// The test is decided in FP32, as the production window does it, and where
// that is in doubt by the reference's FP64 difference and the exact log (host
// libm value or logf): see scan_produce for the bound.
//
// What bounds it: at one warp per SM sub-partition the instructions of the
// warp, and beneath them the chain from one attempt's store to the next one's
// loads and decision.  So the draws come one group of four attempts ahead of the
// scan, in one stretch of code with it and with the sites' and neighbours'
// addresses, and the scan has no branch: an attempt in doubt is noticed at the
// end of its group, whose stores are then taken back and repeated.
//   * a site is split into row and column with FP32 (exact: idx < 2^14); a
//     number in the mantissa of 2^23 goes into the address products as it is,
//     the constant they carry is in the address base;
//   * a word is rotated until its site is at the bottom, and code and
//     direction are the selector of a byte table whose entries 3 and 7 complete
//     the float 2^23 + entry;
//   * lattice columns in shared memory lie a multiple of 32 lanes apart where
//     that fits, so that lanes at different sites meet no bank conflict.
// L = 72, 16384 chains, 85 M attempts: 0.56 ms (224 cycles an attempt and
// warp); 0.68 with the addresses too kept from one group to the next (a move for
// each), selects instead of predicated additions and stores, and a group's
// length tested in its loop; 0.79 with tables of a row's and a column's
// addresses in shared memory; 1.79 with draws, site and test of every attempt on
// one dependency chain.
#include "window.cuh"

#include <algorithm>

namespace muca {

// shared memory: 16 B (read for E = 0, never used) | differences | u32 histogram | lattice
__host__ __device__ inline size_t random_smem_base(uint32_t N)
{
    return 16 + 2 * align16((size_t)(N + 1) * 4);
}

// What a group's draws leave for its scan: the acceptance logarithm, 2^23 + site
// and the selector of the byte tables less the site's code ...
struct RandomDraw {
    float l, ib;
    uint32_t dsel;
};
// ... and with the byte offsets of the site's word and its neighbours', and twice
// their columns (rotations count modulo 32).
struct RandomAttempt {
    float l;
    uint32_t aC, aU, aD, aL, aR, sC, sL, sR, dsel;
};
// Byte tables by code | direction << 2 (window.cuh), entry 3 = 0; entry 7 =
// 0x4B where the value is to be the float 2^23 + entry, else 0.
constexpr uint32_t kRndDV_0 = 0x00000303u, kRndDV_1 = 0x4B010104u;  // s_new - s_old + 2
constexpr uint32_t kRndND_0 = 0x00010002u, kRndND_1 = 0x4B020001u;  // 1 - dDel
constexpr uint32_t kRndD4_0 = 0x00040800u, kRndD4_1 = 0x00000804u;  // 4 dDel + 4
constexpr uint32_t kRndVX_0 = 0x00020301u, kRndVX_1 = 0x00030102u;  // old code ^ new code
constexpr uint32_t kRndSel = 0x7330u;

// SEGMENT: groups between two flushes of the u32 bins (a constant: read from the
// arguments it cost 3 % of the sweep).
template <int R, bool LAT_SMEM, uint32_t SEGMENT>
__global__ void __launch_bounds__(256) k_sweep_random(const RandomArgs a, uint32_t cpb, uint32_t pitch)
{
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t iter = a.iter;
    unsigned long long nup = a.nup;
    if (a.dyn) {
        if (a.dyn[2]) return;
        iter = a.dyn[0];
        nup = a.dyn[1];
    }
    const uint32_t N = a.N, L = a.L, WPR = a.WPR, nt = blockDim.x, tid = threadIdx.x, lane = threadIdx.x;
    float *u = reinterpret_cast<float *>(smem + 16);
    uint32_t *histS = reinterpret_cast<uint32_t *>(smem + 16 + align16((size_t)(N + 1) * 4));
    const uint32_t hist_off = 16u + (uint32_t)align16((size_t)(N + 1) * 4);
    const uint32_t lat_off = (uint32_t)random_smem_base(N);
    const double *__restrict__ w64 = a.w;
    const uint32_t words = L * WPR;
    const bool store = lane < cpb;  // owns its lattice column
    uint32_t *gl = a.lat + (size_t)blockIdx.x * words * cpb + (store ? lane : 0u);
    // the lane's column: its own; without one a padding column, or else lane 0's, which it only reads
    const uint32_t column = LAT_SMEM ? (lane < pitch ? lane : 0u) : (store ? lane : 0u);
    if (LAT_SMEM) {
        uint32_t *latS = reinterpret_cast<uint32_t *>(smem + lat_off) + column;
        if (store) {
            uint32_t d = (uint32_t)__cvta_generic_to_shared(latS);
            for (uint32_t w = 0; w < words; ++w, d += 4u * pitch)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gl + (size_t)w * cpb) : "memory");
        } else if (lane < pitch) {
            for (uint32_t w = 0; w < words; ++w) latS[(size_t)w * pitch] = kZeroWord;
        }
    }
    const float band = stage_differences(w64, N, u) + (float)a.log_eps;
    if (tid == 0) u[-1] = u[N + 1] = 0.0f;  // (u[N + 1]: read by lanes without a chain)
    for (uint32_t i = tid; i <= N; i += nt) histS[i] = 0u;
    if (LAT_SMEM) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const uint32_t chain = blockIdx.x * cpb + lane;
    const bool active = store && chain < a.nchains;
    const uint32_t W = a.worker0 + chain;
    Stream<R> s1, s2, s3;
    s1.init(10u * W + 1000u * a.seed, 0xdecafbadu, 0xbadbad11u, 2u * iter);
    s2.init(100u * W + 4000u * a.seed, 0x20202041u, 0xbadbad11u, 2u * iter);
    s3.init(1000u * W + 10000u * a.seed, 0x11cafeadu, 0xbadbad11u, 2u * iter);
    // lanes without a chain: an infinite logarithm (or a NaN), so they never
    // accept, and E_Delta stays N + 1: they count in the bin after the last,
    // which the rounded-up sizes of the arrays have (N + 1 is no multiple of 4)
    const float ln2 = active ? kLn2 : -INFINITY;
    uint32_t e4 = active ? 4u * (uint32_t)a.edel[chain] : 4u * (N + 1u);
    float ej2 = active ? (float)(2 * a.ej[chain]) : 0.0f;

    unsigned char *const base = LAT_SMEM ? smem : reinterpret_cast<unsigned char *>(a.lat + (size_t)blockIdx.x * words * cpb);
    const uint32_t p4 = 4u * (LAT_SMEM ? pitch : cpb), rs = WPR * p4;  // bytes from a word (row) to the next
    // word q of row r lies at bits(2^23 + r) rs + (bits(2^23 + col) >> 4) p4 + k0
    const uint32_t k0 = (LAT_SMEM ? lat_off : 0u) + 4u * column - 0x4B000000u * rs - 0x04B00000u * p4;
    const float fN = (float)N, fL = (float)L, inv = __frcp_rn(fL), half_inv = 0.5f * inv, magic = 8388608.0f;
    const float last = magic + (fL - 1.0f);

    auto word = [&](uint32_t off) -> uint32_t & { return *reinterpret_cast<uint32_t *>(base + off); };
    auto prep = [&](uint32_t c, RandomDraw (&at)[4]) {
        uint32_t r1[4], r2[4], r3[4];
        const unsigned long long q = (unsigned long long)kPhiloxM0 * c;
        s1.block(q, r1);
        s2.block(q, r2);
        s3.block(q, r3);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            RandomDraw &x = at[t];
            x.l = __fmul_rn(lg2_ftz(u01s(r1[t])), ln2);
            x.ib = __fadd_rz(__fmul_rn(u01s(r2[t]), fN), magic);  // 2^23 + idx, idx = (unsigned)(u N)
            x.dsel = ((r3[t] >> 29) & 4u) | kRndSel;  // u01fixedpt<float>(r3) < 0.5 <=> top bit clear: s + 1
        }
    };
    auto place = [&](const RandomDraw &d) -> RandomAttempt {
        RandomAttempt x;
        x.l = d.l;
        x.dsel = d.dsel;
        // row = floor((idx + 1/2) / L)
        const float rowb = __fadd_rz(__fmaf_rn(__fsub_rn(d.ib, magic), inv, half_inv), magic);
        const float colb = __fmaf_rn(__fsub_rn(rowb, magic), -fL, d.ib);
        const uint32_t col = __float_as_uint(colb), row = __float_as_uint(rowb) * rs + k0;
        uint32_t cl = col - 1u, cr = col + 1u;
        add_if(colb == magic, cl, L);
        add_if(colb == last, cr, 0u - L);
        x.aC = (col >> 4) * p4 + row;
        x.aU = x.aC + rs;
        x.aD = x.aC - rs;
        add_if(rowb == last, x.aU, 0u - L * rs);
        add_if(rowb == magic, x.aD, L * rs);
        x.aL = (cl >> 4) * p4 + row;
        x.aR = (cr >> 4) * p4 + row;
        x.sC = 2u * col;
        x.sL = 2u * cl;
        x.sR = 2u * cr;
        return x;
    };
    // code of the site that the rotation brings to the bottom
    auto code = [](uint32_t w, uint32_t s2x) -> uint32_t { return __funnelshift_r(w, w, s2x) & 3u; };
    struct Move {
        uint32_t word, sel;
        float dv, ns2;
    };
    auto decode = [&](const RandomAttempt &x) -> Move {
        Move m;
        m.word = word(x.aC);
        m.sel = code(m.word, x.sC) | x.dsel;
        const uint32_t nb = code(word(x.aU), x.sC) + code(word(x.aD), x.sC) + code(word(x.aL), x.sL) +
                            code(word(x.aR), x.sR);
        m.ns2 = __fmaf_rn(__uint_as_float(0x4B000000u + nb), 2.0f, -16777224.0f);
        m.dv = __fsub_rn(__uint_as_float(prmt_var(kRndDV_0, kRndDV_1, m.sel)), 8388610.0f);
        return m;
    };
    auto moved = [&](const RandomAttempt &x, const Move &m) -> uint32_t {
        return __funnelshift_l(0u, prmt_var(kRndVX_0, kRndVX_1, m.sel), x.sC);
    };
    const unsigned char *uS = smem + 16;
    auto U = [&](uint32_t e) -> float { return *reinterpret_cast<const float *>(uS + e); };

    uint32_t c0 = 1;
    RandomDraw nx[4];
    prep(c0, nx);
    auto group = [&](uint32_t len, auto rec, auto part) {
        constexpr bool REC = decltype(rec)::value, PART = decltype(part)::value;
        RandomAttempt at[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) at[t] = place(nx[t]);
        if (PART) {
#pragma unroll
            for (int t = 1; t < 4; ++t)
                if ((uint32_t)t >= len) at[t].l = INFINITY;  // never accepted
        }
        prep(c0 + 1u, nx);
        const uint32_t e4_0 = e4;
        const float ej2_0 = ej2;
        uint32_t old[4], Es[4];
        bool near = false;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const RandomAttempt &x = at[t];
            const float um = U(e4 - 4u), up = U(e4);
            const Move m = decode(x);
            const float nd = __fsub_rn(__uint_as_float(prmt_var(kRndND_0, kRndND_1, m.sel)), 8388609.0f);
            // logf(u) - f2 - (w[E + dDel] - w[E]), f2 = -2 dE = dv ns2
            const float g = __fmaf_rn(nd, nd > 0.0f ? um : up, __fmaf_rn(-m.dv, m.ns2, x.l));
            const bool acc = g < 0.0f;
            near |= !(fabsf(g) > band);  // a NaN (differences beyond FP32) is in doubt too
            old[t] = m.word;
            const uint32_t step = prmt_var(kRndD4_0, kRndD4_1, m.sel) - 4u, changed = m.word ^ moved(x, m);
            if (acc) {
                word(x.aC) = changed;
                ej2 = __fmaf_rn(-m.dv, m.ns2, ej2);
            }
            add_if(acc, e4, step);
            Es[t] = e4;
        }
        if (near) {
            // in doubt: the group again, with the reference's FP64
            // difference and exact log
            uint32_t r1[4];
            s1.block((unsigned long long)kPhiloxM0 * c0, r1);
            e4 = e4_0;
            ej2 = ej2_0;
            if (store) {
#pragma unroll
                for (int t = 3; t >= 0; --t) word(at[t].aC) = old[t];
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const Move m = decode(at[t]);
                const int E = (int)(e4 >> 2), d4 = (int)prmt_var(kRndD4_0, kRndD4_1, m.sel) - 4;
                if (active && (uint32_t)t < len) {
                    const double diff = __dsub_rn(__dadd_rn((double)__fmul_rn(m.dv, m.ns2), w64[E + d4 / 4]), w64[E]);
                    bool acc = diff >= 0.0;
                    if (!acc) {
                        const float lg = a.logf_tab ? __ldg(a.logf_tab + (r1[t] >> 9)) : logf(u01s(r1[t]));
                        acc = (double)lg < diff;
                    }
                    if (acc) {
                        word(at[t].aC) = m.word ^ moved(at[t], m);
                        ej2 = __fmaf_rn(-m.dv, m.ns2, ej2);
                        e4 += (uint32_t)d4;
                    }
                }
                Es[t] = e4;
            }
        }
        ++c0;
        if (REC) {
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (!PART || (uint32_t)t < len) atomicAdd(reinterpret_cast<uint32_t *>(smem + hist_off + Es[t]), 1u);
        }
    };
    auto run = [&](unsigned long long n, auto rec) {
        while (n >= 4ull) {
            const uint32_t m = n < 4ull * SEGMENT ? (uint32_t)n / 4u : SEGMENT;
#pragma unroll 2
            for (uint32_t i = 0; i < m; ++i) group(4u, rec, std::false_type{});
            n -= 4ull * m;
            // no more than 256 lanes x 4 x 2^20 = 2^30 entries between two flushes
            if (decltype(rec)::value && n >= 4ull) flush_hist<kModeWeight>(histS, a.hist, N);
        }
        if (n > 0) group((uint32_t)n, rec, std::true_type{});
    };
    run(a.therm, std::false_type{});
    run(nup, std::true_type{});
    if (LAT_SMEM && store) {
        const uint32_t *lat = reinterpret_cast<const uint32_t *>(smem + lat_off) + column;
#pragma unroll 8
        for (uint32_t w = 0; w < words; ++w) gl[(size_t)w * cpb] = lat[(size_t)w * pitch];
    }
    if (active) {
        a.edel[chain] = (int32_t)(e4 >> 2);
        a.ej[chain] = (int32_t)ej2 / 2;
    }
    __syncthreads();
    drain_hist<kModeWeight>(histS, a.hist, N);
}

template <int R, bool LS>
static cudaError_t launch_random_one(const RandomArgs &a, uint32_t cpb, uint32_t pitch, uint32_t blocks, size_t smem,
                                     size_t smem_limit, cudaStream_t s)
{
    // (the test hook's short segments)
    void (*const kern)(const RandomArgs, uint32_t, uint32_t) =
        (a.hooks & kHookFlushRows) ? k_sweep_random<R, LS, 2u> : k_sweep_random<R, LS, 1u << 20>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_limit);
    if (e != cudaSuccess) return e;
    kern<<<blocks, (cpb + 31u) / 32u * 32u, smem, s>>>(a, cpb, pitch);
    return cudaGetLastError();
}

// Block shape of the random-site sweep: one wave of blocks over the SMs with
// the chains spread evenly (ceil(nchains / SMs) per block), each block's
// lattice in shared memory when that many chains' lattices fit beside the
// difference table and the histogram.  The random site makes the lattice
// loads of one attempt depend on the previous attempt's store, so their
// latency is on every attempt's chain: shared memory, not L1/L2.  When the
// lattices do not fit, blocks of up to 128 chains read them from global
// memory.
SweepPlan plan_random(uint32_t L, uint32_t nchains, size_t smem_optin, int sms)
{
    SweepPlan p{};
    p.mode = kModeWeight;
    p.kernel = kKernelGeneric;
    const uint32_t N = L * L, WPR = (L + 15) / 16;
    const size_t per_chain = (size_t)L * WPR * 4, base = random_smem_base(N);
    const size_t optin = smem_optin > 512 ? smem_optin - 512 : 0;
    const size_t cap = optin > base ? (optin - base) / per_chain : 0;
    const uint32_t want = (nchains + (uint32_t)sms - 1) / (uint32_t)sms;
    p.lat_smem = cap >= 1 && want <= cap && want <= 256;
    p.cpb = p.lat_smem ? want : std::min<uint32_t>(128u, want);
    p.blocks = (nchains + p.cpb - 1) / p.cpb;
    p.threads = (p.cpb + 31u) / 32u * 32u;
    p.smem = random_sweep_smem(L, p.cpb, p.lat_smem);
    return p;
}

size_t random_sweep_smem(uint32_t L, uint32_t pitch, bool lat_smem)
{
    const uint32_t WPR = (L + 15) / 16;
    return random_smem_base(L * L) + (lat_smem ? (size_t)L * WPR * 4 * pitch : 0);
}

cudaError_t launch_sweep_random(const RandomArgs &a, uint32_t cpb, uint32_t blocks, int rounds, size_t smem_optin,
                                cudaStream_t s)
{
    if (cpb == 0 || cpb > 256 || a.L < 3) return cudaErrorInvalidValue;
    // (512 B of the opt-in limit stay free for the kernel's static shared memory)
    auto fits = [&](uint32_t pitch) { return random_sweep_smem(a.L, pitch, true) + 512 <= smem_optin; };
    const uint32_t whole = (cpb + 31u) / 32u * 32u, pitch = fits(whole) ? whole : cpb;
    const bool ls = fits(pitch);
    const size_t smem = random_sweep_smem(a.L, pitch, ls);
    if (smem + 512 > smem_optin) return cudaErrorInvalidValue;
    const size_t limit = smem_optin - 512;
    if (rounds == 10)
        return ls ? launch_random_one<10, true>(a, cpb, pitch, blocks, smem, limit, s) : launch_random_one<10, false>(a, cpb, pitch, blocks, smem, limit, s);
    return ls ? launch_random_one<7, true>(a, cpb, pitch, blocks, smem, limit, s) : launch_random_one<7, false>(a, cpb, pitch, blocks, smem, limit, s);
}

}  // namespace muca
