// k_bench.cu -- measurement kernels for the rooflines of the sweep.
//
// The sweep kernels spend most of their issue slots on Philox4x32 blocks
// (two per four Metropolis attempts).  k_philox_peak generates Philox blocks
// in exactly the form the sweeps use them (per-thread key, counter words 1..3
// fixed, word 0 counting) at full occupancy with nothing else to do, so its
// rate is the ceiling of "Philox blocks per second" on this GPU.
//
// k_sweep_floor takes the weight-mode windowed sweep apart and times each
// part per warp in SM cycles (clock64), in the sweep's own geometry at
// 16384 chains: one block of four warps of 32 chains on one SM, one warp per
// SM sub-partition, the L = 72 lattice, the FP32 weights and the u32
// histogram in shared memory (225,824 B).  Each lane runs `windows` full
// 8-site windows:
//   part 0  the sweep's window body: the next window's draws, decode, scan,
//           lattice store and histogram entries (the sweep without its
//           4-site and partial windows and its loop bookkeeping);
//   part 1  the draws and the decode alone, the work off the chain of
//           decisions (its fields folded into one word so none is dead);
//   part 2  the scan, store and histogram entries alone, on two decoded
//           windows held in registers;
//   part 3  the bare chain of decisions of the scan: per attempt a select of
//           the prefetched weight, two adds, one compare, the E_Delta update
//           and the two weight loads one attempt ahead, with the scan's
//           loads at each window start;
//   part 4  the draws alone (four Philox4x32-7 blocks per window);
//   part 5  one dependent FP32 add per "attempt" (its latency);
//   part 6  one dependent shared-memory load per "attempt" (its latency).
// Parts 2 and 3 replay fixed windows, so E_Delta is kept inside the weight
// array by walls: the weights at E_Delta = 0..2 and N-2..N are -1e30, every
// move onto them is rejected, and the loads reach at most three bins beyond
// the current E_Delta.
#include "window.cuh"

namespace muca {

template <int R>
__global__ void __launch_bounds__(256) k_philox_peak(uint32_t blocks_per_thread, uint32_t seed, uint32_t *out)
{
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    RoundKeys<R> k;
    k.init(2u * t, 0xdecafbadu);
    uint32_t acc = 0;
#pragma unroll 4
    for (uint32_t i = 0; i < blocks_per_thread; ++i) {
        const uint4 r = philox<R>(i + 1u, seed, t, kCtrTag, k);
        acc ^= r.x ^ r.y ^ r.z ^ r.w;
    }
    out[t] = acc;
}

cudaError_t launch_philox_peak(int rounds, uint32_t grid, uint32_t blocks_per_thread, uint32_t *out, cudaStream_t s)
{
    if (rounds == 10)
        k_philox_peak<10><<<grid, 256, 0, s>>>(blocks_per_thread, 100u, out);
    else
        k_philox_peak<7><<<grid, 256, 0, s>>>(blocks_per_thread, 100u, out);
    return cudaGetLastError();
}

constexpr uint32_t kFloorL = 72, kFloorWPR = 5, kFloorCpb = 128, kFloorN = kFloorL * kFloorL;
constexpr float kFloorEps = 3.5e-6f;  // twice max |fast_logf(u) - logf(u)| measured on GB300

__device__ __forceinline__ uint32_t floor_hash(uint32_t x)
{
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}

template <int PART>
__global__ void __launch_bounds__(kFloorCpb, 1) k_sweep_floor(uint32_t windows, unsigned long long *cycles,
                                                               uint32_t *sink)
{
    extern __shared__ __align__(16) unsigned char smem[];
    float *wS = reinterpret_cast<float *>(smem);
    const uint32_t hist_off = (uint32_t)align16((size_t)(kFloorN + 1) * 4);
    uint32_t *histS = reinterpret_cast<uint32_t *>(smem + hist_off);
    const uint32_t lane = threadIdx.x;
    uint32_t *lat = reinterpret_cast<uint32_t *>(smem + win_smem_base(kModeWeight, kFloorN, true)) + lane;
    const bool walls = PART >= 2;
    for (uint32_t b = lane; b <= kFloorN; b += blockDim.x) {
        wS[b] = (walls && (b < 3 || b + 3 > kFloorN)) ? -1e30f : 0.0f;
        histS[b] = 0;
    }
    // random spin codes 0..2 in the L sites of each row, code 1 (spin 0) in the padding
    int E = 0;
    for (uint32_t w = 0; w < kFloorL * kFloorWPR; ++w) {
        const uint32_t q = w % kFloorWPR;
        uint32_t word = 0;
        for (uint32_t c = 0; c < 16; ++c) {
            const uint32_t code = (16 * q + c < kFloorL) ? floor_hash(w * 16 + c + 7919u * lane) % 3u : 1u;
            word |= code << (2 * c);
            E += code != 1u;
        }
        lat[(size_t)w * kFloorCpb] = word;
    }
    __syncthreads();
    WState st;
    st.e4 = 4u * (walls ? kFloorN / 2 : (uint32_t)E);
    st.wE = *reinterpret_cast<const float *>(smem + st.e4);
    st.ej2 = 0.0f;
    Draws<7> dr;
    dr.s1.init(2u * lane + 1u, 0xdecafbadu, 100u, 0u);
    dr.s3.init(2u * lane + 3u, 0xdecafbadu, 100u, 0u);
    dr.ln2 = kLn2;
    Ahead ah;
    draw8(dr, 1u, ah);
    uint32_t cc = 2, fold = 0;
    auto decode_at = [&](uint32_t row, uint32_t q, Win<8> &w) {
        const uint32_t *pc = lat + (row * kFloorWPR + q) * kFloorCpb;
        decode<8, 0, false>(pc[0], pc[kFloorWPR * kFloorCpb], *(pc - kFloorWPR * kFloorCpb),
                            q ? *(pc - kFloorCpb) : pc[(kFloorWPR - 1) * kFloorCpb], ah, nullptr, w);
    };
    Win<8> d0, d1;
    if (PART == 2 || PART == 3) {
        decode_at(3, 1, d0);
        draw8(dr, 3u, ah);
        decode_at(5, 2, d1);
    }
    // part 6: a permutation of the bins to chase through shared memory
    if (PART == 6)
        for (uint32_t b = lane; b <= kFloorN; b += blockDim.x) histS[b] = (b * 7u + 3u) % (kFloorN + 1u);
    __syncthreads();
    float fx = 1.0f + u01f(floor_hash(lane)), fy = u01f(floor_hash(lane + 77u));
    int ix = (int)(floor_hash(lane) % (kFloorN + 1u));
    // replay draws never agree with a window's here: the windows are replayed
    // rarely, and with any numbers
    auto redraw = [&](uint32_t(&r1)[8]) {
        dr.s1.block((unsigned long long)kPhiloxM0 * (cc - 1u), r1);
        dr.s1.block((unsigned long long)kPhiloxM0 * cc, r1 + 4);
    };
    auto scan_store = [&](const Win<8> &w, uint32_t *p, uint32_t C) {
        uint32_t Es[8];
        const uint32_t accm = scan_weight<8, true, false>(8u, w, smem, kFloorEps, st, Es, redraw);
#pragma unroll
        for (int t = 0; t < 8; ++t) atomicAdd(reinterpret_cast<uint32_t *>(smem + hist_off + Es[t]), 1u);
        *p = C ^ ((w.ctr ^ w.vnib) & accm);
    };
    const unsigned long long t0 = clock64();
    if (PART == 4) {
#pragma unroll 1
        for (uint32_t k = 0; k < windows; ++k) {
            draw8(dr, cc + 1, ah);
            cc += 2;
            fold ^= ah.dn;
#pragma unroll
            for (int t = 0; t < 8; ++t) fold ^= __float_as_uint(ah.l[t]);
        }
    } else if (PART == 5) {
#pragma unroll 1
        for (uint32_t k = 0; k < windows; ++k) {
#pragma unroll
            for (int t = 0; t < 8; ++t) fx = __fadd_rn(fx, fy);
        }
        fold = __float_as_uint(fx);
    } else if (PART == 6) {
#pragma unroll 1
        for (uint32_t k = 0; k < windows; ++k) {
#pragma unroll
            for (int t = 0; t < 8; ++t) ix = (int)histS[ix];
        }
        fold = (uint32_t)ix;
    } else if (PART <= 1) {
        uint32_t row = 0, q = 0;
#pragma unroll 1
        for (uint32_t k = 0; k < windows; ++k) {
            uint32_t *pc = lat + (row * kFloorWPR + q) * kFloorCpb;
            const uint32_t C = *pc, side = q ? *(pc - kFloorCpb) : pc[(kFloorWPR - 1) * kFloorCpb];
            const uint32_t U = lat[((row + 1 == kFloorL ? 0 : row + 1) * kFloorWPR + q) * kFloorCpb];
            const uint32_t D = lat[((row ? row - 1 : kFloorL - 1) * kFloorWPR + q) * kFloorCpb];
            Win<8> w;
            decode<8, 0, false>(C, U, D, side, ah, nullptr, w);
            draw8(dr, cc + 1, ah);
            cc += 2;
            if (PART == 0) {
                scan_store(w, pc, C);
            } else {
                uint32_t f = w.ctr ^ w.vnib ^ w.code[0];
#pragma unroll
                for (int t = 0; t < 8; ++t)
                    f ^= __float_as_uint(w.ns2[t]) ^ __float_as_uint(w.dv[t]) ^ __float_as_uint(w.l[t]);
                fold += f;
            }
            // the full windows of the L = 72 rows: words 0..3 of each row
            if (++q == 4) {
                q = 0;
                if (++row == kFloorL) row = 0;
            }
        }
    } else if (PART == 2) {
#pragma unroll 1
        for (uint32_t k = 0; k < windows; k += 2) {
            scan_store(d0, lat, 0u);
            scan_store(d1, lat, 0u);
        }
    } else if (PART == 3) {
        auto chain = [&](const Win<8> &d) {
            const uint32_t ddb[2] = {prmt_var(kTabDD4_0, kTabDD4_1, d.code[0]), prmt_var(kTabDD4_0, kTabDD4_1, d.code[1])};
            int dd[8];
            unrolled<8>([&](auto tc) {
                constexpr int t = decltype(tc)::value;
                dd[t] = sbyte<(t & 3)>(ddb[t >> 2]);
            });
            auto W = [&](uint32_t e) -> float { return *reinterpret_cast<const float *>(smem + e); };
            uint32_t e1 = st.e4 + dd[0];
            float A = W(e1), diff = __fsub_rn(__fadd_rn(d.dv[0], A), st.wE);
            float c0 = W(st.e4 + dd[1]), c1 = W(e1 + dd[1]);
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                float x0 = 0.0f, x1 = 0.0f;
                if (t + 1 < 8) {
                    x0 = __fsub_rn(__fadd_rn(d.dv[t + 1], c0), st.wE);
                    x1 = __fsub_rn(__fadd_rn(d.dv[t + 1], c1), A);
                }
                const bool acc = d.l[t] < diff;
                st.e4 = acc ? e1 : st.e4;
                st.wE = acc ? A : st.wE;
                if (t + 1 < 8) {
                    A = acc ? c1 : c0;
                    diff = acc ? x1 : x0;
                    e1 = st.e4 + dd[t + 1];
                    if (t + 2 < 8) {
                        c0 = W(st.e4 + dd[t + 2]);
                        c1 = W(e1 + dd[t + 2]);
                    }
                }
            }
        };
#pragma unroll 1
        for (uint32_t k = 0; k < windows; k += 2) {
            chain(d0);
            chain(d1);
        }
    }
    const unsigned long long t1 = clock64();
    if ((lane & 31u) == 0) cycles[lane >> 5] = t1 - t0;
    sink[lane] = fold + st.e4 + __float_as_uint(st.ej2) + lat[0] + (PART == 6 ? 0u : histS[lane]);
}

cudaError_t launch_sweep_floor(int part, uint32_t windows, unsigned long long *cycles, uint32_t *sink,
                               cudaStream_t s)
{
    const size_t smem = win_smem_base(kModeWeight, kFloorN, true) + (size_t)kFloorL * kFloorWPR * kFloorCpb * 4;
    auto go = [&](auto kern) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<1, kFloorCpb, smem, s>>>(windows, cycles, sink);
        return cudaGetLastError();
    };
    switch (part) {
    case 0: return go(k_sweep_floor<0>);
    case 1: return go(k_sweep_floor<1>);
    case 2: return go(k_sweep_floor<2>);
    case 3: return go(k_sweep_floor<3>);
    case 4: return go(k_sweep_floor<4>);
    case 5: return go(k_sweep_floor<5>);
    default: return go(k_sweep_floor<6>);
    }
}

}  // namespace muca
