// k_mlp.cu -- the learned warm start: a small MLP trained and evaluated by
// hand-written FP32 kernels.
//
// The network maps (L/128, T, Delta, x) to y, where x = E_Delta/N is the
// position on the weight axis and y = (lnW(E_Delta) - mean lnW) / N is the
// log weight per site with its mean removed (lnW is extensive in N, so the
// per-site form is what transfers between lattice sizes).  Three hidden
// layers of 128 SiLU units, one linear output; parameters and arithmetic are
// FP32.  It replaces the trivial (zero) or extrapolated initial weight of the
// reference's `continuing` path (muca_delta_multigpu.cu:223-235); the weight
// recursion then runs to the same flatness criterion.
//
// Parameters live in one flat array, each layer's matrix row-major [out][in]
// followed by its bias (offsets kOff*).  A training step is three launches:
//   k_mlp_points  per tile of 32 points: the minibatch draw, the forward pass,
//                 the loss and the deltas of every layer, with both 128 x 128
//                 matrices and the tile's activations in shared memory; it
//                 leaves the activations and deltas in global memory;
//   k_mlp_wgrad   dW = dZ^T H and db = sum dZ of every layer, the minibatch
//                 split over kWSplit slices;
//   k_mlp_update  sums the slices in a fixed order (no atomics: deterministic)
//                 and applies Adam.
// It used to be thirteen launches (gather, forward, backward, then per layer
// the gradient's slices and their sum, Adam, loss) of a few microseconds each,
// most of them too small to fill the GPU.  Every sum keeps its order, so the
// parameters are the same bit for bit.
// The step reads its step number from device memory, so a CUDA graph of K
// steps can be replayed.  muca_mlp_predict runs k_mlp_forward.
#include "muca_device.cuh"
#include "muca_internal.h"

namespace muca {

constexpr int kIn = 4, kHid = 128;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kHid * kIn;
constexpr int kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid;
constexpr int kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid * kHid;
constexpr int kOffW4 = kOffB3 + kHid, kOffB4 = kOffW4 + kHid;
constexpr int kParams = kOffB4 + 1;
static_assert(kParams == 33793, "parameter layout");
constexpr int kTile = 32;      // points per block in forward/backward
constexpr int kThreads = 256;  // threads per block in forward/backward
constexpr int kPitch = kHid + 4;  // row pitch of a staged layer matrix: 16-byte rows
constexpr int kWSplit = 16;       // minibatch slices of the weight gradients
constexpr int kPtPitch = kTile + 4;  // row pitch of a tile's activations in k_mlp_points: 16-byte rows, and
                                     // 8 rows of one 16-byte column on distinct banks
constexpr int kPartPitch = (kParams + 3) / 4 * 4;  // a slice's partial gradients
static_assert(kThreads == 8 * 32 && kTile == 4 * 8 && kHid == 4 * 32, "4 x 4 register tiles");

size_t mlp_param_count() { return kParams; }

__device__ __forceinline__ float sigm(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigm(z); }
// silu(z) and its derivative
__device__ __forceinline__ void silu_both(float z, float &h, float &d)
{
    const float s = sigm(z);
    h = z * s;
    d = s * (1.0f + z * (1.0f - s));
}

// Stage W [kHid][kHid] (16-byte aligned) transposed into sW[j][o] (row pitch kPitch).
__device__ __forceinline__ void stage_transposed(const float *__restrict__ W, float *sW)
{
    for (int t = threadIdx.x; t < kHid * kHid / 4; t += blockDim.x) {
        const int o = (4 * t) / kHid, j = 4 * t - o * kHid;
        const float4 v = reinterpret_cast<const float4 *>(W)[t];
        sW[(j + 0) * kPitch + o] = v.x;
        sW[(j + 1) * kPitch + o] = v.y;
        sW[(j + 2) * kPitch + o] = v.z;
        sW[(j + 3) * kPitch + o] = v.w;
    }
}
// acc[a][b] += sum over k < kHid of A[k][a0 + a] * Bt[k][b0 + b]: A rows of
// pitch kPitch, Bt rows of kTile (both shared memory, 16-byte aligned), in k
// order.  The lanes of a warp share b0 (a broadcast load) and take 32
// consecutive a0 (one 512-byte row segment).
__device__ __forceinline__ void tile_product(const float *__restrict__ A, const float *__restrict__ Bt, int a0,
                                             int b0, float (&acc)[4][4])
{
#pragma unroll 4
    for (int k = 0; k < kHid; ++k) {
        const float4 a = *reinterpret_cast<const float4 *>(A + k * kPitch + a0);
        const float4 b = *reinterpret_cast<const float4 *>(Bt + k * kTile + b0);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
}

// Forward over B points; Y gets the outputs.  Thread (ty, tx) = (threadIdx.x / 32, threadIdx.x % 32)
// owns units 4 tx .. 4 tx + 3 of points 4 ty .. 4 ty + 3 of the tile.  Shared
// memory leaves room for two blocks per SM; told so, the compiler uses 71
// registers where it else chose 40 and kept fewer loads in flight (a prediction
// of 20000 points 134 us for 156, of 4096 51 for 54.5, copies included).
__global__ void __launch_bounds__(kThreads, 2) k_mlp_forward(const float *__restrict__ P, const float *__restrict__ Xb,
                                                          uint32_t B, float *__restrict__ Y)
{
    extern __shared__ __align__(16) float sm[];
    float *sW = sm;                      // [kHid][kPitch]
    float *hA = sW + kHid * kPitch;      // [kHid][kTile], activations transposed
    float *hB = hA + kHid * kTile;       // [kHid][kTile]
    float *sx = hB + kHid * kTile;       // [kTile][kIn]
    __shared__ float red[kThreads / 32][kTile];
    const uint32_t p0 = blockIdx.x * kTile;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int a0 = 4 * tx, b0 = 4 * ty;
    for (int t = threadIdx.x; t < kTile * kIn; t += blockDim.x) {
        const uint32_t p = p0 + t / kIn;
        sx[t] = p < B ? Xb[(size_t)p0 * kIn + t] : 0.0f;
    }
    __syncthreads();
    // layer 1 (4 inputs): straight from global
    {
        float z[4][4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            float w[kIn];
#pragma unroll
            for (int i = 0; i < kIn; ++i) w[i] = P[kOffW1 + (a0 + a) * kIn + i];
            const float b = P[kOffB1 + a0 + a];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float v = b;
#pragma unroll
                for (int i = 0; i < kIn; ++i) v = fmaf(w[i], sx[(b0 + q) * kIn + i], v);
                z[a][q] = v;
            }
            *reinterpret_cast<float4 *>(hA + (a0 + a) * kTile + b0) =
                make_float4(silu(z[a][0]), silu(z[a][1]), silu(z[a][2]), silu(z[a][3]));
        }
    }
    // layers 2 and 3
    float *hin = hA, *hout = hB;
    for (int l = 0; l < 2; ++l) {
        const float *W = P + (l == 0 ? kOffW2 : kOffW3);
        const float *bias = P + (l == 0 ? kOffB2 : kOffB3);
        __syncthreads();  // previous readers of sW are done; hin is written
        stage_transposed(W, sW);
        __syncthreads();
        float acc[4][4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const float b = bias[a0 + a];
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[a][q] = b;
        }
        tile_product(sW, hin, a0, b0, acc);
#pragma unroll
        for (int a = 0; a < 4; ++a)
            *reinterpret_cast<float4 *>(hout + (a0 + a) * kTile + b0) =
                make_float4(silu(acc[a][0]), silu(acc[a][1]), silu(acc[a][2]), silu(acc[a][3]));
        float *t = hin;
        hin = hout;
        hout = t;
    }
    __syncthreads();
    // output layer: point tx, units 16 ty .. 16 ty + 15, then the 8 partial
    // sums in a fixed order
    {
        float s = 0.0f;
#pragma unroll
        for (int j = 16 * ty; j < 16 * ty + 16; ++j) s = fmaf(P[kOffW4 + j], hin[j * kTile + tx], s);
        red[ty][tx] = s;
    }
    __syncthreads();
    if (ty == 0 && p0 + tx < B) {
        float s = P[kOffB4];
#pragma unroll
        for (int g = 0; g < kThreads / 32; ++g) s += red[g][tx];
        Y[p0 + tx] = s;
    }
}

// Minibatch index of point k in step s: Philox(k, s) mod n.
__device__ __forceinline__ uint32_t minibatch_index(uint32_t k, uint32_t step, uint32_t seed, uint32_t n)
{
    RoundKeys<10> key;
    key.init(seed, 0x4d4c5000u);
    const uint4 r = philox<10>(k, step, 0x57A27u, 0u, key);
    return (uint32_t)(((unsigned long long)r.x * n) >> 32);
}

// acc[a][q] += sum over k < kHid, in k order, of W[tx + 32 a][k] H[k][b0 + q]:
// W rows of pitch kPitch read 4 k at a time (the 8 rows of a quarter warp on
// distinct banks), H rows of pitch kPtPitch (one broadcast per warp).
__device__ __forceinline__ void rows_product(const float *__restrict__ W, const float *__restrict__ H, int tx, int b0,
                                             float (&acc)[4][4])
{
#pragma unroll 2
    for (int k = 0; k < kHid; k += 4) {
        float w[4][4], h[4][4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const float4 v = *reinterpret_cast<const float4 *>(W + (tx + 32 * a) * kPitch + k);
            w[a][0] = v.x; w[a][1] = v.y; w[a][2] = v.z; w[a][3] = v.w;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 v = *reinterpret_cast<const float4 *>(H + (k + j) * kPtPitch + b0);
            h[j][0] = v.x; h[j][1] = v.y; h[j][2] = v.z; h[j][3] = v.w;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[a][q] = fmaf(w[a][j], h[j][q], acc[a][q]);
    }
}
// acc[a][q] += sum over o < kHid, in o order, of W[o][4 tx + a] D[o][b0 + q].
__device__ __forceinline__ void columns_product(const float *__restrict__ W, const float *__restrict__ D, int tx,
                                                int b0, float (&acc)[4][4])
{
#pragma unroll 8
    for (int o = 0; o < kHid; ++o) {
        const float4 w = *reinterpret_cast<const float4 *>(W + o * kPitch + 4 * tx);
        const float4 d = *reinterpret_cast<const float4 *>(D + o * kPtPitch + b0);
        const float wv[4] = {w.x, w.y, w.z, w.w}, dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[a][q] = fmaf(wv[a], dv[q], acc[a][q]);
    }
}
// Starts copying W [kHid][kHid] to sW [kHid][kPitch] as one cp.async group.
__device__ __forceinline__ void stage_async(const float *__restrict__ W, float *sW)
{
    for (int t = threadIdx.x; t < kHid * kHid / 4; t += kThreads) {
        const int o = (4 * t) / kHid, j = 4 * t - o * kHid;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(sW + o * kPitch + j)),
                     "l"(W + 4 * t)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// Forward and backward pass of the minibatch, one tile of 32 points per block.
// Point k is row k of (X, T), or with a step number row
// minibatch_index(k) of n.  Leaves the inputs in Xb [B][kIn], the activations
// in H [3][B][kHid], dL/dz of the hidden layers in D [3][B][kHid] and dL/dy =
// 2 (y - t) / B (of the mean squared error) in Dy [B], and the tile's sum of
// squared errors in lpart.  Threads (ty, tx) = (threadIdx.x / 32, threadIdx.x
// % 32): units tx + 32 a (forward) or 4 tx + a (backward) of points 4 ty .. 4
// ty + 3.
__global__ void __launch_bounds__(kThreads, 1) k_mlp_points(const float *__restrict__ P, const float *__restrict__ X,
                                                            const float *__restrict__ T, uint32_t n, uint32_t B,
                                                            uint32_t *__restrict__ step, uint32_t seed,
                                                            float *__restrict__ Xb, float *__restrict__ H,
                                                            float *__restrict__ D, float *__restrict__ Dy,
                                                            float *__restrict__ lpart)
{
    extern __shared__ __align__(16) float sm[];
    float *sW2 = sm, *sW3 = sW2 + kHid * kPitch;       // [kHid][kPitch]
    float *h1 = sW3 + kHid * kPitch, *h2 = h1 + kHid * kPtPitch;  // activations [kHid][kPtPitch]
    float *d1 = h2 + kHid * kPtPitch, *d2 = d1 + kHid * kPtPitch;  // silu' of layers 1 and 2
    float *sx = d2 + kHid * kPtPitch;                  // [kTile][kIn]
    float *st = sx + kTile * kIn, *sdy = st + kTile;   // targets, dL/dy
    __shared__ float red[kThreads / 32][kTile];
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5, b0 = 4 * ty;
    const uint32_t p0 = blockIdx.x * kTile;
    // the update that follows reads the step number here and advances it there
    const uint32_t s_now = step ? step[0] : 0u;
    if (step && blockIdx.x == 0 && tid == 0) step[2] = s_now;
    if (tid < kTile) {
        const uint32_t p = p0 + tid;
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float t = 0.0f;
        if (p < B) {
            const uint32_t i = step ? minibatch_index(p, s_now, seed, n) : p;
            x = reinterpret_cast<const float4 *>(X)[i];
            t = T[i];
            if (step) reinterpret_cast<float4 *>(Xb)[p] = x;
        }
        reinterpret_cast<float4 *>(sx)[tid] = x;
        st[tid] = t;
    }
    // both matrices on their way (one group each), waited for where they are used
    stage_async(P + kOffW2, sW2);
    stage_async(P + kOffW3, sW3);
    __syncthreads();
    // layer l's activations h of this thread's units and points, to global memory
    auto keep = [&](int l, const float (&h)[4][4]) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (p0 + b0 + q < B)
#pragma unroll
                for (int a = 0; a < 4; ++a) H[((size_t)(l - 1) * B + p0 + b0 + q) * kHid + tx + 32 * a] = h[a][q];
    };
    float h[4][4], d[4][4], acc[4][4];
    // layer 1 (4 inputs)
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int o = tx + 32 * a;
        const float4 w = *reinterpret_cast<const float4 *>(P + kOffW1 + o * kIn);
        const float b = P[kOffB1 + o];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 x = reinterpret_cast<const float4 *>(sx)[b0 + q];
            silu_both(fmaf(w.w, x.w, fmaf(w.z, x.z, fmaf(w.y, x.y, fmaf(w.x, x.x, b)))), h[a][q], d[a][q]);
        }
        *reinterpret_cast<float4 *>(h1 + o * kPtPitch + b0) = make_float4(h[a][0], h[a][1], h[a][2], h[a][3]);
        *reinterpret_cast<float4 *>(d1 + o * kPtPitch + b0) = make_float4(d[a][0], d[a][1], d[a][2], d[a][3]);
    }
    keep(1, h);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    // layer 2
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const float b = P[kOffB2 + tx + 32 * a];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[a][q] = b;
    }
    rows_product(sW2, h1, tx, b0, acc);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int o = tx + 32 * a;
#pragma unroll
        for (int q = 0; q < 4; ++q) silu_both(acc[a][q], h[a][q], d[a][q]);
        *reinterpret_cast<float4 *>(h2 + o * kPtPitch + b0) = make_float4(h[a][0], h[a][1], h[a][2], h[a][3]);
        *reinterpret_cast<float4 *>(d2 + o * kPtPitch + b0) = make_float4(d[a][0], d[a][1], d[a][2], d[a][3]);
    }
    keep(2, h);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // layer 3, over layer 1's activations; its derivatives stay in registers
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const float b = P[kOffB3 + tx + 32 * a];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[a][q] = b;
    }
    rows_product(sW3, h2, tx, b0, acc);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
#pragma unroll
        for (int q = 0; q < 4; ++q) silu_both(acc[a][q], h[a][q], d[a][q]);
        *reinterpret_cast<float4 *>(h1 + (tx + 32 * a) * kPtPitch + b0) =
            make_float4(h[a][0], h[a][1], h[a][2], h[a][3]);
    }
    keep(3, h);
    __syncthreads();
    // output: point tx, units 16 ty .. 16 ty + 15, then the 8 partial sums in a
    // fixed order
    {
        float s = 0.0f;
#pragma unroll
        for (int j = 16 * ty; j < 16 * ty + 16; ++j) s = fmaf(P[kOffW4 + j], h1[j * kPtPitch + tx], s);
        red[ty][tx] = s;
    }
    __syncthreads();
    if (ty == 0) {
        float y = P[kOffB4];
#pragma unroll
        for (int k = 0; k < kThreads / 32; ++k) y += red[k][tx];
        float sq = 0.0f, dy = 0.0f;
        if (p0 + tx < B) {
            const float e = y - st[tx];
            sq = e * e;
            dy = 2.0f * e / (float)B;
            Dy[p0 + tx] = dy;
        }
        sdy[tx] = dy;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (tx == 0) lpart[blockIdx.x] = sq;
    }
    __syncthreads();
    // dz3 = dy W4 silu'(z3), over the activations
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int o = tx + 32 * a;
        const float w = P[kOffW4 + o];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            d[a][q] = sdy[b0 + q] * w * d[a][q];
            if (p0 + b0 + q < B) D[((size_t)2 * B + p0 + b0 + q) * kHid + o] = d[a][q];
        }
        *reinterpret_cast<float4 *>(h1 + o * kPtPitch + b0) = make_float4(d[a][0], d[a][1], d[a][2], d[a][3]);
    }
    __syncthreads();
    // dz2 = (W3^T dz3) silu'(z2) over d2, dz1 = (W2^T dz2) silu'(z1)
#pragma unroll
    for (int l = 2; l >= 1; --l) {
        float *out = l == 2 ? d2 : d1;
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[a][q] = 0.0f;
        columns_product(l == 2 ? sW3 : sW2, l == 2 ? h1 : d2, tx, b0, acc);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            float4 *v = reinterpret_cast<float4 *>(out + (4 * tx + a) * kPtPitch + b0);
            const float4 e = *v;
            acc[a][0] *= e.x;
            acc[a][1] *= e.y;
            acc[a][2] *= e.z;
            acc[a][3] *= e.w;
            if (l == 2) *v = make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (p0 + b0 + q < B)
                *reinterpret_cast<float4 *>(D + ((size_t)(l - 1) * B + p0 + b0 + q) * kHid + 4 * tx) =
                    make_float4(acc[0][q], acc[1][q], acc[2][q], acc[3][q]);
        __syncthreads();
    }
}

// Weight gradients of slice blockIdx.x of the minibatch, summed over its
// points in order, into part + blockIdx.x * kPartPitch.  blockIdx.y 0..7: a 64 x
// 64 tile of layer 2 (0..3) or 3 (4..7), 4 x 4 outputs per thread, chunks of
// 32 points in shared memory, the next chunk's loads in flight meanwhile;
// 8 and 9: 64 units of layer 1, one input per thread, by the same chunks;
// 10: layer 4.  The 128 blocks of the large layers come first, one per SM; the
// small ones fill the rest.
constexpr int kWTile = 64, kWChunk = 32;
__global__ void __launch_bounds__(256) k_mlp_wgrad(const float *__restrict__ Xb, const float *__restrict__ H,
                                                   const float *__restrict__ D, const float *__restrict__ Dy,
                                                   uint32_t B, float *__restrict__ part)
{
    __shared__ __align__(16) float sD[2][kWChunk][kWTile], sH[2][kWChunk][kWTile];
    const int tid = threadIdx.x;
    const uint32_t slice = (B + kWSplit - 1) / kWSplit;
    const uint32_t c0 = min(B, blockIdx.x * slice), c1 = min(B, c0 + slice);
    float *g = part + (size_t)blockIdx.x * kPartPitch;
    if (blockIdx.y == 10) {  // output 128 is the bias, which follows the weights
        if (tid <= kHid) {
            float acc = 0.0f;
#pragma unroll 32
            for (uint32_t p = c0; p < c1; ++p)
                acc = fmaf(Dy[p], tid < kHid ? H[((size_t)2 * B + p) * kHid + tid] : 1.0f, acc);
            g[kOffW4 + tid] = acc;
        }
        return;
    }
    const bool first = blockIdx.y >= 8;  // layer 1
    const int l = blockIdx.y >> 2, o0 = first ? (blockIdx.y & 1) * kWTile : (blockIdx.y >> 1 & 1) * kWTile;
    const int i0 = first ? 0 : (blockIdx.y & 1) * kWTile;
    const float *Dl = D + (first ? 0 : (size_t)(l + 1) * B * kHid) + o0, *Hl = first ? Xb : H + (size_t)l * B * kHid + i0;
    const int ti = tid & 15, to = tid >> 4;
    // thread's share of a chunk: rows r and r + 16, 4 columns
    const int r = tid >> 4, c = 4 * (tid & 15);
    float4 nd[2], nh[2];
    auto fetch = [&](uint32_t p) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t q = p + r + 16 * k;
            nd[k] = nh[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (q < c1) {
                nd[k] = *reinterpret_cast<const float4 *>(Dl + (size_t)q * kHid + c);
                if (!first) nh[k] = *reinterpret_cast<const float4 *>(Hl + (size_t)q * kHid + c);
                else if (c == 0) nh[k] = *reinterpret_cast<const float4 *>(Hl + (size_t)q * kIn);
            }
        }
    };
    float acc[4][4], bias = 0.0f;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.0f;
    fetch(c0);
    int buf = 0;
    for (uint32_t p = c0; p < c1; p += kWChunk, buf ^= 1) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            *reinterpret_cast<float4 *>(&sD[buf][r + 16 * k][c]) = nd[k];
            *reinterpret_cast<float4 *>(&sH[buf][r + 16 * k][c]) = nh[k];
        }
        __syncthreads();  // two buffers: the chunk before last has been read by every thread
        fetch(p + kWChunk);
        if (first) {
#pragma unroll 8
            for (int k = 0; k < kWChunk; ++k) acc[0][0] = fmaf(sD[buf][k][tid & 63], sH[buf][k][tid >> 6], acc[0][0]);
        } else {
#pragma unroll 8
            for (int k = 0; k < kWChunk; ++k) {
                const float4 x = *reinterpret_cast<const float4 *>(&sD[buf][k][4 * to]);
                const float4 y = *reinterpret_cast<const float4 *>(&sH[buf][k][4 * ti]);
                const float xv[4] = {x.x, x.y, x.z, x.w}, yv[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(xv[a], yv[b], acc[a][b]);
            }
        }
        if (i0 == 0 && tid < kWTile)
#pragma unroll
            for (int k = 0; k < kWChunk; ++k) bias += sD[buf][k][tid];
    }
    if (first) {
        g[kOffW1 + (o0 + (tid & 63)) * kIn + (tid >> 6)] = acc[0][0];
        if (tid < kWTile) g[kOffB1 + o0 + tid] = bias;
        return;
    }
    float *gW = g + (l == 0 ? kOffW2 : kOffW3), *gb = g + (l == 0 ? kOffB2 : kOffB3);
#pragma unroll
    for (int a = 0; a < 4; ++a)
        *reinterpret_cast<float4 *>(gW + (size_t)(o0 + 4 * to + a) * kHid + i0 + 4 * ti) =
            make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
    if (i0 == 0 && tid < kWTile) gb[o0 + tid] = bias;
}

// The slices' gradients summed in slice order into G, then (with m, v) Adam
// (Kingma & Ba, 2015, Algorithm 1) with bias correction, t = step + 1.  The
// loss (sum of the tiles' squared errors in order, / B) goes to
// losses[step - *base] when a step is given, else to losses[0]; the step
// number advances.
__global__ void __launch_bounds__(256) k_mlp_update(const float *__restrict__ part, const float *__restrict__ lpart,
                                                    int ntiles, uint32_t B, float *__restrict__ P,
                                                    float *__restrict__ G, float *__restrict__ m,
                                                    float *__restrict__ v, uint32_t *__restrict__ step,
                                                    const uint32_t *__restrict__ base, float lr,
                                                    float *__restrict__ losses, uint32_t losses_cap)
{
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    __shared__ float s_c1, s_c2;
    const uint32_t s_now = step ? step[2] : 0u;  // as k_mlp_points read it
    if (m && threadIdx.x == 0) {
        const float t = (float)(s_now + 1u);
        s_c1 = 1.0f - powf(b1, t);
        s_c2 = 1.0f - powf(b2, t);
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 32) {
        float s = 0.0f;
#pragma unroll 16
        for (int b = 0; b < ntiles; ++b) s += lpart[b];
        const uint32_t k = step ? s_now - (base ? *base : 0u) : 0u;
        if (losses && k < losses_cap) losses[k] = s / (float)B;
        if (step) step[0] = s_now + 1u;
    }
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kParams) return;
    float gr = 0.0f;
#pragma unroll
    for (int z = 0; z < kWSplit; ++z) gr += part[(size_t)z * kPartPitch + i];
    G[i] = gr;
    if (!m) return;
    const float mi = b1 * m[i] + (1.0f - b1) * gr;
    const float vi = b2 * v[i] + (1.0f - b2) * gr * gr;
    m[i] = mi;
    v[i] = vi;
    const float mh = mi / s_c1;
    const float vh = vi / s_c2;
    P[i] -= lr * mh / (sqrtf(vh) + eps);
}

static size_t fwd_smem() { return sizeof(float) * ((size_t)kHid * kPitch + 2 * kTile * kHid + kTile * kIn); }
static size_t points_smem()
{
    return sizeof(float) * (2 * (size_t)kHid * kPitch + 4 * (size_t)kHid * kPtPitch + kTile * kIn + 2 * kTile);
}

cudaError_t mlp_prepare()
{
    cudaError_t e = cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_mlp_points, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)points_smem());
    return e;
}

// Scratch of a minibatch of B points, in floats from the (16-byte aligned)
// base: Xb [B][kIn] at 0, Tb [B] at 4B, Y [B] at 5B (muca_mlp_predict and
// muca_mlp_grad copy into them), then, each 16-byte aligned, H and D [3][B]
// [kHid], Dy [B], the tiles' losses and the slices' gradients.
struct MlpScratch {
    float *Xb, *Tb, *H, *D, *Dy, *lpart, *part;
    size_t floats;
};
static size_t align4f(size_t n) { return (n + 3) / 4 * 4; }
static MlpScratch mlp_scratch_layout(float *base, uint32_t B)
{
    MlpScratch m;
    const size_t h = align4f((size_t)B * kIn + 2ull * B), d = h + 3ull * B * kHid, dy = d + 3ull * B * kHid;
    const size_t lp = dy + align4f(B), pt = lp + align4f((B + kTile - 1) / kTile);
    m.Xb = base;
    m.Tb = base ? base + (size_t)B * kIn : nullptr;
    m.H = base ? base + h : nullptr;
    m.D = base ? base + d : nullptr;
    m.Dy = base ? base + dy : nullptr;
    m.lpart = base ? base + lp : nullptr;
    m.part = base ? base + pt : nullptr;
    m.floats = pt + (size_t)kWSplit * kPartPitch;
    return m;
}

size_t mlp_scratch_floats(uint32_t B) { return mlp_scratch_layout(nullptr, B).floats; }

cudaError_t launch_mlp_forward(const float *P, const float *Xb, uint32_t B, float *Y, cudaStream_t s)
{
    if (B == 0) return cudaSuccess;
    k_mlp_forward<<<(B + kTile - 1) / kTile, kThreads, fwd_smem(), s>>>(P, Xb, B, Y);
    return cudaGetLastError();
}

// One gradient evaluation (and, with m/v, one Adam step): of the minibatch
// drawn from (X, T, n) when gather, else of the B points in scratch.
cudaError_t launch_mlp_step(float *P, float *G, float *m, float *v, const float *X, const float *T, uint32_t n,
                            uint32_t B, uint32_t *step, const uint32_t *base, uint32_t seed, bool gather, float lr,
                            float *scratch, float *losses, uint32_t losses_cap, cudaStream_t s)
{
    const MlpScratch sc = mlp_scratch_layout(scratch, B);
    const int nt = (int)((B + kTile - 1) / kTile);
    uint32_t *st = gather ? step : nullptr;
    k_mlp_points<<<nt, kThreads, points_smem(), s>>>(P, gather ? X : sc.Xb, gather ? T : sc.Tb, n, B, st, seed, sc.Xb,
                                                     sc.H, sc.D, sc.Dy, sc.lpart);
    k_mlp_wgrad<<<dim3(kWSplit, 11), 256, 0, s>>>(sc.Xb, sc.H, sc.D, sc.Dy, B, sc.part);
    k_mlp_update<<<(kParams + 255) / 256, 256, 0, s>>>(sc.part, sc.lpart, nt, B, P, G, m, v, st, base, lr, losses,
                                                       losses_cap);
    return cudaGetLastError();
}

}  // namespace muca
