// Learned lambda warm start: an 8 -> 64 -> 64 -> 64 -> 1 MLP with SiLU, BF16 weights and
// activations on the tensor cores (tcgen05, FP32 accumulation in tensor memory), trained on the
// GPU by its own forward and backward kernels.
//
// Parameters are an FP32 master copy, flattened (offsets below); kernels round W1..W3 to BF16 when
// they stage them in shared memory.  Biases, the output layer (w4, b4) and all element-wise math
// stay FP32.  Rounding points (what the host restatement reproduces):
//   x  = bf16((f - mean) * inv_std)
//   a1 = bf16(silu(x W1^T + b1)),  a2 = bf16(silu(a1 W2^T + b2)),  a3 = silu(a2 W3^T + b3)
//   y  = a3 . w4 + b4,  output = y * out_scale
// Backward of L = (1/n) sum (y - t / out_scale)^2:
//   dy = 2 (y - t') / n;  dz3 = bf16(dy w4 silu'(z3));  dz2 = bf16((dz3 W3) silu'(z2));
//   dz1 = bf16((dz2 W2) silu'(z1));  dW_l = dz_l^T a_{l-1};  db_l = sum dz_l;  dw4 = sum dy a3
//
// The forward kernel: a warpgroup per tile of 128 samples (thread t owns sample row t, TMEM lane t) and
// one 64-column accumulator.  The gradient kernel: 512 threads per tile, one
// 64-column accumulator for z and the input gradients in turn and three for the weight gradients,
// which it accumulates over all tiles it processes before one flush.  Weight gradients are MMAs over
// the batch, D[out][in] = dz[b][out] a[b][in], with a column of ones beside the activations whose
// column of D is the bias gradient (64 output features in an M = 128 MMA: the other rows are not
// read).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "dependent_launch.cuh"
#include "tc05.cuh"

namespace akua::mlp {

constexpr int kIn = 8;
constexpr int kInPad = 16;
constexpr int kHid = 64;
constexpr int kTile = 128;
constexpr int kThreads = 128;

// FP32 parameter offsets.
constexpr int kW1 = 0;                  // [64][8]
constexpr int kB1 = kW1 + kHid * kIn;   // [64]
constexpr int kW2 = kB1 + kHid;         // [64][64]
constexpr int kB2 = kW2 + kHid * kHid;  // [64]
constexpr int kW3 = kB2 + kHid;         // [64][64]
constexpr int kB3 = kW3 + kHid * kHid;  // [64]
constexpr int kW4 = kB3 + kHid;         // [64]
constexpr int kB4 = kW4 + kHid;         // [1]
constexpr int kParams = kB4 + 1;        // 8961
// Normalisation: mean[8], inv_std[8], out_scale, blend (see k_mlp_forward).
constexpr int kNorm = 2 * kIn + 2;
constexpr int kLam0 = 3;  // input feature holding iteration 1's lambda

constexpr int kErrTimeout = 1;

// sigmoid(z) = (1 + tanh(z / 2)) / 2 through the hardware tanh approximation (PTX tanh.approx,
// relative error about 2^-11); training and inference use the same forms.
__device__ __forceinline__ float tanh_hw(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float sigmoid(float z) { return __fmaf_rn(0.5f, tanh_hw(0.5f * z), 0.5f); }
__device__ __forceinline__ float silu(float z) { return z * sigmoid(z); }
// Inference: silu of two values, the tanh evaluated on an FP16 pair (tanh.approx.f16x2: one
// multi-function operation for two activations; its error, about 2^-11 relative, is below the
// BF16 rounding the hidden activations get next).
__device__ __forceinline__ float2 silu2(float2 z) {
    const float2 half = make_float2(0.5f, 0.5f);
    const float2 hz = __fmul2_rn(half, z);
    const __half2 h = __floats2half2_rn(hz.x, hz.y);
    uint32_t in, out;
    memcpy(&in, &h, 4);
    asm("tanh.approx.f16x2 %0, %1;" : "=r"(out) : "r"(in));
    __half2 ht;
    memcpy(&ht, &out, 4);
    return __fmul2_rn(z, __ffma2_rn(half, __half22float2(ht), half));
}
__device__ __forceinline__ float dsilu(float z) {
    const float s = sigmoid(z);
    return s * (1.0f + z * (1.0f - s));
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ uint16_t bf16_bits(float a) {
    const __nv_bfloat16 v = __float2bfloat16_rn(a);
    return *reinterpret_cast<const uint16_t*>(&v);
}
__device__ __forceinline__ float bf16_round(float a) {
    return __bfloat162float(__float2bfloat16_rn(a));
}

// Stages a [64][kin] weight (row-major FP32) as a BF16 K-major B operand with K = kpad columns (zeros
// beyond kin).
__device__ __forceinline__ void stage_weight(uint8_t* dst, const float* __restrict__ w, int kin,
                                             int kpad, int t) {
    for (int e = t; e < kHid * kpad; e += kThreads) {
        const int r = e / kpad, k = e - r * kpad;
        *reinterpret_cast<uint16_t*>(dst + tc::kmajor_offset(r, k, kpad)) =
            bf16_bits(k < kin ? w[r * kin + k] : 0.f);
    }
}

// BF16 operand images of W1, W2, W3 in the kernels' shared-memory layout, built by k_mlp_image when
// parameters are set and kept up to date by k_mlp_adam; a CTA copies them instead of converting.
constexpr int kImageBytes = (kHid * kInPad + 2 * kHid * kHid) * 2;

__global__ void __launch_bounds__(kThreads)
    k_mlp_image(const float* __restrict__ params, uint8_t* __restrict__ image) {
    const int t = threadIdx.x;
    stage_weight(image, params + kW1, kIn, kInPad, t);
    stage_weight(image + kHid * kInPad * 2, params + kW2, kHid, kHid, t);
    stage_weight(image + kHid * kInPad * 2 + kHid * kHid * 2, params + kW3, kHid, kHid, t);
}

// ------------------------------------------------------------------------------------ forward
// Four tiles of 128 samples per CTA, a warpgroup each with its own accumulator, operand tiles and
// barriers; the weights are staged once for all four.
constexpr int kFwdGroups = 4;
constexpr int kFwdThreads = kFwdGroups * kTile;
struct FwdSmem {
    alignas(128) uint8_t w1[kHid * kInPad * 2];
    alignas(128) uint8_t w2[kHid * kHid * 2];
    alignas(128) uint8_t w3[kHid * kHid * 2];
    alignas(128) uint8_t x[kFwdGroups][kTile * kInPad * 2];
    alignas(128) uint8_t h[kFwdGroups][kTile * kHid * 2];
    alignas(16) float b1[kHid], b2[kHid], b3[kHid], w4[kHid];
    float norm[kNorm];
    float b4;
    alignas(8) uint64_t bar[kFwdGroups];
    uint32_t tmem;
};
constexpr size_t kFwdSmem = sizeof(FwdSmem);

// SiLU of 32 columns of this thread's TMEM row plus their biases, two at a time: f(column, values).
template <class F>
__device__ __forceinline__ void silu_columns(uint32_t taddr, const float* b, F&& f) {
    uint32_t r[2][16];
#pragma unroll
    for (int c = 0; c < 2; ++c) tc::tmem_ld16_async(taddr + 16 * c, r[c]);
    tc::tmem_wait_ld();
#pragma unroll
    for (int c = 0; c < 2; ++c) tc::tmem_after_wait(r[c]);
#pragma unroll
    for (int q = 0; q < 32; q += 2) {
        const float2 z = make_float2(__uint_as_float(r[q / 16][q % 16]),
                                     __uint_as_float(r[q / 16][q % 16 + 1]));
        f(q, silu2(__fadd2_rn(z, *reinterpret_cast<const float2*>(b + q))));
    }
}

// Epilogue of a hidden layer: TMEM columns [col, col+64) of this thread's row -> bias, SiLU,
// BF16 -> row t of the next layer's A tile.
__device__ __forceinline__ void hidden_epilogue(uint32_t taddr, const float* b, uint8_t* h, int t) {
#pragma unroll
    for (int c0 = 0; c0 < kHid; c0 += 32) {
        uint32_t v[16];
        silu_columns(taddr + c0, b + c0, [&](int q, float2 a) { v[q / 2] = pack_bf16(a.x, a.y); });
#pragma unroll
        for (int q = 0; q < 16; q += 4)
            *reinterpret_cast<uint4*>(h + tc::kmajor_offset(t, c0 + 2 * q, 64)) =
                make_uint4(v[q], v[q + 1], v[q + 2], v[q + 3]);
    }
}

// Output layer on the FP32 pipe: b4 + sum_c w4[c] silu(z3[c] + b3[c]).
__device__ __forceinline__ float output_layer(uint32_t taddr, const float* b3, const float* w4,
                                              float b4) {
    float y = b4;
#pragma unroll
    for (int c0 = 0; c0 < kHid; c0 += 32)
        silu_columns(taddr + c0, b3 + c0, [&](int q, float2 a) {
            y = __fmaf_rn(w4[c0 + q], a.x, y);
            y = __fmaf_rn(w4[c0 + q + 1], a.y, y);
        });
    return y;
}

__device__ __forceinline__ void load_features(const float* __restrict__ feat, int i, int n,
                                              const float* norm, float (&f)[kIn]) {
    if (i < n) {
        const float4 a = reinterpret_cast<const float4*>(feat)[2 * (size_t)i];
        const float4 b = reinterpret_cast<const float4*>(feat)[2 * (size_t)i + 1];
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
        f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    } else {
#pragma unroll
        for (int k = 0; k < kIn; ++k) f[k] = norm[k];
    }
}

// Features (n x 8, FP32) -> out2[i] = the network's estimate p_i (output * out_scale) and
// out[i] = lambda0_i + blend * (p_i - lambda0_i), lambda0 = feature 3 (blend 1: out = p); the
// latter also into out4[4 i] when given.
//
// Bound by the SiLU epilogues' issue slots and by a tile's chain of three MMAs, which the other
// warpgroups' epilogues fill: two CTAs of four warpgroups per SM (64 registers a thread).
// 1M samples: 74 -> 65 us against five CTAs of one warpgroup with scalar epilogues, 155,648: 20.7 ->
// 12.9 (the hardware tanh of 192 activations a sample alone takes about 40 at 1M).
__global__ void __launch_bounds__(kFwdThreads, 2)
    k_mlp_forward(const float* __restrict__ params, const uint8_t* __restrict__ image,
                  const float* __restrict__ norm, const float* __restrict__ feat, int n,
                  float* __restrict__ out, float* __restrict__ out2, float* __restrict__ out4,
                  uint32_t* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    FwdSmem& S = *reinterpret_cast<FwdSmem*>(smem_raw);
    static_assert(offsetof(FwdSmem, w2) == offsetof(FwdSmem, w1) + sizeof(S.w1) &&
                      offsetof(FwdSmem, w3) == offsetof(FwdSmem, w2) + sizeof(S.w2) &&
                      sizeof(S.w1) + sizeof(S.w2) + sizeof(S.w3) == kImageBytes,
                  "the weight image is w1, w2, w3 back to back");
    const int group = threadIdx.x / kTile, t = threadIdx.x % kTile, warp = t >> 5;
    if (t == 0) tc::mbar_init(&S.bar[group], 1);
    uint8_t* x = S.x[group];
    uint8_t* h = S.h[group];
    // columns 8..15 of the input tile stay zero
    *reinterpret_cast<uint4*>(x + tc::kmajor_offset(t, 8, kInPad)) = make_uint4(0, 0, 0, 0);
    if (threadIdx.x < 32) tc::tmem_alloc(&S.tmem, kFwdGroups * kHid);
    pdl::wait_for_previous(params, image, norm, feat);
    {
        const uint4* src = reinterpret_cast<const uint4*>(image);
        uint4* dst = reinterpret_cast<uint4*>(S.w1);
        for (int k = threadIdx.x; k < kImageBytes / 16; k += kFwdThreads) dst[k] = src[k];
    }
    if (threadIdx.x < kHid) {
        S.b1[t] = params[kB1 + t];
        S.b2[t] = params[kB2 + t];
        S.b3[t] = params[kB3 + t];
        S.w4[t] = params[kW4 + t];
    }
    if (threadIdx.x < kNorm) S.norm[t] = norm[t];
    if (threadIdx.x == 0) S.b4 = params[kB4];
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = S.tmem + kHid * group;
    const uint32_t lane = tmem + ((uint32_t)(warp * 32) << 16);
    constexpr uint32_t idesc = tc::idesc_bf16(128, 64);
    const uint64_t dx = tc::smem_desc(tc::smem_addr(x), 128, kInPad * 16);
    const uint64_t dw1 = tc::smem_desc(tc::smem_addr(S.w1), 128, kInPad * 16);
    const uint32_t sh = tc::smem_addr(h), sw2 = tc::smem_addr(S.w2), sw3 = tc::smem_addr(S.w3);
    uint32_t phase = 0;
    bool ok = true;
    auto publish = [&]() {  // this warpgroup's operand stores and tensor-memory reads are done
        tc::fence_async_smem();
        tc::fence_before_sync();
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kTile) : "memory");
        if (t == 0) tc::fence_after_sync();
    };
    // after a wait that ran out nothing is issued or written any more
    auto wait = [&]() {
        if (ok) ok = tc::mbar_wait(&S.bar[group], phase);
        phase ^= 1;
        tc::fence_after_sync();
    };
    auto layer = [&](uint32_t sw) {
        if (t == 0 && ok) {
#pragma unroll
            for (int s = 0; s < kHid / 16; ++s)
                tc::mma_bf16(tmem, tc::smem_desc(sh + 256 * s, 128, kHid * 16),
                             tc::smem_desc(sw + 256 * s, 128, kHid * 16), idesc, s > 0);
            tc::mma_commit(&S.bar[group]);
        }
        wait();
    };
    const int tiles = (n + kTile - 1) / kTile;
    // tiles in an order that gives every CTA one before any gets a second
    const int first = blockIdx.x + gridDim.x * group, step = gridDim.x * kFwdGroups;
    float fnext[kIn];
    load_features(feat, first * kTile + t, n, S.norm, fnext);
    const float blend = S.norm[2 * kIn + 1];
    for (int tile = first; tile < tiles; tile += step) {
        const int i = tile * kTile + t;
        const float lam0 = fnext[kLam0];
        float f[kIn];
#pragma unroll
        for (int k = 0; k < kIn; ++k) f[k] = (fnext[k] - S.norm[k]) * S.norm[kIn + k];
        if (tile + step < tiles)  // the next tile's features, in flight meanwhile
            load_features(feat, (tile + step) * kTile + t, n, S.norm, fnext);
        *reinterpret_cast<uint4*>(x + tc::kmajor_offset(t, 0, kInPad)) =
            make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]),
                       pack_bf16(f[6], f[7]));
        publish();
        if (t == 0 && ok) {
            tc::mma_bf16(tmem, dx, dw1, idesc, 0);
            tc::mma_commit(&S.bar[group]);
        }
        wait();
        hidden_epilogue(lane, S.b1, h, t);
        publish();
        layer(sw2);
        hidden_epilogue(lane, S.b2, h, t);
        publish();
        layer(sw3);
        const float y = output_layer(lane, S.b3, S.w4, S.b4);
        if (ok && i < n) {
            const float o = y * S.norm[2 * kIn];
            const float used = blend == 1.0f ? o : __fmaf_rn(blend, o - lam0, lam0);
            out[i] = used;
            if (out2) out2[i] = o;
            if (out4) out4[4 * (size_t)i] = used;  // a float4 array's 4th component
        }
    }
    if (!ok) atomicOr(err, (uint32_t)kErrTimeout);
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc::fence_after_sync();
        tc::tmem_free(S.tmem, kFwdGroups * kHid);
    }
}

// ----------------------------------------------------------------------------------- gradient
// One CTA per SM, 16 warps: warp w owns rows 32 (w % 4) .. + 31 of the tile and columns
// 16 (w / 4) .. + 15 of every layer, so a layer's SiLU is spread over 512 threads.  The weight
// gradients' operands are the forward tiles read along the other axis; the bias gradients are a
// column of ones beside the activations.  Per tile five dependent MMAs (z1, z2, z3, da2, da1); the
// weight-gradient MMAs run behind them while the next epilogue works, which is why dz and x have two
// buffers: an MMA's operands are overwritten only after a later commit of the same issue order.
//
// Bound by the chain of a tile (4 us: five MMAs with their epilogues, 33% of the issue slots) and
// about 8 us of start and flush.  65,536 samples (512 tiles, four rounds of 152 CTAs): 95 -> 23 us
// against 4 warps per CTA with transposed copies stored two bytes at a time and dw4 reduced by
// shuffles in every tile; an Adam step, its two kernels together, 110 -> 24 us (29 before each was set
// up while the one before it ends).
constexpr int kGradThreads = 512;
constexpr int kGradCols = 16;  // columns per thread
constexpr uint32_t kColW = 0;                                // z1, z2, z3, da2, da1 in turn
constexpr uint32_t kColG3 = 64, kColG2 = 144, kColG1 = 224;  // 80, 80, 16 columns
constexpr uint32_t kGradTmem = 256;
constexpr int kNT = 80;  // columns of an activation tile: 64 features, ones, zeros
constexpr int kDzBytes = kTile * kHid * 2;
constexpr int kDzPad = 1024;  // rows 64..127 of the M = 128 operand run on past the tile

struct GradSmem {
    alignas(128) uint8_t w1[kHid * kInPad * 2];      // [out][in16], K-major: the image's three
    alignas(128) uint8_t w2[kHid * kHid * 2];        // [out][in]
    alignas(128) uint8_t w3[kHid * kHid * 2];
    alignas(128) uint8_t x[2][kTile * kInPad * 2];   // [b][16]: 8 features, ones, zeros
    alignas(128) uint8_t a1[kTile * kNT * 2];        // [b][80]
    alignas(128) uint8_t a2[kTile * kNT * 2];
    alignas(128) uint8_t dz[2][kDzBytes + kDzPad];   // [b][64]
    float b1[kHid], b2[kHid], b3[kHid], w4[kHid];
    float norm[kNorm];
    float b4;
    float y[4][kTile];     // partial outputs of the four column groups
    float gw4[4][kHid];    // dw4 of the four row quarters
    float gb4, loss;
    alignas(8) uint64_t bar;
    uint32_t tmem;
};

constexpr size_t kGradSmem = sizeof(GradSmem);

// Accumulates into grad[kParams] (dL/dparams) and grad[kParams] += loss.  Targets are in output
// units (lambda); the loss is over `n_total` samples (this call may see a slice of them).  `image`:
// the BF16 operand images of W1..W3 (k_mlp_image).
__global__ void __launch_bounds__(kGradThreads, 1)
    k_mlp_grad(const float* __restrict__ params, const uint8_t* __restrict__ image,
               const float* __restrict__ norm, const float* __restrict__ feat,
               const float* __restrict__ target, int n, float inv_n_total,
               float* __restrict__ grad, uint32_t* __restrict__ err) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    GradSmem& S = *reinterpret_cast<GradSmem*>(smem_raw);
    static_assert(offsetof(GradSmem, w2) == sizeof(S.w1) &&
                      offsetof(GradSmem, w3) == sizeof(S.w1) + sizeof(S.w2),
                  "the weight image is w1, w2, w3 back to back");
    const int t = threadIdx.x, warp = t >> 5;
    const int row = t & (kTile - 1);  // 32 (warp % 4) + lane
    const int group = t / kTile;      // warp / 4
    const int c0 = kGradCols * group;
    if (t == 0) {
        S.gb4 = 0.f;
        S.loss = 0.f;
        tc::mbar_init(&S.bar, 1);
    }
    {  // constant columns of the operand tiles: a one and zeros
        const uint4 ones = make_uint4(pack_bf16(1.0f, 0.0f), 0u, 0u, 0u);
        const uint4 zeros = make_uint4(0u, 0u, 0u, 0u);
        if (group < 2) {
            *reinterpret_cast<uint4*>(S.x[group] + tc::kmajor_offset(row, 8, kInPad)) = ones;
        } else {
            uint8_t* a = group == 2 ? S.a1 : S.a2;
            *reinterpret_cast<uint4*>(a + tc::kmajor_offset(row, kHid, kNT)) = ones;
            *reinterpret_cast<uint4*>(a + tc::kmajor_offset(row, kHid + 8, kNT)) = zeros;
        }
    }
    if (warp == 0) tc::tmem_alloc(&S.tmem, kGradTmem);
    pdl::wait_for_previous(params, image, norm, feat, target);
    for (int k = t; k < kImageBytes / 16; k += kGradThreads)
        reinterpret_cast<uint4*>(S.w1)[k] = reinterpret_cast<const uint4*>(image)[k];
    if (t < kHid) {
        S.b1[t] = params[kB1 + t];
        S.b2[t] = params[kB2 + t];
        S.b3[t] = params[kB3 + t];
        S.w4[t] = params[kW4 + t];
    }
    if (t < kNorm) S.norm[t] = norm[t];
    if (t == 0) S.b4 = params[kB4];
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = S.tmem;
    const uint32_t lane = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    const uint32_t sx = tc::smem_addr(S.x[0]), sw1 = tc::smem_addr(S.w1);
    const uint32_t sa1 = tc::smem_addr(S.a1), sa2 = tc::smem_addr(S.a2);
    const uint32_t sw2 = tc::smem_addr(S.w2), sw3 = tc::smem_addr(S.w3);
    const uint32_t sdz = tc::smem_addr(S.dz[0]);
    constexpr uint32_t kXBytes = kTile * kInPad * 2, kDz = kDzBytes + kDzPad;
    const float inv_scale = 1.0f / S.norm[2 * kIn];
    uint32_t phase = 0;
    uint32_t acc = 0;  // the weight-gradient accumulators hold data
    bool ok = true;

    // issue helpers (thread 0 only); every operand's 8-row groups are `sbo` bytes apart
    auto forward = [&](uint32_t a, uint32_t a_sbo, uint32_t b, int ksteps, uint32_t b_sbo) {
        constexpr uint32_t id = tc::idesc_bf16(kTile, kHid);
        for (int s = 0; s < ksteps; ++s)  // W = A B^T
            tc::mma_bf16(tmem + kColW, tc::smem_desc(a + 256 * s, 128, a_sbo),
                         tc::smem_desc(b + 256 * s, 128, b_sbo), id, s > 0);
        tc::mma_commit(&S.bar);
    };
    auto backward = [&](uint32_t dz, uint32_t w) {  // W[b][in] = dz[b][out] w[out][in]
        constexpr uint32_t id = tc::idesc_bf16(kTile, kHid) | tc::kTransposeB;
#pragma unroll
        for (int s = 0; s < kHid / 16; ++s)
            tc::mma_bf16(tmem + kColW, tc::smem_desc(dz + 256 * s, 128, kHid * 16),
                         tc::smem_desc(w + 2 * kHid * 16 * s, kHid * 16, 128), id, s > 0);
        tc::mma_commit(&S.bar);
    };
    // G[out][in] += dz[b][out] act[b][in], `cols` columns of the activation tile
    auto weights = [&](uint32_t g, uint32_t dz, uint32_t act, uint32_t cols) {
        const uint32_t id = tc::idesc_bf16(kTile, cols) | tc::kTransposeA | tc::kTransposeB;
#pragma unroll
        for (int s = 0; s < kTile / 16; ++s)
            tc::mma_bf16(tmem + g, tc::smem_desc(dz + 2 * kHid * 16 * s, kHid * 16, 128),
                         tc::smem_desc(act + 2 * cols * 16 * s, cols * 16, 128), id, (acc | s) != 0);
    };
    auto publish = [&]() {  // this thread's operand stores and tensor-memory reads are done
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if (t == 0) tc::fence_after_sync();
    };
    // After a wait that ran out nothing waits again; the next tile's check ends the kernel.
    auto wait = [&]() {
        if (ok) ok = tc::mbar_wait(&S.bar, phase);
        phase ^= 1;
        tc::fence_after_sync();
    };
    auto put_x = [&](int buf, const float (&f)[kIn]) {  // row t of the tile, threads 0..127
        float v[kIn];
#pragma unroll
        for (int k = 0; k < kIn; ++k) v[k] = (f[k] - S.norm[k]) * S.norm[kIn + k];
        *reinterpret_cast<uint4*>(S.x[buf] + tc::kmajor_offset(t, 0, kInPad)) =
            make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]),
                       pack_bf16(v[6], v[7]));
    };
    auto put16 = [&](uint8_t* tile, int cols, const float (&v)[kGradCols]) {
        *reinterpret_cast<uint4*>(tile + tc::kmajor_offset(row, c0, cols)) =
            make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]),
                       pack_bf16(v[6], v[7]));
        *reinterpret_cast<uint4*>(tile + tc::kmajor_offset(row, c0 + 8, cols)) =
            make_uint4(pack_bf16(v[8], v[9]), pack_bf16(v[10], v[11]), pack_bf16(v[12], v[13]),
                       pack_bf16(v[14], v[15]));
    };
    // a = silu(z + b) to the activation tile, silu'(z + b) kept
    auto hidden = [&](const float* bias, uint8_t* tile, float (&d)[kGradCols]) {
        float v[kGradCols];
        tc::tmem_ld16(lane + kColW + c0, v);
#pragma unroll
        for (int q = 0; q < kGradCols; ++q) {
            const float z = v[q] + bias[c0 + q];
            v[q] = silu(z);
            d[q] = dsilu(z);
        }
        put16(tile, kNT, v);
    };

    const int tiles = (n + kTile - 1) / kTile;
    float f[kIn], gw4[kGradCols], gb4 = 0.f, loss = 0.f;
#pragma unroll
    for (int q = 0; q < kGradCols; ++q) gw4[q] = 0.f;
    int buf = 0;
    if (t < kTile) {
        load_features(feat, blockIdx.x * kTile + t, n, S.norm, f);
        put_x(0, f);
    }
    publish();
    if (t == 0) forward(sx, kInPad * 16, sw1, 1, kInPad * 16);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int i = tile * kTile + row;
        const bool valid = i < n;
        const float tgt = valid ? target[i] * inv_scale : 0.f;
        const bool more = tile + (int)gridDim.x < tiles;
        if (more && t < kTile) load_features(feat, (tile + gridDim.x) * kTile + t, n, S.norm, f);
        float d1[kGradCols], d2[kGradCols];
        wait();  // z1
        hidden(S.b1, S.a1, d1);
        publish();
        if (t == 0) forward(sa1, kNT * 16, sw2, kHid / 16, kHid * 16);
        wait();  // z2
        hidden(S.b2, S.a2, d2);
        publish();
        if (t == 0) forward(sa2, kNT * 16, sw3, kHid / 16, kHid * 16);
        wait();  // z3
        float a3[kGradCols], v[kGradCols];
        tc::tmem_ld16(lane + kColW + c0, v);
        float part = 0.f;
#pragma unroll
        for (int q = 0; q < kGradCols; ++q) {
            const float z = v[q] + S.b3[c0 + q];
            a3[q] = silu(z);
            v[q] = dsilu(z);
            part = __fmaf_rn(S.w4[c0 + q], a3[q], part);
        }
        S.y[group][row] = part;
        ok = __syncthreads_and(ok);
        if (!ok) break;  // uniform: a wait ran out
        const float y = S.b4 + ((S.y[0][row] + S.y[1][row]) + (S.y[2][row] + S.y[3][row]));
        const float e = valid ? y - tgt : 0.f;
        const float dy = 2.0f * e * inv_n_total;
        if (group == 0) {
            loss = __fmaf_rn(e * e, inv_n_total, loss);
            gb4 += dy;
        }
#pragma unroll
        for (int q = 0; q < kGradCols; ++q) {
            gw4[q] = __fmaf_rn(dy, a3[q], gw4[q]);
            v[q] = dy * S.w4[c0 + q] * v[q];
        }
        put16(S.dz[0], kHid, v);
        publish();
        if (t == 0) {
            backward(sdz, sw3);
            weights(kColG3, sdz, sa2, kNT);
        }
        wait();  // da2
        tc::tmem_ld16(lane + kColW + c0, v);
#pragma unroll
        for (int q = 0; q < kGradCols; ++q) v[q] = v[q] * d2[q];
        put16(S.dz[1], kHid, v);
        publish();
        if (t == 0) {
            backward(sdz + kDz, sw2);
            weights(kColG2, sdz + kDz, sa1, kNT);
        }
        wait();  // da1, and everything issued before it
        tc::tmem_ld16(lane + kColW + c0, v);
#pragma unroll
        for (int q = 0; q < kGradCols; ++q) v[q] = v[q] * d1[q];
        put16(S.dz[0], kHid, v);
        if (more && t < kTile) put_x(buf ^ 1, f);
        publish();
        if (t == 0) {
            weights(kColG1, sdz, sx + buf * kXBytes, kInPad);
            if (more) forward(sx + (buf ^ 1) * kXBytes, kInPad * 16, sw1, 1, kInPad * 16);
            else tc::mma_commit(&S.bar);
        }
        buf ^= 1;
        acc = 1;
    }
    if (ok) wait();  // the last weight gradients
    ok = __syncthreads_and(ok);
    // flush: rows 0..63 of the weight-gradient accumulators are lanes 0..63
    if (ok && row < kHid) {
        const int o = row;  // output feature
        float v[16];
        auto row16 = [&](float* g) {
#pragma unroll
            for (int q = 0; q < 16; q += 4) tc::red_add4(g + q, v[q], v[q + 1], v[q + 2], v[q + 3]);
        };
        tc::tmem_ld16(lane + kColG3 + c0, v);
        row16(grad + kW3 + o * kHid + c0);
        tc::tmem_ld16(lane + kColG2 + c0, v);
        row16(grad + kW2 + o * kHid + c0);
        if (group == 0) {
            tc::tmem_ld16(lane + kColG3 + kHid, v);
            atomicAdd(&grad[kB3 + o], v[0]);
        } else if (group == 1) {
            tc::tmem_ld16(lane + kColG2 + kHid, v);
            atomicAdd(&grad[kB2 + o], v[0]);
        } else if (group == 2) {
            tc::tmem_ld16(lane + kColG1, v);
            tc::red_add4(grad + kW1 + o * kIn, v[0], v[1], v[2], v[3]);
            tc::red_add4(grad + kW1 + o * kIn + 4, v[4], v[5], v[6], v[7]);
            atomicAdd(&grad[kB1 + o], v[kIn]);
        }
    }
    if (ok) {  // dw4, db4 and the loss: sums over the rows
#pragma unroll
        for (int q = 0; q < kGradCols; ++q) {
#pragma unroll
            for (int o = 16; o; o >>= 1) gw4[q] += __shfl_xor_sync(0xffffffffu, gw4[q], o);
            if ((t & 31) == 0) S.gw4[warp & 3][c0 + q] = gw4[q];
        }
        if (group == 0) {
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                gb4 += __shfl_xor_sync(0xffffffffu, gb4, o);
                loss += __shfl_xor_sync(0xffffffffu, loss, o);
            }
            if ((t & 31) == 0) {
                atomicAdd(&S.gb4, gb4);
                atomicAdd(&S.loss, loss);
            }
        }
        __syncthreads();
        if (t < kHid)
            atomicAdd(&grad[kW4 + t],
                      (S.gw4[0][t] + S.gw4[1][t]) + (S.gw4[2][t] + S.gw4[3][t]));
        if (t == 0) {
            atomicAdd(&grad[kB4], S.gb4);
            atomicAdd(&grad[kParams], S.loss);
        }
    }
    if (!ok && t == 0) atomicOr(err, (uint32_t)kErrTimeout);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after_sync();
        tc::tmem_free(tmem, kGradTmem);
    }
}

// Place of parameter k in the operand images (bytes), or -1 for biases and the output layer.
__device__ __forceinline__ int image_offset(int k) {
    if (k < kB1) return (int)tc::kmajor_offset(k / kIn, k % kIn, kInPad);
    if (k >= kW2 && k < kB2)
        return kHid * kInPad * 2 + (int)tc::kmajor_offset((k - kW2) / kHid, (k - kW2) % kHid, kHid);
    if (k >= kW3 && k < kB3)
        return (kHid * kInPad + kHid * kHid) * 2 +
               (int)tc::kmajor_offset((k - kW3) / kHid, (k - kW3) % kHid, kHid);
    return -1;
}

// Adam on the FP32 master parameters; clears the gradient (and the loss slot) afterwards and keeps
// the weights' BF16 images up to date (a kernel of its own took 7 us to rebuild them).
__global__ void k_mlp_adam(float* __restrict__ params, float* __restrict__ grad,
                           float* __restrict__ m, float* __restrict__ v,
                           uint8_t* __restrict__ image, float lr, float beta1, float beta2,
                           float eps, float bc1, float bc2) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    pdl::wait_for_previous(params, grad, m, v);
    if (k > kParams) return;
    if (k == kParams) {
        grad[k] = 0.f;
        return;
    }
    const float g = grad[k];
    const float mk = beta1 * m[k] + (1.0f - beta1) * g;
    const float vk = beta2 * v[k] + (1.0f - beta2) * g * g;
    m[k] = mk;
    v[k] = vk;
    const float p = params[k] - lr * (mk / bc1) / (sqrtf(vk / bc2) + eps);
    params[k] = p;
    grad[k] = 0.f;
    const int at = image_offset(k);
    if (at >= 0) *reinterpret_cast<uint16_t*>(image + at) = bf16_bits(p);
}

}  // namespace akua::mlp
