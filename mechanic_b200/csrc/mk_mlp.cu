// mk_mlp.cu — the network of the learned parts on the 5th-generation tensor
// cores (tcgen05, bf16 operands, f32 accumulation in tensor memory).
//
// One network shape serves both learned parts: 16 inputs (slot 15 is the
// constant 1 that carries the first layer's bias), two hidden layers of 64
// with ReLU, 16 outputs (the caller uses the first few):
//   h1 = relu(W1 x),  h2 = relu(W2 h1 + b2),  y = W3 h2 + b3.
// Parameters are one f32 array (row-major [out][in]): W1 64x16 | W2 64x64 |
// W3 16x64 | b2 64 | b3 16; every CTA rounds the weights to bf16 as it brings
// them into shared memory.
//
// 128 threads take a tile of 128 samples: a training CTA one at a time, a forward CTA
// up to 8 beside one another (1,024 threads).  Thread t of the 128 owns sample t of
// the tile, which is TMEM lane t of every accumulator, so the epilogues are
// one tcgen05.ld per 16 columns and no shuffles.  The backward pass reuses
// the activations where they lie: the same shared-memory tiles are read
// K-major by the data-gradient MMAs and MN-major by the weight-gradient MMAs
// (which reduce over the 128 samples of the tile), so nothing is transposed.
// The two 64-row weight gradients are stacked into one M = 128 MMA
// ([dH2; dH1] x [H1; X]^T), whose off-diagonal blocks are unused except the
// column of the constant input, which is the sum of dH2 over samples (db2).
// Weight gradients accumulate in TMEM across a CTA's tiles; each CTA writes
// one partial, and after a grid barrier the partials are summed in CTA order,
// so the gradient of a batch is deterministic.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>

#include "mk_device.cuh"
#include "mk_internal.h"
#include "mk_mlp.h"
#include "mk_tc.cuh"

namespace mk {
namespace mlp {

constexpr uint32_t kTile = 128, kThreads = 128, kCH = 2048;   // bytes per 8-column chunk of a 128-row tile
constexpr uint32_t kTmemCols = 256;
// accumulator columns: layer 1 / dH1, layer 2 / dH2, layer 3, dW3^T block, [dW2 | db2 | dW1] block
constexpr uint32_t cAcc1 = 0, cAcc2 = 64, cAcc3 = 128, cDB = 144, cDA = 160;
constexpr uint32_t kWaitLimit = 1u << 20;

template <uint32_t kWeightsAt>
struct WeightLayout {
    static constexpr uint32_t W1 = kWeightsAt;
    static constexpr uint32_t W2 = W1 + 2048;
    static constexpr uint32_t W3 = W2 + 8192;
    static constexpr uint32_t B2 = W3 + 2048;
    static constexpr uint32_t B3 = B2 + 256;
    static constexpr uint32_t END = B3 + 64;
};
struct TrainLayout {
    // F: [H1 (chunks 0-7) | X (8-9)]; G: [H2 (0-7) | dH2 (8-15) | dH1 (16-23)]; Y: dY (0-1)
    static constexpr uint32_t F = 0;
    static constexpr uint32_t G = F + 10 * kCH;
    static constexpr uint32_t Y = G + 24 * kCH;
    using W = WeightLayout<Y + 2 * kCH>;
    static constexpr uint32_t RED = W::END;              // 4 warps x 17 floats (db3, loss)
    static constexpr uint32_t BAR = RED + 4 * 17 * 4 + 16;
    static constexpr uint32_t SLOT = BAR + 8;
    static constexpr uint32_t BYTES = SLOT + 8;
};
// Forward only: X, H1 and H2 take one another's place in one tile of 8 chunks (each is
// dead once the MMAs of its layer are complete), and the three accumulators the same 64
// TMEM columns, so that 8 tiles are worked on beside one another on an SM.
constexpr uint32_t kForwardTmem = 64, kForwardGroups = 8;   // columns of a tile, tiles of a CTA
struct ForwardLayout {
    using W = WeightLayout<0>;
    static constexpr uint32_t BAR = W::END;                // one mbarrier per tile
    static constexpr uint32_t SLOT = BAR + 8 * kForwardGroups;
    static constexpr uint32_t H = (SLOT + 8 + 1023) / 1024 * 1024;   // 8 chunks per tile
    static constexpr uint32_t bytes(uint32_t groups) { return H + groups * 8 * kCH; }
};
// A training CTA waits for its peers, so no CTA on its SM may hold it up at the TMEM allocation
// while that one waits for another training launch.  It asks for so much shared memory that
// it never shares an SM with a forward CTA of 512 columns; beside what fits with it, the
// columns are there or come free with a forward CTA that already has its own.
constexpr uint32_t kSmShared = 233472, kCtaReserved = 1024;   // bytes of an SM, of each CTA beyond its own
constexpr uint32_t kTrainBytes =
    std::max(TrainLayout::BYTES, kSmShared - ForwardLayout::bytes(kForwardGroups) - 2 * kCtaReserved + 1024);
static_assert(2 * (kTrainBytes + kCtaReserved) <= kSmShared && 3 * (kTrainBytes + kCtaReserved) > kSmShared,
              "two training CTAs per SM, which have 512 columns between them");

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// Eight consecutive columns of one row into its 16-byte slot of a tile.
__device__ __forceinline__ void store8(unsigned char* buf, uint32_t chunk, uint32_t row, const float* v) {
    uint4 u = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
    *reinterpret_cast<uint4*>(buf + chunk * kCH + (row >> 3) * 128 + (row & 7) * 16) = u;
}
__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__device__ __forceinline__ void publish() {
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
}
// The same among the 128 threads of one tile of the CTA.
__device__ __forceinline__ void group_sync(uint32_t group) {
    tc::fence_before_sync();
    asm volatile("bar.sync %0, 128;" ::"r"(group + 1u) : "memory");
    tc::fence_after_sync();
}
__device__ __forceinline__ void publish(uint32_t group) {
    tc::fence_async_smem();
    group_sync(group);
}

// Weights (rounded to bf16) into the core-matrix layout, W1 64 rows x 2 chunks, W2 64 x 8,
// W3 16 x 8, and the biases.  Units of 8 consecutive parameters are one row of a chunk.
// Read past L1: a training launch rewrites the parameters between its steps.
template <class W, uint32_t kUnits, uint32_t kBlock>   // kBlock: threads of the CTA, 0 if known at the launch only
__device__ __forceinline__ void load_weights(unsigned char* smem, const float* params) {
    const bool rows16 = (reinterpret_cast<uintptr_t>(params) & 15u) == 0;
    const uint32_t block = kBlock ? kBlock : blockDim.x;
    constexpr bool kExact = kBlock != 0 && kWeights / 8 % (kUnits * kBlock + (kBlock == 0)) == 0;
    for (uint32_t u0 = 0; u0 < kWeights / 8; u0 += kUnits * block) {
        float w[kUnits][8];
#pragma unroll
        for (uint32_t k = 0; k < kUnits; ++k) {
            const uint32_t u = u0 + k * block + threadIdx.x;
            if (!kExact && u >= kWeights / 8) continue;
            if (rows16) {
                const float4* q = reinterpret_cast<const float4*>(params + 8 * u);
                const float4 lo = __ldcg(q), hi = __ldcg(q + 1);
                w[k][0] = lo.x; w[k][1] = lo.y; w[k][2] = lo.z; w[k][3] = lo.w;
                w[k][4] = hi.x; w[k][5] = hi.y; w[k][6] = hi.z; w[k][7] = hi.w;
            } else {
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) w[k][i] = __ldcg(params + 8 * u + i);
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < kUnits; ++k) {
            const uint32_t u = u0 + k * block + threadIdx.x;
            if (!kExact && u >= kWeights / 8) continue;
            uint32_t at;
            if (u < 128) at = W::W1 + (u & 1u) * 1024 + (u >> 4) * 128 + ((u >> 1) & 7u) * 16;
            else if (u < 640) at = W::W2 + (u & 7u) * 1024 + ((u - 128) >> 6) * 128 + ((u >> 3) & 7u) * 16;
            else at = W::W3 + (u & 7u) * 256 + ((u - 640) >> 6) * 128 + ((u >> 3) & 7u) * 16;
            *reinterpret_cast<uint4*>(smem + at) =
                make_uint4(pack_bf16(w[k][0], w[k][1]), pack_bf16(w[k][2], w[k][3]), pack_bf16(w[k][4], w[k][5]),
                           pack_bf16(w[k][6], w[k][7]));
        }
    }
    if (threadIdx.x < 64) reinterpret_cast<float*>(smem + W::B2)[threadIdx.x] = __ldcg(params + kB2 + threadIdx.x);
    if (threadIdx.x < 16) reinterpret_cast<float*>(smem + W::B3)[threadIdx.x] = __ldcg(params + kB3 + threadIdx.x);
}

// One sample's inputs (slot 15 is the constant 1); zeros past the end.
__device__ __forceinline__ void load_input(const float* __restrict__ x, uint32_t s, uint32_t n, float* v) {
    if (s < n) {
        const float4* xr = reinterpret_cast<const float4*>(x + (size_t)s * 16);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 f = __ldg(xr + q);
            v[4 * q] = f.x; v[4 * q + 1] = f.y; v[4 * q + 2] = f.z; v[4 * q + 3] = f.w;
        }
        v[15] = 1.0f;
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0.0f;
    }
}

// Forward pass.  A tile is a chain (inputs, three times MMA, read-back, ReLU and store)
// that leaves the SM idle unless other tiles run beside it, so a CTA has up to 8 groups of
// 128 threads with a tile each, which share the weights.  300,001 samples: 51 us with 2
// CTAs of one tile per SM; 28 with 7, whose start is held up (until a CTA has given up its
// right to allocate TMEM, its SM starts no other: 0.75 us between them, 2.5 with the weights
// loaded first); one CTA of 8 tiles, with the next inputs loaded during layer 1, 18
// (16.4 in a run of calls, where the first form took 48.1 and the second 24.6).
__global__ void __launch_bounds__(kThreads * kForwardGroups)
k_mlp_forward(const float* params, const float* __restrict__ x, uint32_t n_host, const uint32_t* n_dev,
              float* __restrict__ y, uint32_t y_cols, uint32_t* __restrict__ error_flags) {
    using L = ForwardLayout;
    extern __shared__ __align__(1024) unsigned char smem[];
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + L::SLOT);
    const float* sb2 = reinterpret_cast<const float*>(smem + L::W::B2);
    const float* sb3 = reinterpret_cast<const float*>(smem + L::W::B3);
    const uint32_t group = threadIdx.x / kThreads, groups = blockDim.x / kThreads;
    const uint32_t tid = threadIdx.x % kThreads, warp = tid >> 5;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::BAR) + group;
    unsigned char* H = smem + L::H + group * 8 * kCH;
    const uint32_t n = n_dev ? *n_dev : n_host;
    const uint32_t tiles = (n + kTile - 1) / kTile;
    if (blockIdx.x >= tiles) return;
    if (threadIdx.x < 32) tc::tmem_alloc(tslot, kForwardTmem * groups);
    const uint32_t first = blockIdx.x + group * gridDim.x, stride = groups * gridDim.x;
    float next[16];
    if (first < tiles) load_input(x, first * kTile + tid, n, next);
    if (tid == 0) tc::mbar_init(bar, 1);
    load_weights<L::W, 1, 0>(smem, params);
    publish();
    const uint32_t tbase = *tslot + kForwardTmem * group;
    const uint32_t tlane = tbase + ((32u * warp) << 16);
    uint32_t phase = 0;
    bool timed_out = false;
    auto mma_wait = [&]() {
        if (!tc::mbar_wait(bar, phase, kWaitLimit) && !timed_out) {
            timed_out = true;
            atomicOr(error_flags, MK_DEVICE_WAIT_TIMEOUT_FLAG);
        }
        phase ^= 1u;
        tc::fence_after_sync();
    };
    const uint32_t sH = tc::smem_u32(H);
    const uint32_t sW1 = tc::smem_u32(smem + L::W::W1), sW2 = tc::smem_u32(smem + L::W::W2);
    const uint32_t sW3 = tc::smem_u32(smem + L::W::W3);
    constexpr uint32_t id64 = tc::idesc_bf16(128, 64, false, false);
    constexpr uint32_t id16 = tc::idesc_bf16(128, 16, false, false);
    const bool rows4 = (y_cols & 3u) == 0u && (reinterpret_cast<uintptr_t>(y) & 15u) == 0;
    for (uint32_t tile = first; tile < tiles; tile += stride) {
        const uint32_t s = tile * kTile + tid;
        store8(H, 0, tid, next);
        store8(H, 1, tid, next + 8);
        publish(group);
        // layer 1: [128 x 16] x W1^T
        if (tid == 0) {
            tc::mma_bf16(tbase, tc::sdesc(sH, kCH, 128), tc::sdesc(sW1, 1024, 128), id64, 0);
            tc::commit(bar);
        }
        if (tile + stride < tiles) load_input(x, s + stride * kTile, n, next);
        mma_wait();
        float v[16];
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            tc::tmem_ld16(tlane + 16 * q, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = v[i] > 0.0f ? v[i] : 0.0f;
            store8(H, 2 * q, tid, v);
            store8(H, 2 * q + 1, tid, v + 8);
        }
        publish(group);
        // layer 2: H1 [128 x 64] x W2^T
        if (tid == 0) {
#pragma unroll
            for (uint32_t ks = 0; ks < 4; ++ks)
                tc::mma_bf16(tbase, tc::sdesc(sH + 2 * ks * kCH, kCH, 128), tc::sdesc(sW2 + 2 * ks * 1024, 1024, 128),
                             id64, ks > 0);
            tc::commit(bar);
        }
        mma_wait();
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            tc::tmem_ld16(tlane + 16 * q, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                v[i] += sb2[16 * q + i];
                v[i] = v[i] > 0.0f ? v[i] : 0.0f;
            }
            store8(H, 2 * q, tid, v);
            store8(H, 2 * q + 1, tid, v + 8);
        }
        publish(group);
        // layer 3: H2 [128 x 64] x W3^T
        if (tid == 0) {
#pragma unroll
            for (uint32_t ks = 0; ks < 4; ++ks)
                tc::mma_bf16(tbase, tc::sdesc(sH + 2 * ks * kCH, kCH, 128), tc::sdesc(sW3 + 2 * ks * 256, 256, 128),
                             id16, ks > 0);
            tc::commit(bar);
        }
        mma_wait();
        tc::tmem_ld16(tlane, v);
#pragma unroll
        for (int o = 0; o < 16; ++o) v[o] += sb3[o];
        if (s < n) {
            float* row = y + (size_t)s * y_cols;
            if (rows4) {
#pragma unroll
                for (uint32_t o = 0; o < 16; o += 4)
                    if (o < y_cols)
                        *reinterpret_cast<float4*>(row + o) = make_float4(v[o], v[o + 1], v[o + 2], v[o + 3]);
            } else {
#pragma unroll
                for (uint32_t o = 0; o < 16; ++o)
                    if (o < y_cols) row[o] = v[o];
            }
        }
        group_sync(group);   // the accumulator is read by all before the next tile's layer 1 overwrites it
    }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) tc::tmem_free(*tslot, kForwardTmem * groups);
}

__device__ __forceinline__ void store16(float* at, const float* v) {
#pragma unroll
    for (int j = 0; j < 16; j += 4)
        *reinterpret_cast<float4*>(at + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
}

// Forward and backward over the tiles of CTA blockIdx.x of `parts`, and its partial.
__device__ __forceinline__ void train_tiles(unsigned char* smem, const float* params, const float* __restrict__ x,
                                            const float* __restrict__ t, const float* __restrict__ out_w, uint32_t n,
                                            uint32_t parts, uint32_t tbase, uint32_t& phase, float* partials,
                                            uint32_t* error_flags) {
    using L = TrainLayout;
    unsigned char* F = smem + L::F;
    unsigned char* G = smem + L::G;
    unsigned char* Yb = smem + L::Y;
    const float* sb2 = reinterpret_cast<const float*>(smem + L::W::B2);
    const float* sb3 = reinterpret_cast<const float*>(smem + L::W::B3);
    float* sred = reinterpret_cast<float*>(smem + L::RED);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::BAR);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t tlane = tbase + ((32u * warp) << 16);
    auto mma_wait = [&]() {
        if (!tc::mbar_wait(bar, phase, kWaitLimit)) atomicOr(error_flags, MK_DEVICE_WAIT_TIMEOUT_FLAG);
        phase ^= 1u;
        tc::fence_after_sync();
    };
    const uint32_t sF = tc::smem_u32(F), sG = tc::smem_u32(G), sY = tc::smem_u32(Yb);
    const uint32_t sW1 = tc::smem_u32(smem + L::W::W1), sW2 = tc::smem_u32(smem + L::W::W2);
    const uint32_t sW3 = tc::smem_u32(smem + L::W::W3);
    constexpr uint32_t id64 = tc::idesc_bf16(128, 64, false, false);
    constexpr uint32_t id16 = tc::idesc_bf16(128, 16, false, false);
    constexpr uint32_t id64_bmn = tc::idesc_bf16(128, 64, false, true);
    constexpr uint32_t id80_mn = tc::idesc_bf16(128, 80, true, true);
    constexpr uint32_t id16_mn = tc::idesc_bf16(128, 16, true, true);

    const float coef = n > 0 ? 2.0f / (float)n : 0.0f;
    const uint32_t tiles = (n + kTile - 1) / kTile;
    float loss = 0.0f;
    float db3[16];
#pragma unroll
    for (int o = 0; o < 16; ++o) db3[o] = 0.0f;
    float next[16];
    load_input(x, blockIdx.x * kTile + tid, n, next);
    load_weights<L::W, kWeights / 8 / kThreads, kThreads>(smem, params);
    uint32_t it = 0;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += parts, ++it) {
        const uint32_t s = tile * kTile + tid;
        const bool valid = s < n;
        store8(F, 8, tid, next);
        store8(F, 9, tid, next + 8);
        publish();
        // layer 1: [128 x 16] x W1^T
        if (tid == 0) {
            tc::mma_bf16(tbase + cAcc1, tc::sdesc(sF + 8 * kCH, kCH, 128), tc::sdesc(sW1, 1024, 128), id64, 0);
            tc::commit(bar);
        }
        float tv[16];
        if (valid) {
            const float4* tr = reinterpret_cast<const float4*>(t + (size_t)s * 16);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 f = __ldg(tr + q);
                tv[4 * q] = f.x; tv[4 * q + 1] = f.y; tv[4 * q + 2] = f.z; tv[4 * q + 3] = f.w;
            }
        }
        mma_wait();
        float v[16];
        uint64_t mask1 = 0, mask2 = 0;
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            tc::tmem_ld16(tlane + cAcc1 + 16 * q, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                if (v[i] > 0.0f) mask1 |= 1ull << (16 * q + i);
                else v[i] = 0.0f;
            }
            store8(F, 2 * q, tid, v);
            store8(F, 2 * q + 1, tid, v + 8);
        }
        publish();
        // layer 2: H1 [128 x 64] x W2^T
        if (tid == 0) {
#pragma unroll
            for (uint32_t ks = 0; ks < 4; ++ks)
                tc::mma_bf16(tbase + cAcc2, tc::sdesc(sF + 2 * ks * kCH, kCH, 128), tc::sdesc(sW2 + 2 * ks * 1024, 1024, 128),
                             id64, ks > 0);
            tc::commit(bar);
        }
        mma_wait();
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            tc::tmem_ld16(tlane + cAcc2 + 16 * q, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                v[i] += sb2[16 * q + i];
                if (v[i] > 0.0f) mask2 |= 1ull << (16 * q + i);
                else v[i] = 0.0f;
            }
            store8(G, 2 * q, tid, v);
            store8(G, 2 * q + 1, tid, v + 8);
        }
        publish();
        // layer 3: H2 [128 x 64] x W3^T
        if (tid == 0) {
#pragma unroll
            for (uint32_t ks = 0; ks < 4; ++ks)
                tc::mma_bf16(tbase + cAcc3, tc::sdesc(sG + 2 * ks * kCH, kCH, 128), tc::sdesc(sW3 + 2 * ks * 256, 256, 128),
                             id16, ks > 0);
            tc::commit(bar);
        }
        mma_wait();
        tc::tmem_ld16(tlane + cAcc3, v);
#pragma unroll
        for (int o = 0; o < 16; ++o) v[o] += sb3[o];
        // dL/dy of L = (1/n) sum w_o (y_o - t_o)^2
#pragma unroll
        for (int o = 0; o < 16; ++o) {
            float d = 0.0f;
            if (valid) {
                const float e = v[o] - tv[o];
                const float w = __ldg(out_w + o);
                loss += w * e * e;
                d = bf16_round(coef * w * e);
            }
            db3[o] += d;
            v[o] = d;
        }
        store8(Yb, 0, tid, v);
        store8(Yb, 1, tid, v + 8);
        publish();
        // dH2 = dY [128 x 16] x W3 (W3 read MN-major)
        if (tid == 0) {
            tc::mma_bf16(tbase + cAcc2, tc::sdesc(sY, kCH, 128), tc::sdesc(sW3, 128, 256), id64_bmn, 0);
            tc::commit(bar);
        }
        mma_wait();
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            tc::tmem_ld16(tlane + cAcc2 + 16 * q, v);
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (!((mask2 >> (16 * q + i)) & 1ull)) v[i] = 0.0f;
            store8(G, 8 + 2 * q, tid, v);
            store8(G, 9 + 2 * q, tid, v + 8);
        }
        publish();
        // dH1 = dH2 [128 x 64] x W2 (W2 read MN-major)
        if (tid == 0) {
#pragma unroll
            for (uint32_t ks = 0; ks < 4; ++ks)
                tc::mma_bf16(tbase + cAcc1, tc::sdesc(sG + (8 + 2 * ks) * kCH, kCH, 128),
                             tc::sdesc(sW2 + ks * 256, 128, 1024), id64_bmn, ks > 0);
            tc::commit(bar);
        }
        mma_wait();
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            tc::tmem_ld16(tlane + cAcc1 + 16 * q, v);
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (!((mask1 >> (16 * q + i)) & 1ull)) v[i] = 0.0f;
            store8(G, 16 + 2 * q, tid, v);
            store8(G, 17 + 2 * q, tid, v + 8);
        }
        publish();
        // weight gradients, reduced over the tile's samples (K = samples):
        //   [dH2; dH1]^T-stack x [H1; X]  -> dW2 | db2 and dW1
        //   [H2; dH2] x dY               -> dW3^T
        if (tid == 0) {
#pragma unroll
            for (uint32_t ks = 0; ks < 8; ++ks) {
                const uint32_t acc = (it > 0 || ks > 0) ? 1u : 0u;
                tc::mma_bf16(tbase + cDA, tc::sdesc(sG + 8 * kCH + ks * 256, 128, kCH),
                             tc::sdesc(sF + ks * 256, 128, kCH), id80_mn, acc);
                tc::mma_bf16(tbase + cDB, tc::sdesc(sG + ks * 256, 128, kCH), tc::sdesc(sY + ks * 256, 128, kCH),
                             id16_mn, acc);
            }
            tc::commit(bar);
        }
        if (tile + parts < tiles) load_input(x, s + parts * kTile, n, next);
        mma_wait();
    }

    // ---- the CTA's partial
    float* part = partials + (size_t)blockIdx.x * kPartialStride;
    float g[16];
    if (warp < 2) {
        const uint32_t i = 32 * warp + lane;   // hidden-2 unit (row of dW2, column of dW3)
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            tc::tmem_ld16(tlane + cDA + 16 * q, g);
            store16(part + kW2 + i * 64 + 16 * q, g);
        }
        tc::tmem_ld16(tlane + cDA + 64, g);
        part[kB2 + i] = g[15];
        tc::tmem_ld16(tlane + cDB, g);
#pragma unroll
        for (int o = 0; o < 16; ++o) part[kW3 + o * 64 + i] = g[o];
    } else {
        const uint32_t i = 32 * (warp - 2) + lane;   // hidden-1 unit (row of dW1)
        tc::tmem_ld16(tlane + cDA + 64, g);
        store16(part + kW1 + i * 16, g);
    }
    // db3 and the loss: fixed-order warp trees, then the warps in order
#pragma unroll
    for (int o = 0; o < 17; ++o) {
        float r = o < 16 ? db3[o] : loss;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) r += __shfl_xor_sync(0xffffffffu, r, d);
        if (lane == 0) sred[warp * 17 + o] = r;
    }
    __syncthreads();
    if (tid < 17) {
        const float r = ((sred[tid] + sred[17 + tid]) + sred[34 + tid]) + sred[51 + tid];
        part[tid < 16 ? kB3 + tid : kLossSlot] = tid < 16 ? r : r * coef * 0.5f;   // loss = sum / n
    }
}

// Gradient, or a run of training steps: forward and backward over the CTA's tiles, one
// partial per CTA, a grid barrier, the sum of the partials in CTA order with the Adam
// update, and a barrier before the next step's weights.  Bound by latency: six MMAs and
// read-backs in a chain, the sums over up to 148 partials, two barriers.  As three launches a
// step (round the weights, tiles, sum and update) a step of 8,192 samples took 23.4 us, of
// which the sum's loads, four at a time, took 6.8; as steps of one cooperative launch, with
// 32 loads at a time and the inputs loaded ahead, it takes 11.
// Takes steps [0, steps) of `plan`; with `grad` non-null a single step that leaves the
// parameters alone.  The tiles' CTAs are the first `parts`; the others only sum.
__global__ void __launch_bounds__(kThreads)
k_mlp_train(float* params, const float* __restrict__ x, const float* __restrict__ t, const float* __restrict__ out_w,
            const __grid_constant__ TrainPlan plan, float* partials, uint32_t parts, float* grad, float* losses,
            float* m, float* v, uint32_t* barrier, uint32_t* __restrict__ error_flags) {
    using L = TrainLayout;
    extern __shared__ __align__(1024) unsigned char smem[];
    uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + L::SLOT);
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    const uint32_t n = plan.batch;
    if (tid == 0) tc::mbar_init(reinterpret_cast<uint64_t*>(smem + L::BAR), 1);
    if (warp == 0) tc::tmem_alloc(tslot, kTmemCols);
    publish();
    const uint32_t tbase = *tslot;
    uint32_t phase = 0, offset = plan.offset;
    for (uint32_t step = 0; step < plan.steps; ++step) {
        if (offset + n > plan.samples) offset = 0;   // batches walk the (pre-shuffled) samples cyclically
        if (blockIdx.x < parts)
            train_tiles(smem, params, x + (size_t)offset * 16, t + (size_t)offset * 16, out_w, n, parts, tbase, phase,
                        partials, error_flags);
        offset += n;
        if (step + 1 < plan.steps) {   // the next step's first tile, into L2 meanwhile
            const uint32_t s = blockIdx.x * kTile + tid;
            if (blockIdx.x < parts && s < n) {
                const size_t at = ((size_t)(offset + n > plan.samples ? 0u : offset) + s) * 16;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(x + at));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(t + at));
            }
        }
        grid_barrier(barrier, error_flags, gridDim.x);
        // ---- sums in CTA order, and the Adam update
        for (uint32_t i = blockIdx.x * kThreads + tid; i <= kLossSlot; i += gridDim.x * kThreads) {
            const bool update = !grad && i != kLossSlot;
            const float m0 = update ? m[i] : 0.0f, v0 = update ? v[i] : 0.0f, p0 = update ? __ldcg(params + i) : 0.0f;
            float g = 0.0f;
#pragma unroll 32
            for (uint32_t c = 0; c < parts; ++c) g += __ldcg(partials + (size_t)c * kPartialStride + i);
            if (grad) grad[i] = g;
            if (i == kLossSlot && losses) losses[step] = g;
            if (update) {
                const float mi = plan.beta1 * m0 + (1.0f - plan.beta1) * g;
                const float vi = plan.beta2 * v0 + (1.0f - plan.beta2) * g * g;
                m[i] = mi;
                v[i] = vi;
                const float mh = mi / plan.bias[step].x, vh = vi / plan.bias[step].y;
                params[i] = p0 - plan.lr * mh / (sqrtf(vh) + plan.eps);
            }
        }
        if (step + 1 < plan.steps) grid_barrier(barrier, error_flags, gridDim.x);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_free(tbase, kTmemCols);
}

static int g_sm_count = 0;

static cudaError_t prepare_attributes() {
    static bool done = false;
    if (done) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrainBytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 ForwardLayout::bytes(kForwardGroups));
    if (e == cudaSuccess) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
        done = true;
    }
    return e;
}

// The barrier word and the partials, in the size that callers have been asked for since the
// weights were kept there too (12 KB, unused now): sizes refused before stay refused.
uint64_t scratch_bytes(uint32_t max_samples) {
    (void)max_samples;
    int sms = g_sm_count > 0 ? g_sm_count : 148;
    return align256((uint64_t)kWeights * 2) + align256((uint64_t)sms * kPartialStride * 4) + align256(4);
}

cudaError_t init(void) { return prepare_attributes(); }

cudaError_t forward(const float* params, const float* x, uint32_t n, const uint32_t* n_dev, uint32_t max_n, float* y,
                    uint32_t y_cols, uint32_t* error_flags, cudaStream_t s) {
    cudaError_t e = prepare_attributes();
    if (e != cudaSuccess) return e;
    // one CTA per SM, with as many tiles beside one another (1, 2, 4 or 8) as there are for it
    const uint32_t tiles = std::max(1u, ((n_dev ? max_n : n) + kTile - 1) / kTile);
    const uint32_t grid = std::min(tiles, (uint32_t)g_sm_count);
    uint32_t groups = 1;
    while (groups < kForwardGroups && groups * grid < tiles) groups *= 2;
    k_mlp_forward<<<grid, kThreads * groups, ForwardLayout::bytes(groups), s>>>(params, x, n, n_dev, y, y_cols,
                                                                                error_flags);
    return cudaGetLastError();
}

cudaError_t train(float* params, const float* x, const float* t, const float* out_w, const TrainPlan& plan,
                  void* scratch, float* grad, float* losses, float* m, float* v, uint32_t* error_flags, cudaStream_t s) {
    cudaError_t e = prepare_attributes();
    if (e != cudaSuccess) return e;
    const uint32_t sms = (uint32_t)g_sm_count;
    const uint32_t tiles = (plan.batch + kTile - 1) / kTile;
    uint32_t parts = std::max(1u, std::min(tiles, sms));
    // at least a thread per parameter for the sums
    const uint32_t grid = std::max(parts, std::min(sms, (kLossSlot + kThreads) / kThreads));
    uint32_t* barrier = reinterpret_cast<uint32_t*>(scratch);
    float* partials = reinterpret_cast<float*>(reinterpret_cast<char*>(scratch) + 256);
    e = cudaMemsetAsync(barrier, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return e;
    TrainPlan by_value = plan;
    void* args[] = {&params, &x,      &t, &out_w, &by_value, &partials,   &parts,
                    &grad,   &losses, &m, &v,     &barrier,  &error_flags};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_mlp_train), dim3(grid), dim3(kThreads), args,
                                       kTrainBytes, s);
}

}  // namespace mlp
}  // namespace mk

// ------------------------------------------------------------------ C ABI
namespace {
int check_mlp(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return MK_OK;
    char msg[256];
    std::snprintf(msg, sizeof(msg), "%s: %s", what, cudaGetErrorString(e));
    mk::set_last_error(msg);
    return MK_ERR_DEVICE_FAILURE;
}
int bad_mlp(const char* msg) {
    mk::set_last_error(msg);
    return MK_ERR_INVALID_ARGUMENT;
}
}  // namespace

extern "C" {

MK_API uint32_t mk_mlp_param_count(void) { return mk::mlp::kParams; }

MK_API uint64_t mk_op_mlp_scratch_bytes(uint32_t max_samples) {
    if (mk::mlp::init() != cudaSuccess) return 0;
    return mk::mlp::scratch_bytes(max_samples);
}

MK_API int mk_op_mlp_forward(const float* params, const float* x, uint32_t n, float* y, uint32_t y_cols, void* scratch,
                             uint64_t scratch_bytes, uint32_t* error_flags, void* stream) {
    if (!params || !scratch || !error_flags || (n && (!x || !y))) return bad_mlp("mlp forward: null pointer");
    if (y_cols == 0 || y_cols > 16) return bad_mlp("mlp forward: y_cols must be 1..16");
    if ((reinterpret_cast<uintptr_t>(x) & 15u) != 0) return bad_mlp("mlp forward: x must be 16-byte aligned");
    if (mk::mlp::init() != cudaSuccess) return check_mlp(cudaGetLastError(), "mlp init");
    if (scratch_bytes < mk::mlp::scratch_bytes(n)) return bad_mlp("mlp forward: scratch too small");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const cudaError_t e = n ? mk::mlp::forward(params, x, n, nullptr, n, y, y_cols, error_flags, s) : cudaSuccess;
    return check_mlp(e, "mlp forward");
}

MK_API int mk_op_mlp_gradient(const float* params, const float* x, const float* targets, const float* out_weights,
                              uint32_t n, float* grad, void* scratch, uint64_t scratch_bytes, uint32_t* error_flags,
                              void* stream) {
    if (!params || !x || !targets || !out_weights || !grad || !scratch || !error_flags || n == 0)
        return bad_mlp("mlp gradient: null pointer or no samples");
    if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(targets)) & 15u) != 0)
        return bad_mlp("mlp gradient: x and targets must be 16-byte aligned");
    if (mk::mlp::init() != cudaSuccess) return check_mlp(cudaGetLastError(), "mlp init");
    if (scratch_bytes < mk::mlp::scratch_bytes(n)) return bad_mlp("mlp gradient: scratch too small");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    mk::mlp::TrainPlan plan{};
    plan.samples = plan.batch = n;
    plan.steps = 1;
    const cudaError_t e = mk::mlp::train(const_cast<float*>(params), x, targets, out_weights, plan, scratch, grad,
                                         nullptr, nullptr, nullptr, error_flags, s);
    return check_mlp(e, "mlp gradient");
}

MK_API int mk_op_mlp_train(float* params, float* adam_m, float* adam_v, const float* x, const float* targets,
                           const float* out_weights, uint32_t n, uint32_t batch, uint32_t steps, float lr,
                           uint32_t first_step, float* losses, void* scratch, uint64_t scratch_bytes,
                           uint32_t* error_flags, void* stream) {
    if (!params || !adam_m || !adam_v || !x || !targets || !out_weights || !scratch || !error_flags || n == 0)
        return bad_mlp("mlp train: null pointer or no samples");
    if (batch == 0 || batch > n) batch = n;
    if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(targets)) & 15u) != 0)
        return bad_mlp("mlp train: x and targets must be 16-byte aligned");
    if (mk::mlp::init() != cudaSuccess) return check_mlp(cudaGetLastError(), "mlp init");
    if (scratch_bytes < mk::mlp::scratch_bytes(batch)) return bad_mlp("mlp train: scratch too small");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const float b1 = 0.9f, b2 = 0.999f;
    cudaError_t e = cudaSuccess;
    mk::mlp::TrainPlan plan{};
    plan.samples = n;
    plan.batch = batch;
    plan.lr = lr;
    plan.beta1 = b1;
    plan.beta2 = b2;
    plan.eps = 1.0e-8f;
    for (uint32_t k = 0; k < steps && e == cudaSuccess; k += plan.steps) {
        plan.steps = std::min(steps - k, mk::mlp::kPlanSteps);
        for (uint32_t j = 0; j < plan.steps; ++j) {
            const float step = (float)(first_step + k + j + 1);
            plan.bias[j] = make_float2(1.0f - std::pow(b1, step), 1.0f - std::pow(b2, step));
        }
        e = mk::mlp::train(params, x, targets, out_weights, plan, scratch, nullptr, losses ? losses + k : nullptr,
                           adam_m, adam_v, error_flags, s);
        for (uint32_t j = 0; j < plan.steps; ++j) plan.offset = (plan.offset + batch > n ? 0u : plan.offset) + batch;
    }
    return check_mlp(e, "mlp train");
}

}  // extern "C"
