// The cut-refinement MLP (16 -> 64 -> 64 -> 64 -> 1, GELU or ReLU, BF16 weights, FP32 accumulation) on
// the 5th-generation tensor cores.  No counterpart in the reference: it predicts, for an 8x8 pixel
// tile and a tree node, whether the cut must refine the node.
//
// Two kernels.  Each CTA walks 128-row tiles of the input (forward: thread t owns row t; training: two
// threads per row):
//   forward   X[128x16] -> tcgen05.mma -> TMEM -> +b, activation -> BF16 core-matrix smem -> next layer;
//             the 64 -> 1 output layer runs on the CUDA cores from registers (mlp_tile.cuh, shared
//             with the fused level kernel of the learned cut).
//   training  the forward pass, then BCE gradient, and the backward pass:
//             dH_l = dZ_{l+1} W_{l+1}                       (M = 128 rows, B read MN-major)
//             dW_l += dZ_l^T H_{l-1}   (accumulated in TMEM over every tile the CTA owns;
//                                       M padded to 128 = out features, A and B read MN-major)
//             bias / output-layer gradients are column sums kept in registers.
// Weights are kept as an FP32 master copy (Adam updates it) and rounded to BF16 into shared
// memory by every CTA.  Every tensor-core result waits on an mbarrier with a bounded wait; the CTA
// stops (and still frees its TMEM) if a wait gives up.
#include <cuda_bf16.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "arc_internal.h"
#include "device_common.cuh"
#include "mlp_tile.cuh"
#include "pcg32.h"
#include "tcgen05.cuh"

namespace arc {
namespace mlp {

// shared-memory carve-up (bytes); dZ is followed by 2 KB because the M-padded weight-gradient
// MMA reads up to that far past it (the extra rows land in D rows 64..127, which are ignored)
constexpr uint32_t sW1 = 0, sW2 = sW1 + 2048, sW3 = sW2 + 8192, sX = sW3 + 8192, sH1 = sX + 4096,
                   sH2 = sH1 + 16384, sDZ = sH2 + 16384, sVecTrain = sDZ + 16384 + 2048;
constexpr uint32_t kVecBytes = 4 * 64 * 4;
constexpr uint32_t kSmemTrain = sVecTrain + kVecBytes;
// inference: weights and vectors | per group the hidden rows of its tile (16 KB), whose first 4 KB hold
// the input rows until layer 1 has read them
constexpr int kInferGroups = 4;
constexpr uint32_t sInH = ((kImageBytes + 127) / 128) * 128, kSmemInfer = sInH + kInferGroups * 16384;

struct Args {
    const float* params;
    const __nv_bfloat16* x;  // [rows][16]
    int64_t rows;
    float* logits;            // [rows] (forward mode)
    const float* labels;      // [rows] (training)
    const float* weights;     // [rows] sample weights or NULL
    float loss_scale;         // 1 / sum of weights
    float* grads;             // [kParams] (atomicAdd)
    float* loss;              // [1]
    int loss_kind;            // arc_mlp_loss
    uint32_t* err;
};

// store 32 values of row r, columns c0 .. c0 + 31, as BF16 into a K-major (K = 64) core-matrix buffer
__device__ __forceinline__ void store_row32(unsigned char* buf, int r, int c0, const float* v) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        uint4 q;
        q.x = pack2(v[8 * c + 0], v[8 * c + 1]);
        q.y = pack2(v[8 * c + 2], v[8 * c + 3]);
        q.z = pack2(v[8 * c + 4], v[8 * c + 5]);
        q.w = pack2(v[8 * c + 6], v[8 * c + 7]);
        *reinterpret_cast<uint4*>(buf + tc::kmajor_offset(r, c0 + 8 * c, 64)) = q;
    }
}

// one 32-lane sum, result in every lane
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums over a warp's 32 rows of 32 columns (one row per lane): lane c returns column c's sum.  Each step
// sends half of what is left to the partner lane, 31 exchanges instead of 32 x 5.
__device__ __forceinline__ float column_sums(float* v, int lane) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const bool up = (lane & s) != 0;
#pragma unroll
        for (int i = 0; i < s; ++i) {
            const float send = up ? v[i] : v[i + s], keep = up ? v[i + s] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
    }
    return v[0];
}

// Forward over every row of the input: persistent CTAs of four 128-thread groups that share the
// weights and otherwise run on their own (named barriers), one 128-row tile each; two CTAs per SM keep
// eight tiles in flight.  A tile is a chain of three tensor-core rounds with barriers and epilogues
// between them, so tiles in flight are what the rate follows; the next tile's rows are loaded while
// the current one is scored.
template <int ACT>
__global__ void __launch_bounds__(128 * kInferGroups, 2) mlp_infer_kernel(Args a) {
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ __align__(8) uint64_t bars[kInferGroups];
    __shared__ uint32_t tmem_base;
    const int t = threadIdx.x & 127, g = threadIdx.x >> 7;
    float* vec = reinterpret_cast<float*>(sm + kWeightBytes);
    load_weights<ACT>(sm, vec, a.params, threadIdx.x, 128 * kInferGroups);
    if (threadIdx.x < 32) tc::alloc(&tmem_base, 64 * kInferGroups);
    if (threadIdx.x == 0) {
        for (int i = 0; i < kInferGroups; ++i) mbar_init(&bars[i], 1);
        fence_mbar_init();
    }
    fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t h = sInH + 16384u * g;
    InferCta c{smem_u32(sm), 0, h, sm, vec, tmem_base + 64u * g, &bars[g], 0u, a.err};
    const GroupSync group{1 + g};
    const int64_t ntiles = (a.rows + kRows - 1) / kRows, step = (int64_t)gridDim.x * kInferGroups;
    uint4 x0, x1;
    auto load_rows = [&](int64_t tile) {
        const int64_t row = tile * kRows + t;
        x0 = x1 = make_uint4(0, 0, 0, 0);
        if (tile < ntiles && row < a.rows) {
            const uint4* xp = reinterpret_cast<const uint4*>(a.x + row * kIn);
            x0 = xp[0];
            x1 = xp[1];
        }
    };
    // consecutive tiles go to different CTAs, so that a small input spreads over the SMs
    int64_t tile = (int64_t)g * gridDim.x + blockIdx.x;
    load_rows(tile);
    for (; tile < ntiles; tile += step) {
        *reinterpret_cast<uint4*>(sm + h + tc::kmajor_offset(t, 0, kIn)) = x0;
        *reinterpret_cast<uint4*>(sm + h + tc::kmajor_offset(t, 8, kIn)) = x1;
        load_rows(tile + step);
        float y;
        if (!group.all(infer_tiles<1, ACT, false>(c, h, t, &y, group))) {  // (the error word says so)
            if (t == 0) drain_mma(c);
            break;
        }
        const int64_t row = tile * kRows + t;
        if (row < a.rows) a.logits[row] = y;
    }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) tc::dealloc(tmem_base, 64 * kInferGroups);
}

// Forward + backward with weight-gradient accumulation in TMEM (training).  256 threads per 128-row
// tile: thread t owns row t % 128 and columns 32 (t / 128) .. + 31 of every layer (a warp reads its
// own quarter of the TMEM lanes, so warps w and w + 4 share a quarter).  A training batch has fewer
// tiles than the chip has SMs, so a tile's latency is the kernel's time: two threads per row halve
// the elementwise work between the tensor-core rounds, the column sums (bias and output-layer
// gradients) stay in one register per lane until the end, pre-activations stay in registers, and
// the weights arrive with independent 16-byte loads.
constexpr int kTrainThreads = 256;

// four consecutive weights of row r (K columns, 4 c ..) as BF16 into a K-major operand
__device__ __forceinline__ void store_weights4(unsigned char* w, const float* params, int i, int K) {
    const float4 v = *reinterpret_cast<const float4*>(params + 4 * i);
    const int r = 4 * i / K, k = 4 * i % K;
    *reinterpret_cast<uint2*>(w + tc::kmajor_offset(r, k, K)) = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
}

// adds four consecutive floats to global memory (16-byte aligned)
__device__ __forceinline__ void red_add4(float* dst, const float* v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
                 : "memory");
}

template <int ACT>
__global__ void __launch_bounds__(kTrainThreads, 2) mlp_train_kernel(Args a) {
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_base;
    __shared__ float s_y[kRows], s_dy[kRows];
    __shared__ float s_col[4][4][64];  // [row quarter][gw4, gb3, gb2, gb1][column]
    __shared__ float s_b4[4];
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const int r = t & (kRows - 1), half = t >> 7, c0 = 32 * half;
    float* vec = reinterpret_cast<float*>(sm + sVecTrain);
    const float* b1 = vec + c0;
    const float* b2 = vec + 64 + c0;
    const float* b3 = vec + 128 + c0;
    const float* w4 = vec + 192 + c0;
    constexpr uint32_t kCols = 256;  // D | dW3 | dW2 | dW1

    // weights -> BF16 core-matrix layouts, vectors -> FP32
    store_weights4(sm + sW1, a.params + oW1, t, kIn);
#pragma unroll
    for (int i = 0; i < kHid * kHid / 4 / kTrainThreads; ++i) {
        store_weights4(sm + sW2, a.params + oW2, i * kTrainThreads + t, kHid);
        store_weights4(sm + sW3, a.params + oW3, i * kTrainThreads + t, kHid);
    }
    vec[t] = a.params[(t < 64 ? oB1 : t < 128 ? oB2 : t < 192 ? oB3 : oW4) + (t & 63)];
    const float b4 = a.params[oB4];
    if (w == 0) tc::alloc(&tmem_base, kCols);
    if (t == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_base;
    const uint32_t taddr = tmem + ((uint32_t)((w & 3) * 32) << 16) + (uint32_t)c0;  // this thread's lane and columns
    const uint32_t base = smem_u32(sm);
    uint32_t phase = 0;
    bool any_tile = false;
    bool gave_up = false;  // a tensor-core wait gave up: its commit may still be in flight
    float gw4 = 0.0f, gb3 = 0.0f, gb2 = 0.0f, gb1 = 0.0f;  // column c0 + lane over this warp's rows
    float gb4 = 0.0f, loss = 0.0f;

    constexpr uint32_t idKK64 = tc::idesc_bf16(128, 64, false, false);
    constexpr uint32_t idKM64 = tc::idesc_bf16(128, 64, false, true);
    constexpr uint32_t idMM64 = tc::idesc_bf16(128, 64, true, true);
    constexpr uint32_t idMM16 = tc::idesc_bf16(128, 16, true, true);

    // wait for the MMAs committed on `bar`; every thread learns whether all threads got there
    auto wait_mma = [&]() -> bool {
        const bool ok = mbar_wait_bounded(&bar, phase, a.err);
        phase ^= 1u;
        tc::fence_after_sync();
        const bool all = __syncthreads_and(ok) != 0;
        if (!all) gave_up = true;
        return all;
    };
    // make this thread's generic-proxy smem writes visible to the tensor cores, then barrier
    auto publish_smem = [&]() {
        fence_proxy_async_smem();
        tc::fence_before_sync();
        __syncthreads();
    };
    // forward layer with K = 64: D = A[128 x 64] B^T
    auto layer64 = [&](uint32_t A, uint32_t B) {
        if (t == 0) {
            tc::fence_after_sync();
#pragma unroll
            for (int s = 0; s < 4; ++s)
                tc::mma(tmem, tc::smem_desc(base + A + 256 * s, 128, 1024), tc::smem_desc(base + B + 256 * s, 128, 1024),
                        idKK64, s > 0);
            tc::commit(&bar);
        }
    };
    // this thread's half row of D
    auto load_d = [&](float* v) { tc::ld32(taddr, v); };
    // the pre-activation rounded to BF16, as the backward pass differentiates it
    auto rounded = [](uint32_t z, int h) { return __uint_as_float(h ? z & 0xffff0000u : z << 16); };

    const int64_t ntiles = (a.rows + kRows - 1) / kRows;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t row = tile * kRows + r;
        const bool valid = row < a.rows;
        uint4 x = make_uint4(0, 0, 0, 0);
        if (valid) x = reinterpret_cast<const uint4*>(a.x + row * kIn)[half];
        *reinterpret_cast<uint4*>(sm + sX + tc::kmajor_offset(r, 8 * half, kIn)) = x;
        float lab = 0.0f, wgt = 0.0f;
        if (valid) {
            lab = a.labels[row];
            wgt = a.weights ? a.weights[row] : 1.0f;
        }

        float z[32], h[32];
        uint32_t z1[16], z2[16];  // pre-activations of the first two layers, BF16 pairs
        // ---- layer 1 (K = 16) ----
        publish_smem();
        if (t == 0) {
            tc::fence_after_sync();
            tc::mma(tmem, tc::smem_desc(base + sX, 128, 256), tc::smem_desc(base + sW1, 128, 256), idKK64, false);
            tc::commit(&bar);
        }
        if (!wait_mma()) break;
        load_d(z);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            z[j] += b1[j];
            h[j] = act<ACT>(z[j]);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) z1[j] = pack2(z[2 * j], z[2 * j + 1]);
        store_row32(sm + sH1, r, c0, h);
        // ---- layer 2 ----
        publish_smem();
        layer64(sH1, sW2);
        if (!wait_mma()) break;
        load_d(z);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            z[j] += b2[j];
            h[j] = act<ACT>(z[j]);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) z2[j] = pack2(z[2 * j], z[2 * j + 1]);
        store_row32(sm + sH2, r, c0, h);
        // ---- layer 3 (kept in registers) ----
        publish_smem();
        layer64(sH2, sW3);
        if (!wait_mma()) break;
        load_d(z);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            z[j] += b3[j];
            h[j] = act<ACT>(z[j]);
        }
        // ---- output layer on the CUDA cores: one sum over the row, columns 0 .. 63 in order ----
        if (half == 0) {
            float y = b4;
#pragma unroll
            for (int j = 0; j < 32; ++j) y = fmaf(h[j], w4[j], y);
            s_y[r] = y;
        }
        __syncthreads();
        if (half == 1) {
            float y = s_y[r];
#pragma unroll
            for (int j = 0; j < 32; ++j) y = fmaf(h[j], w4[j], y);
            // ---- loss and its gradient ----
            float dy = 0.0f;
            if (valid) {
                if (a.loss_kind == ARC_MLP_LOSS_SQUARED) {
                    const float d = y - lab;
                    dy = wgt * 2.0f * d * a.loss_scale;
                    loss += wgt * d * d * a.loss_scale;
                } else {
                    const float p = 1.0f / (1.0f + expf(-y));
                    dy = wgt * (p - lab) * a.loss_scale;
                    loss += wgt * (fmaxf(y, 0.0f) - y * lab + log1pf(expf(-fabsf(y)))) * a.loss_scale;
                }
            }
            gb4 += dy;
            s_dy[r] = dy;
        }
        __syncthreads();
        // ---- output-layer gradients, dZ3 ----
        const float dy = s_dy[r];
        float g[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) g[j] = dy * w4[j] * act_grad<ACT>(z[j]);  // dZ3
        store_row32(sm + sDZ, r, c0, g);
        // dW3 += dZ3^T H2 ; dH2 = dZ3 W3
        publish_smem();
        if (t == 0) {
            tc::fence_after_sync();
#pragma unroll
            for (int s = 0; s < 8; ++s)
                tc::mma(tmem + 64, tc::smem_desc(base + sDZ + 2048 * s, 1024, 128),
                        tc::smem_desc(base + sH2 + 2048 * s, 1024, 128), idMM64, any_tile || s > 0);
#pragma unroll
            for (int s = 0; s < 4; ++s)
                tc::mma(tmem, tc::smem_desc(base + sDZ + 256 * s, 128, 1024), tc::smem_desc(base + sW3 + 2048 * s, 1024, 128),
                        idKM64, s > 0);
            tc::commit(&bar);
        }
        // (the column sums run beside the tensor cores)
        gb3 += column_sums(g, lane);
#pragma unroll
        for (int j = 0; j < 32; ++j) h[j] *= dy;
        gw4 += column_sums(h, lane);
        if (!wait_mma()) break;
        load_d(g);  // dH2
#pragma unroll
        for (int j = 0; j < 32; ++j) g[j] *= act_grad<ACT>(rounded(z2[j / 2], j & 1));  // dZ2
        store_row32(sm + sDZ, r, c0, g);
        // dW2 += dZ2^T H1 ; dH1 = dZ2 W2
        publish_smem();
        if (t == 0) {
            tc::fence_after_sync();
#pragma unroll
            for (int s = 0; s < 8; ++s)
                tc::mma(tmem + 128, tc::smem_desc(base + sDZ + 2048 * s, 1024, 128),
                        tc::smem_desc(base + sH1 + 2048 * s, 1024, 128), idMM64, any_tile || s > 0);
#pragma unroll
            for (int s = 0; s < 4; ++s)
                tc::mma(tmem, tc::smem_desc(base + sDZ + 256 * s, 128, 1024), tc::smem_desc(base + sW2 + 2048 * s, 1024, 128),
                        idKM64, s > 0);
            tc::commit(&bar);
        }
        gb2 += column_sums(g, lane);
        if (!wait_mma()) break;
        load_d(g);  // dH1
#pragma unroll
        for (int j = 0; j < 32; ++j) g[j] *= act_grad<ACT>(rounded(z1[j / 2], j & 1));  // dZ1
        store_row32(sm + sDZ, r, c0, g);
        // dW1 += dZ1^T X  (N = 16)
        publish_smem();
        if (t == 0) {
            tc::fence_after_sync();
#pragma unroll
            for (int s = 0; s < 8; ++s)
                tc::mma(tmem + 192, tc::smem_desc(base + sDZ + 2048 * s, 1024, 128),
                        tc::smem_desc(base + sX + 512 * s, 256, 128), idMM16, any_tile || s > 0);
            tc::commit(&bar);
        }
        gb1 += column_sums(g, lane);
        if (!wait_mma()) break;
        any_tile = true;
    }

    if (any_tile && !gave_up) {
        // weight gradients: D rows 0..63 (= output features) live in TMEM lanes 0..63, which warps
        // 0, 1 (columns 0 .. 31) and 4, 5 (32 .. 63) read
        if ((w & 3) < 2) {
            float v[32];
            tc::ld32(taddr + 64, v);
#pragma unroll
            for (int j = 0; j < 32; j += 4) red_add4(&a.grads[oW3 + r * 64 + c0 + j], v + j);
            tc::ld32(taddr + 128, v);
#pragma unroll
            for (int j = 0; j < 32; j += 4) red_add4(&a.grads[oW2 + r * 64 + c0 + j], v + j);
            if (half == 0) {
                tc::ld16(taddr + 192, v);
#pragma unroll
                for (int j = 0; j < 16; j += 4) red_add4(&a.grads[oW1 + r * 16 + j], v + j);
            }
        }
        float* col = &s_col[w & 3][0][c0 + lane];
        col[0] = gw4;
        col[64] = gb3;
        col[128] = gb2;
        col[192] = gb1;
        const float ls = warp_sum(loss), ds = warp_sum(gb4);
        if (lane == 0 && half == 1) {
            s_b4[w & 3] = ds;
            atomicAdd(a.loss, ls);
        }
        __syncthreads();
        const int k = t >> 6, c = t & 63;
        const float v = (s_col[0][k][c] + s_col[1][k][c]) + (s_col[2][k][c] + s_col[3][k][c]);
        atomicAdd(&a.grads[(k == 0 ? oW4 : k == 1 ? oB3 : k == 2 ? oB2 : oB1) + c], v);
        if (t == 0) atomicAdd(&a.grads[oB4], (s_b4[0] + s_b4[1]) + (s_b4[2] + s_b4[3]));
    }
    // after a wait that gave up (the error word says so), the last commit gets a second bounded
    // wait before the TMEM and shared memory are released (the failed wait flipped the phase)
    if (gave_up && t == 0) mbar_wait_bounded(&bar, phase ^ 1u, a.err);
    tc::fence_before_sync();
    __syncthreads();
    if (w == 0) tc::dealloc(tmem, kCols);
}

__global__ void adam_kernel(float* params, float* grads, float* m, float* v, int n, float lr, float b1, float b2,
                            float eps, float bc1, float bc2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float g = grads[i];
    const float mi = b1 * m[i] + (1.0f - b1) * g;
    const float vi = b2 * v[i] + (1.0f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    params[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    grads[i] = 0.0f;
}

}  // namespace mlp
}  // namespace arc

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
using namespace arc;

struct arc_mlp {
    arc_context* ctx = nullptr;
    float* params = nullptr;  // device FP32 master copy
    float* grads = nullptr;   // kParams, then the loss of arc_mlp_gradients; zero between calls
    float* host = nullptr;    // pinned: what arc_mlp_gradients reads back
    float* adam_m = nullptr;
    float* adam_v = nullptr;
    float* loss = nullptr;
    int64_t step = 0;
    int32_t loss_kind = ARC_MLP_LOSS_BCE;
    int32_t activation = ARC_MLP_ACT_GELU;
};

namespace {

arc_status mlp_launch(arc_mlp* m, bool train, const void* x, int64_t rows, float* logits, const float* labels,
                      const float* weights, float loss_scale) {
    arc_context* ctx = m->ctx;
    mlp::Args a{};
    a.params = m->params;
    a.x = static_cast<const __nv_bfloat16*>(x);
    a.rows = rows;
    a.logits = logits;
    a.labels = labels;
    a.weights = weights;
    a.loss_scale = loss_scale;
    a.grads = m->grads;
    a.loss = m->loss;
    a.loss_kind = m->loss_kind;
    a.err = ctx->d_error;
    const int64_t tiles = (rows + mlp::kRows - 1) / mlp::kRows;
    if (tiles == 0) return ARC_OK;
    // the shared-memory limit is a per-device attribute of the kernel: set it on every call (a
    // host-side call), not once per process, so contexts on other devices get it too
    const bool relu = m->activation == ARC_MLP_ACT_RELU;
    if (train) {
        auto* k = relu ? mlp::mlp_train_kernel<mlp::kActRelu> : mlp::mlp_train_kernel<mlp::kActGelu>;
        ARC_TRY_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp::kSmemTrain));
        // Two CTAs per SM overlap each other's tensor-core rounds once each has several tiles (500,000
        // rows: 140 against 170 us); with few tiles a second CTA only adds weight loads and reductions.
        const int per_sm = tiles >= 8 * (int64_t)ctx->sm_count ? 2 : 1;
        const int grid = (int)std::min<int64_t>(tiles, (int64_t)ctx->sm_count * per_sm);
        stage_begin(ctx, "mlp_train");
        k<<<grid, mlp::kTrainThreads, mlp::kSmemTrain, ctx->stream>>>(a);
        stage_end(ctx, 1);
    } else {
        auto* k = relu ? mlp::mlp_infer_kernel<mlp::kActRelu> : mlp::mlp_infer_kernel<mlp::kActGelu>;
        ARC_TRY_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp::kSmemInfer));
        const int grid = (int)std::min<int64_t>(tiles, (int64_t)ctx->sm_count * 2);
        stage_begin(ctx, "mlp_forward");
        k<<<grid, 128 * mlp::kInferGroups, mlp::kSmemInfer, ctx->stream>>>(a);
        stage_end(ctx, 1);
    }
    ARC_TRY_CUDA(cudaGetLastError());
    return ARC_OK;
}

}  // namespace

namespace arc {
const float* mlp_params(const arc_mlp* m) { return m->params; }
int32_t mlp_loss_kind(const arc_mlp* m) { return m->loss_kind; }
int32_t mlp_activation(const arc_mlp* m) { return m->activation; }
arc_status mlp_forward_device(arc_mlp* m, const void* x, int64_t rows, float* logits) {
    return mlp_launch(m, false, x, rows, logits, nullptr, nullptr, 0.0f);
}
}  // namespace arc

extern "C" {

int32_t arc_mlp_num_params(void) { return mlp::kParams; }

arc_status arc_mlp_create(arc_context* ctx, uint64_t seed, arc_mlp** out) {
    ARC_CHECK_ARG(ctx && out, "NULL argument");
    ARC_TRY_CUDA(cudaSetDevice(ctx->device));
    arc_mlp* m = new arc_mlp();
    m->ctx = ctx;
    const size_t bytes = sizeof(float) * mlp::kParams;
    cudaError_t e = cudaMalloc(&m->params, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&m->grads, bytes + sizeof(float));
    if (e == cudaSuccess) e = cudaMallocHost(&m->host, bytes + sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&m->adam_m, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&m->adam_v, bytes);
    if (e == cudaSuccess) e = cudaMalloc(&m->loss, sizeof(float));
    if (e != cudaSuccess) {
        set_last_error(std::string("arc_mlp_create: ") + cudaGetErrorString(e));
        arc_mlp_destroy(m);
        return ARC_ERR_OUT_OF_MEMORY;
    }
    // uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) from a PCG32 stream
    std::vector<float> p(mlp::kParams, 0.0f);
    arc_pcg32 r;
    arc_pcg32_seed(&r, seed, 0x6d6c70ULL);
    auto fill = [&](int off, int count, int fan_in) {
        const float b = 1.0f / std::sqrt((float)fan_in);
        for (int i = 0; i < count; ++i) p[off + i] = (2.0f * arc_pcg32_float(&r) - 1.0f) * b;
    };
    fill(mlp::oW1, 64 * 16, 16);
    fill(mlp::oB1, 64, 16);
    fill(mlp::oW2, 64 * 64, 64);
    fill(mlp::oB2, 64, 64);
    fill(mlp::oW3, 64 * 64, 64);
    fill(mlp::oB3, 64, 64);
    fill(mlp::oW4, 64, 64);
    fill(mlp::oB4, 1, 64);
    e = cudaMemcpy(m->params, p.data(), bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(m->grads, 0, bytes + sizeof(float));
    if (e == cudaSuccess) e = cudaMemset(m->adam_m, 0, bytes);
    if (e == cudaSuccess) e = cudaMemset(m->adam_v, 0, bytes);
    if (e != cudaSuccess) {
        set_last_error(std::string("arc_mlp_create: ") + cudaGetErrorString(e));
        arc_mlp_destroy(m);
        return ARC_ERR_CUDA;
    }
    *out = m;
    return ARC_OK;
}

arc_status arc_mlp_destroy(arc_mlp* m) {
    if (!m) return ARC_OK;
    if (m->ctx) {
        cudaSetDevice(m->ctx->device);
        cudaStreamSynchronize(m->ctx->stream);
    }
    cudaFree(m->params);
    cudaFree(m->grads);
    cudaFreeHost(m->host);
    cudaFree(m->adam_m);
    cudaFree(m->adam_v);
    cudaFree(m->loss);
    delete m;
    return ARC_OK;
}

arc_status arc_mlp_set_params(arc_mlp* m, const float* host, int32_t n) {
    ARC_CHECK_ARG(m && host && n == mlp::kParams, "parameter count mismatch");
    ARC_TRY_CUDA(cudaSetDevice(m->ctx->device));
    ARC_TRY_CUDA(cudaMemcpyAsync(m->params, host, sizeof(float) * n, cudaMemcpyHostToDevice, m->ctx->stream));
    ARC_TRY_CUDA(cudaStreamSynchronize(m->ctx->stream));
    return ARC_OK;
}

arc_status arc_mlp_get_params(arc_mlp* m, float* host, int32_t n) {
    ARC_CHECK_ARG(m && host && n == mlp::kParams, "parameter count mismatch");
    ARC_TRY_CUDA(cudaSetDevice(m->ctx->device));
    ARC_TRY_CUDA(cudaMemcpyAsync(host, m->params, sizeof(float) * n, cudaMemcpyDeviceToHost, m->ctx->stream));
    ARC_TRY_CUDA(cudaStreamSynchronize(m->ctx->stream));
    return ARC_OK;
}

arc_status arc_mlp_forward(arc_mlp* m, const void* features_bf16, int64_t rows, float* logits) {
    ARC_CHECK_ARG(m && (rows == 0 || (features_bf16 && logits)), "NULL argument");
    ARC_CHECK_ARG(reinterpret_cast<uintptr_t>(features_bf16) % 16 == 0, "features must be 16-byte aligned");
    ARC_TRY_CUDA(cudaSetDevice(m->ctx->device));
    return mlp_launch(m, false, features_bf16, rows, logits, nullptr, nullptr, 0.0f);
}

arc_status arc_mlp_gradients(arc_mlp* m, const void* features_bf16, const float* labels, const float* weights,
                             int64_t rows, float weight_sum, float* host_grads, float* host_loss) {
    ARC_CHECK_ARG(m && features_bf16 && labels && rows > 0 && weight_sum > 0.0f, "bad argument");
    ARC_TRY_CUDA(cudaSetDevice(m->ctx->device));
    // gradients and loss in one buffer: one copy back (to pinned memory), one clear for the next call
    const size_t bytes = sizeof(float) * (mlp::kParams + 1);
    cudaStream_t st = m->ctx->stream;
    float* saved = m->loss;
    m->loss = m->grads + mlp::kParams;
    const arc_status s = mlp_launch(m, true, features_bf16, rows, nullptr, labels, weights, 1.0f / weight_sum);
    m->loss = saved;
    ARC_TRY(s);
    const cudaError_t e = cudaMemcpyAsync(m->host, m->grads, bytes, cudaMemcpyDeviceToHost, st);
    ARC_TRY_CUDA(cudaMemsetAsync(m->grads, 0, bytes, st));
    ARC_TRY_CUDA(e);
    ARC_TRY_CUDA(cudaStreamSynchronize(st));
    if (host_grads) std::memcpy(host_grads, m->host, sizeof(float) * mlp::kParams);
    if (host_loss) *host_loss = m->host[mlp::kParams];
    return ARC_OK;
}

arc_status arc_mlp_set_loss(arc_mlp* m, int32_t kind) {
    ARC_CHECK_ARG(m, "NULL model");
    ARC_CHECK_ARG(kind == ARC_MLP_LOSS_BCE || kind == ARC_MLP_LOSS_SQUARED, "unknown loss");
    m->loss_kind = kind;
    return ARC_OK;
}

int32_t arc_mlp_get_loss(const arc_mlp* m) { return m ? m->loss_kind : -1; }

arc_status arc_mlp_set_activation(arc_mlp* m, int32_t kind) {
    ARC_CHECK_ARG(m, "NULL model");
    ARC_CHECK_ARG(kind == ARC_MLP_ACT_GELU || kind == ARC_MLP_ACT_RELU, "unknown activation");
    m->activation = kind;
    return ARC_OK;
}

int32_t arc_mlp_get_activation(const arc_mlp* m) { return m ? m->activation : -1; }

arc_status arc_mlp_train_step(arc_mlp* m, const void* features_bf16, const float* labels, const float* weights,
                              int64_t rows, float weight_sum, float lr, float* device_loss_accum) {
    ARC_CHECK_ARG(m && features_bf16 && labels && rows > 0 && weight_sum > 0.0f, "bad argument");
    ARC_TRY_CUDA(cudaSetDevice(m->ctx->device));
    float* saved = m->loss;
    if (device_loss_accum) m->loss = device_loss_accum;
    arc_status s = mlp_launch(m, true, features_bf16, rows, nullptr, labels, weights, 1.0f / weight_sum);
    m->loss = saved;
    ARC_TRY(s);
    m->step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float bc1 = 1.0f - std::pow(b1, (float)m->step), bc2 = 1.0f - std::pow(b2, (float)m->step);
    mlp::adam_kernel<<<(mlp::kParams + 255) / 256, 256, 0, m->ctx->stream>>>(m->params, m->grads, m->adam_m, m->adam_v,
                                                                             mlp::kParams, lr, b1, b2, 1e-8f, bc1, bc2);
    m->ctx->launches += 1;
    ARC_TRY_CUDA(cudaGetLastError());
    return ARC_OK;
}

}  // extern "C"
