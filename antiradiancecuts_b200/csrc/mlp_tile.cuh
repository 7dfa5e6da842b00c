// Shared pieces of the cut-refinement MLP (16 -> 64 -> 64 -> 64 -> 1): parameter layout, the
// activations, and the inference of one 128-row tile on the tensor cores, used by the stand-alone
// forward kernel (mlp.cu) and by the fused level kernel of the learned cut (learned.cu).  The
// activation is a property of the model and a template parameter of every kernel (kActGelu,
// kActRelu).
//
// ReLU: max(x, 0).  Inference takes the parameters as they are; a hidden value costs one add
// (bias), and the rounding to BF16 applies the ReLU for free (cvt.rn.relu.bf16x2.f32).
//
// GELU, in its sigmoid form (Hendrycks & Gimpel 2016, x sigma(1.702 x)), written with
// the hardware tanh (tanh.approx.f32):
//     gelu(x) = x/2 (1 + tanh(s x)),   s = 1.702 / 2.
// Training and the FP64 oracle use this function.  Inference folds its constants into the
// parameters (load_weights): with z' = s z the activation is (1 / (2 s)) g(z'), g(z) = z + z tanh(z),
// so layer 1 takes s W1, s b1, the next layers (s / (2 s)) W = W / 2 and s b, and the output layer
// w4 / (2 s); the epilogue is then one add (bias), one tanh and one multiply-add per value.
// (Two forms were measured and dropped: the tanh form of GELU, whose cubic argument costs three
// more operations per value, and a BF16-pair tanh, tanh.approx.bf16x2, whose packing cost more
// issue slots than the special-function work it saved.)
#ifndef ARC_MLP_TILE_CUH_
#define ARC_MLP_TILE_CUH_

#include <cuda_bf16.h>
#include <stdint.h>

#include "device_common.cuh"
#include "tcgen05.cuh"

namespace arc {
namespace mlp {

constexpr int kIn = 16, kHid = 64, kRows = 128;
// parameter layout of the FP32 master copy
constexpr int oW1 = 0, oB1 = oW1 + kHid * kIn, oW2 = oB1 + kHid, oB2 = oW2 + kHid * kHid, oW3 = oB2 + kHid,
              oB3 = oW3 + kHid * kHid, oW4 = oB3 + kHid, oB4 = oW4 + kHid, kParams = oB4 + 1;  // 9473

constexpr int kActGelu = 0, kActRelu = 1;  // arc_mlp_activation
constexpr float kGeluS = 0.851f;                   // 1.702 / 2
constexpr float kGeluOut = 0.5f / 0.851f;          // 1 / (2 s): the folded activation's scale

__device__ __forceinline__ float tanh_hw(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float gelu(float x) {
    const float th = tanh_hw(kGeluS * x);
    const float hx = 0.5f * x;
    return fmaf(hx, th, hx);
}

// d gelu / dx = (1 + th) / 2 + (x / 2) s (1 - th^2)
__device__ __forceinline__ float gelu_grad(float x) {
    const float th = tanh_hw(kGeluS * x);
    return fmaf(0.5f, th, 0.5f) + 0.5f * x * kGeluS * (1.0f - th * th);
}

// activation and its derivative in unfolded form (training)
template <int ACT>
__device__ __forceinline__ float act(float x) {
    if constexpr (ACT == kActRelu) return fmaxf(x, 0.0f);
    else return gelu(x);
}

template <int ACT>
__device__ __forceinline__ float act_grad(float x) {
    if constexpr (ACT == kActRelu) return x > 0.0f ? 1.0f : 0.0f;
    else return gelu_grad(x);
}

// The folded activation of inference for a pair: x = z + b (both already scaled by s), g(x) =
// x + x tanh(x); the result is 2 s gelu of the unscaled value.
__device__ __forceinline__ uint64_t act2(uint64_t z, uint64_t b) {
    const uint64_t x = f2_add(z, b);
    float x0, x1;
    f2_split(x, x0, x1);
    return f2_fma(x, f2(tanh_hw(x0), tanh_hw(x1)), x);
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// {bf16(max(a, 0)), bf16(max(b, 0))}, a in the low half like pack2 (cvt puts its first source in
// the high half)
__device__ __forceinline__ uint32_t pack2_relu(float a, float b) {
    uint32_t d;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(b), "f"(a));
    return d;
}

// One inference hidden value pair: z + b through the activation, rounded to a BF16 pair.
template <int ACT>
__device__ __forceinline__ uint32_t hidden_pair(uint64_t z, uint64_t b) {
    float g0, g1;
    if constexpr (ACT == kActRelu) {
        f2_split(f2_add(z, b), g0, g1);
        return pack2_relu(g0, g1);
    } else {
        f2_split(act2(z, b), g0, g1);
        return pack2(g0, g1);
    }
}

// y + w (activation of z + b) for a pair, FP32 (the output layer)
template <int ACT>
__device__ __forceinline__ uint64_t output_pair(uint64_t z, uint64_t b, uint64_t w, uint64_t y) {
    if constexpr (ACT == kActRelu) {
        float x0, x1;
        f2_split(f2_add(z, b), x0, x1);
        return f2_fma(f2(fmaxf(x0, 0.0f), fmaxf(x1, 0.0f)), w, y);
    } else {
        return f2_fma(act2(z, b), w, y);
    }
}

// Weights of one CTA for inference: W1 | W2 | W3 as BF16 K-major core matrices, then b1, b2,
// b3, w4, b4 as FP32.
constexpr uint32_t kW1 = 0, kW2 = kW1 + 2048, kW3 = kW2 + 8192, kWeightBytes = kW3 + 8192;
constexpr uint32_t kVecBytesInfer = (4 * 64 + 4) * 4;
// weights followed by the vectors: the image a CTA copies into shared memory in one bulk copy
constexpr uint32_t kImageBytes = kWeightBytes + kVecBytesInfer;
static_assert(kImageBytes % 16 == 0, "bulk copies move multiples of 16 bytes");

// Every thread of the CTA (nthreads of them) helps load the weights (into shared memory, or into
// a global image in the same layout): W1 | W2 | W3 in BF16, then b1 | b2 | b3 | w4 | b4 in FP32.
// GELU folds its constants in (see the top of this file): s W1 | W2 / 2 | W3 / 2, then
// s b1 | s b2 | s b3 | w4 / (2 s) | b4; ReLU takes the parameters as they are.
template <int ACT>
__device__ __forceinline__ void load_weights(unsigned char* w, float* vec, const float* params, int t, int nthreads) {
    const float s1 = ACT == kActGelu ? kGeluS : 1.0f, sh = ACT == kActGelu ? 0.5f : 1.0f,
                sb = ACT == kActGelu ? kGeluS : 1.0f, so = ACT == kActGelu ? kGeluOut : 1.0f;
    // four weights per 16-byte load (their offsets in the parameters are multiples of four)
    auto put4 = [&](uint32_t at, int first, int i, int K, float scale) {
        const float4 v = *reinterpret_cast<const float4*>(params + first + 4 * i);
        *reinterpret_cast<uint2*>(w + at + tc::kmajor_offset(4 * i / K, 4 * i % K, K)) =
            make_uint2(pack2(scale * v.x, scale * v.y), pack2(scale * v.z, scale * v.w));
    };
    for (int i = t; i < kHid * kIn / 4; i += nthreads) put4(kW1, oW1, i, kIn, s1);
    for (int i = t; i < kHid * kHid / 4; i += nthreads) {
        put4(kW2, oW2, i, kHid, sh);
        put4(kW3, oW3, i, kHid, sh);
    }
    for (int i = t; i < 64; i += nthreads) {
        vec[i] = sb * params[oB1 + i];
        vec[64 + i] = sb * params[oB2 + i];
        vec[128 + i] = sb * params[oB3 + i];
        vec[192 + i] = so * params[oW4 + i];
    }
    if (t == 0) vec[256] = params[oB4];
}

// Inference state of one 128-thread CTA: the smem base address (shared window), the weight block,
// the 128-row hidden buffer, the FP32 vectors, 64 TMEM columns and one mbarrier.
struct InferCta {
    uint32_t base;     // smem_u32 of the dynamic shared memory
    uint32_t w;        // byte offsets within it
    uint32_t h;        // 16 KB, K-major [128][64]
    unsigned char* sm;
    const float* vec;  // b1 | b2 | b3 | w4 | b4
    uint32_t tmem;
    uint64_t* bar;
    uint32_t phase;  // parity of the next barrier completion
    uint32_t* err;
    bool ok = true;         // this thread's waits have all succeeded
    uint32_t committed = 0; // issuing thread: parity of its last commit
};

// The threads that score together: the whole CTA, or 128 of its threads on named barrier `id` (each such
// group has its own tile, hidden rows, TMEM columns and mbarrier, and never waits for the others).
struct CtaSync {
    __device__ __forceinline__ void sync() const { __syncthreads(); }
    __device__ __forceinline__ bool all(bool ok) const { return __syncthreads_and(ok) != 0; }
};
struct GroupSync {
    int id;
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
    __device__ __forceinline__ bool all(bool ok) const {
        int r;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.b32 q, %1, 0;\n\t"
            "bar.red.and.pred p, %2, 128, q;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(r)
            : "r"((int)ok), "r"(id)
            : "memory");
        return r != 0;
    }
};

// Waits for the MMAs committed on the barrier.  A wait that gives up is remembered in c.ok, without a
// barrier to tell the other threads (three per tile cost 5% of the learned selection): the issuing
// thread issues nothing more, so every thread's next wait gives up too at the latest, and the caller
// learns of it at its own next barrier.
__device__ __forceinline__ void wait_mma(InferCta& c) {
    if (!mbar_wait_bounded(c.bar, c.phase, c.err)) c.ok = false;
    c.phase ^= 1u;
    tc::fence_after_sync();
}

// A CTA that stops after a wait gave up: the issuing thread gives its last commit a second bounded wait
// before the TMEM and the shared memory are released.
__device__ __forceinline__ void drain_mma(const InferCta& c) { mbar_wait_bounded(c.bar, c.committed, c.err); }

// Makes this thread's generic-proxy smem writes visible to the tensor cores, then barrier.
template <class Sync>
__device__ __forceinline__ void publish_smem(const Sync& s) {
    fence_proxy_async_smem();
    tc::fence_before_sync();
    s.sync();
}

// The epilogues read the accumulators as MMA fragments: a thread then holds few columns of several rows
// (2 of every 8 columns, 4 of the warp's 32 rows), so it needs 16 of a layer's 64 biases instead of all
// of them, and a warp stores whole 8 x 8 core matrices with stmatrix.  (With one row per thread the
// broadcast loads of biases and output weights took most of the shared-memory bandwidth that the tensor
// cores' operands also need: L1 at 90%.)

// TMEM address of rows 16 h .. 16 h + 15 of thread t's warp: tile t / 128 owns accumulator columns
// 64 (t / 128) ..+63, and a warp may only read its lane quarter, 32 ((t / 32) % 4) .. +31.
__device__ __forceinline__ uint32_t rows_tmem(const InferCta& c, int t, int h) {
    return c.tmem + ((uint32_t)(((t >> 5) & 3) * 32 + 16 * h) << 16) + 64u * (uint32_t)(t >> 7);
}

// this thread's pairs of a 64-vector: columns 2 (lane % 4), + 1 of each 8-column block of 32
__device__ __forceinline__ void load_pairs(const float* v, int lane, uint64_t* p) {
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const uint64_t*>(v + 8 * i + 2 * (lane & 3));
}

// Hidden layer epilogue for the warp's 32 rows: 32 columns of 16 rows at a time from TMEM, + bias, the
// activation, BF16 into the K-major hidden buffer (rows of all tiles, 64 columns).
template <int ACT>
__device__ __forceinline__ void hidden_epilogue(const InferCta& c, int t, const float* bias) {
    const int lane = t & 31, row0 = t & ~31;
    // address of the core-matrix row this lane stores: 8-row group (lane / 8) % 2, 8-column block lane / 16
    const uint32_t dst = c.base + c.h + tc::kmajor_offset(row0 + (lane & 15), 8 * (lane >> 4), 64);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        uint64_t b[4];
        load_pairs(bias + 32 * q, lane, b);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float z[16];
            tc::ld_frag32(rows_tmem(c, t, h) + 32 * q, z);
#pragma unroll
            for (int i = 0; i < 4; i += 2)
                tc::stmatrix4(dst + 2048 * h + (32 * q / 8 + i) * 128,
                              hidden_pair<ACT>(f2(z[4 * i], z[4 * i + 1]), b[i]),
                              hidden_pair<ACT>(f2(z[4 * i + 2], z[4 * i + 3]), b[i]),
                              hidden_pair<ACT>(f2(z[4 * i + 4], z[4 * i + 5]), b[i + 1]),
                              hidden_pair<ACT>(f2(z[4 * i + 6], z[4 * i + 7]), b[i + 1]));
        }
    }
}

// Layer 3 epilogue and the 64 -> 1 output layer: the logit of row t.
template <int ACT>
__device__ __forceinline__ float output_epilogue(const InferCta& c, int t) {
    const int lane = t & 31;
    uint64_t y2[2][2] = {};  // [row half][row T / 4 or T / 4 + 8], even and odd columns
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        uint64_t b[4], wt[4];
        load_pairs(c.vec + 128 + 32 * q, lane, b);
        load_pairs(c.vec + 192 + 32 * q, lane, wt);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float z[16];
            tc::ld_frag32(rows_tmem(c, t, h) + 32 * q, z);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                y2[h][0] = output_pair<ACT>(f2(z[4 * i], z[4 * i + 1]), b[i], wt[i], y2[h][0]);
                y2[h][1] = output_pair<ACT>(f2(z[4 * i + 2], z[4 * i + 3]), b[i], wt[i], y2[h][1]);
            }
        }
    }
    // sums over the four lanes that share a row, then row t's to thread t
    float y = 0.0f;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float lo, hi;
            f2_split(y2[h][e], lo, hi);
            float v = lo + hi;
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            v = __shfl_sync(0xffffffffu, v, 4 * (lane & 7));
            if ((lane >> 3) == 2 * h + e) y = v;
        }
    return y + c.vec[256];
}

// The same with one row per thread and its columns in order: the sum that the learned selection
// compares with its threshold (another order of the sum, 1e-7 away, decides a few pairs per frame the
// other way, which moves single pixels of the antiradiance by 1e-3).
template <int ACT>
__device__ __forceinline__ float output_in_order(const InferCta& c, int t) {
    const uint32_t taddr = rows_tmem(c, t, 0);
    const float* b3 = c.vec + 128;
    const float* w4 = c.vec + 192;
    uint64_t y2 = f2(c.vec[256], 0.0f);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        float z[16];
        tc::ld16(taddr + 16 * q, z);
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
            const float4 bb = *reinterpret_cast<const float4*>(b3 + 16 * q + j);
            const float4 ww = *reinterpret_cast<const float4*>(w4 + 16 * q + j);
            y2 = output_pair<ACT>(f2(z[j], z[j + 1]), f2(bb.x, bb.y), f2(ww.x, ww.y), y2);
            y2 = output_pair<ACT>(f2(z[j + 2], z[j + 3]), f2(bb.z, bb.w), f2(ww.z, ww.w), y2);
        }
    }
    float y0, y1;
    f2_split(y2, y0, y1);
    return y0 + y1;
}

// Logits of NT 128-row tiles: row t (of 128 NT, one per thread of the group) of the K-major input
// rows at smem offset x (stride between 8-row groups: 256 bytes), hidden rows at c.h (1024 bytes
// between 8-row groups; the input rows may lie in their first 4096 NT bytes), tile u's accumulator in
// TMEM columns 64 u .. 64 u + 63.  Called by all 128 NT threads; returns c.ok: false for a thread whose
// tensor-core wait gave up, after which the CTA calls drain_mma, frees its TMEM and stops.
template <int NT, int ACT, bool IN_ORDER, class Sync>
__device__ __forceinline__ bool infer_tiles(InferCta& c, uint32_t x, int t, float* logit, const Sync& s) {
    constexpr uint32_t id = tc::idesc_bf16(128, 64, false, false);
    // layer 1 (K = 16)
    publish_smem(s);
    if (t == 0 && c.ok) {
        c.committed = c.phase;
        tc::fence_after_sync();
#pragma unroll
        for (int u = 0; u < NT; ++u)
            tc::mma(c.tmem + 64 * u, tc::smem_desc(c.base + x + 4096 * u, 128, 256),
                    tc::smem_desc(c.base + c.w + kW1, 128, 256), id, false);
        tc::commit(c.bar);
    }
    wait_mma(c);
    hidden_epilogue<ACT>(c, t, c.vec);
    // layers 2 and 3 (K = 64); layer 2 overwrites the hidden buffer it read once its MMAs are done
#pragma unroll 1
    for (int l = 0; l < 2; ++l) {
        publish_smem(s);
        if (t == 0 && c.ok) {
            c.committed = c.phase;
            tc::fence_after_sync();
            const uint32_t wb = c.w + (l == 0 ? kW2 : kW3);
#pragma unroll
            for (int u = 0; u < NT; ++u)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    tc::mma(c.tmem + 64 * u, tc::smem_desc(c.base + c.h + 16384 * u + 256 * k, 128, 1024),
                            tc::smem_desc(c.base + wb + 256 * k, 128, 1024), id, k > 0);
            tc::commit(c.bar);
        }
        wait_mma(c);
        if (l == 0) hidden_epilogue<ACT>(c, t, c.vec + 64);
    }
    const float y = IN_ORDER ? output_in_order<ACT>(c, t) : output_epilogue<ACT>(c, t);
    // every thread's TMEM reads are done before the next round's MMAs overwrite the accumulators
    tc::fence_before_sync();
    *logit = y;
    return c.ok;
}

}  // namespace mlp
}  // namespace arc

#endif  // ARC_MLP_TILE_CUH_
