// Brute-force gather: radiance minus antiradiance of every AVPL at every pixel, fused into one
// kernel.  Replaces kernel_radiance_simple + kernel_antiradiance + kernel_combine
// (cudaGather.cu:269-314, 446-557, 782-803) and the cone antiradiance of Shaders/Gather.frag:149-188.
//
// Fast path (Lambertian materials, which every configured scene uses):
//   * AVPLs are first packed into 64-byte records {p, n}, {n, w}, {w, L'}, {A, 1/|w|} with
//     L' = L * (diffuse/pi) of the AVPL's own material (1 for light-source AVPLs), so the AVPL-side
//     BRDF of getRadiance (cudaGather.cu:84-90) is paid once per AVPL instead of once per pair.
//   * The receiver's Lambertian BRDF is constant per pixel and is applied once in the epilogue.
//   * A block owns a 16 x (16*PX) pixel tile; AVPL records are staged chunk by chunk into shared
//     memory with bulk asynchronous copies (cp.async.bulk, no multicast) on an mbarrier.
//   * The default and the all-FP64 precision (no or cone antiradiance) test each staged record once
//     against the tile's bounds and evaluate only the records that can add something to it
//     (gather_bf_culled_kernel, pair_cull.cuh), and the default precision's disk antiradiance is a
//     culled pass of its own (disk_ar.cu); the other precisions, every disk gather of the
//     allocation-free entry point, and gathers of few AVPLs (few_avpls) evaluate every pair
//     (gather_bf_kernel).
//   * Radiance and antiradiance go to separate sums (culled: per-chunk FP32 partials folded into
//     FP64; every pair: into Kahan sums, or per-term Kahan) and are combined in FP64.
// General path (specular materials or geometry-term limits): one thread per pixel evaluating the
// full f_r on both sides of every pair.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <type_traits>

#include "arc_internal.h"
#include "device_common.cuh"
#include "pair_cull.cuh"
#include "pair_math.cuh"

namespace arc {

namespace {

constexpr int kThreads = 256;
constexpr int kTileW = 16;
constexpr int kStages = 2;

struct BfArgs {
    const float4* records;  // 4 float4 per AVPL
    int32_t n;
    const float4* gpos;
    const float4* gnrm;
    int64_t gpitch;
    int32_t width, height;
    const MaterialRecord* mats;
    int32_t num_mats;
    float3 cam;
    PairConsts pc;       // per-pair constants (cone threshold, clamp, disk radius)
    float cos_thr;       // cone: max(cos(half angle), 0.001)
    float eps;           // cone: 0.001 (Gather.frag:10)
    float clamp2;        // dist_clamp^2, or 0
    float disk_r2;       // disk radius^2
    float disk_scale;    // 1 / (pi r^2)
    float lim_rad;       // GeoTermLimitRadiance or +inf
    float lim_ar;        // GeoTermLimitAntiradiance or +inf
    int32_t chunk;       // AVPL records per stage
    float4* out_res;
    float4* out_rad;
    float4* out_ar;
    double* out_res64;
    double* out_ar64;    // antiradiance in FP64 (3 per pixel), used by the cut path
    int64_t opitch;
    uint32_t* err;
    // general path (raw SoA)
    ArcAvplsGpuParam soa;
    // culled path: the AVPLs split over gridDim.z segments, each block's sums of one segment here
    // (NULL with one segment): [tile][segment][6][pixels of a tile]
    double* partial;
};

// ---------------------------------------------------------------------------------------
// pack: SoA -> 64-byte records
// ---------------------------------------------------------------------------------------
// One AVPL's 64-byte record (fields 0..15: p, n, w, L', A, 1/|w|).
__device__ __forceinline__ void bf_record(const ArcAvplsGpuParam& a, const MaterialRecord* mats, int32_t num_mats,
                                          int64_t i, uint32_t* err, float4* r) {
    const float3 p = ld3(a.position, i), nr = ld3(a.normal, i), w = ld3(a.incDirection, i);
    const float3 L = ld3(a.incRadiance, i), A = ld3(a.antiradiance, i);
    int m = a.materialIndex[i];
    if (m < 0 || m >= num_mats) {
        set_error(err, ARC_DEVERR_BAD_MATERIAL);
        m = 0;
    }
    const float4 dif = mats[m].diffuse_exp;
    const float inv_n = rn_div(1.0f, rn_sqrt(rn_dot(nr.x, nr.y, nr.z, nr.x, nr.y, nr.z)));
    const float3 n = f3(rn_mul(nr.x, inv_n), rn_mul(nr.y, inv_n), rn_mul(nr.z, inv_n));
    const float ww = rn_dot(w.x, w.y, w.z, w.x, w.y, w.z);
    const bool light = (ww == 0.0f);
    float3 Lp;
    Lp.x = light ? L.x : rn_mul(L.x, rn_mul(kOneOverPi, dif.x));
    Lp.y = light ? L.y : rn_mul(L.y, rn_mul(kOneOverPi, dif.y));
    Lp.z = light ? L.z : rn_mul(L.z, rn_mul(kOneOverPi, dif.z));
    const float inv_w = light ? 0.0f : rn_div(1.0f, rn_sqrt(ww));
    r[0] = make_float4(p.x, p.y, p.z, n.x);
    r[1] = make_float4(n.y, n.z, w.x, w.y);
    r[2] = make_float4(w.z, Lp.x, Lp.y, Lp.z);
    r[3] = make_float4(A.x, A.y, A.z, inv_w);
}

__global__ void pack_bf_records(ArcAvplsGpuParam a, const MaterialRecord* mats, int32_t num_mats, float4* rec,
                                uint32_t* err) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.numAvpls) return;
    float4 r[4];
    bf_record(a, mats, num_mats, i, err, r);
    float4* d = rec + 4 * i;
    d[0] = r[0];
    d[1] = r[1];
    d[2] = r[2];
    d[3] = r[3];
}

// PREC: 0 = chunk partials folded into Kahan sums, 1 = per-term Kahan, 2 = naive FP32, 3 = FP64.
template <int AR, int PREC, int PX>
__global__ void __launch_bounds__(kThreads) gather_bf_kernel(BfArgs k) {
    using T = typename std::conditional<PREC == 3, double, float>::type;
    extern __shared__ __align__(128) unsigned char smem[];
    float4* stage = reinterpret_cast<float4*>(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)kStages * k.chunk * 64);

    const int tid = threadIdx.x;
    const int tx = tid % kTileW, ty = tid / kTileW;
    const int x = blockIdx.x * kTileW + tx;
    const int rows = kThreads / kTileW;  // 16
    const int ybase = blockIdx.y * rows * PX + ty;

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(&bars[s], 1);
        fence_mbar_init();
    }

    Pixel<T> pix[PX];
    float sc[PX][6];  // Kahan compensation (PREC 0/1)
    float ss[PX][6];  // Kahan running sums (PREC 0)
    bool valid[PX];
    int mat[PX];
#pragma unroll
    for (int j = 0; j < PX; ++j) {
        const int y = ybase + j * rows;
        valid[j] = (x < k.width && y < k.height);
        mat[j] = 0;
        float4 gp = make_float4(0, 0, 0, 0), gn = make_float4(0, 0, 0, 0);
        if (valid[j]) {
            gp = k.gpos[(int64_t)y * k.gpitch + x];
            gn = k.gnrm[(int64_t)y * k.gpitch + x];
            mat[j] = (int)gn.w;
            if (mat[j] <= 0 || mat[j] >= k.num_mats) {
                if (mat[j] != 0) set_error(k.err, ARC_DEVERR_BAD_MATERIAL);
                valid[j] = false;
            }
        }
        T nx = 0, ny = 0, nz = 0;
        if (valid[j]) {
            const T l = rsqrt_t<T>((T)gn.x * gn.x + (T)gn.y * gn.y + (T)gn.z * gn.z);
            nx = gn.x * l;
            ny = gn.y * l;
            nz = gn.z * l;
        }
        pix[j].px = gp.x;
        pix[j].py = gp.y;
        pix[j].pz = gp.z;
        pix[j].nx = nx;
        pix[j].ny = ny;
        pix[j].nz = nz;
        pix[j].r0 = pix[j].r1 = pix[j].r2 = pix[j].a0 = pix[j].a1 = pix[j].a2 = 0;
#pragma unroll
        for (int c = 0; c < 6; ++c) sc[j][c] = ss[j][c] = 0.0f;
    }

    // A warp without a surface pixel skips the pairs, a block without one the records as well (known
    // before the first copy, so that none is in flight when it ends): 960 x 540 x 131,072, half of it
    // background, per-term Kahan 129.5 -> 75.1 ms, naive 91.7 -> 51.8 ms, the same sums.
    bool live = false;
#pragma unroll
    for (int j = 0; j < PX; ++j) live |= valid[j];
    live = __any_sync(0xffffffffu, live);
    const int nchunks = __syncthreads_or(live) ? (k.n + k.chunk - 1) / k.chunk : 0;
    if (tid == 0) {
        for (int c = 0; c < kStages && c < nchunks; ++c) {
            const int cnt = min(k.chunk, k.n - c * k.chunk);
            mbar_arrive_expect_tx(&bars[c], (uint32_t)cnt * 64u);
            bulk_g2s(stage + (size_t)c * k.chunk * 4, k.records + (size_t)c * k.chunk * 4, (uint32_t)cnt * 64u,
                     &bars[c]);
        }
    }

    bool ok = true;
    int fail_c = -1;  // first chunk whose wait gave up
    for (int c = 0; c < nchunks; ++c) {
        const int s = c % kStages;
        const uint32_t parity = (uint32_t)((c / kStages) & 1);
        if (ok) {
            ok = mbar_wait_bounded(&bars[s], parity, k.err);
            if (!ok) fail_c = c;
        }
        if (ok && live) {
            const int cnt = min(k.chunk, k.n - c * k.chunk);
            const float4* rec = stage + (size_t)s * k.chunk * 4;
#pragma unroll 2
            for (int i = 0; i < cnt; ++i) {
                const float4 q0 = rec[4 * i + 0], q1 = rec[4 * i + 1], q2 = rec[4 * i + 2], q3 = rec[4 * i + 3];
#pragma unroll
                for (int j = 0; j < PX; ++j) {
                    T g, ga;
                    pair_terms<AR, T>(q0, q1, q2, q3, pix[j], k.pc, g, ga);
                    if (PREC == 1) {
                        kahan_add(ss[j][0], sc[j][0], (float)(q2.y * g));
                        kahan_add(ss[j][1], sc[j][1], (float)(q2.z * g));
                        kahan_add(ss[j][2], sc[j][2], (float)(q2.w * g));
                        if (AR != ARC_AR_NONE) {
                            kahan_add(ss[j][3], sc[j][3], (float)(q3.x * ga));
                            kahan_add(ss[j][4], sc[j][4], (float)(q3.y * ga));
                            kahan_add(ss[j][5], sc[j][5], (float)(q3.z * ga));
                        }
                    } else {
                        pix[j].r0 += (T)q2.y * g;
                        pix[j].r1 += (T)q2.z * g;
                        pix[j].r2 += (T)q2.w * g;
                        if (AR != ARC_AR_NONE) {
                            pix[j].a0 += (T)q3.x * ga;
                            pix[j].a1 += (T)q3.y * ga;
                            pix[j].a2 += (T)q3.z * ga;
                        }
                    }
                }
            }
            if (PREC == 0) {
#pragma unroll
                for (int j = 0; j < PX; ++j) {
                    kahan_add(ss[j][0], sc[j][0], (float)pix[j].r0);
                    kahan_add(ss[j][1], sc[j][1], (float)pix[j].r1);
                    kahan_add(ss[j][2], sc[j][2], (float)pix[j].r2);
                    kahan_add(ss[j][3], sc[j][3], (float)pix[j].a0);
                    kahan_add(ss[j][4], sc[j][4], (float)pix[j].a1);
                    kahan_add(ss[j][5], sc[j][5], (float)pix[j].a2);
                    pix[j].r0 = pix[j].r1 = pix[j].r2 = pix[j].a0 = pix[j].a1 = pix[j].a2 = 0;
                }
            }
        }
        __syncthreads();  // every thread is done reading stage s before it is refilled
        if (tid == 0 && ok && c + kStages < nchunks) {
            fence_proxy_async_smem();
            const int cn = c + kStages;
            const int cnt = min(k.chunk, k.n - cn * k.chunk);
            mbar_arrive_expect_tx(&bars[s], (uint32_t)cnt * 64u);
            bulk_g2s(stage + (size_t)s * k.chunk * 4, k.records + (size_t)cn * k.chunk * 4, (uint32_t)cnt * 64u,
                     &bars[s]);
        }
    }
    // the copies the ring still has in flight after a wait gave up (only thread 0 issues them)
    if (tid == 0 && fail_c >= 0) drain_ring_bounded(bars, kStages, fail_c, nchunks, k.err);

    // epilogue: receiver BRDF, signed combine, stores
#pragma unroll
    for (int j = 0; j < PX; ++j) {
        const int y = ybase + j * rows;
        if (x >= k.width || y >= k.height) continue;
        double rad[3] = {0, 0, 0}, ar[3] = {0, 0, 0}, res[3] = {0, 0, 0};
        float radf[3] = {0, 0, 0}, arf[3] = {0, 0, 0}, resf[3] = {0, 0, 0};
        if (valid[j]) {
            const float4 d = k.mats[mat[j]].diffuse_exp;
            const float kd[3] = {kOneOverPi * d.x, kOneOverPi * d.y, kOneOverPi * d.z};
            const float arscale = (AR == ARC_AR_DISK) ? k.disk_scale : 1.0f;
            if (PREC == 2) {
                const float S[6] = {(float)pix[j].r0, (float)pix[j].r1, (float)pix[j].r2,
                                    (float)pix[j].a0, (float)pix[j].a1, (float)pix[j].a2};
                for (int c = 0; c < 3; ++c) {
                    radf[c] = kd[c] * S[c];
                    arf[c] = kd[c] * arscale * S[3 + c];
                    resf[c] = radf[c] - arf[c];
                    rad[c] = radf[c];
                    ar[c] = arf[c];
                    res[c] = resf[c];
                }
            } else {
                double S[6];
                if (PREC == 3) {
                    S[0] = (double)pix[j].r0; S[1] = (double)pix[j].r1; S[2] = (double)pix[j].r2;
                    S[3] = (double)pix[j].a0; S[4] = (double)pix[j].a1; S[5] = (double)pix[j].a2;
                } else {
                    for (int c = 0; c < 6; ++c) S[c] = (double)ss[j][c] - (double)sc[j][c];
                }
                for (int c = 0; c < 3; ++c) {
                    rad[c] = (double)kd[c] * S[c];
                    ar[c] = (double)kd[c] * (double)arscale * S[3 + c];
                    res[c] = rad[c] - ar[c];
                    radf[c] = (float)rad[c];
                    arf[c] = (float)ar[c];
                    resf[c] = (float)res[c];
                }
            }
        }
        const int64_t o = (int64_t)y * k.opitch + x;
        if (k.out_res) k.out_res[o] = make_float4(resf[0], resf[1], resf[2], 1.0f);
        if (k.out_rad) k.out_rad[o] = make_float4(radf[0], radf[1], radf[2], 1.0f);
        if (k.out_ar) k.out_ar[o] = make_float4(arf[0], arf[1], arf[2], 1.0f);
        if (k.out_res64) {
            k.out_res64[3 * o + 0] = res[0];
            k.out_res64[3 * o + 1] = res[1];
            k.out_res64[3 * o + 2] = res[2];
        }
    }
}

// A pixel's outputs from its FP64 sums (radiance 0..2, antiradiance 3..5): receiver BRDF, signed
// combine; 0 without a surface (material 0).
__device__ __forceinline__ void write_pixel(const BfArgs& k, int x, int y, int mat, const double* S) {
    double rad[3] = {0, 0, 0}, ar[3] = {0, 0, 0}, res[3] = {0, 0, 0};
    if (mat > 0) {
        const float4 d = k.mats[mat].diffuse_exp;
        const float kd[3] = {kOneOverPi * d.x, kOneOverPi * d.y, kOneOverPi * d.z};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            rad[c] = (double)kd[c] * S[c];
            ar[c] = (double)kd[c] * S[3 + c];
            res[c] = rad[c] - ar[c];
        }
    }
    const int64_t o = (int64_t)y * k.opitch + x;
    if (k.out_res) k.out_res[o] = make_float4((float)res[0], (float)res[1], (float)res[2], 1.0f);
    if (k.out_rad) k.out_rad[o] = make_float4((float)rad[0], (float)rad[1], (float)rad[2], 1.0f);
    if (k.out_ar) k.out_ar[o] = make_float4((float)ar[0], (float)ar[1], (float)ar[2], 1.0f);
    if (k.out_res64)
        for (int c = 0; c < 3; ++c) k.out_res64[3 * o + c] = res[c];
    if (k.out_ar64)
        for (int c = 0; c < 3; ++c) k.out_ar64[3 * o + c] = ar[c];
}

// ---------------------------------------------------------------------------------------
// Culled form of the default precision (T = float: packed FP32x2, per-chunk FP32 partials folded
// into FP64 sums) and of the all-FP64 precision (T = double), no or cone antiradiance.
//
// A block owns a 16 x 16 PX pixel tile and one segment (blockIdx.z) of the AVPLs.  Per chunk of
// staged records: each thread tests one record against the tile's bounds (record_need), the kept
// ones go in AVPL order into a radiance list and a cone list, the next chunk's copy is issued, and
// every thread runs its PX pixels over the two lists.  The sums of several segments are added in
// FP64 by bf_combine_segments.
//
// The default precision's sparse tiles -- at most half of the pixels have a surface, and no more than the
// block has threads -- are worked on differently: the surface pixels move to the front, one per thread, only
// the warps that hold some run the pair loops, and where they are half of the block's warps or fewer the
// rest take the same pixels over every second, fourth or eighth pair of records (the block adds their sums
// in FP64).  With all pixels evaluated a tile costs the same whatever its surface: 960 x 540 x 131,072 AVPLs
// with 1%, 5%, 20% and 50% of scattered surface pixels 42.9, 50.3, 50.9 and 51.1 ms, now 5.2, 6.2, 15.7 and
// 39.9 ms (a kernel over a list of the surface pixels that tests no records: 12.2, 12.2, 23.9 and 47.4 ms).
// Above half the tile's two pixels per thread share each record's loads.
//
// Bound by the FMA pipe: 18 packed FP32x2 operations per two radiance pairs (69% of the pipe's cycles,
// 16.3 instructions per evaluated pair).  1920 x 1080 x 262,144 AVPLs, cone 60 degrees: 133 ms (138 ms before
// the warps without a surface pixel left the pairs out), 352 ms for the kernel that evaluated every pair;
// all FP64, 637 x 359 x 16,381: 3.5 against 20.3 ms.
// ---------------------------------------------------------------------------------------
// staged records | the two lists | FP32: the threads' FP64 sums (their registers hold the pixels and
// the pair loop's operands instead) | mbarrier
template <typename T, int PX>
constexpr int culled_smem(int chunk) {
    return chunk * 64 + 2 * chunk * (int)(kPairFloats / 2 * sizeof(T)) +
           (sizeof(T) == 4 ? 6 * PX * kThreads * (int)sizeof(double) : 0) + 8;
}

// Three resident blocks of up to two pixels per thread hide the pair loop's latencies (24 warps)
template <int AR, typename T, int PX, bool RAD>
__global__ void __launch_bounds__(kThreads, PX <= 2 ? 3 : 1) gather_bf_culled_kernel(BfArgs k) {
    constexpr bool kDouble = sizeof(T) == 8;
    constexpr int kW = kThreads / 32;
    extern __shared__ __align__(128) unsigned char smem[];
    float4* stage = reinterpret_cast<float4*>(smem);
    T* list_r = reinterpret_cast<T*>(smem + (size_t)k.chunk * 64);
    T* list_a = list_r + (size_t)k.chunk * (kPairFloats / 2);
    double* fsum = reinterpret_cast<double*>(list_a + (size_t)k.chunk * (kPairFloats / 2)) + threadIdx.x;
    uint64_t* bar = reinterpret_cast<uint64_t*>(list_a + (size_t)k.chunk * (kPairFloats / 2)) +
                    (kDouble ? 0 : 6 * PX * kThreads);
    __shared__ PixelBounds sb[kW];
    __shared__ int s_cnt[2][2][kW];
    __shared__ int s_live[PX * kW];    // surface pixels per (pixel of a thread, warp)
    __shared__ short s_pix[kThreads];  // a sparse tile's surface pixels: kThreads j + thread
    static_assert(PX * kW <= 32, "one lane per count in the block's sum");

    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int x = blockIdx.x * kTileW + tid % kTileW;
    const int y0 = blockIdx.y * (kThreads / kTileW) * PX + tid / kTileW;
    constexpr int rows = kThreads / kTileW;

    T px_[PX], py_[PX], pz_[PX], nx_[PX], ny_[PX], nz_[PX];
    int mat[PX];  // 0: no surface
    PixelBounds b;
    b.clear();
    bool any = false;
#pragma unroll
    for (int j = 0; j < PX; ++j) {
        const int y = y0 + j * rows;
        const bool in = x < k.width && y < k.height;
        float4 gp = make_float4(0, 0, 0, 0), gn = make_float4(0, 0, 0, 0);
        if (in) {
            gp = k.gpos[(int64_t)y * k.gpitch + x];
            gn = k.gnrm[(int64_t)y * k.gpitch + x];
        }
        mat[j] = (int)gn.w;
        if (mat[j] <= 0 || mat[j] >= k.num_mats) {
            if (mat[j] != 0) set_error(k.err, ARC_DEVERR_BAD_MATERIAL);
            mat[j] = 0;
        }
        nx_[j] = ny_[j] = nz_[j] = (T)0;
        px_[j] = gp.x;
        py_[j] = gp.y;
        pz_[j] = gp.z;
        if (mat[j]) {
            const T l = rsqrt_t<T>((T)gn.x * gn.x + (T)gn.y * gn.y + (T)gn.z * gn.z);
            nx_[j] = gn.x * l;
            ny_[j] = gn.y * l;
            nz_[j] = gn.z * l;
            any = true;
            if constexpr (kDouble)
                b.add(gp.x, gp.y, gp.z, __double2float_rd(nx_[j]), __double2float_rd(ny_[j]),
                      __double2float_rd(nz_[j]), __double2float_ru(nx_[j]), __double2float_ru(ny_[j]),
                      __double2float_ru(nz_[j]));
            else
                b.add(gp.x, gp.y, gp.z, nx_[j], ny_[j], nz_[j], nx_[j], ny_[j], nz_[j]);
        }
    }
    unsigned lm[PX];
#pragma unroll
    for (int j = 0; j < PX; ++j) {
        lm[j] = __ballot_sync(0xffffffffu, mat[j] != 0);
        if (lane == 0) s_live[j * kW + w] = __popc(lm[j]);
    }
    __syncthreads();
    // (counted again where it is needed: a register for it would last through the pair loops)
    auto surfaces = [&] { return __reduce_add_sync(0xffffffffu, lane < PX * kW ? s_live[lane] : 0); };
    const int found = surfaces();
    const bool live = found > 0, sparse = !kDouble && live && found <= min(kThreads, kThreads * PX / 2);
    bool works = __any_sync(0xffffffffu, any);
    if (sparse) {
        const int warps = (found + 31) >> 5;
        works = w < kW / warps * warps;
#pragma unroll
        for (int j = 0; j < PX; ++j) {
            int at = __popc(lm[j] & ((1u << lane) - 1u));
            for (int q = 0; q < j * kW + w; ++q) at += s_live[q];
            if (mat[j]) s_pix[at] = (short)(j * kThreads + tid);
            const int y = y0 + j * rows;
            const double none[6] = {0, 0, 0, 0, 0, 0};
            if (!k.partial && !mat[j] && x < k.width && y < k.height) write_pixel(k, x, y, 0, none);
        }
        __syncthreads();
        nx_[0] = ny_[0] = nz_[0] = (T)0;
        const int at = w % warps * 32 + lane;
        if (at < found) {
            const int px = s_pix[at];
            const int64_t g = (int64_t)(blockIdx.y * rows * PX + px / kTileW) * k.gpitch + blockIdx.x * kTileW + px % kTileW;
            const float4 gp = k.gpos[g], gn = k.gnrm[g];
            px_[0] = gp.x;
            py_[0] = gp.y;
            pz_[0] = gp.z;
            const T l = rsqrt_t<T>((T)gn.x * gn.x + (T)gn.y * gn.y + (T)gn.z * gn.z);
            nx_[0] = gn.x * l;
            ny_[0] = gn.y * l;
            nz_[0] = gn.z * l;
        }
    }

    double sum[PX][6];  // T = double; the FP32 form keeps its sums at fsum[(6 j + c) * kThreads]
#pragma unroll
    for (int j = 0; j < PX; ++j)
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            sum[j][c] = 0.0;
            if (!kDouble) fsum[(6 * j + c) * kThreads] = 0.0;
        }
    // adds a chunk's packed partial (even and odd list entries) to sum c of pixel j
    auto fold = [&](int j, int c, uint64_t acc) {
        float lo, hi;
        f2_split(acc, lo, hi);
        fsum[(6 * j + c) * kThreads] += (double)(lo + hi);
    };
    if (live) {
        // this segment's chunks
        const int nchunks = (k.n + k.chunk - 1) / k.chunk;
        const int c0 = (int)((int64_t)nchunks * blockIdx.z / gridDim.z),
                  c1 = (int)((int64_t)nchunks * (blockIdx.z + 1) / gridDim.z);
        auto copy_chunk = [&](int c) {
            const uint32_t bytes = (uint32_t)min(k.chunk, k.n - c * k.chunk) * 64u;
            mbar_arrive_expect_tx(bar, bytes);
            bulk_g2s(stage, k.records + (size_t)c * k.chunk * 4, bytes, bar);
        };
        if (tid == 0) {
            mbar_init(bar, 1);
            fence_mbar_init();
        }
        b.reduce_warp();
        if (lane == 0) sb[w] = b;
        __syncthreads();
        if (tid == 0 && c0 < c1) copy_chunk(c0);
        if (w == 0) {
            b = sb[lane & (kW - 1)];
            b.reduce_warp();
            if (lane == 0) sb[0] = b;
        }
        __syncthreads();
        const float cos_thr = k.pc.cos_thr, eps = k.pc.eps, inv_clamp2 = k.pc.inv_clamp2;
        // distance floor folded into the FMA chain: l2 + 1e-30 equals max(l2, 1e-30) for l2 above ~1e-23
        const uint64_t tiny2 = f2(1e-30f, 1e-30f);
        PixelPair pp[PX];
        if constexpr (!kDouble) {
#pragma unroll
            for (int j = 0; j < PX; ++j) pp[j] = pixel_pair(px_[j], py_[j], pz_[j], nx_[j], ny_[j], nz_[j]);
        }
        for (int c = c0; c < c1; ++c) {
            const bool ok = mbar_wait_bounded(bar, (uint32_t)((c - c0) & 1), k.err);
            const int cnt = min(k.chunk, k.n - c * k.chunk);
            int nr = 0, na = 0;  // list lengths so far
            bool all_ok = true;
            for (int base = 0; base < cnt; base += kThreads) {
                const int i = base + tid, turn = (base / kThreads) & 1;
                RecordNeed need{false, false};
                float4 q0, q1, q2, q3;
                if (ok && i < cnt) {
                    q0 = stage[4 * i];
                    q1 = stage[4 * i + 1];
                    q2 = stage[4 * i + 2];
                    q3 = stage[4 * i + 3];
                    need = record_need<AR == ARC_AR_CONE>(sb[0], q0, q1, q2, q3, cos_thr);
                    if (!RAD) need.radiance = false;
                }
                const unsigned mr = __ballot_sync(0xffffffffu, need.radiance);
                const unsigned ma = __ballot_sync(0xffffffffu, need.cone);
                if (lane == 0) {
                    s_cnt[turn][0][w] = __popc(mr);
                    s_cnt[turn][1][w] = __popc(ma);
                }
                // also: every thread is done with the lists of the chunk before
                all_ok = __syncthreads_and(ok) != 0;
                if (!all_ok) break;
                int er = nr + __popc(mr & ((1u << lane) - 1u)), ea = na + __popc(ma & ((1u << lane) - 1u));
#pragma unroll
                for (int q = 0; q < kW; ++q) {
                    const int r = s_cnt[turn][0][q], a = s_cnt[turn][1][q];
                    if (q < w) {
                        er += r;
                        ea += a;
                    }
                    nr += r;
                    na += a;
                }
                if constexpr (kDouble) {
                    if (need.radiance) {
                        T* d = list_r + (size_t)er * (kPairFloats / 2);
                        d[0] = q0.x; d[1] = q0.y; d[2] = q0.z;
                        d[3] = q0.w; d[4] = q1.x; d[5] = q1.y;
                        d[6] = q2.y; d[7] = q2.z; d[8] = q2.w;
                    }
                    if (need.cone) {
                        T* d = list_a + (size_t)ea * (kPairFloats / 2);
                        d[0] = q0.x; d[1] = q0.y; d[2] = q0.z;
                        d[3] = q1.z; d[4] = q1.w; d[5] = q2.x;
                        d[6] = q3.x; d[7] = q3.y; d[8] = q3.z;
                    }
                } else {
                    if (need.radiance)
                        put_entry(list_r, er, q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q2.y, q2.z, q2.w);
                    if (need.cone) put_entry(list_a, ea, q0.x, q0.y, q0.z, q1.z, q1.w, q2.x, q3.x, q3.y, q3.z);
                }
            }
            if (!all_ok) {  // the copy gave up: one more bounded wait for it before the block exits
                if (tid == 0) drain_ring_bounded(bar, 1, c - c0, c1 - c0, k.err);
                break;
            }
            if constexpr (!kDouble) {  // an odd list ends with a zero record, which adds exactly 0
                if (tid == 0 && (nr & 1)) put_entry(list_r, nr, 0, 0, 0, 0, 0, 0, 0, 0, 0);
                if (tid == 32 && (na & 1)) put_entry(list_a, na, 0, 0, 0, 0, 0, 0, 0, 0, 0);
            }
            __syncthreads();  // lists complete, staged records no longer read
            if (tid == 0 && c + 1 < c1) {
                fence_proxy_async_smem();
                copy_chunk(c + 1);
            }
            if (!works) continue;
            if constexpr (kDouble) {
                const T clampi = (T)inv_clamp2;
#pragma unroll 2
                for (int i = 0; i < nr; ++i) {
                    const T* d = list_r + (size_t)i * (kPairFloats / 2);
#pragma unroll
                    for (int j = 0; j < PX; ++j) {
                        const T dx = d[0] - px_[j], dy = d[1] - py_[j], dz = d[2] - pz_[j];
                        T l2 = dx * dx + dy * dy + dz * dz;
                        l2 = l2 > (T)1e-30 ? l2 : (T)1e-30;
                        const T inv = (T)1 / l2;
                        const T a = (nx_[j] * dx + ny_[j] * dy + nz_[j] * dz) * inv;
                        const T e = -(d[3] * dx + d[4] * dy + d[5] * dz) * (inv < clampi ? inv : clampi);
                        const T g = (a > (T)0 ? a : (T)0) * (e > (T)0 ? e : (T)0);
                        sum[j][0] += d[6] * g;
                        sum[j][1] += d[7] * g;
                        sum[j][2] += d[8] * g;
                    }
                }
                if (AR == ARC_AR_CONE) {
                    for (int i = 0; i < na; ++i) {
                        const T* d = list_a + (size_t)i * (kPairFloats / 2);
#pragma unroll
                        for (int j = 0; j < PX; ++j) {
                            const T dx = d[0] - px_[j], dy = d[1] - py_[j], dz = d[2] - pz_[j];
                            T l2 = dx * dx + dy * dy + dz * dz;
                            l2 = l2 > (T)1e-30 ? l2 : (T)1e-30;
                            const T r = rsqrt(l2);
                            const T a = (nx_[j] * dx + ny_[j] * dy + nz_[j] * dz) * r;
                            const T cw = -(d[3] * dx + d[4] * dy + d[5] * dz) * r;
                            const T rr = r * r;
                            // (outside the cone 0 times the antiradiance is added: it may not be finite)
                            const T ga = cw > (T)cos_thr && a > (T)eps ? a * (rr < clampi ? rr : clampi) : (T)0;
                            sum[j][3] += d[6] * ga;
                            sum[j][4] += d[7] * ga;
                            sum[j][5] += d[8] * ga;
                        }
                    }
                }
            } else {
                // PX pixels over the whole lists, or (sparse) one over this group's share of them
                auto pairs = [&](auto is_sparse) {
                    constexpr bool kSparse = decltype(is_sparse)::value;
                    constexpr int N = kSparse ? 1 : PX;
                    const int warps = kSparse ? (surfaces() + 31) >> 5 : kW;
                    const int first = kSparse ? w / warps : 0, step = kSparse ? kW / warps : 1;
                    if (RAD) {
                        uint64_t acc[N][3] = {};  // packed zeros
#pragma unroll 2
                        for (int pr = first; 2 * pr < nr; pr += step)
#pragma unroll
                            for (int j = 0; j < N; ++j)
                                radiance_pair(list_r + pr * kPairFloats, pp[j], inv_clamp2, tiny2, acc[j][0], acc[j][1],
                                              acc[j][2]);
#pragma unroll
                        for (int j = 0; j < N; ++j)
#pragma unroll
                            for (int q = 0; q < 3; ++q) fold(j, q, acc[j][q]);
                    }
                    if (AR == ARC_AR_CONE && na > 0) {
                        uint64_t acc[N][3] = {};
#pragma unroll 1
                        for (int pr = first; 2 * pr < na; pr += step)
#pragma unroll
                            for (int j = 0; j < N; ++j)
                                cone_pair(list_a + pr * kPairFloats, pp[j], cos_thr, eps, inv_clamp2, tiny2, acc[j][0],
                                          acc[j][1], acc[j][2]);
#pragma unroll
                        for (int j = 0; j < N; ++j)
#pragma unroll
                            for (int q = 0; q < 3; ++q) fold(j, 3 + q, acc[j][q]);
                    }
                };
                if (sparse)
                    pairs(std::true_type{});
                else
                    pairs(std::false_type{});
            }
        }
    }

    if (sparse) {
        __syncthreads();  // every group's sums, added in group order
        const int count = surfaces(), warps = (count + 31) >> 5;
        if (tid >= count) return;
        double S[6] = {0, 0, 0, 0, 0, 0};
        for (int g = 0; g < kW / warps; ++g)
            for (int c = 0; c < 6; ++c) S[c] += fsum[c * kThreads + g * warps * 32];
        const int px = s_pix[tid], xp = blockIdx.x * kTileW + px % kTileW, yp = blockIdx.y * rows * PX + px / kTileW;
        if (k.partial) {
            double* d = k.partial + (((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * gridDim.z + blockIdx.z) * 6 *
                                        (kThreads * PX) + px;
            for (int c = 0; c < 6; ++c) d[c * (kThreads * PX)] = S[c];
        } else {
            write_pixel(k, xp, yp, (int)k.gnrm[(int64_t)yp * k.gpitch + xp].w, S);
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < PX; ++j) {
        double S[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) S[c] = kDouble ? sum[j][c] : fsum[(6 * j + c) * kThreads];
        if (k.partial) {
            double* d = k.partial + (((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * gridDim.z + blockIdx.z) * 6 *
                                        (kThreads * PX) + j * kThreads + tid;
            if (live)  // (a tile without surface pixels is written by bf_combine_segments alone)
#pragma unroll
                for (int c = 0; c < 6; ++c) d[c * (kThreads * PX)] = S[c];
        } else {
            const int y = y0 + j * rows;
            if (x < k.width && y < k.height) write_pixel(k, x, y, mat[j], S);
        }
    }
}

// The segments' sums of every pixel added in segment order, and the outputs; the grid of
// gather_bf_culled_kernel without its segments.
template <int PX>
__global__ void __launch_bounds__(kThreads) bf_combine_segments(BfArgs k, int segments) {
    const int tid = threadIdx.x;
    const int x = blockIdx.x * kTileW + tid % kTileW;
#pragma unroll
    for (int j = 0; j < PX; ++j) {
        const int y = (blockIdx.y * PX + j) * (kThreads / kTileW) + tid / kTileW;
        if (x >= k.width || y >= k.height) continue;
        int m = (int)k.gnrm[(int64_t)y * k.gpitch + x].w;
        if (m < 0 || m >= k.num_mats) m = 0;
        double S[6] = {0, 0, 0, 0, 0, 0};
        if (m > 0) {
            const double* d = k.partial + ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * segments * 6 *
                                              (kThreads * PX) + j * kThreads + tid;
            for (int s = 0; s < segments; ++s)
#pragma unroll
                for (int c = 0; c < 6; ++c) S[c] += d[(s * 6 + c) * (kThreads * PX)];
        }
        write_pixel(k, x, y, m, S);
    }
}

// ---------------------------------------------------------------------------------------
// General path: full f_r on both sides (cudaGather.cu:59-95), geometry-term limits
// (Gather.frag:182, 190-194); one thread per pixel over the raw SoA arrays.
// ---------------------------------------------------------------------------------------
template <typename T>
struct V {
    T x, y, z;
};
template <typename T>
__device__ __forceinline__ V<T> vsub(V<T> a, V<T> b) {
    return {a.x - b.x, a.y - b.y, a.z - b.z};
}
template <typename T>
__device__ __forceinline__ V<T> vs(T s, V<T> a) {
    return {s * a.x, s * a.y, s * a.z};
}
template <typename T>
__device__ __forceinline__ T vdot(V<T> a, V<T> b) {
    return a.x * b.x + a.y * b.y + a.z * b.z;
}
template <typename T>
__device__ __forceinline__ V<T> vnorm(V<T> a) {
    return vs(rsqrt_t<T>(vdot(a, a)), a);
}

// f_r(w_i, w_o, n, mat) = diffuse/pi + [|spec| > 0] (e+2)/(2 pi) max(0, reflect(-w_i, n).w_o)^e spec
template <typename T>
__device__ __forceinline__ V<T> brdf(V<T> w_i, V<T> w_o, V<T> n, const MaterialRecord& m) {
    V<T> d = {(T)kOneOverPi * m.diffuse_exp.x, (T)kOneOverPi * m.diffuse_exp.y, (T)kOneOverPi * m.diffuse_exp.z};
    if (m.specular_flag.w != 0.0f) {
        const V<T> I = vs((T)-1, w_i);
        const V<T> r = vsub(I, vs((T)2 * vdot(n, I), n));
        T c = vdot(r, w_o);
        c = c > (T)0 ? c : (T)0;
        const T e = m.diffuse_exp.w;
        const T f = (T)0.5 * (T)kOneOverPi * (e + (T)2) * (T)pow(c, e);
        d.x += f * m.specular_flag.x;
        d.y += f * m.specular_flag.y;
        d.z += f * m.specular_flag.z;
    }
    return d;
}

template <int AR, typename T>
__global__ void __launch_bounds__(kThreads) gather_general_kernel(BfArgs k) {
    __shared__ MaterialRecord smat[ARC_MAX_MATERIALS];
    for (int i = threadIdx.x; i < k.num_mats; i += blockDim.x) smat[i] = k.mats[i];
    __syncthreads();
    const int x = blockIdx.x * kTileW + threadIdx.x % kTileW;
    const int y = blockIdx.y * (kThreads / kTileW) + threadIdx.x / kTileW;
    if (x >= k.width || y >= k.height) return;
    const float4 gp = k.gpos[(int64_t)y * k.gpitch + x];
    const float4 gn = k.gnrm[(int64_t)y * k.gpitch + x];
    const int m = (int)gn.w;
    double rad[3] = {0, 0, 0}, ar[3] = {0, 0, 0};
    if (m > 0 && m < k.num_mats) {
        const V<T> p = {(T)gp.x, (T)gp.y, (T)gp.z};
        const V<T> n = vnorm(V<T>{(T)gn.x, (T)gn.y, (T)gn.z});
        const V<T> cam = {(T)k.cam.x, (T)k.cam.y, (T)k.cam.z};
        const V<T> w_o = vnorm(vsub(cam, p));
        T s[6] = {0, 0, 0, 0, 0, 0};
        float c[6] = {0, 0, 0, 0, 0, 0};
        const ArcAvplsGpuParam& a = k.soa;
        for (int i = 0; i < a.numAvpls; ++i) {
            const float3 fpa = ld3(a.position, i), fna = ld3(a.normal, i), fwa = ld3(a.incDirection, i);
            const V<T> pa = {(T)fpa.x, (T)fpa.y, (T)fpa.z};
            const V<T> na = vnorm(V<T>{(T)fna.x, (T)fna.y, (T)fna.z});
            const V<T> wa = {(T)fwa.x, (T)fwa.y, (T)fwa.z};
            int ma = a.materialIndex[i];
            if (ma < 0 || ma >= k.num_mats) ma = 0;
            const V<T> v = vsub(pa, p);
            T l2 = vdot(v, v);
            if (!(l2 > (T)0)) continue;
            const V<T> w = vs(rsqrt_t<T>(l2), v);  // pixel -> AVPL
            const V<T> fr = brdf<T>(w, w_o, n, smat[m]);
            // radiance
            V<T> fl = {1, 1, 1};
            if (vdot(wa, wa) != (T)0) fl = brdf<T>(vs((T)-1, wa), vs((T)-1, w), na, smat[ma]);
            T c1 = vdot(n, w), c2 = -vdot(na, w);
            c1 = c1 < (T)0 ? (T)0 : (c1 > (T)1 ? (T)1 : c1);
            c2 = c2 < (T)0 ? (T)0 : (c2 > (T)1 ? (T)1 : c2);
            const T l2c = l2 < (T)k.clamp2 ? (T)k.clamp2 : l2;
            T g = c1 * c2 / l2c;
            if (g > (T)k.lim_rad) g = (T)k.lim_rad;
            const float3 L = ld3(a.incRadiance, i), A = ld3(a.antiradiance, i);
            T term[6];
            term[0] = (T)L.x * fl.x * fr.x * g;
            term[1] = (T)L.y * fl.y * fr.y * g;
            term[2] = (T)L.z * fl.z * fr.z * g;
            T ga = 0;
            if (AR == ARC_AR_CONE) {
                const T cw = -vdot(w, wa);
                const T cn = vdot(n, w);
                if (cw > (T)k.eps && cn > (T)k.eps && cw > (T)k.cos_thr) {
                    ga = cn / l2c;
                    if (ga > (T)k.lim_ar) ga = (T)k.lim_ar;
                }
            } else if (AR == ARC_AR_DISK) {
                const T wn = vdot(wa, n);
                if (wn != (T)0) {
                    const T t = -vdot(v, n) / wn;
                    const V<T> wu = vnorm(wa);
                    const V<T> h = {pa.x + t * wu.x, pa.y + t * wu.y, pa.z + t * wu.z};
                    const V<T> hp = vsub(h, p);
                    if (t > (T)0 && vdot(hp, hp) < (T)k.disk_r2 && wn < (T)0 && -vdot(w, na) < (T)0) ga = (T)k.disk_scale;
                }
            }
            term[3] = (T)A.x * fr.x * ga;
            term[4] = (T)A.y * fr.y * ga;
            term[5] = (T)A.z * fr.z * ga;
            if (sizeof(T) == 8) {
                for (int q = 0; q < 6; ++q) s[q] += term[q];
            } else {
                for (int q = 0; q < 6; ++q) {
                    float ssq = (float)s[q];
                    kahan_add(ssq, c[q], (float)term[q]);
                    s[q] = (T)ssq;
                }
            }
        }
        for (int q = 0; q < 3; ++q) {
            rad[q] = (double)s[q] - (double)c[q];
            ar[q] = (double)s[3 + q] - (double)c[3 + q];
        }
    }
    const int64_t o = (int64_t)y * k.opitch + x;
    const double res[3] = {rad[0] - ar[0], rad[1] - ar[1], rad[2] - ar[2]};
    if (k.out_res) k.out_res[o] = make_float4((float)res[0], (float)res[1], (float)res[2], 1.0f);
    if (k.out_rad) k.out_rad[o] = make_float4((float)rad[0], (float)rad[1], (float)rad[2], 1.0f);
    if (k.out_ar) k.out_ar[o] = make_float4((float)ar[0], (float)ar[1], (float)ar[2], 1.0f);
    if (k.out_res64) {
        k.out_res64[3 * o + 0] = res[0];
        k.out_res64[3 * o + 1] = res[1];
        k.out_res64[3 * o + 2] = res[2];
    }
}

// Tile shapes selectable by ArcGatherParams::tile_config: pixels per thread x AVPLs per stage.
struct TileShape {
    int px;
    int chunk;
};
constexpr TileShape kTileShapes[] = {{1, 128}, {2, 128}, {2, 256}, {4, 128}, {4, 256}, {1, 256}, {2, 64},
                                     {4, 64},  {1, 512}, {2, 512}, {4, 512}, {1, 1024}, {2, 1024}};
constexpr int kNumTileShapes = sizeof(kTileShapes) / sizeof(kTileShapes[0]);
constexpr int kDefaultTileShape = 2;
constexpr int kFp64Chunk = 256;
// Segments of the culled gather: enough blocks for several waves of resident ones (a grid of one
// partial wave leaves SMs idle: 64 x 64 x 4,096 takes 269 us in one segment and 59 us split, 640 x 360 x
// 16,384 2.14 and 1.30 ms), each segment at least kMinChunks chunks long (a block's set-up -- pixel
// loads, tile bounds -- costs about a chunk), partial sums within kPartialBytes.  Measured:
//   blocks per SM 6 / 12 / 24 / 48: 640 x 360 x 16,384 1.39 / 1.17 / 1.10 / 1.10 ms, 1280 x 720 x 65,536 16.5 /
//     16.7 / 15.1 / 14.4 ms, 1920 x 1080 x 262,144 123.0 / 123.1 / 122.7 / 120.2 ms, smaller ones the same;
//   chunks per segment 1 / 2 / 4: 64 x 64 x 4,096 60 / 71 / 103 us, 256 x 256 x 4,096 204 / 196 / 218 us, larger
//     ones the same.
constexpr int kBlocksPerSm = 24;
constexpr int kMinChunks = 2;
constexpr int64_t kPartialBytes = (int64_t)1 << 30;

// The most records per stage of the tile shapes with PX pixels per thread.  A kernel's limit of dynamic
// shared memory belongs to the device: it is set to what the largest of its shapes needs, the same value
// from every call, so that a call of another context or thread cannot lower it before this one's launch.
template <int PX>
constexpr int max_chunk() {
    int most = 0;
    for (const TileShape& t : kTileShapes)
        if (t.px == PX && t.chunk > most) most = t.chunk;
    return most;
}

constexpr int fast_smem(int chunk) { return kStages * chunk * 64 + kStages * (int)sizeof(uint64_t); }

template <int AR, int PREC, int PX>
arc_status launch_fast(const BfArgs& a, cudaStream_t st) {
    const int smem = fast_smem(a.chunk);
    auto fn = gather_bf_kernel<AR, PREC, PX>;
    if (smem > 48 * 1024)
        ARC_TRY_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, fast_smem(max_chunk<PX>())));
    dim3 grid((a.width + kTileW - 1) / kTileW, (a.height + 16 * PX - 1) / (16 * PX));
    fn<<<grid, kThreads, smem, st>>>(a);
    ARC_TRY_CUDA(cudaGetLastError());
    return ARC_OK;
}

template <int AR, int PREC>
arc_status launch_fast_px(const BfArgs& a, int px, cudaStream_t st) {
    if (px == 1) return launch_fast<AR, PREC, 1>(a, st);
    if (px == 2) return launch_fast<AR, PREC, 2>(a, st);
    return launch_fast<AR, PREC, 4>(a, st);
}

// Few AVPLs: one launch of the kernel that evaluates every pair takes less than the culled kernel's
// barriers and list tests (all FP64), or than the culled radiance, disk pass and combination (default
// precision, disk).  Microseconds, culled / every pair:
//   disk    1 x 1 x 1: 41 / 17, 192 x 192 x 64: 44 / 41, 512 x 512 x 16: 67 / 32, 1920 x 1080 x 16: 201 / 105
//   FP64    1 x 1 x 1: 25 / 16, 192 x 192 x 64: 30 / 30, 512 x 512 x 16: 49 / 37, 1920 x 1080 x 16: 166 / 128
// and beyond the line culled is ahead: 512 x 512 x 128 84 / 131 and 97 / 176, 1920 x 1080 x 64 217 / 438 and
// 228 / 647.
bool few_avpls(int n, int64_t pixels) {
    return n <= 16 || (n <= 64 && n * pixels <= (int64_t)1 << 23);
}

// the culled kernel serves the default and the all-FP64 precision with no or cone antiradiance
bool use_culled(const ArcGatherParams& p, int n, int64_t pixels) {
    if (p.ar_kind == ARC_AR_DISK) return false;
    return p.precision == ARC_PREC_KAHAN || (p.precision == ARC_PREC_FP64 && !few_avpls(n, pixels));
}

dim3 tile_grid(const BfArgs& a, int px) {
    return dim3((a.width + kTileW - 1) / kTileW, (a.height + 16 * px - 1) / (16 * px));
}

template <int AR, typename T, int PX, bool RAD>
arc_status launch_culled_kernel(const BfArgs& a, int segments, cudaStream_t st) {
    const int smem = culled_smem<T, PX>(a.chunk);
    auto fn = gather_bf_culled_kernel<AR, T, PX, RAD>;
    constexpr int most = culled_smem<T, PX>(sizeof(T) == 8 ? kFp64Chunk : max_chunk<PX>());
    ARC_TRY_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    dim3 grid = tile_grid(a, PX);
    grid.z = (unsigned)segments;
    fn<<<grid, kThreads, smem, st>>>(a);
    ARC_TRY_CUDA(cudaGetLastError());
    if (a.partial) {
        bf_combine_segments<PX><<<tile_grid(a, PX), kThreads, 0, st>>>(a, segments);
        ARC_TRY_CUDA(cudaGetLastError());
    }
    return ARC_OK;
}

template <int AR, bool RAD>
arc_status launch_culled_px(const BfArgs& a, int px, int segments, cudaStream_t st) {
    if (px == 1) return launch_culled_kernel<AR, float, 1, RAD>(a, segments, st);
    if (px == 2) return launch_culled_kernel<AR, float, 2, RAD>(a, segments, st);
    return launch_culled_kernel<AR, float, 4, RAD>(a, segments, st);
}

// A culled gather: its pixels per thread and AVPLs per chunk, and how many segments the AVPLs are
// split into.
struct CulledPlan {
    int px, chunk, segments;
};

CulledPlan culled_plan(const BfArgs& a, const ArcGatherParams& p, int shape, int sm_count) {
    CulledPlan c{kTileShapes[shape >= 0 ? shape : kDefaultTileShape].px,
                 kTileShapes[shape >= 0 ? shape : kDefaultTileShape].chunk, 1};
    if (p.precision == ARC_PREC_FP64) c = CulledPlan{1, kFp64Chunk, 1};
    const dim3 g = tile_grid(a, c.px);
    const int64_t tiles = (int64_t)g.x * g.y;
    const int64_t want = ((int64_t)sm_count * kBlocksPerSm + tiles - 1) / tiles;
    const int64_t chunks = (a.n + c.chunk - 1) / c.chunk;
    const int64_t room = kPartialBytes / (tiles * 6 * kThreads * c.px * (int64_t)sizeof(double));
    c.segments = (int)std::max<int64_t>(1, std::min(std::min(want, chunks / kMinChunks), room));
    return c;
}

// dispatch of the culled path (a.records packed); a.partial: room for plan.segments, or NULL with one
arc_status launch_culled(BfArgs a, const ArcGatherParams& p, const CulledPlan& c, cudaStream_t st) {
    a.chunk = c.chunk;
    if (p.precision == ARC_PREC_FP64)
        return p.ar_kind == ARC_AR_NONE ? launch_culled_kernel<0, double, 1, true>(a, c.segments, st)
                                        : launch_culled_kernel<2, double, 1, true>(a, c.segments, st);
    return p.ar_kind == ARC_AR_NONE ? launch_culled_px<0, true>(a, c.px, c.segments, st)
                                    : launch_culled_px<2, true>(a, c.px, c.segments, st);
}

template <int AR>
arc_status launch_fast_prec(const BfArgs& a, int prec, int px, cudaStream_t st) {
    return prec == ARC_PREC_KAHAN_STRICT ? launch_fast_px<AR, 1>(a, px, st) : launch_fast_px<AR, 2>(a, px, st);
}

// dispatch of the kernel that evaluates every pair
arc_status launch_fast_path(const BfArgs& a, const ArcGatherParams& p, int px, cudaStream_t st) {
    if (p.ar_kind == ARC_AR_DISK) {
        if (p.precision == ARC_PREC_KAHAN) return launch_fast_px<1, 0>(a, px, st);
        if (p.precision == ARC_PREC_FP64) return launch_fast<1, 3, 1>(a, st);
        return launch_fast_prec<1>(a, p.precision, px, st);
    }
    if (p.precision == ARC_PREC_FP64)
        return p.ar_kind == ARC_AR_NONE ? launch_fast<0, 3, 1>(a, st) : launch_fast<2, 3, 1>(a, st);
    return p.ar_kind == ARC_AR_NONE ? launch_fast_prec<0>(a, p.precision, px, st)
                                    : launch_fast_prec<2>(a, p.precision, px, st);
}

BfArgs make_args(arc_context* ctx, const GatherLaunch& g);
arc_status pack_records(arc_context* ctx, const GatherLaunch& g, BfArgs& a);
arc_status run_culled(arc_context* ctx, BfArgs& a, const ArcGatherParams& p, int shape, bool rad);

}  // namespace

int bf_num_tile_shapes() { return kNumTileShapes; }

arc_status launch_gather_bruteforce(arc_context* ctx, const GatherLaunch& g) {
    const ArcGatherParams& p = *g.params;
    const ArcGBufferView& gb = *g.gbuffer;
    const ArcOutputView& out = *g.out;
    ARC_CHECK_ARG(p.ar_kind >= 0 && p.ar_kind <= 2, "ar_kind out of range");
    ARC_CHECK_ARG(p.precision >= 0 && p.precision <= 3, "precision out of range");
    ARC_CHECK_ARG(p.tile_config >= -1 && p.tile_config < kNumTileShapes, "tile_config out of range");
    ARC_CHECK_ARG(gb.width > 0 && gb.height > 0 && gb.pitch >= gb.width && gb.position && gb.normal,
                  "bad G-buffer view");
    ARC_CHECK_ARG(out.pitch >= gb.width && (out.result || out.radiance || out.antiradiance || out.result_fp64),
                  "bad output view");
    ARC_CHECK_ARG(g.avpls->numAvpls >= 0, "negative AVPL count");
    ARC_CHECK_ARG(ctx->num_materials > 0, "materials not uploaded");
    ARC_CHECK_ARG(p.ar_kind != ARC_AR_DISK || p.disk_radius > 0.0f, "disk radius must be > 0");
    ARC_CHECK_ARG(reinterpret_cast<uintptr_t>(gb.position) % 16 == 0 && reinterpret_cast<uintptr_t>(gb.normal) % 16 == 0,
                  "G-buffer planes must be 16-byte aligned");

    BfArgs a = make_args(ctx, g);
    const bool general = ctx->any_specular || p.geo_limit_radiance > 0.0f || p.geo_limit_antiradiance > 0.0f;
    cudaStream_t st = ctx->stream;
    if (general) {
        dim3 grid((gb.width + kTileW - 1) / kTileW, (gb.height + 15) / 16);
        stage_begin(ctx, "bf_general");
        if (p.precision == ARC_PREC_FP64) {
            if (p.ar_kind == 0) gather_general_kernel<0, double><<<grid, kThreads, 0, st>>>(a);
            if (p.ar_kind == 1) gather_general_kernel<1, double><<<grid, kThreads, 0, st>>>(a);
            if (p.ar_kind == 2) gather_general_kernel<2, double><<<grid, kThreads, 0, st>>>(a);
        } else {
            if (p.ar_kind == 0) gather_general_kernel<0, float><<<grid, kThreads, 0, st>>>(a);
            if (p.ar_kind == 1) gather_general_kernel<1, float><<<grid, kThreads, 0, st>>>(a);
            if (p.ar_kind == 2) gather_general_kernel<2, float><<<grid, kThreads, 0, st>>>(a);
        }
        stage_end(ctx, 1);
        ARC_TRY_CUDA(cudaGetLastError());
        return ARC_OK;
    }
    ARC_TRY(pack_records(ctx, g, a));
    const int chosen = p.tile_config >= 0 ? p.tile_config : ctx->bf_tile_config;
    const int64_t pixels = (int64_t)gb.width * gb.height;
    if (use_culled(p, a.n, pixels)) return run_culled(ctx, a, p, chosen, true);
    if (p.ar_kind == ARC_AR_DISK && p.precision == ARC_PREC_KAHAN && !few_avpls(a.n, pixels)) {
        // the radiance by the culled gather, the antiradiance by the culled disk pass
        double *rad64 = nullptr, *ar64 = nullptr;
        const size_t bytes = (size_t)gb.height * out.pitch * 3 * sizeof(double);
        ARC_TRY(ctx->arena.get("bf_rad64", bytes, reinterpret_cast<void**>(&rad64)));
        ARC_TRY(ctx->arena.get("bf_ar64", bytes, reinterpret_cast<void**>(&ar64)));
        ArcGatherParams q = p;
        q.ar_kind = ARC_AR_NONE;
        a.out_res = a.out_ar = nullptr;
        a.out_res64 = rad64;
        ARC_TRY(run_culled(ctx, a, q, chosen, true));
        ARC_TRY(launch_disk_antiradiance(ctx, g.avpls, a.records, &gb, &p, false, nullptr, ar64, out.pitch));
        return launch_combine(ctx, rad64, ar64, gb.width, gb.height, &out);
    }
    const TileShape ts = kTileShapes[chosen >= 0 ? chosen : kDefaultTileShape];
    a.chunk = ts.chunk;
    stage_begin(ctx, "bf_gather");
    const arc_status s = launch_fast_path(a, p, ts.px, st);
    stage_end(ctx, 1);
    return s;
}

arc_status launch_pack_records(arc_context* ctx, const ArcAvplsGpuParam* avpls, const float4** records) {
    const int n = avpls->numAvpls;
    float4* rec = nullptr;
    ARC_TRY(ctx->arena.get("bf_records", (size_t)(n + 1) * 64, reinterpret_cast<void**>(&rec)));
    if (n > 0) {
        stage_begin(ctx, "bf_pack");
        pack_bf_records<<<(n + 255) / 256, 256, 0, ctx->stream>>>(*avpls, ctx->d_materials, ctx->num_materials, rec,
                                                                   ctx->d_error);
        stage_end(ctx, 1);
        ARC_TRY_CUDA(cudaGetLastError());
    }
    *records = rec;
    return ARC_OK;
}

arc_status launch_antiradiance_only(arc_context* ctx, const GatherLaunch& g, double* ar64) {
    const ArcGatherParams& p = *g.params;
    if (p.ar_kind == ARC_AR_DISK)
        return launch_disk_antiradiance(ctx, g.avpls, nullptr, g.gbuffer, &p, false, nullptr, ar64, g.out->pitch);
    BfArgs a = make_args(ctx, g);
    a.out_res = nullptr;
    a.out_rad = nullptr;
    a.out_ar = nullptr;
    a.out_res64 = nullptr;
    a.out_ar64 = ar64;
    ARC_TRY(pack_records(ctx, g, a));
    ArcGatherParams q = p;
    q.precision = ARC_PREC_KAHAN;
    return run_culled(ctx, a, q, -1, false);
}

}  // namespace arc

namespace arc {
namespace {

BfArgs make_args(arc_context* ctx, const GatherLaunch& g) {
    const ArcGatherParams& p = *g.params;
    const ArcGBufferView& gb = *g.gbuffer;
    const ArcOutputView& out = *g.out;
    BfArgs a{};
    a.n = g.avpls->numAvpls;
    a.gpos = reinterpret_cast<const float4*>(gb.position);
    a.gnrm = reinterpret_cast<const float4*>(gb.normal);
    a.gpitch = gb.pitch;
    a.width = gb.width;
    a.height = gb.height;
    a.mats = ctx->d_materials;
    a.num_mats = ctx->num_materials;
    a.cam = g.cam;
    a.eps = 0.001f;
    a.cos_thr = fmaxf(cosf(p.cone_half_angle), a.eps);
    a.clamp2 = p.dist_clamp > 0.0f ? p.dist_clamp * p.dist_clamp : 0.0f;
    a.disk_r2 = p.disk_radius * p.disk_radius;
    a.pc.cos_thr = a.cos_thr;
    a.pc.eps = a.eps;
    a.pc.inv_clamp2 = p.dist_clamp > 0.0f ? 1.0f / a.clamp2 : INFINITY;
    a.pc.disk_r2 = a.disk_r2;
    a.disk_scale = p.disk_radius > 0.0f ? 1.0f / (kPi * p.disk_radius * p.disk_radius) : 0.0f;
    a.lim_rad = p.geo_limit_radiance > 0.0f ? p.geo_limit_radiance : INFINITY;
    a.lim_ar = p.geo_limit_antiradiance > 0.0f ? p.geo_limit_antiradiance : INFINITY;
    a.out_res = reinterpret_cast<float4*>(out.result);
    a.out_rad = reinterpret_cast<float4*>(out.radiance);
    a.out_ar = reinterpret_cast<float4*>(out.antiradiance);
    a.out_res64 = out.result_fp64;
    a.opitch = out.pitch;
    a.err = ctx->d_error;
    a.soa = *g.avpls;
    return a;
}

// Pack the AVPL records into the context arena.
arc_status pack_records(arc_context* ctx, const GatherLaunch& g, BfArgs& a) {
    const float4* rec = nullptr;
    ARC_TRY(launch_pack_records(ctx, g.avpls, &rec));
    a.records = rec;
    return ARC_OK;
}

// The culled gather on the context's stream (rad: radiance and antiradiance; else the cone
// antiradiance alone), its partial sums in the context arena.
arc_status run_culled(arc_context* ctx, BfArgs& a, const ArcGatherParams& p, int shape, bool rad) {
    const CulledPlan c = culled_plan(a, p, shape, ctx->sm_count);
    if (c.segments > 1) {
        const dim3 g = tile_grid(a, c.px);
        ARC_TRY(ctx->arena.get("bf_partial", (size_t)g.x * g.y * c.segments * 6 * kThreads * c.px * sizeof(double),
                               reinterpret_cast<void**>(&a.partial)));
    }
    stage_begin(ctx, rad ? "bf_gather" : "bf_antiradiance");
    arc_status s;
    if (rad) {
        s = launch_culled(a, p, c, ctx->stream);
    } else {
        a.chunk = c.chunk;
        s = launch_culled_px<ARC_AR_CONE, false>(a, c.px, c.segments, ctx->stream);
    }
    stage_end(ctx, a.partial ? 2 : 1);
    return s;
}

}  // namespace
}  // namespace arc

// ---------------------------------------------------------------------------------------
// Allocation-free brute-force gather (arc_gather_bruteforce_noalloc).
//
// For hosts that own every byte of device memory themselves and forbid the library from
// allocating: renderer plugins whose host pre-allocates a fixed device budget at start-up, and
// real-time frame loops that must not call cudaMalloc/cudaFree mid-frame (both can synchronise
// the device and stall the frame).  Such a caller cannot create an arc_context (which
// allocates), so this entry point takes a stream instead and keeps its only scratch -- the
// packed AVPL records, the material table and the device error word -- in one file-scope
// __device__ array of fixed size, which every GPU that loads libarc holds until the process
// exits.
// ---------------------------------------------------------------------------------------
#include <mutex>

static constexpr int kNoAllocMaxAvpls = 65536;  // AVPL records the static scratch holds
static constexpr size_t kNoAllocRecordBytes = (size_t)kNoAllocMaxAvpls * 64;
static constexpr size_t kNoAllocMaterialBytes = ARC_MAX_MATERIALS * sizeof(arc::MaterialRecord);
// [records: 64 B x kNoAllocMaxAvpls][materials: 32 B x 64][error word: 256 B]  (4.2 MB)
static constexpr size_t kNoAllocBytes = kNoAllocRecordBytes + kNoAllocMaterialBytes + 256;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

namespace arc {
namespace {

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
// per device: the context the address was looked up in, and the address
void* g_noalloc_ctx[kNoAllocMaxDevices] = {};
unsigned char* g_noalloc_addr[kNoAllocMaxDevices] = {};

using CtxGetCurrentFn = int (*)(void**);  // cuCtxGetCurrent(CUcontext*) -> CUresult

// The driver context current on this thread (NULL if the driver entry point is unavailable).
void* current_driver_context() {
    static CtxGetCurrentFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<CtxGetCurrentFn>(f);
    }();
    void* c = nullptr;
    if (fn && fn(&c) != 0) c = nullptr;
    return c;
}

// Device address of g_noalloc_scratch in the current device's context, looked up with that
// device current the first time a call runs in that context (again after a device reset or in
// another driver context, where the module is loaded anew at another address).  The host-side
// name g_noalloc_scratch is only a stand-in for the symbol and must never be handed to a kernel.
arc_status noalloc_scratch(unsigned char** out) {
    int dev = 0;
    ARC_TRY_CUDA(cudaGetDevice(&dev));
    ARC_CHECK_ARG(dev >= 0 && dev < kNoAllocMaxDevices, "device index beyond the allocation-free path's table");
    // (NULL before the runtime has made the device's primary context current: looked up then)
    const void* c = current_driver_context();
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_addr[dev] || !c || c != g_noalloc_ctx[dev]) {
        void* p = nullptr;
        ARC_TRY_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        g_noalloc_addr[dev] = static_cast<unsigned char*>(p);
        g_noalloc_ctx[dev] = current_driver_context();  // current now, after the lookup
    }
    *out = g_noalloc_addr[dev];
    return ARC_OK;
}

// The material table travels as a kernel argument (no host buffer is read after the call
// returns); the same launch clears the call's error word.
struct NoAllocMaterials {
    MaterialRecord rec[ARC_MAX_MATERIALS];
    int count;
};

__global__ void noalloc_write_materials(NoAllocMaterials t, MaterialRecord* mats, uint32_t* err) {
    const int i = threadIdx.x;
    if (i < t.count) mats[i] = t.rec[i];
    if (i == 0) *err = 0u;
}

}  // namespace
}  // namespace arc

extern "C" arc_status arc_gather_bruteforce_noalloc(void* cuda_stream, const ArcMaterial* materials,
                                                    int32_t num_materials, const ArcAvplsGpuParam* avpls,
                                                    const ArcGBufferView* gbuffer, ArcFloat3 camera_position,
                                                    const ArcGatherParams* params, const ArcOutputView* out,
                                                    uint32_t* device_error_word) {
    using namespace arc;
    ARC_CHECK_ARG(materials && avpls && gbuffer && params && out, "NULL argument");
    const ArcGatherParams& p = *params;
    const ArcGBufferView& gb = *gbuffer;
    ARC_CHECK_ARG(num_materials > 0 && num_materials <= ARC_MAX_MATERIALS,
                  "material count must be in [1, ARC_MAX_MATERIALS]");
    ARC_CHECK_ARG(avpls->numAvpls >= 0, "negative AVPL count");
    if (avpls->numAvpls > kNoAllocMaxAvpls) {
        set_last_error("arc_gather_bruteforce_noalloc: " + std::to_string(avpls->numAvpls) +
                       " AVPLs exceed the allocation-free path's maximum of " + std::to_string(kNoAllocMaxAvpls) +
                       " (use arc_gather_bruteforce)");
        return ARC_ERR_INVALID_ARG;
    }
    ARC_CHECK_ARG(p.ar_kind >= 0 && p.ar_kind <= 2, "ar_kind out of range");
    ARC_CHECK_ARG(p.precision >= 0 && p.precision <= 3, "precision out of range");
    ARC_CHECK_ARG(p.tile_config >= -1 && p.tile_config < kNumTileShapes, "tile_config out of range");
    ARC_CHECK_ARG(gb.width > 0 && gb.height > 0 && gb.pitch >= gb.width && gb.position && gb.normal,
                  "bad G-buffer view");
    ARC_CHECK_ARG(reinterpret_cast<uintptr_t>(gb.position) % 16 == 0 && reinterpret_cast<uintptr_t>(gb.normal) % 16 == 0,
                  "G-buffer planes must be 16-byte aligned");
    ARC_CHECK_ARG(out->pitch >= gb.width && (out->result || out->radiance || out->antiradiance || out->result_fp64),
                  "bad output view");
    ARC_CHECK_ARG(p.ar_kind != ARC_AR_DISK || p.disk_radius > 0.0f, "disk radius must be > 0");

    unsigned char* scratch = nullptr;
    ARC_TRY(noalloc_scratch(&scratch));
    float4* records = reinterpret_cast<float4*>(scratch);
    MaterialRecord* mats = reinterpret_cast<MaterialRecord*>(scratch + kNoAllocRecordBytes);
    uint32_t* err = reinterpret_cast<uint32_t*>(scratch + kNoAllocRecordBytes + kNoAllocMaterialBytes);
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);

    // material table and error word: the scratch keeps the previous call's contents, so both are
    // rewritten here (the records are rewritten by the pack kernel for every AVPL used)
    NoAllocMaterials tab;
    tab.count = num_materials;
    bool spec = false;
    for (int i = 0; i < num_materials; ++i) {
        const ArcMaterial& m = materials[i];
        const float sl = sqrtf(m.specular.x * m.specular.x + m.specular.y * m.specular.y + m.specular.z * m.specular.z);
        tab.rec[i].diffuse_exp = make_float4(m.diffuse.x, m.diffuse.y, m.diffuse.z, m.exponent);
        tab.rec[i].specular_flag = make_float4(m.specular.x, m.specular.y, m.specular.z, sl > 0.0f ? 1.0f : 0.0f);
        spec = spec || sl > 0.0f;
    }
    for (int i = num_materials; i < ARC_MAX_MATERIALS; ++i) {
        tab.rec[i].diffuse_exp = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        tab.rec[i].specular_flag = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    noalloc_write_materials<<<1, ARC_MAX_MATERIALS, 0, st>>>(tab, mats, err);
    ARC_TRY_CUDA(cudaGetLastError());

    BfArgs a{};
    a.n = avpls->numAvpls;
    a.gpos = reinterpret_cast<const float4*>(gb.position);
    a.gnrm = reinterpret_cast<const float4*>(gb.normal);
    a.gpitch = gb.pitch;
    a.width = gb.width;
    a.height = gb.height;
    a.mats = mats;
    a.num_mats = num_materials;
    a.cam = make_float3(camera_position.x, camera_position.y, camera_position.z);
    a.eps = 0.001f;
    a.cos_thr = fmaxf(cosf(p.cone_half_angle), a.eps);
    a.clamp2 = p.dist_clamp > 0.0f ? p.dist_clamp * p.dist_clamp : 0.0f;
    a.disk_r2 = p.disk_radius * p.disk_radius;
    a.pc.cos_thr = a.cos_thr;
    a.pc.eps = a.eps;
    a.pc.inv_clamp2 = p.dist_clamp > 0.0f ? 1.0f / a.clamp2 : INFINITY;
    a.pc.disk_r2 = a.disk_r2;
    a.disk_scale = p.disk_radius > 0.0f ? 1.0f / (kPi * p.disk_radius * p.disk_radius) : 0.0f;
    a.lim_rad = p.geo_limit_radiance > 0.0f ? p.geo_limit_radiance : INFINITY;
    a.lim_ar = p.geo_limit_antiradiance > 0.0f ? p.geo_limit_antiradiance : INFINITY;
    a.out_res = reinterpret_cast<float4*>(out->result);
    a.out_rad = reinterpret_cast<float4*>(out->radiance);
    a.out_ar = reinterpret_cast<float4*>(out->antiradiance);
    a.out_res64 = out->result_fp64;
    a.out_ar64 = nullptr;
    a.opitch = out->pitch;
    a.err = err;
    a.soa = *avpls;
    a.records = records;

    if (spec || p.geo_limit_radiance > 0.0f || p.geo_limit_antiradiance > 0.0f) {
        dim3 grid((gb.width + kTileW - 1) / kTileW, (gb.height + 15) / 16);
        if (p.precision == ARC_PREC_FP64) {
            if (p.ar_kind == 0) gather_general_kernel<0, double><<<grid, kThreads, 0, st>>>(a);
            if (p.ar_kind == 1) gather_general_kernel<1, double><<<grid, kThreads, 0, st>>>(a);
            if (p.ar_kind == 2) gather_general_kernel<2, double><<<grid, kThreads, 0, st>>>(a);
        } else {
            if (p.ar_kind == 0) gather_general_kernel<0, float><<<grid, kThreads, 0, st>>>(a);
            if (p.ar_kind == 1) gather_general_kernel<1, float><<<grid, kThreads, 0, st>>>(a);
            if (p.ar_kind == 2) gather_general_kernel<2, float><<<grid, kThreads, 0, st>>>(a);
        }
        ARC_TRY_CUDA(cudaGetLastError());
    } else {
        if (a.n > 0) {
            pack_bf_records<<<(a.n + 255) / 256, 256, 0, st>>>(*avpls, mats, num_materials, records, err);
            ARC_TRY_CUDA(cudaGetLastError());
        }
        if (use_culled(p, a.n, (int64_t)gb.width * gb.height)) {  // one segment: there is no room for partial sums
            CulledPlan c = culled_plan(a, p, p.tile_config, 1);
            c.segments = 1;
            ARC_TRY(launch_culled(a, p, c, st));
        } else {
            const TileShape ts = kTileShapes[p.tile_config < 0 ? kDefaultTileShape : p.tile_config];
            a.chunk = ts.chunk;
            ARC_TRY(launch_fast_path(a, p, ts.px, st));
        }
    }
    if (device_error_word) {
        uint32_t w = 0;
        ARC_TRY_CUDA(cudaMemcpyAsync(&w, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        ARC_TRY_CUDA(cudaStreamSynchronize(st));
        *device_error_word = w;
    }
    return ARC_OK;
}

// Brute-force launch-shape autotuner (no counterpart in the reference): times every shape of
// kTileShapes on the caller's workload (one warm-up and one timed run each, CUDA events on the
// context's stream) and makes the fastest the context's default for tile_config = -1.
extern "C" int32_t arc_bruteforce_num_tile_shapes(void) { return arc::kNumTileShapes; }

extern "C" arc_status arc_context_set_tile_config(arc_context* ctx, int32_t tile_config) {
    ARC_CHECK_ARG(ctx, "NULL context");
    ARC_CHECK_ARG(tile_config >= -1 && tile_config < arc::kNumTileShapes, "tile_config out of range");
    ctx->bf_tile_config = tile_config;
    return ARC_OK;
}

extern "C" arc_status arc_autotune_bruteforce(arc_context* ctx, const ArcAvplsGpuParam* avpls,
                                              const ArcGBufferView* gbuffer, ArcFloat3 camera_position,
                                              const ArcGatherParams* params, const ArcOutputView* out, int32_t* best,
                                              float* times_ms, int32_t num_shapes) {
    using namespace arc;
    ARC_CHECK_ARG(ctx && avpls && gbuffer && params && out && best, "NULL argument");
    ARC_CHECK_ARG(!times_ms || num_shapes >= kNumTileShapes, "times_ms holds fewer entries than there are shapes");
    ARC_TRY_CUDA(cudaSetDevice(ctx->device));
    ScopedEvents<2> ev;
    ARC_TRY_CUDA(ev.create());
    const cudaEvent_t e0 = ev[0], e1 = ev[1];
    cudaError_t ce = cudaSuccess;
    arc_status s = ARC_OK;
    float best_ms = 0.0f;
    int best_i = -1;
    for (int i = 0; i < kNumTileShapes && s == ARC_OK; ++i) {
        ArcGatherParams p = *params;
        p.tile_config = i;
        s = arc_gather_bruteforce(ctx, avpls, gbuffer, camera_position, &p, out);  // warm-up
        if (s == ARC_OK) ce = cudaEventRecord(e0, ctx->stream);
        if (s == ARC_OK && ce == cudaSuccess) s = arc_gather_bruteforce(ctx, avpls, gbuffer, camera_position, &p, out);
        if (s == ARC_OK && ce == cudaSuccess) ce = cudaEventRecord(e1, ctx->stream);
        if (s == ARC_OK && ce == cudaSuccess) ce = cudaEventSynchronize(e1);
        float ms = -1.0f;
        if (s == ARC_OK && ce == cudaSuccess) ce = cudaEventElapsedTime(&ms, e0, e1);
        if (ce != cudaSuccess && s == ARC_OK) {
            set_last_error(std::string("arc_autotune_bruteforce: ") + cudaGetErrorString(ce));
            s = ARC_ERR_CUDA;
        }
        if (times_ms) times_ms[i] = ms;
        if (s == ARC_OK && (best_i < 0 || ms < best_ms)) {
            best_ms = ms;
            best_i = i;
        }
    }
    ARC_TRY(s);
    ctx->bf_tile_config = best_i;
    *best = best_i;
    return ARC_OK;
}

