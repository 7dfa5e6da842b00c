// Disk antiradiance of every AVPL at every pixel (getAntiradiance, cudaGather.cu:97-144), with the
// AVPLs culled per block of pixels.
//
// A pair contributes only when the AVPL's ray p_a + s w (s > 0) passes within the disk radius of the
// pixel, the AVPL lies in front of the pixel and the pixel behind the AVPL: a handful of AVPLs per
// pixel.  A block owns a pixel tile and walks the AVPLs in order, kStep at a time:
//   1. each thread tests AVPLs' rays against the tile's bounding spheres grown by the radius (two, the
//      halves of a split along the longest axis: a tile across a silhouette has one as deep as the
//      scene), and the block compacts the survivors of several steps in AVPL order;
//   2. each warp tests the survivors, one per lane, against its own pixels' two spheres and their position
//      and normal boxes, and stages the records that remain;
//   3. every lane evaluates those for its pixels with the terms of pair_terms, in AVPL order, with one
//      compensated sum per channel.
// The tests drop a pair only when pair_terms is certain to give 0 (their margins exceed its rounding),
// so the sums are those over every AVPL.  Several blocks share a tile, each with a segment of the AVPLs
// (tiles differ in work); disk_combine adds their sums in FP64.
//
// Bound by latency (a step's loads, ballots and barrier; the lists hold a few per cent of the rays).
// 512 x 512 x 32,768: 0.28 ms, 21.5 ms for the kernel that evaluated every pair.  The work left is the ray tests, 20 operations per (tile,
// AVPL) instead of 45 per (pixel, AVPL).
#include <algorithm>
#include <cfloat>

#include "arc_internal.h"
#include "device_common.cuh"
#include "pair_cull.cuh"
#include "pair_math.cuh"

namespace arc {
namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kPerThread = 2;                     // rays tested per thread and step
constexpr int kStep = kThreads * kPerThread;      // AVPLs per step
constexpr int kList = 1024;                       // survivors collected before the warps go over them
constexpr int kCounts = kPerThread * kWarps;      // survivor counts of a step, one per (pass, warp)
static_assert(kCounts <= 32, "one lane per count in the block's prefix sum");

// 32 x 32 tiles when they make at least this many blocks per SM (a quarter of the ray tests; 1280 x 720 x
// 65,536: 0.55 against 0.99 ms), else 16 x 16 (more, smaller blocks).
constexpr int64_t kBigTilesPerSm = 2;
// Segments: blocks per SM at which the AVPLs are no longer split, the blocks' set-up against their balance
// (512 x 512 x 32,768 / 1280 x 720 x 65,536 / 1920 x 1080 x 65,536 in ms: 0.284 / 0.640 / 1.143 at 8 per SM,
// 0.285 / 0.560 / 0.948 at 16, 0.290 / 0.533 / 0.948 at 24, 0.298 / 0.527 / 0.910 at 32, 0.319 / 0.538 / 0.916 at
// 48), partial sums within kPartialBytes.
constexpr int64_t kBlocksPerSm = 24;
constexpr int64_t kPartialBytes = (int64_t)1 << 30;

struct DiskArgs {
    const float4* records;  // 4 float4 per AVPL (launch_pack_records)
    // 2 float4 per AVPL that can add something: {p, > 0: where its ray passes, < 0: to every pixel},
    // {w / |w|, index}; counts[s] of them from kStep s on
    const float4* rays;
    const int* counts;
    int n;
    const float4* gpos;
    const float4* gnrm;
    int64_t gpitch;
    int width, height;
    const MaterialRecord* mats;
    int num_mats;
    PairConsts pc;
    float radius;
    float disk_scale;
    bool clustered;   // surface pixels as the clustered pass has them (normal.w > 0)
    float4* out_ar;
    double* out_ar64; // 3 per pixel
    double* partial;  // several segments: [channel][segment][height][width]
    int64_t opitch;
    uint32_t* err;
};

// The rays of the packed records, compacted within each step of kStep AVPLs (in AVPL order; counts[s] of
// step s are left).  An AVPL without antiradiance or without a direction adds 0 to every pixel and is
// dropped (half of them); one with a non-finite antiradiance is kept.
__global__ void __launch_bounds__(kStep) disk_rays(const float4* records, int n, float4* rays, int* counts) {
    __shared__ int s_cnt[kStep / 32];
    const int i = blockIdx.x * kStep + threadIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float4 q0, q1, q2, q3;
    bool keep = false, finite = true;
    if (i < n) {
        q0 = records[4 * (size_t)i];
        q1 = records[4 * (size_t)i + 1];
        q2 = records[4 * (size_t)i + 2];
        q3 = records[4 * (size_t)i + 3];
        const float la = fabsf(q3.x) + fabsf(q3.y) + fabsf(q3.z);
        finite = la <= FLT_MAX;
        keep = !(la == 0.0f || (finite && q1.z == 0.0f && q1.w == 0.0f && q2.x == 0.0f));
    }
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) s_cnt[w] = __popc(m);
    __syncthreads();
    static_assert(kStep / 32 <= 32, "one lane per warp's count");
    const int mine = lane < kStep / 32 ? s_cnt[lane] : 0;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const int first = __shfl_sync(0xffffffffu, incl - mine, w);
    if (threadIdx.x == 31) counts[blockIdx.x] = incl;
    if (keep) {
        const size_t d = (size_t)blockIdx.x * kStep + first + __popc(m & ((1u << lane) - 1u));
        rays[2 * d] = make_float4(q0.x, q0.y, q0.z, finite ? 1.0f : -1.0f);
        rays[2 * d + 1] = make_float4(q1.z * q3.w, q1.w * q3.w, q2.x * q3.w, __int_as_float(i));
    }
}

// Whether the ray from r0 along the unit vector r1 can enter the sphere (c, rho); the margin covers the
// rounding of the hit point here and in pair_terms, which both start from a difference of positions (a
// few ulp of the distance).
__device__ __forceinline__ bool ray_near(float4 r0, float4 r1, float cx, float cy, float cz, float rho) {
    const float vx = cx - r0.x, vy = cy - r0.y, vz = cz - r0.z;
    const float s = fmaxf(0.0f, vx * r1.x + vy * r1.y + vz * r1.z);
    const float hx = vx - s * r1.x, hy = vy - s * r1.y, hz = vz - s * r1.z;
    const float reach = rho + 1e-4f * (rho + s + fabsf(vx) + fabsf(vy) + fabsf(vz));
    return !(hx * hx + hy * hy + hz * hz > reach * reach);
}

// A pixel's antiradiance from its FP64 sums; 0 without a surface (material 0).
__device__ __forceinline__ void write_ar(const DiskArgs& a, int x, int y, int mat, const double* S) {
    double ar[3] = {0.0, 0.0, 0.0};
    if (mat > 0) {
        const float4 d = a.mats[mat].diffuse_exp;
        const float kd[3] = {kOneOverPi * d.x, kOneOverPi * d.y, kOneOverPi * d.z};
        for (int c = 0; c < 3; ++c) ar[c] = (double)kd[c] * (double)a.disk_scale * S[c];
    }
    const int64_t o = (int64_t)y * a.opitch + x;
    if (a.out_ar) a.out_ar[o] = make_float4((float)ar[0], (float)ar[1], (float)ar[2], 1.0f);
    if (a.out_ar64)
        for (int c = 0; c < 3; ++c) a.out_ar64[3 * o + c] = ar[c];
}

// PX = 1: 16 x 16 pixel tiles, 8 x 4 pixels per warp; PX = 4: 32 x 32 tiles, 16 x 8 per warp.
template <int PX>
__global__ void __launch_bounds__(kThreads, PX == 1 ? 3 : 2) disk_antiradiance(DiskArgs a) {
    constexpr int kSide = PX == 1 ? 16 : 32, kSub = PX == 1 ? 1 : 2, kIlp = 4 / PX;
    __shared__ float4 s_rec[kWarps][32 * 4];
    __shared__ int s_list[kList];
    __shared__ PixelBounds s_half[2][kWarps];  // (positions only)
    __shared__ int s_cnt[2][kCounts];
    __shared__ PixelBounds s_box[kWarps];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int xb = blockIdx.x * kSide + (w & 1) * 8 * kSub + (lane & 7);
    const int yb = blockIdx.y * kSide + (w >> 1) * 4 * kSub + (lane >> 3);

    Pixel<float> px[PX];
    int mat[PX];  // 0: nothing to gather
    PixelBounds box;
    box.clear();
    bool any = false;
#pragma unroll
    for (int j = 0; j < PX; ++j) {
        const int x = xb + (j % kSub) * 8, y = yb + (j / kSub) * 4;
        float4 gp = make_float4(0, 0, 0, 0), gn = make_float4(0, 0, 0, 0);
        if (x < a.width && y < a.height) {
            gp = a.gpos[(int64_t)y * a.gpitch + x];
            gn = a.gnrm[(int64_t)y * a.gpitch + x];
        }
        mat[j] = (int)gn.w;
        if (mat[j] <= 0 || mat[j] >= a.num_mats) {
            if (a.clustered ? gn.w > 0.0f : mat[j] != 0) set_error(a.err, ARC_DEVERR_BAD_MATERIAL);
            mat[j] = 0;
        }
        const float l = mat[j] ? rsqrtf(gn.x * gn.x + gn.y * gn.y + gn.z * gn.z) : 0.0f;
        px[j].px = gp.x;
        px[j].py = gp.y;
        px[j].pz = gp.z;
        px[j].nx = gn.x * l;
        px[j].ny = gn.y * l;
        px[j].nz = gn.z * l;
        if (mat[j]) {
            any = true;
            box.add(gp.x, gp.y, gp.z, px[j].nx, px[j].ny, px[j].nz, px[j].nx, px[j].ny, px[j].nz);
        }
    }
    float sum[PX][3], comp[PX][3];
#pragma unroll
    for (int j = 0; j < PX; ++j)
#pragma unroll
        for (int c = 0; c < 3; ++c) sum[j][c] = comp[j][c] = 0.0f;

    const bool warp_live = __any_sync(0xffffffffu, any);
    if (__syncthreads_or(any)) {
        box.reduce_warp();
        if (lane == 0) s_box[w] = box;
        __syncthreads();
        PixelBounds tb = s_box[0];
        for (int q = 1; q < kWarps; ++q) tb.merge(s_box[q]);
        // bounding sphere of a box, grown by the disk radius (radius -1: empty).  The half extents are taken
        // from the centre as it is rounded, which far from the origin is off by more than the disk radius.
        auto sphere = [&](const PixelBounds& b) {
            const float cx = 0.5f * (b.pmin[0] + b.pmax[0]), cy = 0.5f * (b.pmin[1] + b.pmax[1]),
                        cz = 0.5f * (b.pmin[2] + b.pmax[2]);
            const float ex = fmaxf(b.pmax[0] - cx, cx - b.pmin[0]), ey = fmaxf(b.pmax[1] - cy, cy - b.pmin[1]),
                        ez = fmaxf(b.pmax[2] - cz, cz - b.pmin[2]);
            return make_float4(cx, cy, cz,
                               b.pmin[0] <= b.pmax[0] ? 1.0001f * sqrtf(ex * ex + ey * ey + ez * ez) + a.radius : -1.0f);
        };
        // the warp's pixels on one side of the middle of a box's longest axis
        auto half = [&](const PixelBounds& whole, int side) {
            const float e[3] = {whole.pmax[0] - whole.pmin[0], whole.pmax[1] - whole.pmin[1],
                                whole.pmax[2] - whole.pmin[2]};
            const int axis = e[0] >= e[1] && e[0] >= e[2] ? 0 : e[1] >= e[2] ? 1 : 2;
            const float mid = 0.5f * (axis == 0   ? whole.pmin[0] + whole.pmax[0]
                                      : axis == 1 ? whole.pmin[1] + whole.pmax[1]
                                                  : whole.pmin[2] + whole.pmax[2]);
            PixelBounds b;
            b.clear();
#pragma unroll
            for (int j = 0; j < PX; ++j) {
                const float v = axis == 0 ? px[j].px : axis == 1 ? px[j].py : px[j].pz;
                if (mat[j] && !(v > mid) == (side == 0))  // (a position that is not a number: side 0)
                    b.add(px[j].px, px[j].py, px[j].pz, 0, 0, 0, 0, 0, 0);
            }
            b.reduce_warp_positions();
            return b;
        };
        const float4 mine0 = sphere(half(box, 0)), mine1 = sphere(half(box, 1));
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const PixelBounds h = half(tb, side);
            if (lane == 0) s_half[side][w] = h;
        }
        __syncthreads();
        float4 tile0, tile1;
        {
            PixelBounds h0 = s_half[0][0], h1 = s_half[1][0];
            for (int q = 1; q < kWarps; ++q) {
                h0.merge(s_half[0][q]);
                h1.merge(s_half[1][q]);
            }
            tile0 = sphere(h0);
            tile1 = sphere(h1);
        }
        auto near_any = [&](float4 ray0, float4 ray1, float4 b0, float4 b1) {
            return ray0.w < 0.0f || (b0.w >= 0.0f && ray_near(ray0, ray1, b0.x, b0.y, b0.z, b0.w)) ||
                   (b1.w >= 0.0f && ray_near(ray0, ray1, b1.x, b1.y, b1.z, b1.w));
        };
        float4* rec = s_rec[w];
        const int steps = (a.n + kStep - 1) / kStep;
        const int first = (int)((int64_t)steps * blockIdx.z / gridDim.z),
                  last = (int)((int64_t)steps * (blockIdx.z + 1) / gridDim.z);
        // rays of one step ahead
        float4 r0[kPerThread], r1[kPerThread];
        int rays = 0;
        auto load_step = [&](int step) {
            rays = step < last ? a.counts[step] : 0;
#pragma unroll
            for (int u = 0; u < kPerThread; ++u) {
                const int i = u * kThreads + tid;
                if (i < rays) {
                    const float4* r = a.rays + 2 * ((size_t)step * kStep + i);
                    r0[u] = r[0];
                    r1[u] = r[1];
                }
            }
        };
        load_step(first);
        int count = 0;  // survivors in the list
        for (int step = first; step < last; ++step) {
            unsigned m[kPerThread];
            int* cnt = s_cnt[step & 1];
#pragma unroll
            for (int u = 0; u < kPerThread; ++u) {
                m[u] = __ballot_sync(0xffffffffu,
                                     u * kThreads + tid < rays && near_any(r0[u], r1[u], tile0, tile1));
                if (lane == 0) cnt[u * kWarps + w] = __popc(m[u]);
            }
            load_step(step + 1);
            __syncthreads();  // the counts; and the list's readers are done
            const int mine = lane < kCounts ? cnt[lane] : 0;
            int incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            const int excl = count + incl - mine;
            count += __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
            for (int u = 0; u < kPerThread; ++u) {
                const int at = __shfl_sync(0xffffffffu, excl, u * kWarps + w) + __popc(m[u] & ((1u << lane) - 1u));
                if (m[u] >> lane & 1u) s_list[at] = step * kStep + u * kThreads + tid;
            }
            if (count + kStep <= kList && step + 1 < last) continue;  // room for another step
            __syncthreads();
            const int listed = count;
            count = 0;
            if (!warp_live) continue;
            for (int k = 0; k < listed; k += 32) {
                float4 q0, q1, q2, q3;
                bool keep = false;
                float4 ray0, ray1;
                if (k + lane < listed) {
                    const float4* r = a.rays + 2 * (size_t)s_list[k + lane];
                    ray0 = r[0];
                    ray1 = r[1];
                    keep = near_any(ray0, ray1, mine0, mine1);
                }
                if (keep) {
                    const float4* q = a.records + 4 * (size_t)__float_as_int(ray1.w);
                    q0 = q[0];
                    q1 = q[1];
                    q2 = q[2];
                    q3 = q[3];
                    {
                        const float p[3] = {q0.x, q0.y, q0.z}, n[3] = {q0.w, q1.x, q1.y};
                        float recv[3], back[3];
#pragma unroll
                        for (int d = 0; d < 3; ++d) {
                            const float lo = p[d] - box.pmax[d], hi = p[d] - box.pmin[d];
                            recv[d] = fmaxf(fmaxf(box.nmin[d] * lo, box.nmin[d] * hi),
                                            fmaxf(box.nmax[d] * lo, box.nmax[d] * hi));
                            back[d] = fmaxf(n[d] * lo, n[d] * hi);
                        }
                        // accepted pairs have n.d > 0 (t = -n.d / w.n > 0 with w.n < 0) and n_a.d > 0
                        keep = !(dot_never_positive(recv[0], recv[1], recv[2]) ||
                                 dot_never_positive(back[0], back[1], back[2]));
                    }
                    keep = keep || !(fabsf(q3.x) + fabsf(q3.y) + fabsf(q3.z) <= FLT_MAX);
                }
                const unsigned mk = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    float4* d = rec + 4 * __popc(mk & ((1u << lane) - 1u));
                    d[0] = q0;
                    d[1] = q1;
                    d[2] = q2;
                    d[3] = q3;
                }
                __syncwarp();
                const int kept = __popc(mk);
                // kIlp records at a time: their tests are independent, the sums then take them in order
                for (int i = 0; i < kept; i += kIlp) {
                    float hit[kIlp][PX];
#pragma unroll
                    for (int u = 0; u < kIlp; ++u) {
                        const float4* r = rec + 4 * min(i + u, kept - 1);
                        const float4 r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3];
#pragma unroll
                        for (int j = 0; j < PX; ++j) {
                            float g;
                            pair_terms<ARC_AR_DISK, float>(r0, r1, r2, r3, px[j], a.pc, g, hit[u][j]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < kIlp; ++u) {
                        if (i + u >= kept) break;
                        const float4 r3 = rec[4 * (i + u) + 3];
#pragma unroll
                        for (int j = 0; j < PX; ++j) {
                            // (0 times a non-finite antiradiance is added too, except by the clustered pass)
                            const float ga = hit[u][j], x = r3.x * ga, y = r3.y * ga, z = r3.z * ga;
                            if (ga != 0.0f || (!a.clustered && !(x == 0.0f && y == 0.0f && z == 0.0f))) {
                                kahan_add(sum[j][0], comp[j][0], x);
                                kahan_add(sum[j][1], comp[j][1], y);
                                kahan_add(sum[j][2], comp[j][2], z);
                            }
                        }
                    }
                }
                __syncwarp();
            }
        }
    }

#pragma unroll
    for (int j = 0; j < PX; ++j) {
        const int x = xb + (j % kSub) * 8, y = yb + (j / kSub) * 4;
        if (x >= a.width || y >= a.height) continue;
        double S[3];
        for (int c = 0; c < 3; ++c) S[c] = (double)sum[j][c] - (double)comp[j][c];
        if (gridDim.z > 1) {
            double* d = a.partial + ((int64_t)blockIdx.z * a.height + y) * a.width + x;
            const int64_t plane = (int64_t)gridDim.z * a.height * a.width;
            if (mat[j] > 0)  // (other pixels are written by disk_combine alone)
                for (int c = 0; c < 3; ++c) d[c * plane] = S[c];
        } else {
            write_ar(a, x, y, mat[j], S);
        }
    }
}

// The segments' sums of every pixel added in segment order, and the outputs.
__global__ void __launch_bounds__(kThreads) disk_combine(DiskArgs a, int segments) {
    const int x = blockIdx.x * 32 + threadIdx.x % 32, y = blockIdx.y * (kThreads / 32) + threadIdx.x / 32;
    if (x >= a.width || y >= a.height) return;
    int m = (int)a.gnrm[(int64_t)y * a.gpitch + x].w;
    if (m < 0 || m >= a.num_mats) m = 0;
    double S[3] = {0.0, 0.0, 0.0};
    if (m > 0) {
        const int64_t image = (int64_t)a.height * a.width;
        const double* d = a.partial + (int64_t)y * a.width + x;
        for (int s = 0; s < segments; ++s)
            for (int c = 0; c < 3; ++c) S[c] += d[(c * segments + s) * image];
    }
    write_ar(a, x, y, m, S);
}

}  // namespace

arc_status launch_disk_antiradiance(arc_context* ctx, const ArcAvplsGpuParam* avpls, const float4* records,
                                    const ArcGBufferView* gb, const ArcGatherParams* gp, bool clustered, float* out_ar,
                                    double* out_ar64, int64_t opitch) {
    if (!records) ARC_TRY(launch_pack_records(ctx, avpls, &records));
    DiskArgs a{};
    a.records = records;
    a.n = avpls->numAvpls;
    float4* rays = nullptr;
    const int steps = (a.n + kStep - 1) / kStep;
    int* counts = nullptr;
    ARC_TRY(ctx->arena.get("disk_rays", ((size_t)steps * kStep + 1) * 2 * sizeof(float4),
                           reinterpret_cast<void**>(&rays)));
    ARC_TRY(ctx->arena.get("disk_ray_counts", (size_t)(steps + 1) * sizeof(int), reinterpret_cast<void**>(&counts)));
    a.rays = rays;
    a.counts = counts;
    a.gpos = reinterpret_cast<const float4*>(gb->position);
    a.gnrm = reinterpret_cast<const float4*>(gb->normal);
    a.gpitch = gb->pitch;
    a.width = gb->width;
    a.height = gb->height;
    a.mats = ctx->d_materials;
    a.num_mats = ctx->num_materials;
    a.pc.eps = 0.001f;
    a.pc.inv_clamp2 = gp->dist_clamp > 0.0f ? 1.0f / (gp->dist_clamp * gp->dist_clamp) : INFINITY;
    a.pc.disk_r2 = gp->disk_radius * gp->disk_radius;
    a.radius = gp->disk_radius;
    a.disk_scale = gp->disk_radius > 0.0f ? 1.0f / (kPi * gp->disk_radius * gp->disk_radius) : 0.0f;
    a.clustered = clustered;
    a.out_ar = reinterpret_cast<float4*>(out_ar);
    a.out_ar64 = out_ar64;
    a.opitch = opitch;
    a.err = ctx->d_error;
    cudaStream_t st = ctx->stream;
    stage_begin(ctx, "disk_antiradiance");
    if (a.n > 0) disk_rays<<<steps, kStep, 0, st>>>(records, a.n, rays, counts);
    dim3 grid((a.width + 31) / 32, (a.height + 31) / 32);
    const bool big = (int64_t)grid.x * grid.y >= kBigTilesPerSm * ctx->sm_count;
    if (!big) grid = dim3((a.width + 15) / 16, (a.height + 15) / 16);
    const int64_t blocks = (int64_t)grid.x * grid.y, image = (int64_t)a.width * a.height;
    grid.z = (unsigned)std::max<int64_t>(
        1, std::min({(kBlocksPerSm * ctx->sm_count + blocks - 1) / blocks, (int64_t)steps,
                     kPartialBytes / (image * 3 * (int64_t)sizeof(double))}));
    if (grid.z > 1)
        ARC_TRY(ctx->arena.get("disk_partial", (size_t)(image * 3 * grid.z) * sizeof(double),
                               reinterpret_cast<void**>(&a.partial)));
    if (big)
        disk_antiradiance<4><<<grid, kThreads, 0, st>>>(a);
    else
        disk_antiradiance<1><<<grid, kThreads, 0, st>>>(a);
    if (grid.z > 1)
        disk_combine<<<dim3((a.width + 31) / 32, (a.height + 7) / 8), kThreads, 0, st>>>(a, (int)grid.z);
    stage_end(ctx, (a.n > 0 ? 2 : 1) + (grid.z > 1));
    ARC_TRY_CUDA(cudaGetLastError());
    return ARC_OK;
}

}  // namespace arc
