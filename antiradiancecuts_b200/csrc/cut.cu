// Cut gathers over the LBVH.
//
// ARC_CUT_SOLID_ANGLE: the lightcut of kernel_bvh (cudaGather.cu:316-444), one thread per pixel, a
//   warp sharing the walk:
//   DFS from the root; a leaf adds its exact radiance; an inner node is skipped when both of its
//   box corners lie behind the receiver (cudaGather.cu:405-408), used whole when the solid angle
//   2 pi (1 - d / sqrt(r^2 + d^2)) of its bounding sphere seen from the representative is below
//   the threshold, and refined otherwise.  The stack holds 64 entries (the reference's 32
//   overflows for large trees); overflow paints the reference's magenta pixel and sets
//   ARC_DEVERR_STACK_OVERFLOW.  Antiradiance comes from the brute-force pass, as in the
//   reference's non-clustered run() path.
// ARC_CUT_ERROR_BOUND: one cut per 8x8 pixel tile, chosen by one block that walks the tree
//   cooperatively (128 nodes per step, ballot/popc compaction of accepted nodes and of the
//   children to push).  A node is refined while an upper bound of its contribution to any pixel
//   of the tile exceeds eps times the tile's coarse radiance estimate.  Every pixel of the tile
//   then evaluates the same node list, so the evaluation is fully coherent.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>

#include "arc_internal.h"
#include "cut_bounds.cuh"
#include "device_common.cuh"
#include "pair_cull.cuh"
#include "pair_math.cuh"

namespace arc {

arc_status launch_antiradiance_only(arc_context* ctx, const GatherLaunch& g, double* ar64);
arc_status launch_cut_select_learned(arc_context* ctx, const arc_lbvh* bvh, const ArcGatherParams* gp,
                                     const ArcCutParams* cp, const float4* tiles_info, const float4* extra,
                                     int tiles_x, int tiles_y, const CutPool& pool);

namespace {

constexpr int kTile = 8;
constexpr int kSolidStack = 64;
constexpr int kSolidThreads = 64;
constexpr int kChunkSize = 1024;  // cut entries per pool chunk
constexpr int kSetupWarps = 4;
constexpr int kSelThreads = 128;
constexpr int kSelStack = 8192;  // nodes waiting per tile
constexpr int kSelBlocksPerSm = 6;
constexpr int kCoarseDepth = 5;

struct MatSmem {
    MaterialRecord m[ARC_MAX_MATERIALS];
};

// ---------------------------------------------------------------------------------------
// Solid-angle lightcut (reference semantics)
// ---------------------------------------------------------------------------------------
struct SolidArgs {
    const float4* gpos;
    const float4* gnrm;
    int64_t gpitch;
    int width, height;
    const MaterialRecord* mats;
    int num_mats;
    float3 cam;
    int n;
    const float4* bounds;
    const float4* records;
    ArcAvplBvhNodeDataParam nd;
    float thresh;
    float cos2, cos2_margin;  // (1 - thresh / 2 pi)^2; distance from it at which the approximate test holds
    float clamp2;
    double* rad64;
    float4* out_rad;
    int64_t opitch;
    int dbg_x, dbg_y;
    int32_t* used;
    uint32_t* err;
};

__device__ __forceinline__ float3 brdf_f(float3 w_i, float3 w_o, float3 n, const MaterialRecord& m) {
    float3 d = f3(kOneOverPi * m.diffuse_exp.x, kOneOverPi * m.diffuse_exp.y, kOneOverPi * m.diffuse_exp.z);
    if (m.specular_flag.w != 0.0f) {
        const float3 I = -1.0f * w_i;
        const float3 r = I - (2.0f * dot(n, I)) * n;
        const float c = fmaxf(0.0f, dot(r, w_o));
        const float e = m.diffuse_exp.w;
        const float f = 0.5f * kOneOverPi * (e + 2.0f) * powf(c, e);
        d = d + f * f3(m.specular_flag.x, m.specular_flag.y, m.specular_flag.z);
    }
    return d;
}

__device__ __forceinline__ float3 norm3(float3 v) { return rsqrtf(dot(v, v)) * v; }

// getRadiance (cudaGather.cu:78-95) for node-data element idx
__device__ __forceinline__ float3 node_radiance(const SolidArgs& a, const MatSmem& sm, float3 p, float3 n, int mat,
                                                float3 w_o, int idx) {
    const float3 pa = ld3(a.nd.position, idx), na = ld3(a.nd.normal, idx), wa = ld3(a.nd.incDirection, idx);
    const float3 L = ld3(a.nd.incRadiance, idx);
    int ma = a.nd.materialIndex[idx];
    if (ma < 0 || ma >= a.num_mats) ma = 0;
    const float3 v = pa - p;
    const float l2 = dot(v, v);
    if (!(l2 > 0.0f)) return f3(0, 0, 0);
    const float3 w = rsqrtf(l2) * v;
    float3 fl = f3(1, 1, 1);
    if (dot(wa, wa) != 0.0f) fl = brdf_f(-1.0f * wa, -1.0f * w, norm3(na), sm.m[ma]);
    const float3 fr = brdf_f(w, w_o, n, sm.m[mat]);
    const float c1 = fminf(fmaxf(dot(n, w), 0.0f), 1.0f);
    const float c2 = fminf(fmaxf(-dot(norm3(na), w), 0.0f), 1.0f);
    const float g = c1 * c2 / fmaxf(l2, a.clamp2);
    return f3(L.x * fl.x * fr.x * g, L.y * fl.y * fr.y * g, L.z * fl.z * fr.z * g);
}

__device__ __forceinline__ float rcp_approx(float x) {  // 1 ulp
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The same without specular materials, leaving out the receiver's diffuse / pi (a constant of the pixel):
// L f_l max(n.d, 0) max(-n_a.d, 0) / (d^2 max(d^2, clamp^2)), d = p_a - p.  The 1/|d| factors of the two
// cosines are one reciprocal of d^2.
__device__ __forceinline__ float3 node_radiance_diffuse(const SolidArgs& a, const MatSmem& sm, float3 p, float3 n,
                                                        int idx) {
    const float4 q0 = a.records[4 * (size_t)idx], q1 = a.records[4 * (size_t)idx + 1];  // p_a, n_a
    const float3 wa = ld3(a.nd.incDirection, idx), L = ld3(a.nd.incRadiance, idx);
    int ma = a.nd.materialIndex[idx];
    if (ma < 0 || ma >= a.num_mats) ma = 0;
    const float3 v = f3(q0.x, q0.y, q0.z) - p, na = f3(q0.w, q1.x, q1.y);
    const float l2 = dot(v, v);
    if (!(l2 > 0.0f)) return f3(0, 0, 0);
    float3 f = L;
    if (dot(wa, wa) != 0.0f) {
        const float4 d = sm.m[ma].diffuse_exp;
        f = f3(L.x * (kOneOverPi * d.x), L.y * (kOneOverPi * d.y), L.z * (kOneOverPi * d.z));
    }
    const float c1 = fmaxf(dot(n, v) * rcp_approx(l2), 0.0f);
    const float c2 = fmaxf(-dot(na, v) * rsqrtf(dot(na, na)) * rcp_approx(fmaxf(l2, a.clamp2)), 0.0f);
    return (c1 * c2) * f;
}

// One warp per 8 x 4 pixels walks the tree once for all of them: an entry of its stack is a node and the
// mask of the pixels that visit it.  Each pixel visits the nodes of its own walk in its own order (the
// sums are the same), but a node's data are loaded once per warp from one address instead of by 32 lanes
// from as many, and neighbouring pixels' walks coincide almost everywhere.
template <bool SPECULAR>
__global__ void __launch_bounds__(kSolidThreads) cut_solid_angle_kernel(SolidArgs a) {
    __shared__ MatSmem sm;
    __shared__ int s_node[kSolidThreads / 32][kSolidStack];
    __shared__ unsigned s_mask[kSolidThreads / 32][kSolidStack];
    for (int i = threadIdx.x; i < a.num_mats; i += blockDim.x) sm.m[i] = a.mats[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // a block's two warps: 8 x 8 pixels (small blocks, because neighbouring tiles' walks differ in length)
    const int x = blockIdx.x * 8 + (lane & 7);
    const int y = blockIdx.y * 8 + w * 4 + (lane >> 3);
    const bool inside = x < a.width && y < a.height;
    float4 gp = make_float4(0, 0, 0, 0), gn = make_float4(0, 0, 0, 0);
    if (inside) {
        gp = a.gpos[(int64_t)y * a.gpitch + x];
        gn = a.gnrm[(int64_t)y * a.gpitch + x];
    }
    const int mat = (int)gn.w;
    float s[3] = {0, 0, 0}, c[3] = {0, 0, 0};
    const bool surface = mat > 0 && mat < a.num_mats;
    if (mat != 0 && !surface) set_error(a.err, ARC_DEVERR_BAD_MATERIAL);
    const float3 p = f3(gp.x, gp.y, gp.z);
    const float3 nraw = f3(gn.x, gn.y, gn.z);
    const float3 n = norm3(nraw);
    const float3 w_o = norm3(a.cam - p);
    const bool dbg = a.used && x == a.dbg_x && y == a.dbg_y;
    const float two_pi = rn_mul(2.0f, kPi);
    int* nodes = s_node[w];
    unsigned* masks = s_mask[w];
    const unsigned start = __ballot_sync(0xffffffffu, surface);
    unsigned failed = 0;  // pixels whose walk was given up
    int sp = 0;
    if (start) {
        if (lane == 0) {
            nodes[0] = -1;
            masks[0] = start;
        }
        sp = 1;
    }
    __syncwarp();
    // every node is visited at most once in a valid tree: 2n - 1 pops bound the walk
    int budget = 2 * a.n;
    while (sp > 0) {
        --sp;
        const int node = nodes[sp];
        const unsigned mask = masks[sp] & ~failed;
        __syncwarp();  // read by every lane before the children overwrite the entry
        if (--budget < 0 || node >= a.n || node < -(a.n - 1)) {
            failed |= mask;
            if (lane == 0) set_error(a.err, ARC_DEVERR_BAD_NODE);
            if (budget < 0) break;
            continue;
        }
        bool use = mask >> lane & 1u;
        int idx = node;
        if (node < 0) {
            const int k = -(node + 1);
            idx = a.n + k;
            const float4 b0 = a.bounds[4 * (size_t)k], b1 = a.bounds[4 * (size_t)k + 1];
            const float4 q0 = a.records[4 * (size_t)idx];  // the representative's position
            // visibility of the box corners (cudaGather.cu:405-408); the sign of
            // n.normalize(v) is the sign of n.v
            use = use &&
                  (rn_dot(nraw.x, nraw.y, nraw.z, rn_sub(b1.x, p.x), rn_sub(b1.y, p.y), rn_sub(b1.z, p.z)) > 0.0f ||
                   rn_dot(nraw.x, nraw.y, nraw.z, rn_sub(b0.x, p.x), rn_sub(b0.y, p.y), rn_sub(b0.z, p.z)) > 0.0f);
            const float ex = rn_sub(b1.x, b0.x), ey = rn_sub(b1.y, b0.y), ez = rn_sub(b1.z, b0.z);
            const float vx = rn_sub(q0.x, p.x), vy = rn_sub(q0.y, p.y), vz = rn_sub(q0.z, p.z);
            const float d2 = rn_dot(vx, vy, vz, vx, vy, vz), e2 = rn_dot(ex, ey, ez, ex, ey, ez);
            // solid angle < threshold <=> d^2 / (d^2 + r^2) > cos^2, without the square roots and the
            // division unless the two sides are closer than the rounding of the test as written
            const float h2 = fmaf(0.25f, e2, d2), gap = fmaf(-a.cos2, h2, d2);
            bool below = gap > 0.0f;
            if (use && !(fabsf(gap) > a.cos2_margin * h2)) {
                const float radius = rn_mul(0.5f, rn_sqrt(e2)), dist = rn_sqrt(d2);
                below = rn_mul(two_pi, rn_sub(1.0f, rn_div(dist, rn_sqrt(rn_add(rn_mul(radius, radius),
                                                                                rn_mul(dist, dist)))))) < a.thresh;
            }
            const bool refine = use && !below;
            use = use && !refine;
            const unsigned down = __ballot_sync(0xffffffffu, refine);
            if (down) {
                if (sp + 2 > kSolidStack) {
                    failed |= down;
                    if (lane == 0) set_error(a.err, ARC_DEVERR_STACK_OVERFLOW);
                } else {
                    if (lane < 2) {
                        nodes[sp + lane] = __float_as_int(lane == 0 ? b0.w : b1.w);
                        masks[sp + lane] = down;
                    }
                    sp += 2;
                }
            }
        }
        if (use) {
            const float3 t = SPECULAR ? node_radiance(a, sm, p, n, mat, w_o, idx)
                                      : node_radiance_diffuse(a, sm, p, n, idx);
            kahan_add(s[0], c[0], t.x);
            kahan_add(s[1], c[1], t.y);
            kahan_add(s[2], c[2], t.z);
            if (dbg) a.used[idx] = 1;
        }
        __syncwarp();  // the pushes
    }
    if (!inside) return;
    const int64_t o = (int64_t)y * a.opitch + x;
    double r[3];
    for (int q = 0; q < 3; ++q) r[q] = (double)s[q] - (double)c[q];
    if (!SPECULAR) {
        const float4 d = sm.m[surface ? mat : 0].diffuse_exp;
        const float kd[3] = {kOneOverPi * d.x, kOneOverPi * d.y, kOneOverPi * d.z};
        for (int q = 0; q < 3; ++q) r[q] = surface ? r[q] * (double)kd[q] : 0.0;
    }
    // (a walk whose budget ran out was its warp's: what its other pixels still had to visit is not known)
    if ((failed >> lane & 1u) || (surface && budget < 0)) {
        r[0] = 100000.0;
        r[1] = 0.0;
        r[2] = 100000.0;
    }
    a.rad64[3 * o + 0] = r[0];
    a.rad64[3 * o + 1] = r[1];
    a.rad64[3 * o + 2] = r[2];
    if (a.out_rad) a.out_rad[o] = make_float4((float)r[0], (float)r[1], (float)r[2], 1.0f);
}

// ---------------------------------------------------------------------------------------
// Tile set-up: bounds of the tile, receiver normal cone, max receiver albedo, coarse estimate
// ---------------------------------------------------------------------------------------
struct TileArgs {
    const float4* gpos;
    const float4* gnrm;
    int64_t gpitch;
    int width, height;
    const MaterialRecord* mats;
    int num_mats;
    int n;
    const float4* bounds;
    const float4* records;
    float eps_bound;
    float clamp2;
    int tiles_x, tiles_y;
    float4* info;  // [tiles][4]
    // expected cut size of the error-bound selection per tile (optional), from:
    int* estimate;
    const float4* extra;  // NodeExtra per inner node
    BoundParams bp;
    uint32_t* err;
};

__device__ __forceinline__ float coarse_g(float px, float py, float pz, float nx, float ny, float nz, const float4 q0,
                                          const float4 q1, float clamp2) {
    const float dx = rn_sub(q0.x, px), dy = rn_sub(q0.y, py), dz = rn_sub(q0.z, pz);
    const float l2 = rn_dot(dx, dy, dz, dx, dy, dz);
    if (!(l2 > 0.0f)) return 0.0f;
    const float r = rn_div(1.0f, rn_sqrt(l2));
    const float c1 = fmaxf(0.0f, rn_mul(rn_dot(nx, ny, nz, dx, dy, dz), r));
    const float c2 = fmaxf(0.0f, rn_mul(-rn_dot(q0.w, q1.x, q1.y, dx, dy, dz), r));
    return rn_div(rn_mul(c1, c2), fmaxf(l2, clamp2));
}

__global__ void __launch_bounds__(32 * kSetupWarps) cut_tile_setup(TileArgs a) {
    __shared__ float sp[kSetupWarps][64][7];  // p.xyz, n.xyz, valid
    __shared__ float skd[kSetupWarps][64][3];
    __shared__ float sest[kSetupWarps][64];
    __shared__ int scoarse[kSetupWarps][1 << kCoarseDepth];
    __shared__ int sncoarse[kSetupWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x * kSetupWarps + warp;
    if (tile >= a.tiles_x * a.tiles_y) return;
    const int tx0 = (tile % a.tiles_x) * kTile, ty0 = (tile / a.tiles_x) * kTile;
    float tmin[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, tmax[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    float kdl = 0.0f;
    int nvalid = 0;
    for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h;
        const int x = tx0 + i % kTile, y = ty0 + i / kTile;
        float4 gp = make_float4(0, 0, 0, 0), gn = make_float4(0, 0, 0, 0);
        bool v = x < a.width && y < a.height;
        if (v) {
            gp = a.gpos[(int64_t)y * a.gpitch + x];
            gn = a.gnrm[(int64_t)y * a.gpitch + x];
            const int m = (int)gn.w;
            v = m > 0 && m < a.num_mats;
            if (!v && m != 0) set_error(a.err, ARC_DEVERR_BAD_MATERIAL);  // gathers 0, as brute force does
            if (v) {
                const float4 d = a.mats[m].diffuse_exp;
                skd[warp][i][0] = rn_mul(kOneOverPi, d.x);
                skd[warp][i][1] = rn_mul(kOneOverPi, d.y);
                skd[warp][i][2] = rn_mul(kOneOverPi, d.z);
                kdl = fmaxf(kdl, lum3(skd[warp][i][0], skd[warp][i][1], skd[warp][i][2]));
                tmin[0] = fminf(tmin[0], gp.x); tmin[1] = fminf(tmin[1], gp.y); tmin[2] = fminf(tmin[2], gp.z);
                tmax[0] = fmaxf(tmax[0], gp.x); tmax[1] = fmaxf(tmax[1], gp.y); tmax[2] = fmaxf(tmax[2], gp.z);
                nvalid += 1;
            }
        }
        sp[warp][i][0] = gp.x; sp[warp][i][1] = gp.y; sp[warp][i][2] = gp.z;
        sp[warp][i][3] = gn.x; sp[warp][i][4] = gn.y; sp[warp][i][5] = gn.z;
        sp[warp][i][6] = v ? 1.0f : 0.0f;
    }
    for (int o = 16; o > 0; o >>= 1) {
        for (int k = 0; k < 3; ++k) {
            tmin[k] = fminf(tmin[k], __shfl_xor_sync(0xffffffffu, tmin[k], o));
            tmax[k] = fmaxf(tmax[k], __shfl_xor_sync(0xffffffffu, tmax[k], o));
        }
        kdl = fmaxf(kdl, __shfl_xor_sync(0xffffffffu, kdl, o));
        nvalid += __shfl_xor_sync(0xffffffffu, nvalid, o);
    }
    // coarse cut: the nodes at depth kCoarseDepth (or leaves above it), left-first DFS order
    if (lane == 0) {
        int st[2 * kCoarseDepth + 2][2];
        int top = 0, cnt = 0;
        st[top][0] = a.n;  // root inner node 0 in node-record index space
        st[top][1] = 0;
        ++top;
        while (top > 0) {
            --top;
            const int node = st[top][0], depth = st[top][1];
            if (node < a.n || depth == kCoarseDepth) {
                scoarse[warp][cnt++] = node;
                continue;
            }
            const int k = node - a.n;
            const float4 b0 = a.bounds[4 * (size_t)k], b1 = a.bounds[4 * (size_t)k + 1];
            const int lc = __float_as_int(b0.w), rc = __float_as_int(b1.w);
            st[top][0] = rc >= 0 ? rc : a.n - (rc + 1);
            st[top][1] = depth + 1;
            ++top;
            st[top][0] = lc >= 0 ? lc : a.n - (lc + 1);
            st[top][1] = depth + 1;
            ++top;
        }
        sncoarse[warp] = cnt;
    }
    __syncwarp();
    const int ncoarse = sncoarse[warp];
    for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h;
        float est = 0.0f;
        if (sp[warp][i][6] != 0.0f) {
            for (int j = 0; j < ncoarse; ++j) {
                const int node = scoarse[warp][j];
                const float4 q0 = a.records[4 * (size_t)node], q1 = a.records[4 * (size_t)node + 1];
                const float4 q2 = a.records[4 * (size_t)node + 2];
                const float g = coarse_g(sp[warp][i][0], sp[warp][i][1], sp[warp][i][2], sp[warp][i][3], sp[warp][i][4],
                                         sp[warp][i][5], q0, q1, a.clamp2);
                const float l = lum3(rn_mul(skd[warp][i][0], q2.y), rn_mul(skd[warp][i][1], q2.z),
                                     rn_mul(skd[warp][i][2], q2.w));
                est = rn_add(est, rn_mul(l, g));
            }
        }
        sest[warp][i] = est;
    }
    __syncwarp();
    TileInfo ti;
    if (lane == 0) {
        float sum = 0.0f;
        float4 cone = make_float4(0, 0, 0, -2.0f);  // -2: empty
        for (int i = 0; i < 64; ++i) {
            if (sp[warp][i][6] == 0.0f) continue;
            sum = rn_add(sum, sest[warp][i]);
            const float4 ci = make_float4(sp[warp][i][3], sp[warp][i][4], sp[warp][i][5], 1.0f);
            if (cone.w < -1.5f) {
                cone = ci;
            } else {
                // cone union (same as the bottom-up build)
                if (cone.w <= -1.0f) continue;
                const float sx = rn_add(cone.x, ci.x), sy = rn_add(cone.y, ci.y), sz = rn_add(cone.z, ci.z);
                const float l2 = rn_dot(sx, sy, sz, sx, sy, sz);
                if (!(l2 > 1e-12f)) {
                    cone = make_float4(0, 0, 0, -1.0f);
                    continue;
                }
                const float inv = rn_div(1.0f, rn_sqrt(l2));
                const float ax = rn_mul(sx, inv), ay = rn_mul(sy, inv), az = rn_mul(sz, inv);
                float res = 1.0f;
                const float4 cc[2] = {cone, ci};
                for (int q = 0; q < 2; ++q) {
                    float d = rn_dot(ax, ay, az, cc[q].x, cc[q].y, cc[q].z);
                    d = fminf(fmaxf(d, -1.0f), 1.0f);
                    const float sd = rn_sqrt_z(fmaxf(0.0f, rn_sub(1.0f, rn_mul(d, d))));
                    const float si = rn_sqrt_z(fmaxf(0.0f, rn_sub(1.0f, rn_mul(cc[q].w, cc[q].w))));
                    const float v = cc[q].w < -d ? -1.0f : rn_sub(rn_mul(d, cc[q].w), rn_mul(sd, si));
                    res = fminf(res, v);
                }
                cone = make_float4(ax, ay, az, res);
            }
        }
        if (cone.w < -1.5f) cone = make_float4(0, 0, 0, -1.0f);
        const float mean = nvalid > 0 ? rn_div(sum, (float)nvalid) : 0.0f;
        float4* info = a.info + 4 * (size_t)tile;
        info[0] = make_float4(tmin[0], tmin[1], tmin[2], kdl);
        info[1] = make_float4(tmax[0], tmax[1], tmax[2], rn_mul(a.eps_bound, mean));
        info[2] = cone;
        info[3] = make_float4(__int_as_float(nvalid), mean,
                              half_diagonal(rn_sub(tmax[0], tmin[0]), rn_sub(tmax[1], tmin[1]), rn_sub(tmax[2], tmin[2])),
                              cone_sine(cone.w));
        ti.ncone = cone;
        ti.tau = rn_mul(a.eps_bound, mean);
        ti.sn = cone_sine(cone.w);
    }
    if (a.estimate) {
        // A node whose bound is M contributes about M / tau nodes to the cut (its parts' bounds add up
        // to M and each stays below tau), at most its leaves; one coarse node per lane.
        ti.ncone.x = __shfl_sync(0xffffffffu, ti.ncone.x, 0);
        ti.ncone.y = __shfl_sync(0xffffffffu, ti.ncone.y, 0);
        ti.ncone.z = __shfl_sync(0xffffffffu, ti.ncone.z, 0);
        ti.ncone.w = __shfl_sync(0xffffffffu, ti.ncone.w, 0);
        ti.tau = __shfl_sync(0xffffffffu, ti.tau, 0);
        ti.sn = __shfl_sync(0xffffffffu, ti.sn, 0);
        for (int k = 0; k < 3; ++k) {
            ti.tmin[k] = tmin[k];
            ti.tmax[k] = tmax[k];
        }
        ti.kdl = kdl;
        ti.valid = nvalid;
        ti.rt = half_diagonal(tmax[0] - tmin[0], tmax[1] - tmin[1], tmax[2] - tmin[2]);
        float e = 0.0f;
        if (nvalid > 0 && lane < ncoarse) {
            const int node = scoarse[warp][lane];
            e = 1.0f;
            if (node >= a.n) {
                const int k = node - a.n;
                const float4* b = a.bounds + 4 * (size_t)k;
                const float m = node_bound_fast(ti, b[0], b[1], b[2], b[3], load_node_extra(a.extra, k), a.bp).m;
                e = fminf(a.records[4 * (size_t)node + 3].w, fmaxf(1.0f, m / ti.tau));
            }
        }
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
        if (lane == 0) a.estimate[tile] = (int)fminf(e, 1e9f);
    }
}

// NodeExtra of every inner node k (bounds at 4 k, record at 4 (n + k)), for node_geom / node_bound
__global__ void cut_node_extra(int n, const float4* bounds, const float4* records, float4* ext) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n - 1) return;
    const float4 b0 = bounds[4 * (size_t)k], b1 = bounds[4 * (size_t)k + 1];
    const float4 nc = bounds[4 * (size_t)k + 2], wc = bounds[4 * (size_t)k + 3];
    const float4 q2 = records[4 * ((size_t)n + k) + 2], q3 = records[4 * ((size_t)n + k) + 3];
    const float rn = half_diagonal(rn_sub(b1.x, b0.x), rn_sub(b1.y, b0.y), rn_sub(b1.z, b0.z));
    ext[2 * (size_t)k] = make_float4(rn, cone_sine(nc.w), cone_sine(wc.w), lum3(q2.y, q2.z, q2.w));
    ext[2 * (size_t)k + 1] = make_float4(lum3(q3.x, q3.y, q3.z), rn_mul(0.5f, rn_add(b0.x, b1.x)),
                                         rn_mul(0.5f, rn_add(b0.y, b1.y)), rn_mul(0.5f, rn_add(b0.z, b1.z)));
}

__device__ __forceinline__ TileInfo load_tile(const float4* info, int tile) {
    const float4 i0 = info[4 * (size_t)tile], i1 = info[4 * (size_t)tile + 1], i2 = info[4 * (size_t)tile + 2],
                 i3 = info[4 * (size_t)tile + 3];
    TileInfo t;
    t.tmin[0] = i0.x; t.tmin[1] = i0.y; t.tmin[2] = i0.z; t.kdl = i0.w;
    t.tmax[0] = i1.x; t.tmax[1] = i1.y; t.tmax[2] = i1.z; t.tau = i1.w;
    t.ncone = i2;
    t.valid = __float_as_int(i3.x);
    t.rt = i3.z;
    t.sn = i3.w;
    return t;
}

// Tiles in decreasing order of (expected) cut size (buckets of floor(log2(count)), empty tiles last), so that
// the blocks with the longest cuts start first and the short ones fill the tail of the launch.
// One block; the order within a bucket is arbitrary (each tile's result does not depend on it).
__global__ void __launch_bounds__(1024) tile_order_kernel(const int32_t* counts, int tiles, int* order) {
    __shared__ int hist[33], off[33];
    const int t = threadIdx.x;
    if (t < 33) hist[t] = 0;
    __syncthreads();
    for (int i = t; i < tiles; i += blockDim.x) {
        const int c = counts[i];
        atomicAdd(&hist[c > 0 ? 32 - __clz(c) : 0], 1);
    }
    __syncthreads();
    if (t == 0) {
        int s = 0;
        for (int b = 32; b >= 0; --b) {
            off[b] = s;
            s += hist[b];
        }
    }
    __syncthreads();
    for (int i = t; i < tiles; i += blockDim.x) {
        const int c = counts[i];
        order[atomicAdd(&off[c > 0 ? 32 - __clz(c) : 0], 1)] = i;
    }
}

// ---------------------------------------------------------------------------------------
// Error-bound cut selection: one block per tile at a time, tiles from a work counter
// ---------------------------------------------------------------------------------------
struct SelArgs {
    int n;
    const float4* bounds;
    const float4* records;
    const float4* info;
    const float4* extra;  // NodeExtra per inner node
    BoundParams bp;
    int tiles;
    const int* order;     // tiles, largest expected cut first
    int* next_tile;       // tiles handed out
    CutPool pool;
    uint32_t* err;
};

// The rounded bound of (tile, inner node k), for the pairs that node_bound_fast leaves open.
__device__ __noinline__ float rounded_bound(const float4* info, int tile, const float4* bounds, const float4* extra,
                                            int k, const BoundParams& bp) {
    const TileInfo t = load_tile(info, tile);
    const NodeExtra ne = load_node_extra(extra, k);
    const float4* b = bounds + 4 * (size_t)k;
    const NodeGeom g = node_geom(t, b[0], b[1], b[2], b[3], ne, bp);
    return node_bound(t, g, ne.Ls, ne.As, bp);
}

// A tile's walk: the block pops up to 128 nodes of a shared stack, one per thread, appends the accepted
// ones to the tile's list in the cut pool and pushes the others' children.  Four warps share a walk
// because the largest tiles take 10 times the mean (with one warp per tile the last of them ran
// alone for a quarter of the launch), and tiles start in decreasing order of their expected cut.  A
// step pops all it can, so the stack grows by at most 128 nodes per level of the tree: kSelStack holds
// trees of 62 levels, and Morton codes of 32 bits over 2^25 leaves make 57.
//
// Bound by instruction issue and latency (56% issue, ALU 49%, 390 instructions per 32 nodes).  1280 x 720 x
// 65,536 AVPLs, bound 0.01: 5.0 ms with one warp per tile and 12 warps per SM (16 KB of stack each), 3.8 ms
// with 28, 3.5 ms with the approximate bound, 3.2 ms with the expected cuts first, 2.9 ms as it is.
__global__ void __launch_bounds__(kSelThreads, kSelBlocksPerSm) cut_select_bound(SelArgs a) {
    constexpr int kW = kSelThreads / 32;
    __shared__ int stack[kSelStack];
    __shared__ int s_acc[2][kW], s_ref[2][kW];
    __shared__ int s_tile, s_chunk;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned lt = (1u << lane) - 1u;
    for (;;) {
        if (tid == 0) {
            const int i = atomicAdd(a.next_tile, 1);
            s_tile = i < a.tiles ? a.order[i] : -1;
            stack[0] = a.n;  // root
        }
        __syncthreads();
        const int tile = s_tile;
        if (tile < 0) return;
        const TileInfo t = load_tile(a.info, tile);
        int32_t* table = a.pool.tables + (size_t)tile * a.pool.max_chunks;
        int count = 0, chunk = -1;  // list length; pool chunk of its last entry
        bool overflow = false;
        int sp = t.valid ? 1 : 0;
        int budget = 2 * a.n;  // node visits of a valid tree
        for (int turn = 0; sp > 0; turn ^= 1) {
            if (budget <= 0) {
                if (tid == 0) set_error(a.err, ARC_DEVERR_BAD_NODE);
                break;
            }
            const int m = min(kSelThreads, sp);
            budget -= m;
            sp -= m;
            int node = -1, lc = 0, rc = 0;
            bool accept = false, refine = false;
            if (tid < m) {
                node = stack[sp + m - 1 - tid];
                if (node < a.n) {
                    accept = node >= 0;
                } else {
                    const int k = node - a.n;
                    const float4 b0 = a.bounds[4 * (size_t)k], b1 = a.bounds[4 * (size_t)k + 1];
                    const float4 nc = a.bounds[4 * (size_t)k + 2], wc = a.bounds[4 * (size_t)k + 3];
                    const NodeExtra ne = load_node_extra(a.extra, k);
                    int over = exceeds(node_bound_fast(t, b0, b1, nc, wc, ne, a.bp), t.tau);
                    if (over < 0) over = rounded_bound(a.info, tile, a.bounds, a.extra, k, a.bp) > t.tau;
                    refine = over != 0;
                    accept = over == 0;
                    const int l = __float_as_int(b0.w), r = __float_as_int(b1.w);
                    lc = l >= 0 ? l : a.n - (l + 1);
                    rc = r >= 0 ? r : a.n - (r + 1);
                }
            }
            unsigned am = __ballot_sync(0xffffffffu, accept);
            const unsigned rm = __ballot_sync(0xffffffffu, refine);
            if (lane == 0) {
                s_acc[turn][warp] = __popc(am);
                s_ref[turn][warp] = __popc(rm);
            }
            __syncthreads();  // the counts; and every popped node has been read
            int before_a = 0, before_r = 0, na = 0, nref = 0;
#pragma unroll
            for (int q = 0; q < kW; ++q) {
                const int x = s_acc[turn][q], y = s_ref[turn][q];
                if (q < warp) {
                    before_a += x;
                    before_r += y;
                }
                na += x;
                nref += y;
            }
            if (sp + 2 * nref > kSelStack) {  // no room: use the nodes whole
                accept = accept || refine;
                refine = false;
                am |= rm;
                before_a += before_r;
                na += nref;
                nref = 0;
                overflow = true;
            }
            if (na > 0) {  // append to the list, which starts at most one new chunk (128 < kChunkSize)
                const int first_new = (count + kChunkSize - 1) / kChunkSize, last = (count + na - 1) / kChunkSize;
                const bool fresh = last >= first_new;
                int id = chunk;
                if (fresh) {
                    if (tid == 0) {
                        const int c = last < a.pool.max_chunks ? atomicAdd(a.pool.next, 1) : a.pool.num_chunks;
                        if (c < a.pool.num_chunks) table[last] = c;
                        s_chunk = c;
                    }
                    __syncthreads();
                    id = s_chunk;
                }
                if (accept) {
                    const int pos = count + before_a + __popc(am & lt);
                    const int c = pos / kChunkSize == last && fresh ? id : chunk;
                    if (c >= 0 && c < a.pool.num_chunks)
                        a.pool.entries[(size_t)c * kChunkSize + pos % kChunkSize] = node;
                }
                chunk = id;
                if (fresh && id >= a.pool.num_chunks) overflow = true;
                // (past the pool only the entries that landed in a chunk are kept)
                count = chunk >= a.pool.num_chunks ? min(count + na, last * kChunkSize) : count + na;
            }
            if (refine) {
                const int q = sp + 2 * (before_r + __popc(rm & lt));
                stack[q] = rc;
                stack[q + 1] = lc;
            }
            sp += 2 * nref;
            __syncthreads();  // the pushes
        }
        if (tid == 0) {
            if (overflow) set_error(a.err, ARC_DEVERR_CUT_OVERFLOW);
            a.pool.counts[tile] = count;
        }
        __syncthreads();  // every thread has read s_tile and left the stack
    }
}

// ---------------------------------------------------------------------------------------
// Cut evaluation: one 64-thread block per tile, one pixel per thread
// ---------------------------------------------------------------------------------------
struct EvalArgs {
    const float4* gpos;
    const float4* gnrm;
    int64_t gpitch;
    int width, height;
    const MaterialRecord* mats;
    int num_mats;
    const float4* records;
    int tiles_x;
    CutPool pool;
    PairConsts pc;
    float disk_scale;
    float4* out_res;
    float4* out_rad;
    float4* out_ar;
    double* out_res64;
    int64_t opitch;
    const int* order;  // block b evaluates tile order[b]
};

template <int AR>
__global__ void __launch_bounds__(64) cut_eval_kernel(EvalArgs a) {
    constexpr int kChunk = 256;
    __shared__ float4 srec[kChunk * 4];
    const int tile = a.order[blockIdx.x];
    const int i = threadIdx.x;
    const int x = (tile % a.tiles_x) * kTile + i % kTile, y = (tile / a.tiles_x) * kTile + i / kTile;
    bool valid = x < a.width && y < a.height;
    float4 gp = make_float4(0, 0, 0, 0), gn = make_float4(0, 0, 0, 0);
    int mat = 0;
    if (valid) {
        gp = a.gpos[(int64_t)y * a.gpitch + x];
        gn = a.gnrm[(int64_t)y * a.gpitch + x];
        mat = (int)gn.w;
        valid = mat > 0 && mat < a.num_mats;
    }
    Pixel<float> px;
    px.px = gp.x;
    px.py = gp.y;
    px.pz = gp.z;
    if (valid) {
        const float l = rsqrtf(gn.x * gn.x + gn.y * gn.y + gn.z * gn.z);
        px.nx = gn.x * l;
        px.ny = gn.y * l;
        px.nz = gn.z * l;
    } else {
        px.nx = px.ny = px.nz = 0.0f;
    }
    px.r0 = px.r1 = px.r2 = px.a0 = px.a1 = px.a2 = 0.0f;
    float ss[6] = {0, 0, 0, 0, 0, 0}, sc[6] = {0, 0, 0, 0, 0, 0};
    const int count = a.pool.counts[tile];
    for (int base = 0; base < count; base += kChunk) {
        const int cnt = min(kChunk, count - base);
        // kChunk divides kChunkSize: a sub-chunk never straddles two pool chunks
        const int32_t* nodes = a.pool.entries + (size_t)a.pool.tables[(size_t)tile * a.pool.max_chunks + base / kChunkSize] *
                                                    kChunkSize + base % kChunkSize;
        __syncthreads();
        for (int j = i; j < cnt * 4; j += 64) {
            const int node = nodes[j / 4];
            float4 q = a.records[4 * (size_t)node + (j & 3)];
            if (AR == ARC_AR_DISK && (j & 3) == 3) {
                const float4 q1 = a.records[4 * (size_t)node + 1], q2 = a.records[4 * (size_t)node + 2];
                const float ww = q1.z * q1.z + q1.w * q1.w + q2.x * q2.x;
                q.w = ww > 0.0f ? rsqrtf(ww) : 0.0f;
            }
            srec[j] = q;
        }
        __syncthreads();
        for (int j = 0; j < cnt; ++j) {
            float g, ga;
            const float4* q = srec + 4 * j;
            pair_terms<AR, float>(q[0], q[1], q[2], q[3], px, a.pc, g, ga);
            px.r0 += q[2].y * g;
            px.r1 += q[2].z * g;
            px.r2 += q[2].w * g;
            px.a0 += q[3].x * ga;
            px.a1 += q[3].y * ga;
            px.a2 += q[3].z * ga;
        }
        kahan_add(ss[0], sc[0], px.r0);
        kahan_add(ss[1], sc[1], px.r1);
        kahan_add(ss[2], sc[2], px.r2);
        kahan_add(ss[3], sc[3], px.a0);
        kahan_add(ss[4], sc[4], px.a1);
        kahan_add(ss[5], sc[5], px.a2);
        px.r0 = px.r1 = px.r2 = px.a0 = px.a1 = px.a2 = 0.0f;
    }
    if (x >= a.width || y >= a.height) return;
    double rad[3] = {0, 0, 0}, ar[3] = {0, 0, 0};
    if (valid) {
        const float4 d = a.mats[mat].diffuse_exp;
        const double kd[3] = {(double)(kOneOverPi * d.x), (double)(kOneOverPi * d.y), (double)(kOneOverPi * d.z)};
        const double as = AR == ARC_AR_DISK ? (double)a.disk_scale : 1.0;
        for (int c = 0; c < 3; ++c) {
            rad[c] = kd[c] * ((double)ss[c] - (double)sc[c]);
            ar[c] = kd[c] * as * ((double)ss[3 + c] - (double)sc[3 + c]);
        }
    }
    const int64_t o = (int64_t)y * a.opitch + x;
    const double res[3] = {rad[0] - ar[0], rad[1] - ar[1], rad[2] - ar[2]};
    if (a.out_res) a.out_res[o] = make_float4((float)res[0], (float)res[1], (float)res[2], 1.0f);
    if (a.out_rad) a.out_rad[o] = make_float4((float)rad[0], (float)rad[1], (float)rad[2], 1.0f);
    if (a.out_ar) a.out_ar[o] = make_float4((float)ar[0], (float)ar[1], (float)ar[2], 1.0f);
    if (a.out_res64) {
        a.out_res64[3 * o + 0] = res[0];
        a.out_res64[3 * o + 1] = res[1];
        a.out_res64[3 * o + 2] = res[2];
    }
}

// Cut evaluation with packed FP32 pairs (no or cone antiradiance): one 128-thread block per tile, two
// pixels per lane, so that each warp holds the whole tile and walks its own share of the cut (stages
// of kEvalStage nodes, every fourth one) without a barrier until the warps' sums are added.  Per
// stage a warp copies the nodes' 64-byte records into shared memory (16-byte cp.async, four lanes per
// record, one stage ahead), each lane tests two nodes against the tile's bounds (pair_cull.cuh), the
// nodes that can contribute go into a radiance and a cone list, and the packed pair loops run over
// the lists.  FP32 partials of up to 256 nodes are folded into FP64 sums.  Bound by the FMA pipe's
// issue (59-64% active, 22 instructions per evaluated pair of which 16 are the pair's own); four
// blocks of 128 registers per SM measured 24.2 ms, five with spills 24.8 ms, and the kernel that
// evaluated every pair 57.4 ms (1920 x 1080 x 1,048,576 AVPLs, learned cut).
constexpr int kEvalWarps = 4, kEvalStage = 64;
constexpr int kEvalFold = 4;  // stages per FP32 partial

struct EvalWarp {
    float4 raw[kEvalStage * 4];  // records; 16-byte quarter q of record m at 4 m + (q ^ (m / 2 % 4))
    float list_r[kEvalStage / 2 * kPairFloats];
    float list_a[kEvalStage / 2 * kPairFloats];
};

template <int AR>
__global__ void __launch_bounds__(32 * kEvalWarps, 4) cut_eval_culled_kernel(EvalArgs a) {
    __shared__ __align__(16) EvalWarp sw[kEvalWarps];
    static_assert(sizeof(sw) >= kEvalWarps * 64 * 6 * sizeof(double), "the warps' sums reuse the stages");
    const int tile = a.order[blockIdx.x];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int x = (tile % a.tiles_x) * kTile + lane % kTile, y0 = (tile / a.tiles_x) * kTile + lane / kTile;
    const int count = a.pool.counts[tile];
    const int nstages = (count + kEvalStage - 1) / kEvalStage;
    const int32_t* table = a.pool.tables + (size_t)tile * a.pool.max_chunks;
    EvalWarp& e = sw[w];
    // node ids of stage s: entries lane and lane + 32 (kEvalStage divides the pool's chunks)
    auto load_ids = [&](int s, int& id0, int& id1) {
        id0 = id1 = -1;
        if (s >= nstages) return;
        const int base = s * kEvalStage;
        const int32_t* nodes = a.pool.entries + (size_t)table[base / kChunkSize] * kChunkSize + base % kChunkSize;
        if (base + lane < count) id0 = nodes[lane];
        if (base + 32 + lane < count) id1 = nodes[32 + lane];
    };
    auto copy_records = [&](int id0, int id1) {
#pragma unroll
        for (int g = 0; g < kEvalStage / 8; ++g) {
            const int m = g * 8 + (lane >> 2), q = lane & 3;
            const int id = __shfl_sync(0xffffffffu, g < 4 ? id0 : id1, m & 31);
            if (id >= 0) cp_async16(&e.raw[4 * m + (q ^ (m >> 1 & 3))], a.records + 4 * (size_t)id + q);
        }
        cp_async_commit();
    };
    int id0, id1, next0, next1;
    load_ids(w, id0, id1);
    copy_records(id0, id1);
    load_ids(w + kEvalWarps, next0, next1);

    PixelPair pp[2];
    int mat[2];
    PixelBounds box;
    box.clear();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int y = y0 + 4 * j;
        float4 gp = make_float4(0, 0, 0, 0), gn = make_float4(0, 0, 0, 0);
        if (x < a.width && y < a.height) {
            gp = a.gpos[(int64_t)y * a.gpitch + x];
            gn = a.gnrm[(int64_t)y * a.gpitch + x];
        }
        mat[j] = (int)gn.w;
        if (mat[j] <= 0 || mat[j] >= a.num_mats) mat[j] = 0;
        float nx = 0.0f, ny = 0.0f, nz = 0.0f;
        if (mat[j]) {
            const float l = rsqrtf(gn.x * gn.x + gn.y * gn.y + gn.z * gn.z);
            nx = gn.x * l;
            ny = gn.y * l;
            nz = gn.z * l;
            box.add(gp.x, gp.y, gp.z, nx, ny, nz, nx, ny, nz);
        }
        pp[j] = pixel_pair(gp.x, gp.y, gp.z, nx, ny, nz);
    }
    box.reduce_warp();
    const float cos_thr = a.pc.cos_thr, eps = a.pc.eps, inv_clamp2 = a.pc.inv_clamp2;
    // distance floor folded into the FMA chain: l2 + 1e-30 equals max(l2, 1e-30) for l2 above ~1e-23
    const uint64_t tiny2 = f2(1e-30f, 1e-30f);
    double sum[2][6] = {};
    uint64_t acc[2][6] = {};  // packed zeros
    int held = 0;             // stages in acc
    const unsigned lt = (1u << lane) - 1u;
    for (int s = w; s < nstages; s += kEvalWarps) {
        const int left = count - s * kEvalStage;
        cp_async_wait<0>();
        __syncwarp();  // every lane's copies; and the lists' readers are done
        int nr = 0, na = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = 32 * h + lane, sz = m >> 1 & 3;
            RecordNeed need{false, false};
            float4 q0, q1, q2, q3;
            if (m < left) {
                q0 = e.raw[4 * m + sz];
                q1 = e.raw[4 * m + (1 ^ sz)];
                q2 = e.raw[4 * m + (2 ^ sz)];
                q3 = e.raw[4 * m + (3 ^ sz)];
                need = record_need<AR == ARC_AR_CONE>(box, q0, q1, q2, q3, cos_thr);
            }
            const unsigned mr = __ballot_sync(0xffffffffu, need.radiance);
            const unsigned ma = __ballot_sync(0xffffffffu, need.cone);
            if (need.radiance)
                put_entry(e.list_r, nr + __popc(mr & lt), q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q2.y, q2.z, q2.w);
            if (need.cone)
                put_entry(e.list_a, na + __popc(ma & lt), q0.x, q0.y, q0.z, q1.z, q1.w, q2.x, q3.x, q3.y, q3.z);
            nr += __popc(mr);
            na += __popc(ma);
        }
        // an odd list ends with a zero record, which adds exactly 0
        if (lane == 0 && (nr & 1)) put_entry(e.list_r, nr, 0, 0, 0, 0, 0, 0, 0, 0, 0);
        if (lane == 1 && (na & 1)) put_entry(e.list_a, na, 0, 0, 0, 0, 0, 0, 0, 0, 0);
        __syncwarp();  // the lists are complete, the records read
        copy_records(next0, next1);
        load_ids(s + 2 * kEvalWarps, next0, next1);
#pragma unroll 2
        for (int pr = 0; 2 * pr < nr; ++pr)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                radiance_pair(e.list_r + pr * kPairFloats, pp[j], inv_clamp2, tiny2, acc[j][0], acc[j][1], acc[j][2]);
        if (AR == ARC_AR_CONE) {
#pragma unroll 1
            for (int pr = 0; 2 * pr < na; ++pr)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    cone_pair(e.list_a + pr * kPairFloats, pp[j], cos_thr, eps, inv_clamp2, tiny2, acc[j][3], acc[j][4],
                              acc[j][5]);
        }
        if (++held == kEvalFold || s + kEvalWarps >= nstages) {
            held = 0;
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    float lo, hi;
                    f2_split(acc[j][c], lo, hi);
                    sum[j][c] += (double)(lo + hi);
                    acc[j][c] = 0;
                }
        }
    }
    cp_async_wait<0>();
    __syncthreads();  // every warp is done with its stages
    double* ws = reinterpret_cast<double*>(sw);  // [warp][channel][pixel]
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int c = 0; c < 6; ++c) ws[(w * 6 + c) * 64 + 32 * j + lane] = sum[j][c];
    __syncthreads();
    if (w >= 2) return;
    const int y = y0 + 4 * w;  // warp w writes pixels 32 w ... 32 w + 31
    if (x >= a.width || y >= a.height) return;
    double rad[3] = {0, 0, 0}, ar[3] = {0, 0, 0};
    const int m = w ? mat[1] : mat[0];
    if (m) {
        const float4 d = a.mats[m].diffuse_exp;
        const double kd[3] = {(double)(kOneOverPi * d.x), (double)(kOneOverPi * d.y), (double)(kOneOverPi * d.z)};
        for (int c = 0; c < 3; ++c)
            for (int q = 0; q < kEvalWarps; ++q) {
                rad[c] += ws[(q * 6 + c) * 64 + 32 * w + lane];
                ar[c] += ws[(q * 6 + 3 + c) * 64 + 32 * w + lane];
            }
        for (int c = 0; c < 3; ++c) {
            rad[c] *= kd[c];
            ar[c] *= kd[c];
        }
    }
    const int64_t o = (int64_t)y * a.opitch + x;
    const double res[3] = {rad[0] - ar[0], rad[1] - ar[1], rad[2] - ar[2]};
    if (a.out_res) a.out_res[o] = make_float4((float)res[0], (float)res[1], (float)res[2], 1.0f);
    if (a.out_rad) a.out_rad[o] = make_float4((float)rad[0], (float)rad[1], (float)rad[2], 1.0f);
    if (a.out_ar) a.out_ar[o] = make_float4((float)ar[0], (float)ar[1], (float)ar[2], 1.0f);
    if (a.out_res64) {
        a.out_res64[3 * o + 0] = res[0];
        a.out_res64[3 * o + 1] = res[1];
        a.out_res64[3 * o + 2] = res[2];
    }
}

// result = radiance - antiradiance in FP64 (kernel_combine, cudaGather.cu:782-803)
__global__ void combine_kernel(const double* rad64, const double* ar64, int width, int height, float4* out_res,
                               float4* out_ar, double* out_res64, int64_t opitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= width || y >= height) return;
    const int64_t o = (int64_t)y * opitch + x;
    double r[3];
    for (int c = 0; c < 3; ++c) r[c] = rad64[3 * o + c] - (ar64 ? ar64[3 * o + c] : 0.0);
    if (out_res) out_res[o] = make_float4((float)r[0], (float)r[1], (float)r[2], 1.0f);
    if (out_ar) {
        if (ar64)
            out_ar[o] = make_float4((float)ar64[3 * o], (float)ar64[3 * o + 1], (float)ar64[3 * o + 2], 1.0f);
        else
            out_ar[o] = make_float4(0, 0, 0, 1.0f);
    }
    if (out_res64)
        for (int c = 0; c < 3; ++c) out_res64[3 * o + c] = r[c];
}

}  // namespace

arc_status launch_combine(arc_context* ctx, const double* rad64, const double* ar64, int width, int height,
                          const ArcOutputView* out) {
    stage_begin(ctx, "combine");
    combine_kernel<<<dim3((width + 31) / 32, (height + 7) / 8), dim3(32, 8), 0, ctx->stream>>>(
        rad64, ar64, width, height, reinterpret_cast<float4*>(out->result),
        reinterpret_cast<float4*>(out->antiradiance), out->result_fp64, out->pitch);
    stage_end(ctx, 1);
    ARC_TRY_CUDA(cudaGetLastError());
    return ARC_OK;
}

arc_status launch_tile_setup(arc_context* ctx, const arc_lbvh* bvh, const ArcGBufferView* gb, const ArcGatherParams* gp,
                             const ArcCutParams* cp, float4** info_out, float4** extra_out, int* estimate) {
    const int W = gb->width, H = gb->height;
    const int tiles_x = (W + kTile - 1) / kTile, tiles_y = (H + kTile - 1) / kTile, tiles = tiles_x * tiles_y;
    float4* info = nullptr;
    ARC_TRY(ctx->arena.get("tile_info", (size_t)tiles * 4 * sizeof(float4), reinterpret_cast<void**>(&info)));
    TileArgs ta;
    ta.gpos = reinterpret_cast<const float4*>(gb->position);
    ta.gnrm = reinterpret_cast<const float4*>(gb->normal);
    ta.gpitch = gb->pitch;
    ta.width = W;
    ta.height = H;
    ta.mats = ctx->d_materials;
    ta.num_mats = ctx->num_materials;
    ta.n = bvh->n;
    ta.bounds = reinterpret_cast<const float4*>(bvh->view.bounds);
    ta.records = reinterpret_cast<const float4*>(bvh->view.records);
    ta.eps_bound = cp->error_bound;
    ta.clamp2 = gp->dist_clamp > 0.0f ? gp->dist_clamp * gp->dist_clamp : 0.0f;
    ta.tiles_x = tiles_x;
    ta.tiles_y = tiles_y;
    ta.info = info;
    ta.err = ctx->d_error;
    float4* extra = nullptr;
    ARC_TRY(ctx->arena.get("node_extra", (size_t)(bvh->n - 1) * 2 * sizeof(float4), reinterpret_cast<void**>(&extra)));
    ta.estimate = estimate;
    ta.extra = extra;
    ta.bp = bound_params(gp, cp);
    stage_begin(ctx, "cut_setup");
    cut_node_extra<<<(bvh->n - 1 + 255) / 256, 256, 0, ctx->stream>>>(bvh->n, ta.bounds, ta.records, extra);
    cut_tile_setup<<<(tiles + kSetupWarps - 1) / kSetupWarps, 32 * kSetupWarps, 0, ctx->stream>>>(ta);
    stage_end(ctx, 2);
    ARC_TRY_CUDA(cudaGetLastError());
    *info_out = info;
    *extra_out = extra;
    return ARC_OK;
}

arc_status launch_gather_cut(arc_context* ctx, const arc_lbvh* bvh, const ArcAvplsGpuParam* avpls,
                             const ArcGBufferView* gb, float3 cam, const ArcGatherParams* gp, const ArcCutParams* cp,
                             const ArcOutputView* out) {
    ARC_CHECK_ARG(bvh->n >= 2, "LBVH not built");
    ARC_CHECK_ARG(cp->kind >= 0 && cp->kind <= 2, "cut kind out of range");
    ARC_CHECK_ARG(gp->ar_kind >= 0 && gp->ar_kind <= 2, "ar_kind out of range");
    ARC_CHECK_ARG(gb->width > 0 && gb->height > 0 && gb->pitch >= gb->width && gb->position && gb->normal,
                  "bad G-buffer view");
    ARC_CHECK_ARG(out->pitch >= gb->width, "bad output view");
    ARC_CHECK_ARG(ctx->num_materials > 0, "materials not uploaded");
    cudaStream_t st = ctx->stream;
    const int W = gb->width, H = gb->height;
    const float clamp2 = gp->dist_clamp > 0.0f ? gp->dist_clamp * gp->dist_clamp : 0.0f;

    if (cp->kind == ARC_CUT_SOLID_ANGLE) {
        double *rad64 = nullptr, *ar64 = nullptr;
        const size_t np = (size_t)H * out->pitch;
        ARC_TRY(ctx->arena.get("cut_rad64", np * 3 * sizeof(double), reinterpret_cast<void**>(&rad64)));
        SolidArgs a;
        a.gpos = reinterpret_cast<const float4*>(gb->position);
        a.gnrm = reinterpret_cast<const float4*>(gb->normal);
        a.gpitch = gb->pitch;
        a.width = W;
        a.height = H;
        a.mats = ctx->d_materials;
        a.num_mats = ctx->num_materials;
        a.cam = cam;
        a.n = bvh->n;
        a.bounds = reinterpret_cast<const float4*>(bvh->view.bounds);
        a.records = reinterpret_cast<const float4*>(bvh->view.records);
        a.nd = bvh->view.node_data;
        a.thresh = cp->solid_angle_threshold;
        const double cosine = 1.0 - (double)a.thresh / (2.0 * 3.14159265358979);
        a.cos2 = (float)(cosine * cosine);
        // the test as written is within 5e-7 of the cosine (a dozen roundings of values <= 1)
        a.cos2_margin = cosine >= 0.0 && cosine <= 1.0 ? 4e-6f : INFINITY;
        a.clamp2 = clamp2;
        a.rad64 = rad64;
        a.out_rad = reinterpret_cast<float4*>(out->radiance);
        a.opitch = out->pitch;
        a.dbg_x = cp->debug_pixel_x;
        a.dbg_y = cp->debug_pixel_y;
        a.used = cp->used_nodes;
        a.err = ctx->d_error;
        dim3 grid((W + 7) / 8, (H + 7) / 8);
        stage_begin(ctx, "cut_solid_angle");
        if (ctx->any_specular)
            cut_solid_angle_kernel<true><<<grid, kSolidThreads, 0, st>>>(a);
        else
            cut_solid_angle_kernel<false><<<grid, kSolidThreads, 0, st>>>(a);
        stage_end(ctx, 1);
        ARC_TRY_CUDA(cudaGetLastError());
        if (gp->ar_kind != ARC_AR_NONE) {
            ARC_CHECK_ARG(avpls != nullptr, "ARC_CUT_SOLID_ANGLE with antiradiance needs the AVPL arrays");
            ARC_TRY(ctx->arena.get("cut_ar64", np * 3 * sizeof(double), reinterpret_cast<void**>(&ar64)));
            GatherLaunch g{avpls, gb, cam, gp, out};
            ARC_TRY(launch_antiradiance_only(ctx, g, ar64));
        }
        return launch_combine(ctx, rad64, ar64, W, H, out);
    }

    // tile cuts
    const int tiles_x = (W + kTile - 1) / kTile, tiles_y = (H + kTile - 1) / kTile, tiles = tiles_x * tiles_y;
    const int max_cut = cp->max_cut_nodes > 0 ? cp->max_cut_nodes : (1 << 20);
    CutPool pool;
    pool.max_chunks = (max_cut + kChunkSize - 1) / kChunkSize;
    const int64_t pool_entries = cp->cut_pool_entries > 0 ? cp->cut_pool_entries : (int64_t)tiles * 32768;
    pool.num_chunks = (int32_t)std::min<int64_t>((pool_entries + kChunkSize - 1) / kChunkSize, INT32_MAX / kChunkSize);
    ARC_TRY(ctx->arena.get("cut_pool", (size_t)pool.num_chunks * kChunkSize * sizeof(int32_t),
                           reinterpret_cast<void**>(&pool.entries)));
    ARC_TRY(ctx->arena.get("cut_tables", (size_t)tiles * pool.max_chunks * sizeof(int32_t),
                           reinterpret_cast<void**>(&pool.tables)));
    ARC_TRY(ctx->arena.get("cut_counts", (size_t)tiles * sizeof(int32_t), reinterpret_cast<void**>(&pool.counts)));
    // the pool's allocation counter and the selection's work counter
    ARC_TRY(ctx->arena.get("cut_pool_next", 2 * sizeof(int32_t), reinterpret_cast<void**>(&pool.next)));
    ARC_TRY_CUDA(cudaMemsetAsync(pool.next, 0, 2 * sizeof(int32_t), st));
    float4* info = nullptr;
    float4* extra = nullptr;
    int* order = nullptr;     // tiles in the order the selection, then the evaluation takes them
    int* estimate = nullptr;  // expected cut size per tile
    ARC_TRY(ctx->arena.get("cut_order", (size_t)tiles * sizeof(int), reinterpret_cast<void**>(&order)));
    if (cp->kind == ARC_CUT_ERROR_BOUND)
        ARC_TRY(ctx->arena.get("cut_estimate", (size_t)tiles * sizeof(int), reinterpret_cast<void**>(&estimate)));
    ARC_TRY(launch_tile_setup(ctx, bvh, gb, gp, cp, &info, &extra, estimate));

    if (cp->kind == ARC_CUT_ERROR_BOUND) {
        SelArgs sa;
        sa.n = bvh->n;
        sa.bounds = reinterpret_cast<const float4*>(bvh->view.bounds);
        sa.records = reinterpret_cast<const float4*>(bvh->view.records);
        sa.info = info;
        sa.extra = extra;
        sa.bp = bound_params(gp, cp);
        sa.order = order;
        sa.tiles = tiles;
        sa.pool = pool;
        sa.err = ctx->d_error;
        sa.next_tile = pool.next + 1;
        stage_begin(ctx, "cut_select");
        tile_order_kernel<<<1, 1024, 0, st>>>(estimate, tiles, order);
        cut_select_bound<<<std::min(tiles, ctx->sm_count * kSelBlocksPerSm), kSelThreads, 0, st>>>(sa);
        stage_end(ctx, 2);
        ARC_TRY_CUDA(cudaGetLastError());
    } else {
        ARC_CHECK_ARG(cp->model != nullptr, "ARC_CUT_LEARNED needs a model");
        ARC_TRY(launch_cut_select_learned(ctx, bvh, gp, cp, info, extra, tiles_x, tiles_y, pool));
    }

    EvalArgs ea;
    ea.gpos = reinterpret_cast<const float4*>(gb->position);
    ea.gnrm = reinterpret_cast<const float4*>(gb->normal);
    ea.gpitch = gb->pitch;
    ea.width = W;
    ea.height = H;
    ea.mats = ctx->d_materials;
    ea.num_mats = ctx->num_materials;
    ea.records = reinterpret_cast<const float4*>(bvh->view.records);
    ea.tiles_x = tiles_x;
    ea.pool = pool;
    ea.pc.cos_thr = fmaxf(cosf(gp->cone_half_angle), 0.001f);
    ea.pc.eps = 0.001f;
    ea.pc.inv_clamp2 = clamp2 > 0.0f ? 1.0f / clamp2 : INFINITY;
    ea.pc.disk_r2 = gp->disk_radius * gp->disk_radius;
    ea.disk_scale = gp->disk_radius > 0.0f ? 1.0f / (kPi * gp->disk_radius * gp->disk_radius) : 0.0f;
    ea.out_res = reinterpret_cast<float4*>(out->result);
    ea.out_rad = reinterpret_cast<float4*>(out->radiance);
    ea.out_ar = reinterpret_cast<float4*>(out->antiradiance);
    ea.out_res64 = out->result_fp64;
    ea.opitch = out->pitch;
    ea.order = order;
    stage_begin(ctx, "cut_eval");
    tile_order_kernel<<<1, 1024, 0, st>>>(pool.counts, tiles, order);
    if (gp->ar_kind == 0) cut_eval_culled_kernel<0><<<tiles, 32 * kEvalWarps, 0, st>>>(ea);
    if (gp->ar_kind == 1) cut_eval_kernel<1><<<tiles, 64, 0, st>>>(ea);
    if (gp->ar_kind == 2) cut_eval_culled_kernel<2><<<tiles, 32 * kEvalWarps, 0, st>>>(ea);
    stage_end(ctx, 2);
    ARC_TRY_CUDA(cudaGetLastError());
    ctx->last_cut.num_tiles = tiles;
    ctx->last_cut.pool = pool;
    return ARC_OK;
}

}  // namespace arc
