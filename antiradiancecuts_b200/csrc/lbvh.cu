// LBVH build over AVPLs (AvplBvh / Bvh::create, bvh.cu:325-454, 673-808; morton.h).
//
//   1. lbvh_bbox        min/max reduction (only for the reference's AVPL-box normalisation and
//                       for 6D codes), ordered-integer atomics
//   2. lbvh_morton      normalise with IEEE division (bvh.cu:73-81), quantise and interleave
//                       (morton.h:82-107), write (code, index) and the digit histograms of all
//                       four sort passes
//   3. radix sort       4 x 8-bit stable LSD passes, one kernel each: tiles ranked with warp
//                       match/ballot, tile offsets by decoupled look-back with bounded waits
//   4. lbvh_topology    Karras inner node i (bvh.cu:189-266)
//   5. lbvh_blocks      per 128 sorted leaves: the gather of the leaves (the reference's zip-iterator
//                       payload sort, bvh.cu:793-808) and every inner node over them (kernel_innerNodes
//                       + cluster, bvh.cu:280-316, 726-744), merged height by height in shared memory
//   6. lbvh_climb       the other inner nodes: from each block's roots, the second-arriving thread merges
//                       the two children, with release/acquire ordering that the reference lacks (no
//                       fence before its atomic); lbvh_top_nodes writes their data
//
// Every floating-point result is computed with explicitly rounded operations in a fixed order,
// so codes, topology, bounds, sums, representatives and cones equal the CPU build bit for bit.
#include <algorithm>
#include <cfloat>
#include <cstdio>

#include "arc_internal.h"
#include "device_common.cuh"
#include "pcg32.h"

namespace arc {

namespace {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1;

__device__ __forceinline__ uint32_t float_to_ordered(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ordered_to_float(uint32_t u) {
    const uint32_t b = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    return __uint_as_float(b);
}

// bbox slots: [0..2] pos min, [3..5] pos max, [6..8] normal min, [9..11] normal max
__global__ void lbvh_bbox_init(uint32_t* bb) {
    const int t = threadIdx.x;
    if (t < 12) {
        const int which = (t / 3) % 2;  // 0 = min, 1 = max
        // max is seeded with FLT_MIN as numeric_limits<float>::min() in bvh.cu:349-350, 357-358
        bb[t] = which == 0 ? float_to_ordered(FLT_MAX) : float_to_ordered(FLT_MIN);
    }
}

__global__ void lbvh_bbox(ArcAvplsGpuParam a, uint32_t* bb, int with_normals) {
    float mn[6], mx[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        mn[k] = FLT_MAX;
        mx[k] = FLT_MIN;
    }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.numAvpls;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float3 p = ld3(a.position, i);
        mn[0] = fminf(mn[0], p.x); mn[1] = fminf(mn[1], p.y); mn[2] = fminf(mn[2], p.z);
        mx[0] = fmaxf(mx[0], p.x); mx[1] = fmaxf(mx[1], p.y); mx[2] = fmaxf(mx[2], p.z);
        if (with_normals) {
            const float3 n = ld3(a.normal, i);
            mn[3] = fminf(mn[3], n.x); mn[4] = fminf(mn[4], n.y); mn[5] = fminf(mn[5], n.z);
            mx[3] = fmaxf(mx[3], n.x); mx[4] = fmaxf(mx[4], n.y); mx[5] = fmaxf(mx[5], n.z);
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
            mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
        }
    }
    if ((threadIdx.x & 31) == 0) {
        for (int k = 0; k < 3; ++k) {
            atomicMin(&bb[k], float_to_ordered(mn[k]));
            atomicMax(&bb[3 + k], float_to_ordered(mx[k]));
            if (with_normals) {
                atomicMin(&bb[6 + k], float_to_ordered(mn[3 + k]));
                atomicMax(&bb[9 + k], float_to_ordered(mx[3 + k]));
            }
        }
    }
}

__device__ __forceinline__ uint32_t spread3(uint32_t v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__device__ __forceinline__ uint32_t quant10(float v) {
    const float q = fminf(fmaxf(rn_mul(v, 1024.0f), 0.0f), 1023.0f);
    return (uint32_t)q;
}

struct MortonArgs {
    ArcAvplsGpuParam a;
    const uint32_t* bb;  // ordered-int bbox (when computed)
    float3 smin, smax;   // scene box
    int use_avpl_box;
    int consider_normals;
    uint32_t* keys;
    int32_t* vals;
    uint32_t* hist;  // [4][256]
};

__global__ void __launch_bounds__(256) lbvh_morton(MortonArgs m) {
    __shared__ uint32_t sh[4][256];
    for (int i = threadIdx.x; i < 1024; i += blockDim.x) (&sh[0][0])[i] = 0;
    __syncthreads();
    float mn[3], mx[3], nmn[3], nmx[3];
    if (m.use_avpl_box) {
        for (int k = 0; k < 3; ++k) {
            mn[k] = ordered_to_float(m.bb[k]);
            mx[k] = ordered_to_float(m.bb[3 + k]);
        }
    } else {
        mn[0] = m.smin.x; mn[1] = m.smin.y; mn[2] = m.smin.z;
        mx[0] = m.smax.x; mx[1] = m.smax.y; mx[2] = m.smax.z;
    }
    if (m.consider_normals)
        for (int k = 0; k < 3; ++k) {
            nmn[k] = ordered_to_float(m.bb[6 + k]);
            nmx[k] = ordered_to_float(m.bb[9 + k]);
        }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m.a.numAvpls;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float3 p = ld3(m.a.position, i);
        const float pv[3] = {p.x, p.y, p.z};
        uint32_t q[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) q[k] = quant10(rn_div(rn_sub(pv[k], mn[k]), rn_sub(mx[k], mn[k])));
        uint32_t code;
        if (!m.consider_normals) {
            code = spread3(q[0]) | (spread3(q[1]) << 1) | (spread3(q[2]) << 2);
        } else {
            // six 10-bit values interleaved into 64 bits (bit i of value k -> bit 6i + k),
            // truncated to the low 32 bits (MC_SIZE uint32_t, bvh.h:17)
            const float3 n = ld3(m.a.normal, i);
            const float nv[3] = {n.x, n.y, n.z};
            uint32_t u[6] = {q[0], q[1], q[2], 0, 0, 0};
#pragma unroll
            for (int k = 0; k < 3; ++k) u[3 + k] = quant10(rn_div(rn_sub(nv[k], nmn[k]), rn_sub(nmx[k], nmn[k])));
            uint64_t c = 0;
#pragma unroll
            for (int b = 0; b < 10; ++b)
#pragma unroll
                for (int k = 0; k < 6; ++k) c |= (uint64_t)((u[k] >> b) & 1u) << (6 * b + k);
            code = (uint32_t)c;
        }
        m.keys[i] = code;
        m.vals[i] = (int32_t)i;
#pragma unroll
        for (int pass = 0; pass < 4; ++pass) atomicAdd(&sh[pass][(code >> (8 * pass)) & 0xffu], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 1024; i += blockDim.x) {
        const uint32_t v = (&sh[0][0])[i];
        if (v) atomicAdd(&m.hist[i], v);
    }
}

// exclusive scan of each pass's 256-bin histogram (in place), one block of 256 threads
__global__ void lbvh_scan_hist(uint32_t* hist) {
    __shared__ uint32_t s[256];
    for (int pass = 0; pass < 4; ++pass) {
        const uint32_t v = hist[pass * 256 + threadIdx.x];
        s[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < 256; o <<= 1) {
            const uint32_t t = threadIdx.x >= o ? s[threadIdx.x - o] : 0u;
            __syncthreads();
            s[threadIdx.x] += t;
            __syncthreads();
        }
        hist[pass * 256 + threadIdx.x] = s[threadIdx.x] - v;
        __syncthreads();
    }
}

struct SortPassArgs {
    const uint32_t* keys_in;
    const int32_t* vals_in;
    uint32_t* keys_out;
    int32_t* vals_out;
    const uint32_t* digit_base;  // 256 exclusive offsets of this pass
    uint32_t* status;            // [tiles][256]
    uint32_t* tile_counter;
    int32_t n;
    int shift;
    int pass;
    uint32_t spin_limit;  // polls of the look-back before it gives up
    uint32_t* abort;      // the build's abort word: 1 + the pass whose look-back gave up, or 0
    uint32_t* err;
};

template <int kSortKPT>
__global__ void __launch_bounds__(kSortThreads) lbvh_sort_pass(SortPassArgs s) {
    __shared__ uint32_t warp_cnt[kSortWarps][256];
    __shared__ uint32_t tile_off[256];
    __shared__ int tile_sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // An earlier pass gave up (its output is not a permutation, so this pass's digit offsets,
    // counted from the unsorted keys, no longer bound its writes): the build stops here.  CTAs of
    // the pass that gave up keep going, so that none of its tiles waits on a tile that left.
    const uint32_t ab = *reinterpret_cast<volatile uint32_t*>(s.abort);
    if (ab != 0u && ab <= (uint32_t)s.pass) return;
    if (tid == 0) tile_sh = (int)atomicAdd(s.tile_counter, 1u);
    for (int i = tid; i < kSortWarps * 256; i += kSortThreads) (&warp_cnt[0][0])[i] = 0;
    __syncthreads();
    const int tile = tile_sh;
    const int64_t base = (int64_t)tile * kSortThreads * kSortKPT + (int64_t)warp * 32 * kSortKPT;

    uint32_t key[kSortKPT], digit[kSortKPT], rank[kSortKPT];
    unsigned peers[kSortKPT];
    int32_t val[kSortKPT];
    const unsigned lt = (1u << lane) - 1u;
    // (all loads before the first shared-memory update, which the compiler would not move them across)
#pragma unroll
    for (int j = 0; j < kSortKPT; ++j) {
        const int64_t idx = base + j * 32 + lane;
        key[j] = idx < s.n ? s.keys_in[idx] : 0xffffffffu;
        val[j] = idx < s.n ? s.vals_in[idx] : 0;
    }
    // lanes with the same digit, by a ballot per bit (match.any takes a step per distinct digit)
#pragma unroll
    for (int j = 0; j < kSortKPT; ++j) {
        const bool in = base + j * 32 + lane < s.n;
        digit[j] = in ? ((key[j] >> s.shift) & 0xffu) : 256u;
        const unsigned active = __ballot_sync(0xffffffffu, in);
        peers[j] = in ? active : ~active;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const unsigned m = __ballot_sync(0xffffffffu, (digit[j] >> b) & 1u);
            peers[j] &= (digit[j] >> b) & 1u ? m : ~m;
        }
    }
#pragma unroll
    for (int j = 0; j < kSortKPT; ++j) {
        const bool in = digit[j] < 256u;
        const uint32_t before = in ? warp_cnt[warp][digit[j]] : 0u;
        rank[j] = before + __popc(peers[j] & lt);
        __syncwarp();
        if (in && lane == __ffs(peers[j]) - 1) warp_cnt[warp][digit[j]] = before + __popc(peers[j]);
        __syncwarp();
    }
    __syncthreads();
    // per digit: exclusive offsets across warps, tile total, then decoupled look-back
    {
        const int d = tid;  // 256 threads, one digit each
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            const uint32_t c = warp_cnt[w][d];
            warp_cnt[w][d] = run;
            run += c;
        }
        const uint32_t total = run;
        volatile uint32_t* st = s.status;
        uint32_t excl = 0;
        if (tile == 0) {
            st[d] = kFlagPrefix | total;
        } else {
            st[(size_t)tile * 256 + d] = kFlagAgg | total;
            // kWindow tiles' words are loaded at once: the walk back to the nearest known prefix is a
            // chain of loads, and its length times their latency was most of a pass
            constexpr int kWindow = 16;
            int t = tile - 1;
            uint32_t spins = 0;
            bool walking = true;
            while (walking) {
                uint32_t v[kWindow];
#pragma unroll
                for (int q = 0; q < kWindow; ++q)
                    v[q] = t - q >= 0 ? (uint32_t)st[(size_t)(t - q) * 256 + d] : (uint32_t)kFlagPrefix;  // before the first tile: 0
                int used = 0;
#pragma unroll
                for (int q = 0; q < kWindow; ++q) {
                    if (walking && used == q && (v[q] & ~kValueMask) != 0) {
                        excl += v[q] & kValueMask;
                        used = q + 1;
                        if (v[q] & kFlagPrefix) walking = false;
                    }
                }
                t -= used;
                if (walking && used < kWindow && ++spins > s.spin_limit) {
                    // publish what was summed: later tiles' offsets stay within the digit's
                    // range, and the passes after this one do not run
                    set_error(s.err, ARC_DEVERR_TIMEOUT);
                    atomicMax(s.abort, (uint32_t)s.pass + 1u);
                    break;
                }
            }
            __threadfence();
            st[(size_t)tile * 256 + d] = kFlagPrefix | (excl + total);
        }
        tile_off[d] = s.digit_base[d] + excl;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortKPT; ++j) {
        if (digit[j] < 256u) {
            const uint32_t pos = tile_off[digit[j]] + warp_cnt[warp][digit[j]] + rank[j];
            s.keys_out[pos] = key[j];
            s.vals_out[pos] = val[j];
        }
    }
}

// delta(i, j) (cuda_delta, bvh.cu:124-135)
__device__ __forceinline__ int kdelta(const uint32_t* __restrict__ m, int num_nodes, int i, int64_t j) {
    if (j < 0 || j > num_nodes) return -1;
    int d = __clz(m[i] ^ m[j]);
    if (d == 32) d += __clz((uint32_t)(i ^ (int)j));
    return d;
}

struct TopologyArgs {
    const uint32_t* morton;
    int32_t n;
    int32_t* left;
    int32_t* right;
    int32_t* parents;
    int32_t* range;
    const uint32_t* abort;  // set when the sort gave up: its order is not a permutation
};

__global__ void __launch_bounds__(256) lbvh_topology(TopologyArgs k) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = k.n, num_nodes = n - 1;
    if (i >= num_nodes || *k.abort != 0u) return;
    const uint32_t* m = k.morton;
    const int d = (kdelta(m, num_nodes, i, i + 1) - kdelta(m, num_nodes, i, i - 1)) < 0 ? -1 : 1;
    const int delta_min = kdelta(m, num_nodes, i, i - d);
    int64_t l_max = 128;
    while (kdelta(m, num_nodes, i, i + l_max * d) > delta_min) l_max *= 4;
    int64_t l = 0;
    for (int64_t t = l_max / 2; t > 0; t /= 2)
        if (kdelta(m, num_nodes, i, i + (l + t) * d) > delta_min) l += t;
    const int64_t j = i + l * d;
    const int delta_node = kdelta(m, num_nodes, i, j);
    int64_t s = 0, kk = 2, t = (l + kk - 1) / kk;
    while (true) {
        if (kdelta(m, num_nodes, i, i + (s + t) * d) > delta_node) s += t;
        if (t <= 1) break;
        kk *= 2;
        t = (l + kk - 1) / kk;
    }
    const int split = (int)(i + s * d + min(d, 0));
    const int lo = (int)min((int64_t)i, j), hi = (int)max((int64_t)i, j);
    const int lc = lo == split ? split : -(split + 1);
    const int rc = hi == split + 1 ? split + 1 : -(split + 2);
    k.left[i] = lc;
    k.right[i] = rc;
    k.range[2 * i] = lo;
    k.range[2 * i + 1] = hi;
    k.parents[lc >= 0 ? lc : n - (lc + 1)] = i;
    k.parents[rc >= 0 ? rc : n - (rc + 1)] = i;
    if (i == 0) k.parents[n] = -1;
}

// union of two cones; same operation order as the CPU build's cone_union
__device__ __forceinline__ float4 cone_union(float4 c1, float4 c2) {
    if (c1.w <= -1.0f || c2.w <= -1.0f) return make_float4(0.0f, 0.0f, 0.0f, -1.0f);
    const float sx = rn_add(c1.x, c2.x), sy = rn_add(c1.y, c2.y), sz = rn_add(c1.z, c2.z);
    const float l2 = rn_dot(sx, sy, sz, sx, sy, sz);
    if (!(l2 > 1e-12f)) return make_float4(0.0f, 0.0f, 0.0f, -1.0f);
    const float inv = rn_div(1.0f, rn_sqrt(l2));
    const float ax = rn_mul(sx, inv), ay = rn_mul(sy, inv), az = rn_mul(sz, inv);
    float res = 1.0f;
    const float4 ci[2] = {c1, c2};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        float d = rn_dot(ax, ay, az, ci[q].x, ci[q].y, ci[q].z);
        d = fminf(fmaxf(d, -1.0f), 1.0f);
        const float sd = rn_sqrt_z(fmaxf(0.0f, rn_sub(1.0f, rn_mul(d, d))));
        const float si = rn_sqrt_z(fmaxf(0.0f, rn_sub(1.0f, rn_mul(ci[q].w, ci[q].w))));
        const float v = ci[q].w < -d ? -1.0f : rn_sub(rn_mul(d, ci[q].w), rn_mul(sd, si));
        res = fminf(res, v);
    }
    return make_float4(ax, ay, az, res);
}

// What a merge needs of a node, and what the node's outputs are made of.  Representatives are kept as
// leaves, so that a merge moves two indices instead of their positions, normals and directions.
struct NodeState {
    float bb[6];          // box
    float L[3];           // summed radiance
    float Lp[3], A[3];    // the packed record's sums
    float4 dir;           // direction statistics {S, a}
    float4 cn, cw;        // normal and direction cones
    int size, rep, arep;  // leaves below; radiance and antiradiance representative (sorted leaf)
};
constexpr int kStateWords = 30;

// Merges two children into inner node t (record index); same operations and order as the CPU build's
// bottom-up pass.  In three independent parts, which lbvh_blocks gives to three threads: everything but
// the cones, and the two cones.
__device__ __forceinline__ void merge_sums(NodeState& o, const NodeState& l, const NodeState& r, uint32_t seed, int t,
                                           float* rnd_out) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        o.bb[q] = fminf(l.bb[q], r.bb[q]);
        o.bb[3 + q] = fmaxf(l.bb[3 + q], r.bb[3 + q]);
        o.L[q] = rn_add(l.L[q], r.L[q]);
        o.Lp[q] = rn_add(l.Lp[q], r.Lp[q]);
        o.A[q] = rn_add(l.A[q], r.A[q]);
    }
    // representative (cluster, bvh.cu:726-744)
    const float i1 = rn_sqrt_z(rn_dot(l.L[0], l.L[1], l.L[2], l.L[0], l.L[1], l.L[2]));
    const float i2 = rn_sqrt_z(rn_dot(r.L[0], r.L[1], r.L[2], r.L[0], r.L[1], r.L[2]));
    const float rnd = arc_node_random(seed, (uint32_t)t);
    const bool right = rnd > rn_div_z(i1, rn_add(i1, i2));
    o.rep = right ? r.rep : l.rep;
    o.size = l.size + r.size;
    // direction statistics, and the antiradiance representative: drawn in proportion to
    // antiradiance luminance with the same random number; its direction is the record's w
    o.dir = make_float4(rn_add(l.dir.x, r.dir.x), rn_add(l.dir.y, r.dir.y), rn_add(l.dir.z, r.dir.z),
                        rn_add(l.dir.w, r.dir.w));
    const bool aright = o.dir.w > 0.0f ? rnd > rn_div_z(l.dir.w, o.dir.w) : right;
    o.arep = aright ? r.arep : l.arep;
    *rnd_out = rnd;
}

struct BlockArgs {
    const uint32_t* abort;  // set when the sort gave up: its order is not a permutation
    uint32_t* err;
    const int32_t* sorted_index;
    ArcAvplsGpuParam a;
    const MaterialRecord* mats;
    int32_t num_mats;
    int32_t n;
    uint32_t seed;
    const int32_t* left;
    const int32_t* right;
    const int32_t* parents;
    const int32_t* range;  // [N-1][2]: first and last leaf of each inner node
    float4* records;       // [2N-1][4]
    float4* dirstat;       // [2N-1] {S.xyz, a}: a = sum of antiradiance luminances, S = sum of a_i w_i / |w_i|
    float4* bounds;        // [N-1][4]
    ArcAvplBvhNodeDataParam nd;
    ArcFloat3* sorted_pos;
    ArcFloat3* sorted_nrm;
    // the nodes that reach over a block's leaves, and the nodes below them
    float4* state;         // [cap][8]: NodeState of the blocks' roots from the front, of the top nodes from the end
    int32_t cap;           // >= roots + top nodes
    int32_t* visit;        // [N-1] of a top node: 1 + the state of the child that arrived first
    int32_t* roots;        // record indices of every block's roots
    int32_t* top;          // inner nodes above them
    int32_t* top_slot;     // [N-1] of a top node: its place in top
    int32_t* counts;       // roots, top nodes
};

__device__ __forceinline__ void store3(ArcFloat3* p, int64_t i, float x, float y, float z) {
    float* f = reinterpret_cast<float*>(p) + 3 * i;
    f[0] = x;
    f[1] = y;
    f[2] = z;
}

__device__ __forceinline__ void store_state(float4* state, int node, const NodeState& s) {
    float4* d = state + 8 * (size_t)node;
    d[0] = make_float4(s.bb[0], s.bb[1], s.bb[2], s.bb[3]);
    d[1] = make_float4(s.bb[4], s.bb[5], s.L[0], s.L[1]);
    d[2] = make_float4(s.L[2], s.Lp[0], s.Lp[1], s.Lp[2]);
    d[3] = make_float4(s.A[0], s.A[1], s.A[2], __int_as_float(s.size));
    d[4] = s.dir;
    d[5] = s.cn;
    d[6] = s.cw;
    d[7] = make_float4(__int_as_float(s.rep), __int_as_float(s.arep), 0.0f, 0.0f);
}

// (states are written and read by different blocks of one launch: through L2)
__device__ __forceinline__ NodeState load_state(const float4* state, int node) {
    const float4* p = state + 8 * (size_t)node;
    const float4 a = __ldcg(p), b = __ldcg(p + 1), c = __ldcg(p + 2), d = __ldcg(p + 3), h = __ldcg(p + 7);
    NodeState s;
    s.bb[0] = a.x; s.bb[1] = a.y; s.bb[2] = a.z; s.bb[3] = a.w;
    s.bb[4] = b.x; s.bb[5] = b.y;
    s.L[0] = b.z; s.L[1] = b.w; s.L[2] = c.x;
    s.Lp[0] = c.y; s.Lp[1] = c.z; s.Lp[2] = c.w;
    s.A[0] = d.x; s.A[1] = d.y; s.A[2] = d.z;
    s.size = __float_as_int(d.w);
    s.dir = __ldcg(p + 4);
    s.cn = __ldcg(p + 5);
    s.cw = __ldcg(p + 6);
    s.rep = __float_as_int(h.x);
    s.arep = __float_as_int(h.y);
    return s;
}

// Inner node k's outputs: record (representative p / n, antiradiance representative's w, summed L' and A,
// count), direction statistics, bounds and the reference's node data.
__device__ __forceinline__ void write_node(const BlockArgs& b, int k, int lc, int rc, const NodeState& s, float rnd,
                                           float3 p, float3 nr, float3 w, float3 aw, int mat) {
    const int64_t t = (int64_t)b.n + k;
    float4* rec = b.records + 4 * t;
    rec[0] = make_float4(p.x, p.y, p.z, nr.x);
    rec[1] = make_float4(nr.y, nr.z, aw.x, aw.y);
    rec[2] = make_float4(aw.z, s.Lp[0], s.Lp[1], s.Lp[2]);
    rec[3] = make_float4(s.A[0], s.A[1], s.A[2], (float)s.size);
    b.dirstat[t] = s.dir;
    float4* bd = b.bounds + 4 * (size_t)k;
    bd[0] = make_float4(s.bb[0], s.bb[1], s.bb[2], __int_as_float(lc));
    bd[1] = make_float4(s.bb[3], s.bb[4], s.bb[5], __int_as_float(rc));
    bd[2] = s.cn;
    bd[3] = s.cw;
    b.nd.randomNumbers[t] = rnd;
    b.nd.size[t] = s.size;
    b.nd.materialIndex[t] = mat;
    store3(b.nd.incRadiance, t, s.L[0], s.L[1], s.L[2]);
    store3(b.nd.position, t, p.x, p.y, p.z);
    store3(b.nd.normal, t, nr.x, nr.y, nr.z);
    store3(b.nd.incDirection, t, w.x, w.y, w.z);
}

constexpr int kBlockLeaves = 128;
constexpr int kMaxHeight = 63;  // a radix tree of 32-bit codes over 2^29 leaves has at most 61 levels
constexpr int kWRow = kStateWords;  // three more rows (leaves only): w as given
constexpr int kBlockSmem = (kStateWords * 2 + 3) * kBlockLeaves * 4;

// Bound by the latency of its phases and by the L1 / L2 accesses of 41 sectors per leaf (54% of L1, 604 MB of
// DRAM traffic): 1,000,003 leaves take 262 us, where one thread per leaf climbing through global memory took
// 600 us.  128 leaves per block leave five blocks per SM to overlap (256 leaves, three blocks: 396 us).
// One block per 128 sorted leaves; thread j owns leaf base + j and inner node base + j.  An inner node is
// one end of its own leaf range, so the nodes whose range lies inside the block are among those 128.
// They are merged by height (the longest path down), all nodes of a height in consecutive threads:
// climbing from the leaves instead keeps one or two lanes of every warp busy for the whole height.
__global__ void __launch_bounds__(kBlockLeaves) lbvh_blocks(BlockArgs b) {
    extern __shared__ float st[];  // [word][local node]: leaf j at j, inner node base + j at 128 + j
    __shared__ int s_mat[kBlockLeaves], s_src[kBlockLeaves];
    __shared__ int s_up[2 * kBlockLeaves];  // local parent (0 .. 127) or -1
    __shared__ short2 s_child[kBlockLeaves], s_rep[kBlockLeaves];
    __shared__ int2 s_link[kBlockLeaves];
    __shared__ int s_arrived[kBlockLeaves], s_height[kBlockLeaves];
    __shared__ int s_first[kMaxHeight + 2], s_list[kBlockLeaves];
    __shared__ float s_rnd[kBlockLeaves];
    __shared__ int s_count[2], s_base[2];
    if (*b.abort != 0u) return;  // uniform over the CTA: before any barrier
    const int j = threadIdx.x, base = blockIdx.x * kBlockLeaves, i = base + j, n = b.n;
    constexpr int kN = 2 * kBlockLeaves;
    auto put_sums = [&](int id, const NodeState& s) {
        float* d = st + id;
#pragma unroll
        for (int q = 0; q < 6; ++q) d[q * kN] = s.bb[q];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            d[(6 + q) * kN] = s.L[q];
            d[(9 + q) * kN] = s.Lp[q];
            d[(12 + q) * kN] = s.A[q];
        }
        d[15 * kN] = s.dir.x; d[16 * kN] = s.dir.y; d[17 * kN] = s.dir.z; d[18 * kN] = s.dir.w;
        d[27 * kN] = __int_as_float(s.size);
        d[28 * kN] = __int_as_float(s.rep);
        d[29 * kN] = __int_as_float(s.arep);
    };
    auto get_sums = [&](int id, NodeState& s) {
        const float* d = st + id;
#pragma unroll
        for (int q = 0; q < 6; ++q) s.bb[q] = d[q * kN];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            s.L[q] = d[(6 + q) * kN];
            s.Lp[q] = d[(9 + q) * kN];
            s.A[q] = d[(12 + q) * kN];
        }
        s.dir = make_float4(d[15 * kN], d[16 * kN], d[17 * kN], d[18 * kN]);
        s.size = __float_as_int(d[27 * kN]);
        s.rep = __float_as_int(d[28 * kN]);
        s.arep = __float_as_int(d[29 * kN]);
    };
    // which: 0 the normal cone, 1 the direction cone
    auto put_cone = [&](int id, int which, float4 c) {
        float* d = st + (19 + 4 * which) * kN + id;
        d[0] = c.x; d[kN] = c.y; d[2 * kN] = c.z; d[3 * kN] = c.w;
    };
    auto get_cone = [&](int id, int which) {
        const float* d = st + (19 + 4 * which) * kN + id;
        return make_float4(d[0], d[kN], d[2 * kN], d[3 * kN]);
    };
    auto get = [&](int id) {
        NodeState s;
        get_sums(id, s);
        s.cn = get_cone(id, 0);
        s.cw = get_cone(id, 1);
        return s;
    };
    // ---- topology of the block ----
    int lc = 0, rc = 0;
    bool local = false;
    if (i < n - 1) {
        const int2 rg = *reinterpret_cast<const int2*>(b.range + 2 * (size_t)i);
        lc = b.left[i];
        rc = b.right[i];
        local = rg.x >= base && rg.y < base + kBlockLeaves;
    }
    s_up[j] = s_up[kBlockLeaves + j] = -1;
    s_arrived[j] = s_height[j] = 0;
    static_assert(kBlockLeaves >= kMaxHeight + 2, "one thread per entry of s_first");
    if (j < kMaxHeight + 2) s_first[j] = 0;
    if (j < 2) s_count[j] = 0;
    __syncthreads();
    auto local_id = [&](int c) { return c >= 0 ? c - base : kBlockLeaves - (c + 1) - base; };
    if (local) {
        s_up[local_id(lc)] = j;
        s_up[local_id(rc)] = j;
        s_child[j] = make_short2((short)local_id(lc), (short)local_id(rc));
    }
    // ---- sorted leaf i ----
    // The three components of a vector are loaded by neighbouring lanes, so that each random access costs
    // the sectors it touches once, not once per component.
    s_src[j] = i < n ? b.sorted_index[i] : -1;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const int e = j + q * kBlockLeaves, m = e / 3, c = e - 3 * m, src = s_src[m];
        if (src >= 0) {
            auto f = [&](const ArcFloat3* v) { return reinterpret_cast<const float*>(v)[3 * (int64_t)src + c]; };
            const float p = f(b.a.position), nr = f(b.a.normal), w = f(b.a.incDirection), L = f(b.a.incRadiance),
                        A = f(b.a.antiradiance);
            st[c * kN + m] = p;
            st[(3 + c) * kN + m] = p;
            st[(19 + c) * kN + m] = nr;
            st[kWRow * kN + c * kBlockLeaves + m] = w;
            st[(6 + c) * kN + m] = L;
            st[(12 + c) * kN + m] = A;
        }
    }
    __syncthreads();
    if (i < n) {
        int mat = b.a.materialIndex[s_src[j]];
        if (mat < 0 || mat >= b.num_mats) {
            set_error(b.err, ARC_DEVERR_BAD_MATERIAL);
            mat = 0;
        }
        auto vec = [&](int r) { return f3(st[r * kN + j], st[(r + 1) * kN + j], st[(r + 2) * kN + j]); };
        const float3 p = vec(0), nr = vec(19), L = vec(6), A = vec(12);
        const float3 w = f3(st[kWRow * kN + j], st[kWRow * kN + kBlockLeaves + j], st[kWRow * kN + 2 * kBlockLeaves + j]);
        const float4 dif = b.mats[mat].diffuse_exp;
        const bool light = (w.x == 0.0f && w.y == 0.0f && w.z == 0.0f);
        NodeState s;
        s.bb[0] = s.bb[3] = p.x;
        s.bb[1] = s.bb[4] = p.y;
        s.bb[2] = s.bb[5] = p.z;
        s.L[0] = L.x; s.L[1] = L.y; s.L[2] = L.z;
        s.Lp[0] = light ? L.x : rn_mul(L.x, rn_mul(kOneOverPi, dif.x));
        s.Lp[1] = light ? L.y : rn_mul(L.y, rn_mul(kOneOverPi, dif.y));
        s.Lp[2] = light ? L.z : rn_mul(L.z, rn_mul(kOneOverPi, dif.z));
        s.A[0] = A.x; s.A[1] = A.y; s.A[2] = A.z;
        // leaf cones: (n, 1) and (w/|w|, 1), or the whole sphere when w = 0
        s.cn = make_float4(nr.x, nr.y, nr.z, 1.0f);
        const float ww = rn_dot(w.x, w.y, w.z, w.x, w.y, w.z);
        const float a_lum = rn_add(rn_add(rn_mul(0.2126f, A.x), rn_mul(0.7152f, A.y)), rn_mul(0.0722f, A.z));
        if (ww > 0.0f) {
            const float inv = rn_div(1.0f, rn_sqrt(ww));
            s.cw = make_float4(rn_mul(w.x, inv), rn_mul(w.y, inv), rn_mul(w.z, inv), 1.0f);
            s.dir = make_float4(rn_mul(a_lum, s.cw.x), rn_mul(a_lum, s.cw.y), rn_mul(a_lum, s.cw.z), a_lum);
        } else {
            s.cw = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
            s.dir = make_float4(0.0f, 0.0f, 0.0f, a_lum);
        }
        s.size = 1;
        s.rep = s.arep = i;
        put_sums(j, s);
        put_cone(j, 0, s.cn);
        put_cone(j, 1, s.cw);
        s_mat[j] = mat;
        b.dirstat[i] = s.dir;
        b.nd.size[i] = 1;
        b.nd.materialIndex[i] = mat;
        b.nd.randomNumbers[i] = arc_node_random(b.seed, (uint32_t)i);
    }
    __syncthreads();
    // ---- heights: the second arrival at a node carries its height up ----
    if (i < n) {
        int h = 0;
        for (int u = s_up[j]; u >= 0; u = s_up[kBlockLeaves + u]) {
            atomicMax(&s_height[u], h + 1);
            __threadfence_block();
            if (atomicAdd(&s_arrived[u], 1) == 0) break;
            __threadfence_block();
            h = *reinterpret_cast<volatile int*>(&s_height[u]);
        }
    }
    __syncthreads();
    const int height = local ? min(s_height[j], kMaxHeight) : 0;
    int rank = 0;
    if (local) rank = atomicAdd(&s_first[height + 1], 1);
    __syncthreads();
    if (j < 32) {  // s_first[h]: nodes of height < h, h = 1 .. 64 (two per lane)
        static_assert(kMaxHeight + 1 == 64, "two entries per lane");
        const int x = s_first[1 + 2 * j], y = s_first[2 + 2 * j];
        int incl = x + y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (j >= o) incl += v;
        }
        s_first[1 + 2 * j] = incl - y;
        s_first[2 + 2 * j] = incl;
    }
    __syncthreads();
    if (local) s_list[s_first[height] + rank] = j;
    __syncthreads();
    const int total = s_first[kMaxHeight + 1];
    // ---- merges, height by height ----
    for (int h = 1; s_first[h] < total; ++h) {
        const int first = s_first[h], count = s_first[h + 1] - first;
        // three threads per node: the sums, the normal cone, the direction cone
        for (int q = j; q < 3 * count; q += kBlockLeaves) {
            const int part = q >= 2 * count ? 2 : q >= count ? 1 : 0;
            const int k = s_list[first + q - part * count];
            const short2 c = s_child[k];
            if (part == 0) {
                NodeState l, r, o;
                get_sums(c.x, l);
                get_sums(c.y, r);
                merge_sums(o, l, r, b.seed, n + base + k, &s_rnd[k]);
                put_sums(kBlockLeaves + k, o);
            } else {
                put_cone(kBlockLeaves + k, part - 1, cone_union(get_cone(c.x, part - 1), get_cone(c.y, part - 1)));
            }
        }
        __syncthreads();
    }
    // ---- outputs, consecutive threads to consecutive words ----
    // (32-byte sectors half written by each store of a thread's own record cost 50 sector accesses per
    // leaf instead of 20.)  The slots of inner nodes that reach over the block are written too, with
    // values that lbvh_top_nodes replaces.
    const int leaves = min(kBlockLeaves, n - base), nodes = min(kBlockLeaves, n - 1 - base);
    const bool has_node = i < n - 1;
    NodeState s;
    if (local) s = get(kBlockLeaves + j);
    const int rl = local ? s.rep - base : 0, al = local ? s.arep - base : 0;  // both lie in the node's range
    s_rep[j] = make_short2((short)rl, (short)al);
    if (has_node) {
        const int64_t t = (int64_t)n + i;
        b.dirstat[t] = local ? s.dir : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        b.nd.size[t] = local ? s.size : 0;
        b.nd.randomNumbers[t] = local ? s_rnd[j] : 0.0f;
        b.nd.materialIndex[t] = s_mat[rl];
    }
    s_link[j] = make_int2(lc, rc);
    __syncthreads();
    {
        // 16-byte quarter of a record or bounds entry that this thread writes (the same for each pass)
        const int quarter = j & 3;
        auto w_at = [&](int c, int leaf) { return st[kWRow * kN + c * kBlockLeaves + leaf]; };
        auto row = [&](int r, int id) { return st[r * kN + id]; };
        for (int e = j; e < 4 * kBlockLeaves; e += kBlockLeaves) {
            const int m = e >> 2, own = kBlockLeaves + m;
            const int r = s_rep[m].x, ar = s_rep[m].y;
            float4 lf, nf, bf;
            if (quarter == 0) {
                lf = make_float4(row(0, m), row(1, m), row(2, m), row(19, m));
                nf = make_float4(row(0, r), row(1, r), row(2, r), row(19, r));
                bf = make_float4(row(0, own), row(1, own), row(2, own), __int_as_float(s_link[m].x));
            } else if (quarter == 1) {
                lf = make_float4(row(20, m), row(21, m), w_at(0, m), w_at(1, m));
                nf = make_float4(row(20, r), row(21, r), w_at(0, ar), w_at(1, ar));
                bf = make_float4(row(3, own), row(4, own), row(5, own), __int_as_float(s_link[m].y));
            } else if (quarter == 2) {
                lf = make_float4(w_at(2, m), row(9, m), row(10, m), row(11, m));
                nf = make_float4(w_at(2, ar), row(9, own), row(10, own), row(11, own));
                bf = make_float4(row(19, own), row(20, own), row(21, own), row(22, own));
            } else {
                lf = make_float4(row(12, m), row(13, m), row(14, m), 1.0f);
                nf = make_float4(row(12, own), row(13, own), row(14, own), (float)__float_as_int(row(27, own)));
                bf = make_float4(row(23, own), row(24, own), row(25, own), row(26, own));
            }
            if (m < leaves) b.records[4 * (size_t)base + e] = lf;
            if (m < nodes) {
                b.records[4 * ((size_t)n + base) + e] = nf;
                b.bounds[4 * (size_t)base + e] = bf;
            }
        }
        // reference node-data layout (AvplBvhNodeData, bvh.cu:673-724, sorted as bvh.cu:793-808)
        for (int e = j; e < 3 * kBlockLeaves; e += kBlockLeaves) {
            const int m = e / 3, c = e - 3 * m, own = kBlockLeaves + m, r = s_rep[m].x;
            const int64_t lo = 3 * (int64_t)base + e, no = 3 * ((int64_t)n + base) + e;
            auto f = [](ArcFloat3* p) { return reinterpret_cast<float*>(p); };
            if (m < leaves) {
                const float p = row(c, m), nr = row(19 + c, m);
                f(b.nd.position)[lo] = p;
                f(b.nd.normal)[lo] = nr;
                f(b.nd.incRadiance)[lo] = row(6 + c, m);
                f(b.nd.incDirection)[lo] = w_at(c, m);
                f(b.sorted_pos)[lo] = p;
                f(b.sorted_nrm)[lo] = nr;
            }
            if (m < nodes) {
                f(b.nd.position)[no] = row(c, r);
                f(b.nd.normal)[no] = row(19 + c, r);
                f(b.nd.incRadiance)[no] = row(6 + c, own);
                f(b.nd.incDirection)[no] = w_at(c, r);
            }
        }
    }
    // ---- what is left to lbvh_climb: roots of the block (nodes whose parent reaches over it) ----
    const bool leaf_root = i < n && s_up[j] < 0, node_root = local && s_up[kBlockLeaves + j] < 0;
    const bool above = has_node && !local;
    int slot[3] = {0, 0, 0};
    if (leaf_root) slot[0] = atomicAdd(&s_count[0], 1);
    if (node_root) slot[1] = atomicAdd(&s_count[0], 1);
    if (above) slot[2] = atomicAdd(&s_count[1], 1);
    __syncthreads();
    if (j < 2) s_base[j] = atomicAdd(&b.counts[j], s_count[j]);
    __syncthreads();
    // (all within cap in a valid tree, see state_capacity)
    bool fits = true;
    if (leaf_root) {
        const int q = s_base[0] + slot[0];
        fits = q < b.cap;
        if (fits) {
            b.roots[q] = i;
            store_state(b.state, q, get(j));
        }
    }
    if (node_root) {
        const int q = s_base[0] + slot[1];
        fits = fits && q < b.cap;
        if (q < b.cap) {
            b.roots[q] = n + i;
            store_state(b.state, q, s);
        }
    }
    if (above) {
        const int q = s_base[1] + slot[2];
        fits = fits && q < b.cap;
        if (q < b.cap) b.top[q] = i;
        b.top_slot[i] = q;
        b.visit[i] = 0;
    }
    if (!fits) set_error(b.err, ARC_DEVERR_BAD_NODE);
}

// States that a tree of `blocks` blocks keeps: a node over a boundary between two blocks is one of a chain of at
// most kMaxHeight such nodes, T of them in all; they have T + 1 roots below them.  (126 B per leaf; a state
// for every node would take 256.)
inline int32_t state_capacity(int32_t n, int blocks) {
    return (int32_t)std::min<int64_t>(2 * (int64_t)n - 1, 2 * (int64_t)kMaxHeight * (blocks - 1) + 1);
}

// From every block root towards the tree's root: at each inner node above the blocks the first thread to
// arrive leaves its state's place and stops, and the second merges the two states.
__global__ void __launch_bounds__(128) lbvh_climb(BlockArgs b) {
    if (*b.abort != 0u) return;
    const int n = b.n, roots = min(b.counts[0], b.cap);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < roots; q += gridDim.x * blockDim.x) {
        int node = b.roots[q], own = q;
        int parent = b.parents[node];
        // a valid tree reaches the root within n - 1 steps; the bound guards against a corrupt one
        for (int steps = 0; parent >= 0; ++steps) {
            if (steps >= n || parent >= n - 1) {
                set_error(b.err, ARC_DEVERR_BAD_NODE);
                break;
            }
            const int k = parent;
            const int lc = b.left[k], slot = b.top_slot[k];
            parent = b.parents[n + k];
            __threadfence();  // release this thread's state of the child
            const int other = atomicExch(&b.visit[k], own + 1) - 1;
            if (other < 0) break;
            __threadfence();  // acquire the sibling's
            if (other >= b.cap || (unsigned)slot >= (unsigned)b.cap) {
                set_error(b.err, ARC_DEVERR_BAD_NODE);
                break;
            }
            const bool is_left = (lc >= 0 ? lc : n - (lc + 1)) == node;
            const NodeState l = load_state(b.state, is_left ? own : other),
                            r = load_state(b.state, is_left ? other : own);
            float rnd;
            NodeState o;
            merge_sums(o, l, r, b.seed, n + k, &rnd);
            o.cn = cone_union(l.cn, r.cn);
            o.cw = cone_union(l.cw, r.cw);
            node = n + k;
            own = b.cap - 1 - slot;
            store_state(b.state, own, o);
        }
    }
}

// Outputs of the nodes above the blocks, one thread each.
__global__ void __launch_bounds__(128) lbvh_top_nodes(BlockArgs b) {
    if (*b.abort != 0u) return;
    const int n = b.n, count = min(b.counts[1], b.cap);
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
        const int k = b.top[q];
        const NodeState s = load_state(b.state, b.cap - 1 - q);
        const float4* r = b.records + 4 * (size_t)s.rep;
        const float4* ra = b.records + 4 * (size_t)s.arep;
        const float4 q0 = r[0], q1 = r[1], a1 = ra[1];
        write_node(b, k, b.left[k], b.right[k], s, arc_node_random(b.seed, (uint32_t)(n + k)), f3(q0.x, q0.y, q0.z),
                   f3(q0.w, q1.x, q1.y), f3(q1.z, q1.w, r[2].x), f3(a1.z, a1.w, ra[2].x),
                   b.nd.materialIndex[s.rep]);
    }
}

__global__ void lbvh_reference_nodes(int32_t num_nodes, const float4* bounds, ArcBvhNode* nodes) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= num_nodes) return;
    const float4 b0 = bounds[4 * (size_t)k], b1 = bounds[4 * (size_t)k + 1];
    ArcBvhNode nd;
    nd.left = __float_as_int(b0.w);
    nd.right = __float_as_int(b1.w);
    nd.bbMin = ArcFloat3{b0.x, b0.y, b0.z};
    nd.bbMax = ArcFloat3{b1.x, b1.y, b1.z};
    nd.visited = 2;  // both children merged
    nodes[k] = nd;
}

template <typename T>
arc_status get(arc_lbvh* bvh, const char* name, size_t count, T** out) {
    return bvh->arena.get(name, sizeof(T) * (count > 0 ? count : 1), reinterpret_cast<void**>(out));
}

}  // namespace

arc_status launch_lbvh_build(arc_lbvh* bvh, const ArcAvplsGpuParam* avpls, const ArcLbvhParams* p) {
    arc_context* ctx = bvh->ctx;
    const int32_t n = avpls->numAvpls;
    if (n < 2) {
        set_last_error("not enough points for bvh construction (need >= 2 AVPLs)");
        return ARC_ERR_TOO_FEW_AVPLS;
    }
    ARC_CHECK_ARG(n < (1 << 29), "too many AVPLs for the LBVH (max 2^29 - 1)");
    ARC_CHECK_ARG(ctx->num_materials > 0, "materials not uploaded");
    ARC_CHECK_ARG(p->bbox_mode == ARC_BBOX_SCENE || p->bbox_mode == ARC_BBOX_AVPL_REFERENCE, "bad bbox_mode");
    cudaStream_t st = ctx->stream;
    const int total = 2 * n - 1;
    // Keys per thread of a sort pass: few for small inputs, whose passes are one tile's latency (four
    // passes over 16,384 keys: 36 / 37 / 50 us with 4 / 8 / 16), many for large ones, whose tiles wait on
    // each other in a row (262,144: 66 / 52 / 59 us; 1,000,003: 273 / 153 / 109 us).
    const int kpt = n <= (1 << 16) ? 4 : n <= (1 << 19) ? 8 : 16;
    const int tiles = (n + kSortThreads * kpt - 1) / (kSortThreads * kpt);

    uint32_t *keys0, *keys1, *hist, *status, *bb;
    int32_t *vals0, *vals1, *left, *right, *parents, *range;
    float4 *records, *bounds, *dirstat;
    BlockArgs bu;
    ARC_TRY(get(bvh, "keys0", n, &keys0));
    ARC_TRY(get(bvh, "keys1", n, &keys1));
    ARC_TRY(get(bvh, "vals0", n, &vals0));
    ARC_TRY(get(bvh, "vals1", n, &vals1));
    // hist[4*256] | tile counters[4] | root and top node counts[2] | abort word | bbox[12] share one block,
    // zeroed but for the box
    ARC_TRY(get(bvh, "hist", 1024 + 4 + 2 + 1 + 12, &hist));
    ARC_TRY(get(bvh, "status", (size_t)4 * tiles * 256, &status));
    ARC_TRY(get(bvh, "left", n - 1, &left));
    ARC_TRY(get(bvh, "right", n - 1, &right));
    ARC_TRY(get(bvh, "parents", total, &parents));
    ARC_TRY(get(bvh, "range", 2 * (n - 1), &range));
    ARC_TRY(get(bvh, "visit", n - 1, &bu.visit));
    const int blocks = (n + kBlockLeaves - 1) / kBlockLeaves;
    bu.cap = state_capacity(n, blocks);
    ARC_TRY(get(bvh, "roots", bu.cap, &bu.roots));
    ARC_TRY(get(bvh, "top", bu.cap, &bu.top));
    ARC_TRY(get(bvh, "top_slot", n - 1, &bu.top_slot));
    ARC_TRY(get(bvh, "records", (size_t)4 * total, &records));
    ARC_TRY(get(bvh, "dirstat", total, &dirstat));
    ARC_TRY(get(bvh, "bounds", (size_t)4 * (n - 1), &bounds));
    ARC_TRY(get(bvh, "state", (size_t)8 * bu.cap, &bu.state));
    ArcAvplBvhNodeDataParam nd;
    ARC_TRY(get(bvh, "nd_size", total, &nd.size));
    ARC_TRY(get(bvh, "nd_mat", total, &nd.materialIndex));
    ARC_TRY(get(bvh, "nd_rand", total, &nd.randomNumbers));
    ARC_TRY(get(bvh, "nd_pos", total, &nd.position));
    ARC_TRY(get(bvh, "nd_nrm", total, &nd.normal));
    ARC_TRY(get(bvh, "nd_L", total, &nd.incRadiance));
    ARC_TRY(get(bvh, "nd_w", total, &nd.incDirection));
    ARC_TRY(get(bvh, "sorted_pos", n, &bvh->sorted_positions));
    ARC_TRY(get(bvh, "sorted_nrm", n, &bvh->sorted_normals));
    uint32_t* tile_counters = hist + 1024;
    bu.counts = reinterpret_cast<int32_t*>(hist + 1024 + 4);
    uint32_t* abort = hist + 1024 + 4 + 2;
    bb = abort + 1;

    ARC_TRY_CUDA(cudaMemsetAsync(hist, 0, sizeof(uint32_t) * (1024 + 4 + 2 + 1), st));
    ARC_TRY_CUDA(cudaMemsetAsync(status, 0, sizeof(uint32_t) * 4 * (size_t)tiles * 256, st));

    const int grid_stride_blocks = ctx->sm_count * 4;
    stage_begin(ctx, "lbvh_morton");
    const bool need_box = p->bbox_mode == ARC_BBOX_AVPL_REFERENCE || p->consider_normals;
    if (need_box) {
        lbvh_bbox_init<<<1, 32, 0, st>>>(bb);
        lbvh_bbox<<<grid_stride_blocks, 256, 0, st>>>(*avpls, bb, p->consider_normals);
        ARC_TRY_CUDA(cudaGetLastError());
    }
    MortonArgs m;
    m.a = *avpls;
    m.bb = bb;
    m.smin = make_float3(p->scene_min.x, p->scene_min.y, p->scene_min.z);
    m.smax = make_float3(p->scene_max.x, p->scene_max.y, p->scene_max.z);
    m.use_avpl_box = p->bbox_mode == ARC_BBOX_AVPL_REFERENCE;
    m.consider_normals = p->consider_normals;
    m.keys = keys0;
    m.vals = vals0;
    m.hist = hist;
    lbvh_morton<<<grid_stride_blocks, 256, 0, st>>>(m);
    lbvh_scan_hist<<<1, 256, 0, st>>>(hist);
    stage_end(ctx, need_box ? 4 : 2);
    ARC_TRY_CUDA(cudaGetLastError());
    stage_begin(ctx, "lbvh_sort");

    uint32_t* kin = keys0;
    uint32_t* kout = keys1;
    int32_t* vin = vals0;
    int32_t* vout = vals1;
    for (int pass = 0; pass < 4; ++pass) {
        SortPassArgs s;
        s.keys_in = kin;
        s.vals_in = vin;
        s.keys_out = kout;
        s.vals_out = vout;
        s.digit_base = hist + 256 * pass;
        s.status = status + (size_t)pass * tiles * 256;
        s.tile_counter = tile_counters + pass;
        s.n = n;
        s.shift = 8 * pass;
        s.pass = pass;
        s.spin_limit = p->wait_limit ? p->wait_limit : (1u << 26);
        s.abort = abort;
        s.err = ctx->d_error;
        auto* pass_kernel = kpt == 4 ? lbvh_sort_pass<4> : kpt == 8 ? lbvh_sort_pass<8> : lbvh_sort_pass<16>;
        pass_kernel<<<tiles, kSortThreads, 0, st>>>(s);
        ARC_TRY_CUDA(cudaGetLastError());
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    // after 4 passes the sorted data is back in keys0 / vals0
    stage_end(ctx, 4);
    stage_begin(ctx, "lbvh_karras");

    TopologyArgs k;
    k.morton = kin;
    k.n = n;
    k.left = left;
    k.right = right;
    k.parents = parents;
    k.range = range;
    k.abort = abort;
    lbvh_topology<<<(n - 1 + 255) / 256, 256, 0, st>>>(k);
    stage_end(ctx, 1);
    ARC_TRY_CUDA(cudaGetLastError());

    bu.abort = abort;
    bu.err = ctx->d_error;
    bu.sorted_index = vin;
    bu.a = *avpls;
    bu.mats = ctx->d_materials;
    bu.num_mats = ctx->num_materials;
    bu.n = n;
    bu.seed = p->repr_seed;
    bu.left = left;
    bu.right = right;
    bu.parents = parents;
    bu.range = range;
    bu.records = records;
    bu.dirstat = dirstat;
    bu.bounds = bounds;
    bu.nd = nd;
    bu.sorted_pos = bvh->sorted_positions;
    bu.sorted_nrm = bvh->sorted_normals;
    stage_begin(ctx, "lbvh_bottom_up");
    ARC_TRY_CUDA(cudaFuncSetAttribute(lbvh_blocks, cudaFuncAttributeMaxDynamicSharedMemorySize, kBlockSmem));
    lbvh_blocks<<<blocks, kBlockLeaves, kBlockSmem, st>>>(bu);
    // One block settles its whole tree: nothing is left to climb (128 leaves 64 us, 129 with the two
    // launches 90 us).
    if (blocks > 1) {
        // (a block has about ten roots)
        const int top_blocks = std::min(blocks, ctx->sm_count * 8);
        lbvh_climb<<<top_blocks, 128, 0, st>>>(bu);
        lbvh_top_nodes<<<top_blocks, 128, 0, st>>>(bu);
    }
    stage_end(ctx, blocks > 1 ? 3 : 1);
    ARC_TRY_CUDA(cudaGetLastError());

    bvh->n = n;
    ArcLbvhView& v = bvh->view;
    v.num_leaves = n;
    v.num_nodes = n - 1;
    v.morton = kin;
    v.sorted_index = vin;
    v.left = left;
    v.right = right;
    v.parents = parents;
    v.range = range;
    v.bounds = reinterpret_cast<const float*>(bounds);
    v.records = reinterpret_cast<const float*>(records);
    v.node_data = nd;
    v.dirstat = reinterpret_cast<const float*>(dirstat);
    bvh->has_reference_nodes = false;
    if (p->wait_limit != 0) {
        // a caller-chosen wait limit: learn now whether the sort gave up, and if it did leave the
        // object unbuilt (its arrays hold no tree) and report the timeout
        uint32_t aborted = 0;
        ARC_TRY_CUDA(cudaMemcpyAsync(&aborted, abort, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        ARC_TRY_CUDA(cudaStreamSynchronize(st));
        if (aborted) {
            bvh->n = 0;
            set_last_error("LBVH build: the radix sort's look-back gave up after " + std::to_string(p->wait_limit) +
                           " polls (pass " + std::to_string(aborted - 1) + ")");
            return ARC_ERR_TIMEOUT;
        }
    }
    return ARC_OK;
}

arc_status launch_lbvh_reference_nodes(arc_lbvh* bvh) {
    const int32_t n = bvh->n;
    ArcBvhNode* nodes = nullptr;
    ARC_TRY(bvh->arena.get("ref_nodes", sizeof(ArcBvhNode) * (size_t)(n - 1), reinterpret_cast<void**>(&nodes)));
    stage_begin(bvh->ctx, "lbvh_reference_nodes");
    lbvh_reference_nodes<<<(n - 1 + 255) / 256, 256, 0, bvh->ctx->stream>>>(
        n - 1, reinterpret_cast<const float4*>(bvh->view.bounds), nodes);
    stage_end(bvh->ctx, 1);
    ARC_TRY_CUDA(cudaGetLastError());
    bvh->ref_param.numLeafs = n;
    bvh->ref_param.numNodes = n - 1;
    bvh->ref_param.nodes = nodes;
    bvh->ref_param.positions = bvh->sorted_positions;
    bvh->ref_param.normals = bvh->sorted_normals;
    bvh->ref_data = bvh->view.node_data;
    bvh->has_reference_nodes = true;
    return ARC_OK;
}

}  // namespace arc
