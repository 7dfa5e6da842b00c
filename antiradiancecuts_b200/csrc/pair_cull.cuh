// Exact culling of (pixel, record) pairs a block at a time, for the gathers that evaluate every
// record for a block of pixels.
//
// A pair adds radiance only when the record lies in front of the pixel and faces it (n.d > 0 and
// n_a.d < 0, d = p_a - p), and antiradiance only when the pixel also lies inside the record's cone
// -- in a room about half of the records never light a given 16 x 16 pixel tile and 2-7% of them
// reach it with antiradiance (a record carries no antiradiance after a direct hit and no radiance
// after its path ended).  So each thread first tests one record against the bounds of the block's
// pixels, the block keeps the records that can contribute in two compact lists, and the pair loops
// run over those: the radiance loop without the cone test, the cone loop over the few records
// that need it.
//
// A record is dropped only when every pair with it is certain to add exactly 0:
//   * the terms of n.d are bounded per axis over the pixels' position and normal boxes; when every
//     bound is <= 0 each pair's product terms are <= 0 whatever the rounding, and otherwise the sum
//     must clear the rounding of a three-term dot product (4 ulp of the terms' magnitudes);
//   * a record with a non-finite radiance or antiradiance is kept (0 times it is not 0), and every
//     comparison with a NaN keeps the record.
#ifndef ARC_PAIR_CULL_CUH_
#define ARC_PAIR_CULL_CUH_

#include <cfloat>

#include "device_common.cuh"

namespace arc {

// Bounds of a group of pixels: positions and unit normals, per axis.
struct PixelBounds {
    float pmin[3], pmax[3], nmin[3], nmax[3];

    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            pmin[k] = nmin[k] = FLT_MAX;
            pmax[k] = nmax[k] = -FLT_MAX;
        }
    }
    __device__ __forceinline__ void add(float px, float py, float pz, float nx0, float ny0, float nz0, float nx1,
                                        float ny1, float nz1) {
        const float p[3] = {px, py, pz}, a[3] = {nx0, ny0, nz0}, b[3] = {nx1, ny1, nz1};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            pmin[k] = fminf(pmin[k], p[k]);
            pmax[k] = fmaxf(pmax[k], p[k]);
            nmin[k] = fminf(nmin[k], a[k]);
            nmax[k] = fmaxf(nmax[k], b[k]);
        }
    }
    // over the 32 lanes of a warp, result in every lane
    __device__ __forceinline__ void reduce_warp() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                pmin[k] = fminf(pmin[k], __shfl_xor_sync(0xffffffffu, pmin[k], o));
                pmax[k] = fmaxf(pmax[k], __shfl_xor_sync(0xffffffffu, pmax[k], o));
                nmin[k] = fminf(nmin[k], __shfl_xor_sync(0xffffffffu, nmin[k], o));
                nmax[k] = fmaxf(nmax[k], __shfl_xor_sync(0xffffffffu, nmax[k], o));
            }
    }
    __device__ __forceinline__ void reduce_warp_positions() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                pmin[k] = fminf(pmin[k], __shfl_xor_sync(0xffffffffu, pmin[k], o));
                pmax[k] = fmaxf(pmax[k], __shfl_xor_sync(0xffffffffu, pmax[k], o));
            }
    }
    __device__ __forceinline__ void merge(const PixelBounds& b) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            pmin[k] = fminf(pmin[k], b.pmin[k]);
            pmax[k] = fmaxf(pmax[k], b.pmax[k]);
            nmin[k] = fminf(nmin[k], b.nmin[k]);
            nmax[k] = fmaxf(nmax[k], b.nmax[k]);
        }
    }
};

// Whether a dot product whose terms are at most v0, v1, v2 is certain to round to a value <= 0.
__device__ __forceinline__ bool dot_never_positive(float v0, float v1, float v2) {
    return (v0 <= 0.0f && v1 <= 0.0f && v2 <= 0.0f) ||
           v0 + v1 + v2 <= -1e-6f * (fabsf(v0) + fabsf(v1) + fabsf(v2));
}

struct RecordNeed {
    bool radiance, cone;
};

// Which sums the record {p, n}, {n, w}, {w, L'}, {A, .} can add to for the pixels within b.
// CONE: whether cone antiradiance is gathered (cos_thr: max(cos(half angle), 0.001)).
template <bool CONE>
__device__ __forceinline__ RecordNeed record_need(const PixelBounds& b, float4 q0, float4 q1, float4 q2, float4 q3,
                                                  float cos_thr) {
    const float p[3] = {q0.x, q0.y, q0.z}, n[3] = {q0.w, q1.x, q1.y}, w[3] = {q1.z, q1.w, q2.x};
    float recv[3], face[3], lo[3], hi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        lo[k] = p[k] - b.pmax[k];  // d = p_a - p lies in [lo, hi]
        hi[k] = p[k] - b.pmin[k];
        recv[k] = fmaxf(fmaxf(b.nmin[k] * lo[k], b.nmin[k] * hi[k]), fmaxf(b.nmax[k] * lo[k], b.nmax[k] * hi[k]));
        face[k] = fmaxf(-n[k] * lo[k], -n[k] * hi[k]);
    }
    const bool behind = dot_never_positive(recv[0], recv[1], recv[2]);
    const float ll = fabsf(q2.y) + fabsf(q2.z) + fabsf(q2.w);
    RecordNeed r;
    r.radiance = !(ll <= FLT_MAX) || (ll != 0.0f && !behind && !dot_never_positive(face[0], face[1], face[2]));
    r.cone = false;
    if (CONE) {
        // cos(angle) <= max of -w.d over the box / the distance to the box
        float u = 0.0f, s = 0.0f, d2 = 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float x = -w[k] * lo[k], y = -w[k] * hi[k];
            u += fmaxf(x, y);
            s += fmaxf(fabsf(x), fabsf(y));
            const float gap = fmaxf(0.0f, fmaxf(lo[k], -hi[k]));
            d2 += gap * gap;
        }
        const bool outside = u + 1e-5f * s < 0.99999f * cos_thr * sqrtf(d2);
        const float la = fabsf(q3.x) + fabsf(q3.y) + fabsf(q3.z);
        r.cone = !(la <= FLT_MAX) || (la != 0.0f && !behind && !outside);
    }
    return r;
}

// rsqrt of a normal positive number in one instruction: rsqrtf(x) without its denormal path (three
// more instructions per call without -ftz), the same result for the distances here, which are
// >= 1e-30.
__device__ __forceinline__ float rsqrt_normal(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// 1 / x in one instruction (1 ulp); x >= 1e-30, results below the smallest normal flush to 0
__device__ __forceinline__ float rcp_normal(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The packed FP32x2 pair loops, over lists of records interleaved two by two (kPairFloats floats
// per pair of records: float 2 f + h holds field f of record h).
//   radiance list: p, n, L' (9 fields);  cone list: p, w, A (9 fields)
constexpr int kPairFloats = 20;

// Writes one record's 9 fields as entry e of a list.
__device__ __forceinline__ void put_entry(float* list, int e, float a0, float a1, float a2, float b0, float b1,
                                          float b2, float c0, float c1, float c2) {
    float* d = list + (e >> 1) * kPairFloats + (e & 1);
    d[0] = a0; d[2] = a1; d[4] = a2;
    d[6] = b0; d[8] = b1; d[10] = b2;
    d[12] = c0; d[14] = c1; d[16] = c2;
}

// One pixel's packed constants: -p and the unit normal, each in both halves.
struct PixelPair {
    uint64_t px, py, pz, nx, ny, nz;
};

__device__ __forceinline__ PixelPair pixel_pair(float px, float py, float pz, float nx, float ny, float nz) {
    return PixelPair{f2(-px, -px), f2(-py, -py), f2(-pz, -pz), f2(nx, nx), f2(ny, ny), f2(nz, nz)};
}

// Radiance of two records: acc += L' max(n.d, 0) max(-n_a.d, 0) / (d^2 max(d^2, clamp^2)).  The
// two cosines' 1/|d| factors are taken together as one reciprocal of d^2 (no square root), and the
// maxima come after the products, so that a NaN or 0 x inf factor adds 0.
__device__ __forceinline__ void radiance_pair(const float* rec, const PixelPair& s, float inv_clamp2, uint64_t tiny2,
                                              uint64_t& r0, uint64_t& r1, uint64_t& r2) {
    const ulonglong2* q = reinterpret_cast<const ulonglong2*>(rec);
    const ulonglong2 f01 = q[0], f23 = q[1], f45 = q[2], f67 = q[3];
    const uint64_t f8 = *reinterpret_cast<const uint64_t*>(q + 4);
    const uint64_t dx = f2_add(f01.x, s.px), dy = f2_add(f01.y, s.py), dz = f2_add(f23.x, s.pz);
    float l0, l1;
    f2_split(f2_fma(dz, dz, f2_fma(dy, dy, f2_fma(dx, dx, tiny2))), l0, l1);  // >= 1e-30
    const float i0 = rcp_normal(l0), i1 = rcp_normal(l1);
    const uint64_t nd = f2_fma(s.nz, dz, f2_fma(s.ny, dy, f2_mul(s.nx, dx)));
    const uint64_t nad = f2_fma(f45.y, dz, f2_fma(f45.x, dy, f2_mul(f23.y, dx)));
    float a0, a1, b0, b1;
    f2_split(f2_mul(nd, f2(i0, i1)), a0, a1);
    f2_split(f2_mul(nad, f2(fminf(i0, inv_clamp2), fminf(i1, inv_clamp2))), b0, b1);
    const uint64_t g = f2_mul(f2(fmaxf(a0, 0.0f), fmaxf(a1, 0.0f)), f2(fmaxf(-b0, 0.0f), fmaxf(-b1, 0.0f)));
    r0 = f2_fma(f67.x, g, r0);
    r1 = f2_fma(f67.y, g, r1);
    r2 = f2_fma(f8, g, r2);
}

// Cone antiradiance of two records (the tests and the term of pair_terms).
__device__ __forceinline__ void cone_pair(const float* rec, const PixelPair& s, float cos_thr, float eps,
                                          float inv_clamp2, uint64_t tiny2, uint64_t& a0, uint64_t& a1, uint64_t& a2) {
    const ulonglong2* q = reinterpret_cast<const ulonglong2*>(rec);
    const ulonglong2 f01 = q[0], f23 = q[1], f45 = q[2], f67 = q[3];
    const uint64_t f8 = *reinterpret_cast<const uint64_t*>(q + 4);
    const uint64_t dx = f2_add(f01.x, s.px), dy = f2_add(f01.y, s.py), dz = f2_add(f23.x, s.pz);
    float l0, l1;
    f2_split(f2_fma(dz, dz, f2_fma(dy, dy, f2_fma(dx, dx, tiny2))), l0, l1);  // >= 1e-30
    const uint64_t r = f2(rsqrt_normal(l0), rsqrt_normal(l1));
    const uint64_t c1 = f2_mul(f2_fma(s.nz, dz, f2_fma(s.ny, dy, f2_mul(s.nx, dx))), r);
    const uint64_t wdr = f2_mul(f2_fma(f45.y, dz, f2_fma(f45.x, dy, f2_mul(f23.y, dx))), r);  // -cos
    float c1a, c1b, wa, wb, ra, rb, ia, ib;
    f2_split(c1, c1a, c1b);
    f2_split(wdr, wa, wb);
    f2_split(f2_mul(r, r), ra, rb);
    f2_split(f2_mul(c1, f2(fminf(ra, inv_clamp2), fminf(rb, inv_clamp2))), ia, ib);
    const uint64_t ga = f2((-wa > cos_thr && c1a > eps) ? ia : 0.0f, (-wb > cos_thr && c1b > eps) ? ib : 0.0f);
    a0 = f2_fma(f67.x, ga, a0);
    a1 = f2_fma(f67.y, ga, a1);
    a2 = f2_fma(f8, ga, a2);
}

}  // namespace arc

#endif  // ARC_PAIR_CULL_CUH_
