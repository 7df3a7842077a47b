// traverse.cuh - closest-hit and any-hit traversal of the two-level BVH4.
//
// Restates traceRayTracked / traceInstance / traceTriangle /
// intersectTriangle (shaders/traversal.slang:349-811) and traceOccluded /
// occludedInstance / occludedTriangle (shaders/traversal.slang:826-1046) on
// a 4-wide BVH whose child boxes are the reference's binary node boxes.
// Hit distances, triangles and instances are produced by the same watertight
// triangle test as the reference; equal distances resolve to the smaller
// (instance, triangle), which makes the answer independent of tree shape.
#pragma once
#include <type_traits>

#include "lux_internal.h"
#include "lux_math.cuh"

namespace lux {

constexpr uint32_t kMaxSteps = 4096u;  // MAX_TRAVERSAL_STEPS, shaders/traversal.slang:8
constexpr int kStack = 64;  // default traversal stack depth (entries)
// Stack of the flattened walk; deeper trees are not flattened.
constexpr int kFlatStack = 64;

struct Hit {
    float t;
    uint32_t tri, inst, errors;
    float b1, b2;
};

struct TraceCounters {
    uint32_t nodes, triangles, instances;
};

// boxRayInterval, shaders/traversal.slang:349-369, for one box.
__device__ __forceinline__ bool box_interval(f3 o, f3 d, float lx, float ly, float lz, float hx, float hy,
                                             float hz, float limit, float &entry, float &exit) {
    float near_t = 0.0f, far_t = limit;
    float lo[3] = {lx, ly, lz}, hi[3] = {hx, hy, hz};
    float oo[3] = {o.x, o.y, o.z}, dd[3] = {d.x, d.y, d.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (dd[a] == 0.0f) {
            if (oo[a] < lo[a] || oo[a] > hi[a]) {
                entry = 0.0f;
                exit = 0.0f;
                return false;
            }
        } else {
            float ta = (lo[a] - oo[a]) / dd[a];
            float tb = (hi[a] - oo[a]) / dd[a];
            float ax = fmaxf(ta, tb);
            near_t = fmaxf(near_t, fminf(ta, tb));
            far_t = fminf(far_t, ax + fabsf(ax) * 3.5762791e-7f);
        }
    }
    entry = near_t;
    exit = far_t;
    return near_t <= far_t;
}

// Per-ray slab constants for the BVH4 child tests.  The reference divides
// by the direction for every slab (shaders/traversal.slang:360-361); here a
// plane P of an axis lies at t = P / d - o / d, one fused multiply-add
// fma(P, inv, c) with inv = 1 / d and c = -o inv, and the child tests only
// have to be conservative: culling decides which triangles are tested, hit
// distances come from the exact triangle test.  The two constants of an axis
// are moved apart by e = kSlabPad (|o| + M) |inv|, M the largest coordinate
// magnitude of the boxes (the TLAS root box, or the instance's BLAS root box):
// the reciprocal (1 ulp), the product o inv, the sum c and the result round by
// at most 3.6e-7 (|o| + M) |inv| together, so each end keeps at least 6e-7
// |P - o| |inv| = 6e-7 t of margin, what a multiply by the correctly rounded
// reciprocal with 7.2e-7 relative padding kept.
//
// Why this form: the walk is bound by instruction issue at the occupancy its
// registers allow, and this needs both fewest: 24 multiply-adds per node for
// 24 subtracts and 24 multiplies, the padding in the constants, tmin and the
// limit folded into three-operand min / max, nine constants per ray.  Packed
// fma.rn.f32x2 (12 per node) was slower: its constants take register pairs
// (closest hits of the 1280x720 frame 1.26 ms against 1.18, visibility 2.90
// against 2.77).
//
// A zero (or below 1e-30) direction component takes inv = +-1e30: planes on
// either side of the origin are then beyond any distance, a box wholly on one
// side misses, and within e of the origin the axis does not constrain (the
// reference's inside test).  Constants that overflow, a direction too short
// for that (below 1e-15) or a component above 1e30 leave the axis
// unconstrained: inv = +-1e-30 with constants -+3e38, so every finite plane
// lies outside any interval while an empty slot's infinite planes (near +inf,
// far -inf on every axis) still fail the test.
constexpr float kSlabPad = 1.9e-6f;

struct SlabRay {
    float ix, iy, iz;       // 1 / d
    float nx, ny, nz;       // near planes: -o / d - e
    float fx, fy, fz;       // far planes: -o / d + e
};  // the sign bit of an inv selects the high plane as near

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// The rare rays of slab_ray: an axis whose fast constants are not finite (or
// below 1e-30 in inv).
__device__ __forceinline__ void slab_special(float o, float d, float pad, bool tiny, float &inv, float &near_c,
                                          float &far_c) {
    inv = fabsf(d) < 1e-30f ? copysignf(1e30f, d) : rcp_approx(d);
    const float c = o * inv, e = __fmaf_rn(fabsf(o), kSlabPad, pad) * fabsf(inv);
    near_c = -c - e;
    far_c = e - c;
    if (tiny || !(fabsf(c) + e < 1e37f) || fabsf(inv) < 1e-30f) {
        inv = copysignf(1e-30f, d);
        near_c = -3e38f;
        far_c = 3e38f;
    }
}

// pad: kSlabPad x M; with kEven the whole padding, the same on every axis.
template <bool kEven = false>
__device__ __forceinline__ SlabRay slab_ray(f3 o, f3 d, float pad) {
    SlabRay r;
    r.ix = rcp_approx(d.x);
    r.iy = rcp_approx(d.y);
    r.iz = rcp_approx(d.z);
    const float cx = o.x * r.ix, ex = (kEven ? pad : __fmaf_rn(fabsf(o.x), kSlabPad, pad)) * fabsf(r.ix);
    const float cy = o.y * r.iy, ey = (kEven ? pad : __fmaf_rn(fabsf(o.y), kSlabPad, pad)) * fabsf(r.iy);
    const float cz = o.z * r.iz, ez = (kEven ? pad : __fmaf_rn(fabsf(o.z), kSlabPad, pad)) * fabsf(r.iz);
    r.nx = -cx - ex;
    r.fx = ex - cx;
    r.ny = -cy - ey;
    r.fy = ey - cy;
    r.nz = -cz - ez;
    r.fz = ez - cz;
    // Common rays: every constant finite (an axis of d between 1e-30 and
    // 1e30 with room for the products) and the direction at least 1e-15 long.
    const float largest = max3(fabsf(r.ix), fabsf(r.iy), fabsf(r.iz)), least = min3(fabsf(r.ix), fabsf(r.iy), fabsf(r.iz));
    const float bound = (fabsf(cx) + ex) + (fabsf(cy) + ey) + (fabsf(cz) + ez);
    if (!(largest <= 1e30f && least >= 1e-30f && least <= 1e15f && bound < 1e37f)) {
        const bool tiny = max3(fabsf(d.x), fabsf(d.y), fabsf(d.z)) < 1e-15f;
        slab_special(o.x, d.x, pad, tiny, r.ix, r.nx, r.fx);
        slab_special(o.y, d.y, pad, tiny, r.iy, r.ny, r.fy);
        slab_special(o.z, d.z, pad, tiny, r.iz, r.nz, r.fz);
    }
    return r;
}

// Child tests of one BVH4 node.  Returns the hit mask and conservative entry
// distances (at least tmin >= 0); children that end before tmin or start
// after `limit` are culled, and so are empty slots.
__device__ __forceinline__ uint32_t node_test(const Bvh4Node *__restrict__ nodes, uint32_t index, const SlabRay &r,
                                              float limit, float tmin, float entry[4], uint32_t child[4]) {
    // Node rows: lo_x, hi_x, lo_y, hi_y, lo_z, hi_z, child.
    const float4 *p = reinterpret_cast<const float4 *>(nodes + index);
    const uint32_t sx = as_uint(r.ix) >> 31, sy = as_uint(r.iy) >> 31, sz = as_uint(r.iz) >> 31;
    const float4 nx = __ldg(p + sx), fx = __ldg(p + (1u - sx));
    const float4 ny = __ldg(p + 2u + sy), fy = __ldg(p + (3u - sy));
    const float4 nz = __ldg(p + 4u + sz), fz = __ldg(p + (5u - sz));
    const uint4 ch = __ldg(reinterpret_cast<const uint4 *>(p + 6));
    child[0] = ch.x;
    child[1] = ch.y;
    child[2] = ch.z;
    child[3] = ch.w;
    const float NX[4] = {nx.x, nx.y, nx.z, nx.w}, FX[4] = {fx.x, fx.y, fx.z, fx.w};
    const float NY[4] = {ny.x, ny.y, ny.z, ny.w}, FY[4] = {fy.x, fy.y, fy.z, fy.w};
    const float NZ[4] = {nz.x, nz.y, nz.z, nz.w}, FZ[4] = {fz.x, fz.y, fz.z, fz.w};
    uint32_t mask = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float near_t = max3(__fmaf_rn(NX[i], r.ix, r.nx), __fmaf_rn(NY[i], r.iy, r.ny),
                                  fmaxf(__fmaf_rn(NZ[i], r.iz, r.nz), tmin));
        const float far_t = min3(__fmaf_rn(FX[i], r.ix, r.fx), __fmaf_rn(FY[i], r.iy, r.fy),
                                 fminf(__fmaf_rn(FZ[i], r.iz, r.fz), limit));
        entry[i] = near_t;
        mask |= near_t <= far_t ? (1u << i) : 0u;
    }
    return mask;
}

// Slab tests of rays from far outside the scene: t = (plane - o) * inv with
// the correctly rounded reciprocal carries under 2 ulp, and the interval grows
// by 7.2e-7 relative on both ends.  SlabRay's padding is a part of the origin's
// magnitude on every axis; where that is many times the boxes, a walk meets so
// many of them that it runs into its step budget (2e5 units from a scene of 2
// units and 131,072 triangles: 790 nodes per ray and 16% of the rays abandoned;
// so 180 and none).  A zero direction component gives an infinite reciprocal:
// planes on either side of the origin give -inf/+inf (no constraint), a box
// wholly on one side misses, and a plane through the origin gives NaN, which
// fmaxf/fminf ignore.
struct FarSlabRay {
    float ox, oy, oz;
    float ix, iy, iz;
};
__device__ __forceinline__ void make_slab(FarSlabRay &r, f3 o, f3 d, float) {
    r = FarSlabRay{o.x, o.y, o.z, __frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z)};
}
__device__ __forceinline__ void make_slab(SlabRay &r, f3 o, f3 d, float pad) { r = slab_ray(o, d, pad); }
__device__ __forceinline__ uint32_t node_test(const Bvh4Node *__restrict__ nodes, uint32_t index, const FarSlabRay &r,
                                              float limit, float tmin, float entry[4], uint32_t child[4]) {
    const float4 *p = reinterpret_cast<const float4 *>(nodes + index);
    const uint32_t sx = as_uint(r.ix) >> 31, sy = as_uint(r.iy) >> 31, sz = as_uint(r.iz) >> 31;
    const float4 nx = __ldg(p + sx), fx = __ldg(p + (1u - sx));
    const float4 ny = __ldg(p + 2u + sy), fy = __ldg(p + (3u - sy));
    const float4 nz = __ldg(p + 4u + sz), fz = __ldg(p + (5u - sz));
    const uint4 ch = __ldg(reinterpret_cast<const uint4 *>(p + 6));
    child[0] = ch.x;
    child[1] = ch.y;
    child[2] = ch.z;
    child[3] = ch.w;
    const float NX[4] = {nx.x, nx.y, nx.z, nx.w}, FX[4] = {fx.x, fx.y, fx.z, fx.w};
    const float NY[4] = {ny.x, ny.y, ny.z, ny.w}, FY[4] = {fy.x, fy.y, fy.z, fy.w};
    const float NZ[4] = {nz.x, nz.y, nz.z, nz.w}, FZ[4] = {fz.x, fz.y, fz.z, fz.w};
    uint32_t mask = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float ax = (NX[i] - r.ox) * r.ix, bx = (FX[i] - r.ox) * r.ix;
        const float ay = (NY[i] - r.oy) * r.iy, by = (FY[i] - r.oy) * r.iy;
        const float az = (NZ[i] - r.oz) * r.iz, bz = (FZ[i] - r.oz) * r.iz;
        float near_t = fmaxf(fmaxf(ax, ay), fmaxf(az, 0.0f));
        float far_t = fminf(fminf(bx, by), bz);
        near_t = near_t - fabsf(near_t) * 7.2e-7f;
        far_t = far_t + fabsf(far_t) * 7.2e-7f;
        // An empty slot's inverted infinities come out NaN: every comparison fails.
        const bool hit = near_t <= far_t && near_t <= limit && far_t >= tmin;
        entry[i] = hit ? near_t : 0.0f;
        mask |= hit ? (1u << i) : 0u;
    }
    return mask;
}

// Whether a caller's ray starts so far outside (more than 8 times the scene
// box's largest coordinate magnitude M) that its padding would be large against
// the triangles: it takes the two-level walk then, by FarSlabRay.
constexpr float kFarOrigin = 8.0f;
__device__ __forceinline__ float largest_component(f3 v) { return max3(fabsf(v.x), fabsf(v.y), fabsf(v.z)); }
constexpr uint32_t kFarSteps = 0xffffffffu;  // `steps` of such a ray's walker
constexpr uint32_t kFarRay = 0x80000000u;    // and the errors it returns

struct TriRay {
    uint32_t kx, ky, kz;
    float sx, sy;
    bool valid;
};

// triangleRay, shaders/traversal.slang:399-413.
__device__ __forceinline__ TriRay triangle_ray(f3 d) {
    TriRay r{0, 0, 0, 0.0f, 0.0f, false};
    float mx = fabsf(d.x), my = fabsf(d.y), mz = fabsf(d.z);
    r.kz = mx > my ? (mx > mz ? 0u : 2u) : (my > mz ? 1u : 2u);
    float dz = comp(d, r.kz);
    r.valid = dz != 0.0f;
    if (!r.valid) return r;
    r.kx = (r.kz + 1u) % 3u;
    r.ky = (r.kx + 1u) % 3u;
    if (dz < 0.0f) {
        uint32_t t = r.kx;
        r.kx = r.ky;
        r.ky = t;
    }
    r.sx = comp(d, r.kx) / dz;
    r.sy = comp(d, r.ky) / dz;
    return r;
}

// orientedEdge, shaders/traversal.slang:379-392.
__device__ __forceinline__ float oriented_edge(float ax, float ay, float bx, float by) {
    bool reverse = ax > bx || (ax == bx && ay > by);
    float fx = reverse ? bx : ax, fy = reverse ? by : ay;
    float sx = reverse ? ax : bx, sy = reverse ? ay : by;
    float pa = fx * sy;
    float pb = fy * sx;
    float edge = pa - pb;
    float error = (fabsf(pa) + fabsf(pb)) * 2.3841858e-7f;
    if (fabsf(edge) <= error) edge = 0.0f;
    return reverse ? -edge : edge;
}

// intersectTriangle, shaders/traversal.slang:415-443.  Returns distance or -1.
__device__ __forceinline__ float intersect_triangle(f3 o, f3 d, const TriRay &ray, f3 A, f3 B, f3 C, float &w1,
                                                    float &w2) {
    if (!ray.valid) return -1.0f;
    f3 a = A - o, b = B - o, c = C - o;
    float akz = comp(a, ray.kz), bkz = comp(b, ray.kz), ckz = comp(c, ray.kz);
    float pax = comp(a, ray.kx) - ray.sx * akz, pay = comp(a, ray.ky) - ray.sy * akz;
    float pbx = comp(b, ray.kx) - ray.sx * bkz, pby = comp(b, ray.ky) - ray.sy * bkz;
    float pcx = comp(c, ray.kx) - ray.sx * ckz, pcy = comp(c, ray.ky) - ray.sy * ckz;
    float largest = fmaxf(fmaxf(fmaxf(fabsf(pax), fabsf(pay)), fmaxf(fabsf(pbx), fabsf(pby))),
                          fmaxf(fabsf(pcx), fabsf(pcy)));
    if (largest == 0.0f || !isfinite(largest)) return -1.0f;
    uint32_t exponent = (as_uint(largest) >> 23) & 255u;
    exponent = exponent < 1u ? 1u : (exponent > 253u ? 253u : exponent);
    float scale = as_float((254u - exponent) << 23);
    pax *= scale;
    pay *= scale;
    pbx *= scale;
    pby *= scale;
    pcx *= scale;
    pcy *= scale;
    float e0 = oriented_edge(pbx, pby, pcx, pcy);
    float e1 = oriented_edge(pcx, pcy, pax, pay);
    float e2 = oriented_edge(pax, pay, pbx, pby);
    bool any_neg = e0 < 0.0f || e1 < 0.0f || e2 < 0.0f;
    bool any_pos = e0 > 0.0f || e1 > 0.0f || e2 > 0.0f;
    if (any_neg && any_pos) return -1.0f;
    float det = (e0 + e1) + e2;
    if (det == 0.0f || !isfinite(det)) return -1.0f;
    float wx = e0 / det, wy = e1 / det, wz = e2 / det;
    float dist = ((wx * akz + wy * bkz) + wz * ckz) / comp(d, ray.kz);
    if (!isfinite(dist)) return -1.0f;
    w1 = wy;
    w2 = wz;
    return dist;
}

__device__ __forceinline__ bool hit_better(float t, uint32_t inst, uint32_t tri, const Hit &h) {
    if (t < h.t) return true;
    if (t > h.t || h.tri == kEmpty) return false;
    if (inst != h.inst) return inst < h.inst;
    return tri < h.tri;
}

// Face culling of traceTriangle / occludedTriangle (shaders/traversal.slang:449-453).
__device__ __forceinline__ bool cull_reject(uint32_t flags, f3 A, f3 B, f3 C, f3 d) {
    if ((flags & 3u) == 0u) return false;
    float facing = dot(cross(B - A, C - A), d) * ((flags & 4u) != 0u ? -1.0f : 1.0f);
    return ((flags & 1u) != 0u && facing >= 0.0f) || ((flags & 2u) != 0u && facing <= 0.0f);
}

__device__ __forceinline__ void load_triangle(const float4 *__restrict__ tris, uint32_t t, f3 &A, f3 &B, f3 &C) {
    float4 a = __ldg(tris + 3 * (size_t)t), b = __ldg(tris + 3 * (size_t)t + 1), c = __ldg(tris + 3 * (size_t)t + 2);
    A = f3{a.x, a.y, a.z};
    B = f3{b.x, b.y, b.z};
    C = f3{c.x, c.y, c.z};
}

// Local ray, shaders/traversal.slang:481-488.
__device__ __forceinline__ void local_ray(const DeviceInstance &I, f3 o, f3 d, f3 &lo, f3 &ld) {
    float r[3][4];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int c = 0; c < 4; ++c) r[k][c] = I.row[k][c];
    lo = f3{((r[0][0] * o.x + r[0][1] * o.y) + r[0][2] * o.z) + r[0][3] * 1.0f,
            ((r[1][0] * o.x + r[1][1] * o.y) + r[1][2] * o.z) + r[1][3] * 1.0f,
            ((r[2][0] * o.x + r[2][1] * o.y) + r[2][2] * o.z) + r[2][3] * 1.0f};
    ld = f3{((r[0][0] * d.x + r[0][1] * d.y) + r[0][2] * d.z) + r[0][3] * 0.0f,
            ((r[1][0] * d.x + r[1][1] * d.y) + r[1][2] * d.z) + r[1][3] * 0.0f,
            ((r[2][0] * d.x + r[2][1] * d.y) + r[2][2] * d.z) + r[2][3] * 0.0f};
}

__device__ __forceinline__ DeviceInstance load_instance(const DeviceInstance *__restrict__ inst, uint32_t i) {
    const float4 *p = reinterpret_cast<const float4 *>(inst + i);
    float4 r0 = __ldg(p), r1 = __ldg(p + 1), r2 = __ldg(p + 2);
    uint4 w = __ldg(reinterpret_cast<const uint4 *>(p + 3));
    DeviceInstance I;
    I.row[0][0] = r0.x; I.row[0][1] = r0.y; I.row[0][2] = r0.z; I.row[0][3] = r0.w;
    I.row[1][0] = r1.x; I.row[1][1] = r1.y; I.row[1][2] = r1.z; I.row[1][3] = r1.w;
    I.row[2][0] = r2.x; I.row[2][1] = r2.y; I.row[2][2] = r2.z; I.row[2][3] = r2.w;
    I.root = w.x;
    I.first = w.y;
    I.extent = as_float(w.z);
    I.flags = w.w;
    return I;
}

// Triangles of an instance, from its record in the scene words (word 8).
__device__ __forceinline__ uint32_t instance_triangles(const SceneView &S, uint32_t inst) {
    const uint4 h = __ldg(S.scene_words);
    return __ldg(S.scene_words + h.y + (size_t)inst * h.w + 8u).z;
}

// Largest coordinate magnitude of a box.
__device__ __forceinline__ float box_magnitude(f3 lo, f3 hi) {
    return fmaxf(max3(fabsf(lo.x), fabsf(lo.y), fabsf(lo.z)), max3(fabsf(hi.x), fabsf(hi.y), fabsf(hi.z)));
}

// Child ordering keys: the entry distance's bits (entries are >= 0, so the
// bits order like the values) with the low two bits replaced by the child
// slot; missed children get ~0 and sort last.  Truncating two mantissa bits
// only lowers a stored entry, which keeps the closest-hit pop test
// (skip when entry > best distance) conservative.
__device__ __forceinline__ uint32_t child_key(uint32_t mask, const float entry[4], int i) {
    return (mask & (1u << i)) ? ((as_uint(entry[i]) & ~3u) | (uint32_t)i) : 0xffffffffu;
}

__device__ __forceinline__ void key_swap(uint32_t &a, uint32_t &b) {
    uint32_t lo = min(a, b), hi = max(a, b);
    a = lo;
    b = hi;
}

__device__ __forceinline__ uint32_t key_child(uint32_t key, const uint32_t child[4]) {
    uint32_t s = key & 3u;
    return s == 0u ? child[0] : (s == 1u ? child[1] : (s == 2u ? child[2] : child[3]));
}

__device__ __forceinline__ float key_entry(uint32_t key) { return as_float(key & ~3u); }

// The barycentrics of a closest hit, worked out once when the query is
// complete: the winning triangle's test again from the same local ray.
__device__ __forceinline__ void hit_barycentrics(const SceneView &S, f3 o, f3 d, Hit &hit) {
    if (hit.tri == kEmpty) return;
    const DeviceInstance I = load_instance(S.instances, hit.inst);
    f3 lo, ld, A, B, C;
    local_ray(I, o, d, lo, ld);
    load_triangle(S.triangles, hit.tri, A, B, C);
    intersect_triangle(lo, ld, triangle_ray(ld), A, B, C, hit.b1, hit.b2);
}

// One warp's scratch for the cooperative leaf pass (shared memory): slot k is
// the k-th lane of the warp that reached a leaf in this round, and only that
// lane writes it.
struct LeafScratch {
    float ox[32], oy[32], oz[32], dx[32], dy[32], dz[32], sx[32], sy[32], lower[32], limit[32];
    uint32_t axes[32], flags[32], first[32];  // first: leaf's first triangle - the lane's pair prefix
    unsigned long long best[32];
};

    // The BLAS leaves that the lanes of the warp reached in this step, tested
    // by the whole warp: the lanes with a leaf publish their rays in lane
    // order, the warp's sum(count) (ray, triangle) pairs are dealt out to its
    // lanes in turn, 32 at a time, and each owner then takes the best of its
    // candidates.  A pair's owner comes from the owners' prefixes as bits of
    // one word (their union over the warp, counted up to the pair), not from
    // a search in shared memory.  The closest candidate is the minimum of
    // (distance bits, triangle index) over triangles of one instance, which
    // is the order hit_better applies, so the hit is the one the in-order
    // loop of test_leaf keeps.  For any hit the lowest blocking triangle index
    // is the one the in-order loop stops at, and the owner counts the
    // triangles that loop would have tested.
    // Returns true when the lane's any-hit query is complete.
    //
// lo, ld, flags, inst: the lane's local ray at its leaf, and the instance's
// cull flags and index; tmin as the walk's.
template <bool kAnyHit>
__device__ __forceinline__ bool leaf_pass(const SceneView &S, LeafScratch *L, uint32_t first, uint32_t count, f3 lo,
                                          f3 ld, uint32_t flags, uint32_t inst, float tmin, Hit &hit,
                                          TraceCounters &cn) {
        const unsigned group = 0xffffffffu;  // every lane of the warp takes part
        const uint32_t lane = threadIdx.x & 31u;
        const unsigned below = (1u << lane) - 1u;
        const unsigned owners = __ballot_sync(group, count != 0u);
        if (owners == 0u) return false;
        uint32_t pre = 0, total = 0;
#pragma unroll
        for (int b = 0; b < 5; ++b) {  // leaf counts are at most 16
            const unsigned v = __ballot_sync(group, (count >> b) & 1u);
            pre += (uint32_t)__popc(v & below) << b;
            total += (uint32_t)__popc(v) << b;
        }
        const uint32_t rank = (uint32_t)__popc(owners & below);
        if (count) {
            const TriRay tri_ray = triangle_ray(ld);
            L->ox[rank] = lo.x;
            L->oy[rank] = lo.y;
            L->oz[rank] = lo.z;
            L->dx[rank] = ld.x;
            L->dy[rank] = ld.y;
            L->dz[rank] = ld.z;
            L->sx[rank] = tri_ray.sx;
            L->sy[rank] = tri_ray.sy;
            L->axes[rank] = tri_ray.kx | (tri_ray.ky << 2) | (tri_ray.kz << 4) | (tri_ray.valid ? 64u : 0u);
            L->flags[rank] = flags;
            L->first[rank] = first - pre;
            if (!kAnyHit) L->lower[rank] = fmaxf(tmin, 0.000025f);
            if (kAnyHit) L->limit[rank] = hit.t;
            L->best[rank] = ~0ull;
        }
        __syncwarp(group);
        for (uint32_t base = 0; base < total; base += 32u) {
            const uint32_t at = pre - base;  // this lane's first pair within the 32
            const unsigned starts = __reduce_or_sync(group, count && at < 32u ? 1u << at : 0u);
            const uint32_t before = base ? (uint32_t)__popc(__ballot_sync(group, count && pre < base)) : 0u;
            const uint32_t p = base + lane;
            if (p >= total) continue;
            const uint32_t o = before + (uint32_t)__popc(starts & (below | (1u << lane))) - 1u;
            const uint32_t t = L->first[o] + p;
            f3 A, B, C;
            load_triangle(S.triangles, t, A, B, C);
            const f3 rd{L->dx[o], L->dy[o], L->dz[o]};
            if (cull_reject(L->flags[o], A, B, C, rd)) continue;
            TriRay tr;
            const uint32_t ax = L->axes[o];
            tr.kx = ax & 3u;
            tr.ky = (ax >> 2) & 3u;
            tr.kz = (ax >> 4) & 3u;
            tr.valid = (ax & 64u) != 0u;
            tr.sx = L->sx[o];
            tr.sy = L->sy[o];
            float w1 = 0.0f, w2 = 0.0f;
            const float dist = intersect_triangle(f3{L->ox[o], L->oy[o], L->oz[o]}, rd, tr, A, B, C, w1, w2);
            if (kAnyHit) {
                if (dist > 0.000025f && dist < L->limit[o]) atomicMin(&L->best[o], (unsigned long long)t);
            } else if (dist > L->lower[o]) {
                atomicMin(&L->best[o], ((unsigned long long)as_uint(dist) << 32) | t);
            }
        }
        __syncwarp(group);
        bool done = false;
        if (count) {
            const unsigned long long b = L->best[rank];
            if (kAnyHit) {
                if (b != ~0ull) {
                    const uint32_t t = (uint32_t)b;
                    cn.triangles += t - first + 1u;
                    hit.tri = t;
                    hit.inst = inst;
                    hit.errors &= ~kQueryUnsupported;
                    done = true;
                } else {
                    cn.triangles += count;
                }
            } else {
                cn.triangles += count;
                if (b != ~0ull) {
                    const float dist = as_float((uint32_t)(b >> 32));
                    const uint32_t t = (uint32_t)b;
                    if (hit_better(dist, inst, t, hit)) {
                        hit.t = dist;
                        hit.tri = t;
                        hit.inst = inst;
                    }
                }
            }
        }
        __syncwarp(group);  // the scratch is rewritten by the next pass
        return done;
    }

// traceRayTracked + traceInstance (kAnyHit = false) and traceOccluded +
// occludedInstance (kAnyHit = true) as one resumable walk over one stack.  A
// TLAS leaf enters its first instance (the rest of the leaf is pushed back);
// the BLAS walk runs on the same stack above `blas_base` in the instance's
// local space and returns to world space when the stack drops back to it.
// Each step traverses inner nodes until a leaf is reached, then processes
// that leaf (the while-while order), so the lanes of a warp stay in step and
// a lane whose ray finished can take a new ray between steps.
//
// Error bits follow the reference: 4 when a walk exceeds MAX_TRAVERSAL_STEPS
// (per TLAS walk and per instance walk), 2 / 1 when the stack is exhausted in
// the TLAS / a BLAS, after which the walk continues over every instance / every
// triangle of the instance in order (shaders/traversal.slang:498-517, :729-745).
template <bool kAnyHit, int kDepth = kStack, typename Slab = SlabRay>
struct Walker {
    Hit hit;
    f3 o, d, lo, ld;  // world ray; the current instance's local ray
    float tmin;       // at least 0
    float pad;        // kSlabPad x the largest coordinate magnitude of the TLAS root box
    Slab r;           // slab constants of the current space's ray
    uint32_t inst, inst_flags, inst_first;
    int blas_base;        // stack depth at instance entry; -1 = TLAS space
    uint32_t tlas_next;   // TLAS fallback: next instance to scan in order
    uint32_t blas_next;   // BLAS fallback: next triangle to scan in order
    uint32_t steps;       // of the current walk (TLAS, or the instance's)
    uint32_t tlas_steps;  // the TLAS walk's, while inside an instance
    int sp;  // depth of the caller's stack: kDepth entries of (payload, entry distance bits)
    uint32_t cur;
    bool have;

    // Returns false when the query is already complete (no instances, the ray
    // misses the TLAS root box: traceRayTracked's early exits; or a ray that is
    // not finite or has no interval, NaN bounds included, which the child tests'
    // three-operand minima would drop: no hit satisfies them).  kLeaveFar: so do far
    // rays, with `steps` kFarSteps.
    template <bool kLeaveFar = false>
    __device__ __forceinline__ bool start(const SceneView &S, f3 origin, f3 direction, float t_min, float limit) {
        hit.t = limit;
        hit.tri = kEmpty;
        hit.inst = kEmpty;
        hit.errors = 0;
        hit.b1 = 0.0f;
        hit.b2 = 0.0f;
        if (S.instance_count == 0) return false;
        if (!(finite3(origin) && finite3(direction) && t_min <= limit)) return false;
        // The TLAS root box is read from the live scene words (node 0), so a
        // device-side refit takes effect without a host round trip.
        float re, rx;
        uint4 ra = __ldg(S.scene_words + 1), rb = __ldg(S.scene_words + 2);
        const f3 rl{as_float(ra.x), as_float(ra.y), as_float(ra.z)}, rh{as_float(rb.x), as_float(rb.y), as_float(rb.z)};
        if (!box_interval(origin, direction, rl.x, rl.y, rl.z, rh.x, rh.y, rh.z, limit, re, rx)) return false;
        const float magnitude = box_magnitude(rl, rh);
        if (kLeaveFar && largest_component(origin) > kFarOrigin * magnitude) {
            steps = kFarSteps;
            return false;
        }
        pad = magnitude * kSlabPad;
        o = origin;
        d = direction;
        tmin = fmaxf(t_min, 0.0f);
        make_slab(r, o, d, pad);
        lo = o;
        ld = d;
        inst = kEmpty;
        inst_flags = inst_first = 0;
        blas_base = -1;
        tlas_next = blas_next = kEmpty;
        steps = tlas_steps = 0;
        sp = 0;
        cur = S.tlas_root;
        have = true;
        return true;
    }

    // Stack exhausted: the TLAS walk scans every instance in order, an
    // instance's walk every triangle of it.
    __device__ __forceinline__ void overflow() {
        if (blas_base < 0) {
            hit.errors |= 2u;
            sp = 0;
            tlas_next = 0;
        } else {
            hit.errors |= 1u;
            sp = blas_base;
            blas_next = inst_first;
        }
        have = false;
    }

    // One step: inner nodes down to a leaf, that leaf, then the next pending
    // entry.  Returns true when the query is complete.
    // The stack lives outside the walker so the walker's fields stay in
    // registers; only the stack itself is addressed dynamically.
    // One inner node of the descent: its child tests, the farther hit
    // children pushed, the nearest taken.  Clears `have` at a dead end, an
    // instance's step budget or a stack overflow (the ordered-scan
    // fallback); returns true when the whole query is abandoned (the TLAS
    // step budget).
    __device__ __forceinline__ bool node_step(const SceneView &S, uint2 *stack, TraceCounters &cn) {
        if (++steps > kMaxSteps) {
            hit.errors |= kQueryUnsupported;
            if (blas_base < 0) return true;  // abandon the whole query
            sp = blas_base;                  // abandon this instance
            have = false;
            return false;
        }
        float entry[4];
        uint32_t child[4];
        cn.nodes++;
        const uint32_t mask = node_test(S.nodes, cur, r, hit.t, tmin, entry, child);
        if (mask == 0u) {
            have = false;
            return false;
        }
        const int n = __popc(mask);
        if (sp + n - 1 > kDepth) {
            overflow();
            return false;
        }
        if (kAnyHit) {
            // Visibility needs a blocker, not the nearest one: the hit
            // children are taken in slot order without sorting (1.6% less
            // trace time at the bench frame than nearest first).
            const int first = __ffs(mask) - 1;
#pragma unroll
            for (int i = 3; i >= 1; --i)
                if (((mask >> i) & 1u) && i != first) stack[sp++] = make_uint2(child[i], 0u);
            cur = first == 0 ? child[0] : (first == 1 ? child[1] : (first == 2 ? child[2] : child[3]));
            return false;
        }
        uint32_t k0 = child_key(mask, entry, 0), k1 = child_key(mask, entry, 1);
        uint32_t k2 = child_key(mask, entry, 2), k3 = child_key(mask, entry, 3);
        key_swap(k0, k1);
        key_swap(k2, k3);
        key_swap(k0, k2);
        key_swap(k1, k3);
        key_swap(k1, k2);
        if (n > 3) stack[sp++] = make_uint2(key_child(k3, child), k3 & ~3u);
        if (n > 2) stack[sp++] = make_uint2(key_child(k2, child), k2 & ~3u);
        if (n > 1) stack[sp++] = make_uint2(key_child(k1, child), k1 & ~3u);
        cur = key_child(k0, child);
        return false;
    }

    // A TLAS leaf (first, count): enter its first instance (the rest of the
    // leaf waits on the stack).
    // The instance's slab constants are set here and the world ray's again in
    // next(); the triangle constants wait for a leaf.
    __device__ __forceinline__ void enter_instance(const SceneView &S, uint2 *stack, TraceCounters &cn, uint32_t first,
                                                   uint32_t count) {
        if (count > 1u) {
            if (sp < kDepth) {
                stack[sp++] = make_uint2(kLeafBit | ((first + 1u) & kLeafFirstMask) | ((count - 2u) << 27), 0u);
            } else {
                // Stack exhausted: after this instance, scan every instance.
                hit.errors |= 2u;
                sp = 0;
                tlas_next = 0;
            }
        }
        const DeviceInstance I = load_instance(S.instances, first);
        local_ray(I, o, d, lo, ld);
        cn.instances++;
        if (!isfinite(((fabsf(lo.x) + fabsf(lo.y)) + fabsf(lo.z)) + ((fabsf(ld.x) + fabsf(ld.y)) + fabsf(ld.z))))
            return;  // no triangle test accepts such a ray
        make_slab(r, lo, ld, I.extent * kSlabPad);
        inst = first;
        inst_flags = I.flags;
        inst_first = I.first;
        blas_base = sp;
        tlas_steps = steps;
        steps = 0;
        cur = I.root;
        have = true;
    }

    // Inner nodes down to a leaf and that leaf's kind: a TLAS leaf enters its
    // first instance; a BLAS leaf within the step budget is returned as
    // (first, count) for its triangle tests (count 0: none).  Returns true
    // when the query is complete.
    __device__ __forceinline__ bool descend(const SceneView &S, uint2 *stack, TraceCounters &cn, uint32_t &leaf_first,
                                            uint32_t &leaf_count) {
        leaf_first = 0;
        leaf_count = 0;
        while (have && (cur & kLeafBit) == 0u)
            if (node_step(S, stack, cn)) return true;
        if (have) {
            uint32_t first = cur & kLeafFirstMask;
            uint32_t count = ((cur >> 27) & 15u) + 1u;
            have = false;
            if (blas_base < 0) {
                enter_instance(S, stack, cn, first, count);
                return false;
            }
            // BLAS leaf (traceTriangle / occludedTriangle).
            if (++steps > kMaxSteps) {
                hit.errors |= kQueryUnsupported;
                sp = blas_base;
            } else {
                leaf_first = first;
                leaf_count = count;
            }
        }
        return false;
    }

    // The triangles of one BLAS leaf in order; true when an any-hit query is
    // complete.
    __device__ __forceinline__ bool test_leaf(const SceneView &S, uint32_t first, uint32_t count, TraceCounters &cn) {
        const TriRay tri_ray = triangle_ray(ld);
        const float lower = fmaxf(tmin, 0.000025f);
        for (uint32_t t = first; t < first + count; ++t) {
            f3 A, B, C;
            load_triangle(S.triangles, t, A, B, C);
            cn.triangles++;
            if (cull_reject(inst_flags, A, B, C, ld)) continue;
            float w1 = 0.0f, w2 = 0.0f;
            float dist = intersect_triangle(lo, ld, tri_ray, A, B, C, w1, w2);
            if (kAnyHit) {
                if (dist > 0.000025f && dist < hit.t) {
                    // Any accepted blocker is a complete proof
                    // (shaders/traversal.slang:786-792, :1035-1040).
                    hit.tri = t;
                    hit.inst = inst;
                    hit.errors &= ~kQueryUnsupported;
                    return true;
                }
            } else if (dist > lower && hit_better(dist, inst, t, hit)) {
                hit.t = dist;
                hit.tri = t;
                hit.inst = inst;
            }
        }
        return false;
    }

    // The next pending entry, leaving instances and fallbacks as needed; true
    // when the query is complete.
    __device__ __forceinline__ bool next(const SceneView &S, uint2 *stack) {
        while (!have) {
            if (blas_base >= 0 && sp == blas_base) {
                if (blas_next != kEmpty) {  // ordered scan: the instance's triangle count from its record
                    const uint32_t end = inst_first + instance_triangles(S, inst);
                    if (blas_next < end) {
                        const uint32_t c = min(kLeafMaxCount, end - blas_next);
                        cur = kLeafBit | (blas_next & kLeafFirstMask) | ((c - 1u) << 27);
                        blas_next += c;
                        have = true;
                        break;
                    }
                    blas_next = kEmpty;
                }
                blas_base = -1;
                steps = tlas_steps;
                make_slab(r, o, d, pad);
                inst = kEmpty;
                continue;
            }
            if (sp == 0) {
                if (tlas_next != kEmpty && tlas_next < S.instance_count) {
                    cur = kLeafBit | (tlas_next & kLeafFirstMask);
                    ++tlas_next;
                    have = true;
                    break;
                }
                return true;
            }
            uint2 top = stack[--sp];
            if (!kAnyHit && as_float(top.y) > hit.t) continue;
            cur = top.x;
            have = true;
        }
        return false;
    }

    // One step: inner nodes down to a leaf, that leaf, then the next pending
    // entry.  Returns true when the query is complete.
    // The stack lives outside the walker so the walker's fields stay in
    // registers; only the stack itself is addressed dynamically.
    __device__ __forceinline__ bool step(const SceneView &S, uint2 *stack, TraceCounters &cn) {
        uint32_t first, count;
        if (descend(S, stack, cn, first, count)) return true;
        if (count && test_leaf(S, first, count, cn)) return true;
        return next(S, stack);
    }

    // step() for walks of a whole warp: every lane calls it in every round
    // (alive = the lane still has a query), so the leaf pass runs over the
    // full warp.  Returns true when the lane's query is complete (or it has
    // none).
    __device__ __forceinline__ bool step_warp(const SceneView &S, uint2 *stack, TraceCounters &cn, LeafScratch *L,
                                              bool alive) {
        uint32_t first = 0, count = 0;
        bool complete = !alive;
        if (alive) complete = descend(S, stack, cn, first, count);
        if (complete) count = 0;
        if (leaf_pass<kAnyHit>(S, L, first, count, lo, ld, inst_flags, inst, tmin, hit, cn)) complete = true;
        if (complete) return true;
        return next(S, stack);
    }
};

// Closest hit (kAnyHit = false) or any hit of one ray.  kDepth is the stack
// depth: a shallower stack uses less local memory per thread, and a walk that
// overflows it continues with the reference's ordered scan (same answers).
template <bool kAnyHit, int kDepth = kStack>
__device__ void trace(const SceneView &S, f3 o, f3 d, float tmin, float limit, Hit &hit, TraceCounters &cn) {
    Walker<kAnyHit, kDepth> w;
    uint2 stack[kDepth];
    if (w.start(S, o, d, tmin, limit))
        while (!w.step(S, stack, cn)) {
        }
    hit = w.hit;
    if (!kAnyHit) hit_barycentrics(S, o, d, hit);
}

// Walk over the flattened tree (SceneView::flat_nodes): the TLAS with a
// world-space copy of every instance's nodes below it, so a ray is transformed
// only at the leaves it tests and one set of slab constants serves the whole
// query.  Against the two-level walk this drops the instance entry and exit
// (a transform and two sets of slab constants, run by a few lanes of a warp at
// a time), the rounds that end at an instance, and the registers of the second
// ray.  Hits are the same: the triangles are tested in the instance's local
// space from the same local ray, the copies' boxes are padded (scene.cu), and
// so is the ray, by kFlatPad (max|o| + M) on every axis, since a rotated
// instance's local ray mixes the axes and rounds by the largest.  With u =
// 2^-24 and sum_j |M_ij| sum_k |R_jk| <= 4 (flat_conditioned): the local
// origin rounds by 3.5 u, the direction by 3 u over the distance, the matrix
// itself by u, the triangle test's differences by u and its shear by 2 u, each
// at most four times that in world space, 42 u of max|o|; the hit distance
// takes 4 u and the slab constants 6 u: 52 u, and less of M.  (With |o| of the
// axis alone, rays along an axis lost hits from 1,000 scene sizes on.)
// Measured at the 1280x720 frame (262,144 triangles, 1.97 M interval rays, 8.8 M
// visibility queries): closest hits 1.73 -> 1.20 ms, visibility 3.53 -> 2.59
// ms; 1920x1080 and 1,048,576 triangles: whole frame 20.7 -> 15.7 ms.
//
// The stack cannot overflow (a flattened tree is built only when three pending
// children per level fit kFlatStack).  The step budgets of the two-level walk
// (4096 per TLAS walk and per instance) cannot be exceeded before 4096 steps
// in all; a query that gets there starts over with the two-level walk's
// accounting (careful_step), whose state lives behind the stack in local
// memory so that the common walk keeps no register for it.
constexpr float kFlatPad = 3.814697265625e-6f;  // 64 u

template <bool kAnyHit>
struct FlatWalker {
    // A pending child: its payload, and for closest hits its entry distance.
    struct Near {
        uint2 v;
        __device__ __forceinline__ void set(uint32_t payload, uint32_t entry) { v = make_uint2(payload, entry); }
        __device__ __forceinline__ uint32_t payload() const { return v.x; }
        __device__ __forceinline__ float entry() const { return as_float(v.y); }
    };
    struct Any {
        uint32_t v;
        __device__ __forceinline__ void set(uint32_t payload, uint32_t) { v = payload; }
        __device__ __forceinline__ uint32_t payload() const { return v; }
        __device__ __forceinline__ float entry() const { return 0.0f; }
    };
    using Entry = typename std::conditional<kAnyHit, Any, Near>::type;
    // Behind the stack: the query's limit, and careful_step's state.
    enum Slot { kLimit = kFlatStack, kTlasSteps, kInstance, kBase, kInstanceSteps, kErrors, kEntries };

    Hit hit;  // errors: set by finish()
    f3 o, d;
    float tmin;
    SlabRay r;
    uint32_t steps;
    int sp;
    uint32_t cur;
    bool have;

    template <bool kLeaveFar = false>
    __device__ __forceinline__ bool start(const SceneView &S, Entry *stack, f3 origin, f3 direction, float t_min,
                                          float limit) {
        if (!(finite3(origin) && finite3(direction) && t_min <= limit)) return false;
        float re, rx;
        uint4 ra = __ldg(S.scene_words + 1), rb = __ldg(S.scene_words + 2);
        const f3 rl{as_float(ra.x), as_float(ra.y), as_float(ra.z)}, rh{as_float(rb.x), as_float(rb.y), as_float(rb.z)};
        if (!box_interval(origin, direction, rl.x, rl.y, rl.z, rh.x, rh.y, rh.z, limit, re, rx)) return false;
        const float magnitude = box_magnitude(rl, rh), out = largest_component(origin);
        if (kLeaveFar && out > kFarOrigin * magnitude) {
            steps = kFarSteps;
            return false;
        }
        o = origin;
        d = direction;
        tmin = fmaxf(t_min, 0.0f);
        r = slab_ray<true>(o, d, (out + magnitude) * kFlatPad);
        if (!kAnyHit) stack[kLimit].set(as_uint(limit), 0u);
        sp = 0;
        cur = S.tlas_root;
        have = true;
        return true;
    }

    // A step past kMaxSteps in all.  The first time the query starts over
    // (false, with the root to go on from); then every step (the inner node
    // `cur`, or a leaf of instance `leaf_inst`) counts against its walk's
    // budget, as Walker counts it.  False when the step is not taken: its
    // instance is abandoned, or the query (`done`).
    __device__ __forceinline__ bool careful_step(const SceneView &S, Entry *stack, uint32_t leaf_inst, bool &done) {
        const bool first = steps == kMaxSteps + 1u;
        steps = kMaxSteps + 1u;  // the next step counts one up: careful again, not the first time
        if (first) {
            if (!kAnyHit) {
                hit.t = as_float(stack[kLimit].payload());
                hit.tri = hit.inst = kEmpty;
            }
            stack[kTlasSteps].set(0u, 0u);
            stack[kInstance].set(kEmpty, 0u);
            stack[kErrors].set(0u, 0u);
            sp = 0;
            cur = S.tlas_root;
            have = true;
            return false;
        }
        uint32_t inst = leaf_inst;
        if (inst == kEmpty && cur >= S.flat_tlas) {
            uint32_t lo = 0, hi = S.instance_count;  // the instance whose copy holds the node
            while (hi - lo > 1u) {
                const uint32_t mid = (lo + hi) >> 1;
                if (__ldg(&S.flat_inst[mid].x) <= cur)
                    lo = mid;
                else
                    hi = mid;
            }
            inst = lo;
        }
        if (inst == kEmpty) {
            const uint32_t n = stack[kTlasSteps].payload() + 1u;
            stack[kTlasSteps].set(n, 0u);
            if (n <= kMaxSteps) return true;
            done = true;  // abandon the whole query
        } else {
            if (inst != stack[kInstance].payload()) {
                stack[kInstance].set(inst, 0u);
                stack[kBase].set((uint32_t)sp, 0u);
                stack[kInstanceSteps].set(0u, 0u);
            }
            const uint32_t n = stack[kInstanceSteps].payload() + 1u;
            stack[kInstanceSteps].set(n, 0u);
            if (n <= kMaxSteps) return true;
            sp = (int)stack[kBase].payload();  // abandon this instance
        }
        stack[kErrors].set(kQueryUnsupported, 0u);
        have = false;
        return false;
    }

    // Inner nodes down to the next leaf (its payload in `leaf`) or to a dead
    // end; true when the query is abandoned.
    __device__ __forceinline__ bool descend(const SceneView &S, Entry *stack, TraceCounters &cn, uint32_t &leaf) {
        while (have && (cur & kLeafBit) == 0u) {
            if (++steps > kMaxSteps) {
                bool done = false;
                if (!careful_step(S, stack, kEmpty, done)) {
                    if (done) return true;
                    continue;
                }
            }
            float entry[4];
            uint32_t child[4];
            cn.nodes++;
            const uint32_t mask = node_test(S.flat_nodes, cur, r, hit.t, tmin, entry, child);
            if (mask == 0u) {
                have = false;
                break;
            }
            if (kAnyHit) {  // slot order, as the two-level walk
                const int first = __ffs(mask) - 1;
#pragma unroll
                for (int i = 3; i >= 1; --i)
                    if (((mask >> i) & 1u) && i != first) stack[sp++].set(child[i], 0u);
                cur = first == 0 ? child[0] : (first == 1 ? child[1] : (first == 2 ? child[2] : child[3]));
            } else {
                uint32_t k0 = child_key(mask, entry, 0), k1 = child_key(mask, entry, 1);
                uint32_t k2 = child_key(mask, entry, 2), k3 = child_key(mask, entry, 3);
                key_swap(k0, k1);
                key_swap(k2, k3);
                key_swap(k0, k2);
                key_swap(k1, k3);
                key_swap(k1, k2);
                const int n = __popc(mask);
                if (n > 3) stack[sp++].set(key_child(k3, child), k3 & ~3u);
                if (n > 2) stack[sp++].set(key_child(k2, child), k2 & ~3u);
                if (n > 1) stack[sp++].set(key_child(k1, child), k1 & ~3u);
                cur = key_child(k0, child);
            }
        }
        if (have) {
            leaf = cur;
            have = false;
        }
        return false;
    }

    // The next pending entry; true when there is none.
    __device__ __forceinline__ bool next(Entry *stack) {
        while (!have) {
            if (sp == 0) return true;
            const Entry top = stack[--sp];
            if (!kAnyHit && top.entry() > hit.t) continue;
            cur = top.payload();
            have = true;
        }
        return false;
    }

    // One round of a whole warp's walks (Walker::step_warp's contract).
    __device__ __forceinline__ bool step_warp(const SceneView &S, Entry *stack, TraceCounters &cn, LeafScratch *L,
                                              bool alive) {
        uint32_t leaf = 0, first = 0, count = 0, flags = 0, inst = kEmpty;
        bool complete = !alive;
        if (alive) complete = descend(S, stack, cn, leaf);
        f3 lo{0.0f, 0.0f, 0.0f}, ld{0.0f, 0.0f, 0.0f};
        if (leaf) {
            const uint2 at = __ldg(S.flat_leaves + (leaf & kLeafFirstMask));
            inst = at.x;
            first = at.y;
            count = ((leaf >> 27) & 15u) + 1u;
            const DeviceInstance I = load_instance(S.instances, inst);
            local_ray(I, o, d, lo, ld);
            flags = I.flags;
            cn.instances++;
            if (++steps > kMaxSteps) {
                bool done = false;
                if (!careful_step(S, stack, inst, done)) count = 0;
            }
        }
        if (leaf_pass<kAnyHit>(S, L, first, count, lo, ld, flags, inst, tmin, hit, cn)) complete = true;
        if (complete) return true;
        return next(stack);
    }

    __device__ __forceinline__ void finish(const Entry *stack) {
        if (steps > kMaxSteps && !(kAnyHit && hit.tri != kEmpty)) hit.errors = stack[kErrors].payload();
    }
};

// trace() for a whole warp: every lane of the warp calls it (active: the lane
// has a query), and the BLAS leaves reached in each round are tested by the
// whole warp (leaf_pass).  A lane without a query returns no hit.
// kFar: the rays are a caller's and may start far outside the scene; one that
// does returns no hit and errors = kFarRay, and is traced after the others
// (trace_warp with FarSlabRay) where that costs the walk beside it least.
template <bool kAnyHit, int kDepth = kStack, bool kFar = false, typename Slab = SlabRay>
__device__ __forceinline__ void trace_warp(const SceneView &S, bool active, f3 o, f3 d, float tmin, float limit,
                                           Hit &hit, TraceCounters &cn, LeafScratch *L) {
    Walker<kAnyHit, kDepth, Slab> w;
    w.hit = Hit{limit, kEmpty, kEmpty, 0u, 0.0f, 0.0f};
    w.steps = 0;
    uint2 stack[kDepth];
    bool alive = active && w.template start<kFar>(S, o, d, tmin, limit);
    while (__any_sync(0xffffffffu, alive)) {
        const bool complete = w.step_warp(S, stack, cn, L, alive);
        alive = alive && !complete;
    }
    if (kFar && w.steps == kFarSteps) w.hit.errors = kFarRay;
    hit = w.hit;
    if (!kAnyHit) hit_barycentrics(S, o, d, hit);
}

// trace_warp over the flattened tree.  (The two-level walk is in kernels of its
// own: the flattened walk loses its registers to a second walk in the same
// loop, even one that is hardly ever called: closest hits 1.51 ms against 1.26.)
template <bool kAnyHit, bool kFar = false>
__device__ __forceinline__ void trace_warp_flat(const SceneView &S, bool active, f3 o, f3 d, float tmin, float limit,
                                                Hit &hit, TraceCounters &cn, LeafScratch *L) {
    FlatWalker<kAnyHit> w;
    w.hit = Hit{limit, kEmpty, kEmpty, 0u, 0.0f, 0.0f};
    w.steps = 0;
    typename FlatWalker<kAnyHit>::Entry stack[FlatWalker<kAnyHit>::kEntries];
    bool alive = active && w.template start<kFar>(S, stack, o, d, tmin, limit);
    while (__any_sync(0xffffffffu, alive)) {
        const bool complete = w.step_warp(S, stack, cn, L, alive);
        alive = alive && !complete;
    }
    if (kFar && w.steps == kFarSteps)
        w.hit.errors = kFarRay;
    else
        w.finish(stack);
    hit = w.hit;
    if (!kAnyHit) hit_barycentrics(S, o, d, hit);
}

// A persistent warp's loop with per-lane refill: whenever lanes are idle, the
// warp takes that many new rays from `counter` (one atomic per refill) and
// keeps stepping until the counter passes `n` and every lane is done.
// gen(id, o, d, tmin, limit) produces ray `id`; done(id, hit) consumes it.
// The warp's walks step together and the leaves of each round are tested by
// the whole warp.
template <bool kAnyHit, typename Gen, typename Done>
__device__ __forceinline__ void trace_refill(const SceneView &S, uint32_t *counter, uint32_t n, Gen &&gen, Done &&done,
                                             TraceCounters &cn, LeafScratch *L) {
    const uint32_t lane = threadIdx.x & 31u;
    Walker<kAnyHit> w;
    uint2 stack[kStack];
    bool active = false;
    bool exhausted = false;  // the counter passed n: no further rays for this warp
    uint32_t id = 0;
    while (true) {
        uint32_t need = __ballot_sync(0xffffffffu, !active && !exhausted);
        if (need) {
            uint32_t leader = __ffs(need) - 1u;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(need));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (base + (uint32_t)__popc(need) > n) exhausted = true;  // uniform across the warp
            if (!active && (need & (1u << lane))) {
                id = base + (uint32_t)__popc(need & ((1u << lane) - 1u));
                if (id < n) {
                    f3 o, d;
                    float tmin, limit;
                    gen(id, o, d, tmin, limit);
                    active = w.start(S, o, d, tmin, limit);
                    if (!active) done(id, w.hit);
                }
            }
        }
        if (!__any_sync(0xffffffffu, active)) {
            if (exhausted) break;
            continue;
        }
        const bool complete = w.step_warp(S, stack, cn, L, active);
        if (active && complete) {
            if (!kAnyHit) hit_barycentrics(S, w.o, w.d, w.hit);
            done(id, w.hit);
            active = false;
        }
    }
}

}  // namespace lux
