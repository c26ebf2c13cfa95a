// cpt_trace.cuh — closest-hit traversal of the BVH2 layout and primitive intersection in
// FP32 (traverseIterative BVH.cuh:282-332, Hittable::hit Hittable.cuh:487-503).
//
// The traversal returns the closest hit like the reference but orders children near-first
// and prunes boxes beyond the closest hit so far (the reference tests every box the ray
// line crosses).  Leaves are tested as soon as their box is hit, with [0.001, closest], as
// in the reference; only exact ties may resolve to a different primitive.
#pragma once

#include "cpt_device.cuh"
#include "cpt_fetch.h"

namespace cpt {

struct Hit {
    float t, u, v;
    int leaf;   // sorted leaf index, -1 on a miss
};

__device__ __forceinline__ float4 ldg4(const float4* p) { return __ldg(p); }

// Möller–Trumbore exactly as Triangle::hit (Hittable.cuh:85-111): eps 1e-8 on the
// determinant, inclusive u, v, u+v and t bounds.
__device__ __forceinline__ bool hit_triangle(float3 o, float3 d, float3 p0, float3 e1, float3 e2, float tmin,
                                             float tmax, float& t, float& u, float& v)
{
    float3 h = cross3(d, e2);
    float a = dot3(e1, h);
    if (fabsf(a) < 1e-8f) return false;
    float f = 1.0f / a;
    float3 s = o - p0;
    u = f * dot3(s, h);
    if (u < 0.0f || u > 1.0f) return false;
    float3 q = cross3(s, e1);
    v = f * dot3(d, q);
    if (v < 0.0f || u + v > 1.0f) return false;
    t = f * dot3(e2, q);
    return !(t < tmin || t > tmax);
}

// Sphere::hit (Hittable.cuh:27-44).
__device__ __forceinline__ bool hit_sphere(float3 o, float3 d, float3 c, float r, float tmin, float tmax, float& t)
{
    float3 oc = o - c;
    float a = dot3(d, d);
    float b = dot3(d, oc);
    float cc = dot3(oc, oc) - r * r;
    float disc = b * b - a * cc;
    if (disc < 0.0f) return false;
    float sq = sqrtf(disc);
    t = (-b - sq) / a;
    if (t < tmin || t > tmax) t = (-b + sq) / a;
    return !(t < tmin || t > tmax);
}

// Light::hit (Hittable.cuh:367-398): one-sided rectangle, only when visible.
__device__ __forceinline__ bool hit_light(const DevLight& L, float3 o, float3 d, float tmin, float tmax, float& t)
{
    if (!L.visible) return false;
    float denom = dot3(d, L.normal);
    if (fabsf(denom) < 1e-6f || denom > 0.0f) return false;
    t = dot3(L.center - o, L.normal) / denom;
    if (t < tmin || t > tmax) return false;
    float3 hp = o + t * d;
    float3 diff = hp - L.center;
    float u = dot3(diff, L.eu), v = dot3(diff, L.ev);
    return fabsf(u) <= L.w / 2.0f && fabsf(v) <= L.h / 2.0f;
}

// Hit of leaf k in [0.001, tmax]; with SKIP the light `skip` is never hit.
template <bool SKIP = false>
__device__ __forceinline__ bool hit_leaf(const SceneView& s, int k, float3 o, float3 d, float tmax, float& t, float& u,
                                         float& v, int skip = -1)
{
    const float4* r = s.leaf_rec + 3 * (size_t)k;
    float4 r0 = ldg4(r), r1 = ldg4(r + 1);
    int kind = __float_as_int(r1.w);
    if (kind == CPT_KIND_TRI) {
        float4 r2 = ldg4(r + 2);
        return hit_triangle(o, d, f3(r0.x, r0.y, r0.z), f3(r1.x, r1.y, r1.z), f3(r2.x, r2.y, r2.z), 0.001f, tmax, t, u,
                            v);
    }
    u = v = 0.f;
    if (kind == CPT_KIND_SPHERE) return hit_sphere(o, d, f3(r0.x, r0.y, r0.z), r1.x, 0.001f, tmax, t);
    const int li = __float_as_int(r1.x);
    return (!SKIP || li != skip) && hit_light(s.lights[li], o, d, 0.001f, tmax, t);
}

// Occlusion test of leaf k for a shadow ray aimed at light `skip`: any primitive hit in
// [0.001, tmax] occludes, except that light itself.
__device__ __forceinline__ bool occludes_leaf(const SceneView& s, int k, float3 o, float3 d, float tmax, int skip)
{
    const float4* r = s.leaf_rec + 3 * (size_t)k;
    float4 r0 = ldg4(r), r1 = ldg4(r + 1);
    int kind = __float_as_int(r1.w);
    float t, u, v;
    if (kind == CPT_KIND_TRI) {
        float4 r2 = ldg4(r + 2);
        return hit_triangle(o, d, f3(r0.x, r0.y, r0.z), f3(r1.x, r1.y, r1.z), f3(r2.x, r2.y, r2.z), 0.001f, tmax, t, u,
                            v);
    }
    if (kind == CPT_KIND_SPHERE) return hit_sphere(o, d, f3(r0.x, r0.y, r0.z), r1.x, 0.001f, tmax, t);
    int li = __float_as_int(r1.x);
    return li != skip && hit_light(s.lights[li], o, d, 0.001f, tmax, t);
}

// What a traversal asks: the closest hit, any occluder of a shadow ray, or either, per ray.
enum Query { Q_CLOSEST, Q_ANY, Q_EITHER };

// One leaf reached by a traversal.  Closest-hit queries keep the nearest hit in [0.001, best];
// occlusion queries (Q_ANY, or Q_EITHER with any set) return true at the first occluder.
template <Query Q>
__device__ __forceinline__ bool visit_leaf(const SceneView& s, int leaf, float3 o, float3 d, float& best, Hit& hit,
                                           int skip, bool any)
{
    if (Q == Q_ANY) {
        if (!occludes_leaf(s, leaf, o, d, best, skip)) return false;
        hit.leaf = leaf;
        return true;
    }
    float t, u, v;
    if (hit_leaf<Q == Q_EITHER>(s, leaf, o, d, best, t, u, v, skip)) {
        best = t; hit.t = t; hit.u = u; hit.v = v; hit.leaf = leaf;
        return Q == Q_EITHER && any;
    }
    return false;
}

// Inverse direction for slab tests.  A zero component (an axis-parallel ray, e.g. a cosine
// sample with r1 = 1 from a floor) would make 1/d infinite and turn slab distances into NaN,
// which the min/max chain then drops: boxes are wrongly accepted or rejected.  Components
// below 1e-20 in magnitude are replaced by +-1e-20 (the limit of a nearly parallel ray); the
// primitive tests keep the exact direction.
__device__ __forceinline__ float3 safe_inverse(float3 d)
{
    const float e = 1e-20f;
    float x = fabsf(d.x) < e ? copysignf(e, d.x) : d.x;
    float y = fabsf(d.y) < e ? copysignf(e, d.y) : d.y;
    float z = fabsf(d.z) < e ? copysignf(e, d.z) : d.z;
    return f3(1.0f / x, 1.0f / y, 1.0f / z);
}

// 32 bytes of read-only memory (32-byte aligned) in one load: the traversals are divergent, so each
// load is an L1 request of its own lines per lane (the 64-byte BVH2 nodes take two of these in place of
// four 16-byte loads: 10M queries of a 1.31M-triangle mesh 2 % faster at best, which runs differ by too).
__device__ __forceinline__ void ldg8(const float4* p, float4& a, float4& b)
{
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

__device__ __forceinline__ float max3f(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

__device__ __forceinline__ float min3f(float a, float b, float c)
{
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Byte k of w as the float 1 + byte * 2^-15: one byte permute instead of an extraction and a
// conversion.
template <int K>
__device__ __forceinline__ float byte_float(uint32_t w)
{
    return __uint_as_float(__byte_perm(w, 0x3F800000u, 0x7604u | (K << 4)));
}

// r[i] = byte_float<K + i>(w) * a + b for i = 0, 1 in one packed multiply-add.
template <int K>
__device__ __forceinline__ void planes(uint32_t w, float a, float b, float (&r)[2])
{
    asm("{\n .reg .b64 q, m, c;\n mov.b64 q, {%2, %3};\n mov.b64 m, {%4, %4};\n mov.b64 c, {%5, %5};\n"
        " fma.rn.f32x2 q, q, m, c;\n mov.b64 {%0, %1}, q;\n}\n"
        : "=f"(r[0]), "=f"(r[1])
        : "f"(byte_float<K>(w)), "f"(byte_float<K + 1>(w)), "f"(a), "f"(b));
}

// Bit p of each byte of v moves to bit p ^ o (o in 0..7).
__device__ __forceinline__ uint32_t xor_bits(uint32_t v, uint32_t o)
{
    if (o & 1u) v = ((v & 0x55555555u) << 1) | ((v >> 1) & 0x55555555u);
    if (o & 2u) v = ((v & 0x33333333u) << 2) | ((v >> 2) & 0x33333333u);
    if (o & 4u) v = ((v & 0x0F0F0F0Fu) << 4) | ((v >> 4) & 0x0F0F0F0Fu);
    return v;
}

// Closest hit through the compressed 8-wide BVH (layout in wide.cu).  A visit decodes the 8
// 8-bit quantised child boxes and tests them; hit children are recorded in a byte mask at bit
// positions slot ^ (7 ^ octant), which orders them roughly front to back for this ray (the slots
// were assigned by direction at build time).  Leaf children are tested at once, nearest bit
// first (the reference tests leaves as it reaches them); the traversal continues with the first
// internal child and keeps the rest as one node-group entry (first child's number, node's internal
// mask, remaining hit bits) on the stack, as in compressed wide BVH traversal (Ylitie et al. 2017);
// a popped group yields its next child without touching memory.  Boxes are tested against the
// closest hit so far, so far subtrees are culled.  An occlusion query (visit_leaf) stops at the
// first occluder.  The walk advances one node per step() so that a
// warp can refill finished lanes (dynamic fetching); Stack64 keeps group entries (in shared and
// local memory, or local only).
//
// The walk is bound by issue slots and the integer/min-max pipe (58-62 % and 52-57 % busy with 17 to 20
// of 32 lanes active, against 5 % of DRAM; before this visit 65-69 % of the issue slots), so a visit is written for few such instructions: planes are
// taken in the ray's order (no min/max per plane pair), bytes become floats by one permute, two
// children share a packed multiply-add, three-input min/max, and a miss is the sign bit of the
// interval's length shifted into a mask.  On the 64-spp 1080p frame of 4.1M triangles: 365 ms with
// byte conversions, min/max per pair and stored child references, 292 ms with this visit and
// scalar multiply-adds, 283 ms packed.  Measured and left out: prefetching the next node before the
// leaf tests (+4 %), testing the three interval conditions by sign instead of min/max with tmin and
// best (+2 %).
//
// LEAVES_FIRST tests a visit's leaves before it chooses the next node; the results are the same.
// Walks with dynamic fetching choose the node first (2 to 4 % faster: a batch of eight renders
// over 8-wide layouts 36.5 -> 35.0 ms).  A loop that traces one ray to its end
// (trace_closest_wide) tests leaves first: the other way round, the lanes whose stack ran empty
// parted from their warp before the leaf tests (4.6 of 32 lanes active), Cornell 400x400 37.5
// instead of 13.5 ms.
template <Query Q, typename Stack64, bool LEAVES_FIRST = false>
struct WideWalk {
    float3 o, d, idir;
    float tmin, best;
    uint32_t first, node;
    int sp, skip;
    bool any;   // Q_EITHER: this ray asks for any occluder
    Hit hit;
    Stack64 stack;

    __device__ __forceinline__ void start(float3 o_, float3 d_, float tmin_, float tmax_, int skip_, bool any_ = false)
    {
        o = o_;
        d = d_;
        idir = safe_inverse(d_);
        first = 7u ^ ((d.x < 0.f ? 1u : 0u) | (d.y < 0.f ? 2u : 0u) | (d.z < 0.f ? 4u : 0u));
        tmin = tmin_;
        best = tmax_;
        node = 0;
        sp = 0;
        skip = skip_;
        any = any_;
        hit.leaf = -1;
        hit.t = tmax_;
        hit.u = hit.v = 0.f;
    }

    // Slab distances along one axis as multiplier and offsets for byte_float values.  A byte q
    // stands for the plane p + q * scale at t = (p - o) * idir + q * a with a = scale * idir; with
    // byte_float(q) = 1 + q * 2^-15 that is byte_float(q) * A + (b - A), A = 2^15 a, b = (p - o) * idir.
    // b - A is rounded to half a unit of 2^-24 |b - A|, 2^-9 |a| while |b| is not above |A|, so the near
    // offset is moved down and the far offset up by 2^-7 |a| (under 1 % of a grid step): for origins within
    // 2^17 grid steps of the node the tested box contains the stored one but for the roundings of b and of
    // the final multiply-add, which every slab test has.  Farther out b - A adds one such rounding more,
    // and a grazing ray may miss the box by it.  That is left so: with a slack of 2^-20 on the distances no
    // ray misses, but rays from 30,000 units away then report hits of spheres (their boxes are not padded)
    // that only the FP32 sphere test sees, which the binary layout does not report.
    __device__ __forceinline__ static void axis(float p, float o, float scale, float idir, float& A, float& bn, float& bf)
    {
        A = scale * idir * 32768.0f;
        const float c = (p - o) * idir - A;
        const float e = fabsf(A) * 0x1p-22f;
        bn = c - e;
        bf = c + e;
    }

    // Visits one node; returns true when the traversal has finished.
    __device__ __forceinline__ bool step(const SceneView& s, int* err)
    {
        const float4* np = s.wide + CPT_WIDE_F4 * (size_t)node;
        float4 f0, f1, qx, qy, qz, f5;
        ldg8(np, f0, f1);
        ldg8(np + 2, qx, qy);
        ldg8(np + 4, qz, f5);
        float ax, ay, az, nbx, nby, nbz, fbx, fby, fbz;
        axis(f0.x, o.x, f0.w, idir.x, ax, nbx, fbx);
        axis(f0.y, o.y, f1.x, idir.y, ay, nby, fby);
        axis(f0.z, o.z, f1.y, idir.z, az, nbz, fbz);
        // planes in the order the ray meets them: the near plane of an axis is the box's maximum
        // when the ray runs towards smaller coordinates
        const bool sx = idir.x < 0.f, sy = idir.y < 0.f, sz = idir.z < 0.f;
        uint32_t misses = 0;   // bit 7 - slot
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t xl = __float_as_uint(h ? qx.y : qx.x), xh = __float_as_uint(h ? qx.w : qx.z);
            const uint32_t yl = __float_as_uint(h ? qy.y : qy.x), yh = __float_as_uint(h ? qy.w : qy.z);
            const uint32_t zl = __float_as_uint(h ? qz.y : qz.x), zh = __float_as_uint(h ? qz.w : qz.z);
            const uint32_t xn = sx ? xh : xl, xf = sx ? xl : xh, yn = sy ? yh : yl, yf = sy ? yl : yh,
                           zn = sz ? zh : zl, zf = sz ? zl : zh;
            // children K and K + 1 of this half
#define CPT_WIDE_PAIR(K)                                                                          \
    {                                                                                             \
        float nx[2], ny[2], nz[2], fx[2], fy[2], fz[2];                                           \
        planes<K>(xn, ax, nbx, nx);                                                               \
        planes<K>(yn, ay, nby, ny);                                                               \
        planes<K>(zn, az, nbz, nz);                                                               \
        planes<K>(xf, ax, fbx, fx);                                                               \
        planes<K>(yf, ay, fby, fy);                                                               \
        planes<K>(zf, az, fbz, fz);                                                               \
        _Pragma("unroll") for (int i = 0; i < 2; ++i)                                             \
        {                                                                                         \
            const float tn = fmaxf(max3f(nx[i], ny[i], nz[i]), tmin);                             \
            const float tf = fminf(min3f(fx[i], fy[i], fz[i]), best);                             \
            misses = __funnelshift_l(__float_as_uint(tf - tn), misses, 1); /* sign set: a miss */ \
        }                                                                                         \
    }
            CPT_WIDE_PAIR(0)
            CPT_WIDE_PAIR(2)
#undef CPT_WIDE_PAIR
        }
        // (internal mask, leaf mask) of the hit slots, from bit 7 - slot to bit slot ^ first
        const uint32_t masks = __float_as_uint(f5.x);
        const uint32_t hits = xor_bits(masks & ((~misses & 0xFFu) * 0x0101u), first ^ 7u);
        const uint32_t ihits = hits & 0xFFu;
        uint32_t lhits = (hits >> 8) & 0xFFu;
        // Tests the hit leaves; true when an any-hit ray has its answer.
        const auto leaves = [&]() -> bool {
            const uint32_t leaf0 = __float_as_uint(f1.w), lmask = (masks >> 8) & 0xFFu;
            while (lhits) {
                const uint32_t slot = (uint32_t)(__ffs(lhits) - 1) ^ first;
                lhits &= lhits - 1;
                if (visit_leaf<Q>(s, (int)(leaf0 + __popc(lmask >> (8u - slot))), o, d, best, hit, skip, any)) return true;
            }
            return false;
        };
        if (LEAVES_FIRST && leaves()) return true;
        // Continue with the first hit internal child; the others stay on the stack as one group.
        bool done = false;
        uint64_t g = (uint64_t)__float_as_uint(f1.z) | ((uint64_t)(ihits | ((masks & 0xFFu) << 8)) << 32);
        if (!ihits) {
            done = sp == 0;
            if (!done) g = stack.get(--sp);
        }
        if (!done) {
            const uint32_t m = (uint32_t)(g >> 32);
            const uint32_t slot = (uint32_t)(__ffs(m & 0xFFu) - 1) ^ first;
            // internal children are numbered in slot order
            node = (uint32_t)g + __popc((m >> 8) >> (8u - slot));
            const uint32_t rest = m & 0xFFu & ((m & 0xFFu) - 1u);
            if (rest) {
                if (sp >= CPT_WSTACK) {
                    if (err) atomicOr(err, CPT_DEVERR_STACK);
                    done = true;
                } else {
                    stack.put(sp++, (uint64_t)(uint32_t)g | ((uint64_t)(rest | (m & 0xFF00u)) << 32));
                }
            }
        }
        if (!LEAVES_FIRST && leaves()) return true;
        return done;
    }
};

// Group-entry stacks of the wide traversal: the whole stack in local memory, or the bottom SHORT
// entries in the block's dynamic shared memory (wide_short_stack_bytes) and the rest in local
// memory; thread t owns the column t, t + T, ... of 64-bit words.
struct LocalStack64 {
    uint64_t s[CPT_WSTACK];
    __device__ __forceinline__ void init() {}
    __device__ __forceinline__ void put(int i, uint64_t v) { s[i] = v; }
    __device__ __forceinline__ uint64_t get(int i) const { return s[i]; }
};

template <int SHORT>
struct ShortStack64 {
    uint64_t* col;
    int stride;
    uint64_t spill[CPT_WSTACK - SHORT];
    __device__ __forceinline__ void init()
    {
        extern __shared__ int cpt_short_stack_smem[];
        const int t = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
        col = reinterpret_cast<uint64_t*>(cpt_short_stack_smem) + t;
        stride = blockDim.x * blockDim.y * blockDim.z;
    }
    __device__ __forceinline__ void put(int i, uint64_t v)
    {
        if (i < SHORT) col[i * stride] = v;
        else spill[i - SHORT] = v;
    }
    __device__ __forceinline__ uint64_t get(int i) const { return i < SHORT ? col[i * stride] : spill[i - SHORT]; }
};

template <bool ANY>
__device__ __forceinline__ bool trace_closest_wide(const SceneView& s, float3 o, float3 d, float tmin, float tmax,
                                                   Hit& hit, int* err, int skip)
{
    WideWalk<ANY ? Q_ANY : Q_CLOSEST, LocalStack64, true> w;
    w.stack.init();
    w.start(o, d, tmin, tmax, skip);
    while (!w.step(s, err)) {}
    hit = w.hit;
    return hit.leaf >= 0;
}

// Slab distances of both children of BVH2 node `node` (t = box * idir - o * idir per axis) and
// their references, from the full 64-byte node or the compressed 32-byte one (s.node_q).
struct Bvh2Slabs {
    float ax0, ax1, ay0, ay1, az0, az1, bx0, bx1, by0, by1, bz0, bz1;
    int ca, cb;
};

__device__ __forceinline__ float u8f(uint32_t w, int k) { return (float)((w >> (8 * k)) & 0xFFu); }

__device__ __forceinline__ void bvh2_slabs(const SceneView& s, int node, float3 o, float3 idir, float3 ood,
                                           Bvh2Slabs& r)
{
    if (s.node_q) {
        float4 q0, q1;
        ldg8(s.nodes + 2 * (size_t)node, q0, q1);
        const uint32_t e = __float_as_uint(q0.w);
        const float sx = __uint_as_float((e & 0xFFu) << 23) * idir.x;
        const float sy = __uint_as_float(((e >> 8) & 0xFFu) << 23) * idir.y;
        const float sz = __uint_as_float(((e >> 16) & 0xFFu) << 23) * idir.z;
        const float bx = (q0.x - o.x) * idir.x, by = (q0.y - o.y) * idir.y, bz = (q0.z - o.z) * idir.z;
        const uint32_t w0 = __float_as_uint(q1.x), w1 = __float_as_uint(q1.y), w2 = __float_as_uint(q1.z);
        const int split = __float_as_int(q1.w);
        r.ax0 = fmaf(u8f(w0, 0), sx, bx); r.ax1 = fmaf(u8f(w0, 3), sx, bx);
        r.ay0 = fmaf(u8f(w0, 1), sy, by); r.ay1 = fmaf(u8f(w1, 0), sy, by);
        r.az0 = fmaf(u8f(w0, 2), sz, bz); r.az1 = fmaf(u8f(w1, 1), sz, bz);
        r.bx0 = fmaf(u8f(w1, 2), sx, bx); r.bx1 = fmaf(u8f(w2, 1), sx, bx);
        r.by0 = fmaf(u8f(w1, 3), sy, by); r.by1 = fmaf(u8f(w2, 2), sy, by);
        r.bz0 = fmaf(u8f(w2, 0), sz, bz); r.bz1 = fmaf(u8f(w2, 3), sz, bz);
        r.ca = ((e >> 24) & 1u) ? ~split : split;
        r.cb = ((e >> 25) & 1u) ? ~(split + 1) : split + 1;
        return;
    }
    const float4* np = s.nodes + 4 * (size_t)node;
    float4 n0, n1, n2, n3;
    ldg8(np, n0, n1);
    ldg8(np + 2, n2, n3);
    r.ax0 = fmaf(n0.x, idir.x, -ood.x); r.ax1 = fmaf(n0.y, idir.x, -ood.x);
    r.ay0 = fmaf(n0.z, idir.y, -ood.y); r.ay1 = fmaf(n0.w, idir.y, -ood.y);
    r.az0 = fmaf(n2.x, idir.z, -ood.z); r.az1 = fmaf(n2.y, idir.z, -ood.z);
    r.bx0 = fmaf(n1.x, idir.x, -ood.x); r.bx1 = fmaf(n1.y, idir.x, -ood.x);
    r.by0 = fmaf(n1.z, idir.y, -ood.y); r.by1 = fmaf(n1.w, idir.y, -ood.y);
    r.bz0 = fmaf(n2.z, idir.z, -ood.z); r.bz1 = fmaf(n2.w, idir.z, -ood.z);
    r.ca = __float_as_int(n3.x);
    r.cb = __float_as_int(n3.y);
}

// Binary-node traversal (Aila–Laine node layout): near child first, far child pushed.  The
// stack (ShortStack: shared memory, then local memory) holds at most one entry per level.  ANY as in
// trace_closest_wide.
template <bool ANY, typename Stack>
__device__ __forceinline__ bool trace_closest_bvh2(const SceneView& s, float3 o, float3 d, float tmin, float tmax,
                                                   Hit& hit, int* err, int skip)
{
    const float3 idir = safe_inverse(d);
    const float3 ood = f3(o.x * idir.x, o.y * idir.y, o.z * idir.z);
    Stack stack;
    stack.init();
    int sp = 0;
    int node = 0;
    float best = tmax;
    for (;;) {
        Bvh2Slabs r;
        bvh2_slabs(s, node, o, idir, ood, r);
        float an = fmaxf(fmaxf(fminf(r.ax0, r.ax1), fminf(r.ay0, r.ay1)), fmaxf(fminf(r.az0, r.az1), tmin));
        float af = fminf(fminf(fmaxf(r.ax0, r.ax1), fmaxf(r.ay0, r.ay1)), fminf(fmaxf(r.az0, r.az1), best));
        float bn = fmaxf(fmaxf(fminf(r.bx0, r.bx1), fminf(r.by0, r.by1)), fmaxf(fminf(r.bz0, r.bz1), tmin));
        float bf = fminf(fminf(fmaxf(r.bx0, r.bx1), fmaxf(r.by0, r.by1)), fminf(fmaxf(r.bz0, r.bz1), best));
        int ca = r.ca, cb = r.cb;
        bool ha = an <= af, hb = bn <= bf;
        if (ha && ca < 0 && visit_leaf<ANY ? Q_ANY : Q_CLOSEST>(s, ~ca, o, d, best, hit, skip, ANY)) return true;
        if (hb && cb < 0 && visit_leaf<ANY ? Q_ANY : Q_CLOSEST>(s, ~cb, o, d, best, hit, skip, ANY)) return true;
        bool ta = ha && ca >= 0, tb = hb && cb >= 0;
        if (ta && tb) {
            bool anear = an <= bn;
            if (sp >= CPT_STACK) {
                if (err) atomicOr(err, CPT_DEVERR_STACK);
                break;
            }
            stack.put(sp++, anear ? cb : ca);
            node = anear ? ca : cb;
        } else if (ta) {
            node = ca;
        } else if (tb) {
            node = cb;
        } else {
            if (sp == 0) break;
            node = stack.get(--sp);
        }
    }
    return hit.leaf >= 0;
}

// ---------------------------------------------------------------- step-wise BVH2 traversal
// One ray's traversal state, advanced one node per call, so that a warp can refill lanes whose
// ray finished with new rays instead of waiting for its slowest lane (dynamic ray fetching,
// Aila & Laine 2009).  The visit order and pruning are those of trace_closest_bvh2.
template <Query Q, typename Stack>
struct Bvh2Walk {
    float3 o, d, idir, ood;
    float tmin, best;
    int node, sp, skip;
    bool any;   // Q_EITHER: this ray asks for any occluder
    Hit hit;
    Stack stack;   // init() once per kernel, before the first start()

    __device__ __forceinline__ void start(float3 o_, float3 d_, float tmin_, float tmax_, int skip_, bool any_ = false)
    {
        o = o_;
        d = d_;
        idir = safe_inverse(d_);
        ood = f3(o.x * idir.x, o.y * idir.y, o.z * idir.z);
        tmin = tmin_;
        best = tmax_;
        node = 0;
        sp = 0;
        skip = skip_;
        any = any_;
        hit.leaf = -1;
        hit.t = tmax_;
        hit.u = hit.v = 0.f;
    }

    // Visits one node; returns true when the traversal has finished.
    __device__ __forceinline__ bool step(const SceneView& s, int* err)
    {
        Bvh2Slabs r;
        bvh2_slabs(s, node, o, idir, ood, r);
        float an = fmaxf(fmaxf(fminf(r.ax0, r.ax1), fminf(r.ay0, r.ay1)), fmaxf(fminf(r.az0, r.az1), tmin));
        float af = fminf(fminf(fmaxf(r.ax0, r.ax1), fmaxf(r.ay0, r.ay1)), fminf(fmaxf(r.az0, r.az1), best));
        float bn = fmaxf(fmaxf(fminf(r.bx0, r.bx1), fminf(r.by0, r.by1)), fmaxf(fminf(r.bz0, r.bz1), tmin));
        float bf = fminf(fminf(fmaxf(r.bx0, r.bx1), fmaxf(r.by0, r.by1)), fminf(fmaxf(r.bz0, r.bz1), best));
        int ca = r.ca, cb = r.cb;
        bool ha = an <= af, hb = bn <= bf;
        if (ha && ca < 0 && visit_leaf<Q>(s, ~ca, o, d, best, hit, skip, any)) return true;
        if (hb && cb < 0 && visit_leaf<Q>(s, ~cb, o, d, best, hit, skip, any)) return true;
        bool ta = ha && ca >= 0, tb = hb && cb >= 0;
        if (ta && tb) {
            bool anear = an <= bn;
            if (sp >= CPT_STACK) {
                if (err) atomicOr(err, CPT_DEVERR_STACK);
                return true;
            }
            stack.put(sp++, anear ? cb : ca);
            node = anear ? ca : cb;
        } else if (ta) {
            node = ca;
        } else if (tb) {
            node = cb;
        } else {
            if (sp == 0) return true;
            node = stack.get(--sp);
        }
        return false;
    }
};

__device__ __forceinline__ uint32_t lane_mask_lt()
{
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Traces work items [0, n) through the BVH2 with dynamic fetching: every loop trip each busy lane
// advances its ray by one node, and once CPT_REFILL lanes (or all) are idle they take the next
// items from *fetch (one atomic per warp).  load(i, o, d, tmin, tmax, skip, scene) supplies item
// i's ray (skip: the light an occlusion query aims at; scene: which of views(scene) it traverses,
// for batches that mix scenes), store(i, hit) takes its result (for ANY, hit.leaf >= 0 means
// occluded).  All 32 lanes of every warp must call this together.  Returns the number of rays
// traced by the lane.
constexpr int CPT_REFILL = 8;

// SPREAD: fewer items than lanes are spread over all warps (a warp with one ray steps without
// divergence, so a few rays are answered in the time of their own steps).
template <typename Walk, bool SPREAD = false, typename Views, typename Load, typename Store>
__device__ __forceinline__ uint32_t trace_items_walk(const Views& views, int n, int* fetch, int* err, Load load,
                                                     Store store)
{
    const int lane = threadIdx.x & 31;
    Walk w;
    w.stack.init();
    int item = -1, scene = 0;
    bool exhausted = false;
    uint32_t rays = 0;
    int lanes = 32;   // of this warp that take items
    if (SPREAD) lanes = spread_lanes(n, (int)(gridDim.x * (blockDim.x >> 5)));
    for (;;) {
        const bool idle = item < 0 && (!SPREAD || lane < lanes);
        const uint32_t m = __ballot_sync(0xffffffffu, idle);
        // refill once at least CPT_REFILL lanes are idle (one atomic and one divergent ray load per
        // batch instead of per finished ray): 1 -> 8 lanes is +10 % on the 1080p render (16: same)
        if (__popc(m) >= (SPREAD ? min(CPT_REFILL, lanes) : CPT_REFILL) && !exhausted) {
            uint32_t base = 0;
            if (lane == 0) base = (uint32_t)atomicAdd(fetch, __popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (fetch_ends(base, __popc(m), n)) exhausted = true;
            if (idle) {
                const uint32_t r = base + (uint32_t)__popc(m & lane_mask_lt());
                if (is_item(r, n)) {
                    float3 o, d;
                    float tmn, tmx;
                    int skip = -1;
                    item = (int)r;
                    load(item, o, d, tmn, tmx, skip, scene);
                    w.start(o, d, tmn, tmx, skip);
                    rays++;
                }
            }
        }
        if (__all_sync(0xffffffffu, item < 0)) break;
        if (item >= 0 && w.step(views(scene), err)) {
            store(item, w.hit, scene);
            item = -1;
        }
    }
    return rays;
}

template <bool ANY, typename Stack, bool SPREAD = false, typename Views, typename Load, typename Store>
__device__ __forceinline__ uint32_t trace_items_bvh2_views(const Views& views, int n, int* fetch, int* err, Load load,
                                                           Store store)
{
    return trace_items_walk<Bvh2Walk<ANY ? Q_ANY : Q_CLOSEST, Stack>, SPREAD>(views, n, fetch, err, load, store);
}

// Dynamic fetching over the 8-wide BVH (the same refill policy).
template <bool ANY, typename Stack64, bool SPREAD = false, typename Views, typename Load, typename Store>
__device__ __forceinline__ uint32_t trace_items_wide_views(const Views& views, int n, int* fetch, int* err, Load load,
                                                           Store store)
{
    return trace_items_walk<WideWalk<ANY ? Q_ANY : Q_CLOSEST, Stack64>, SPREAD>(views, n, fetch, err, load, store);
}

// Closest hit over [tmin (boxes), tmax]; false on a miss.  WIDE selects the traversal layout at
// compile time (each kernel is instantiated for the layout the scene was built with), so a
// kernel carries the registers and code of one traversal only.  *err gets CPT_DEVERR_STACK if a
// fixed stack would overflow.  With ANY the query is an occlusion test (see occluded).  Stack is
// where the binary traversal keeps its stack (ShortStack needs short_stack_bytes at launch).
template <bool WIDE, bool ANY = false, typename Stack = ShortStack>
__device__ __forceinline__ bool trace_closest(const SceneView& s, float3 o, float3 d, float tmin, float tmax, Hit& hit,
                                              int* err, int skip = -1)
{
    hit.leaf = -1;
    hit.t = tmax;
    hit.u = hit.v = 0.f;
    if (s.n_prims <= 0) return false;
    if (s.n_internal == 0) {
        float best = tmax;
        visit_leaf<ANY ? Q_ANY : Q_CLOSEST>(s, 0, o, d, best, hit, skip, ANY);
        return hit.leaf >= 0;
    }
    if (WIDE) return trace_closest_wide<ANY>(s, o, d, tmin, tmax, hit, err, skip);
    return trace_closest_bvh2<ANY, Stack>(s, o, d, tmin, tmax, hit, err, skip);
}

// Visibility of light `light` along a shadow ray whose hit on that light is at t_light (from
// hit_light with the same origin and direction).  The reference's test is "the closest hit is
// that light" (Render.cu:178-181); except for exact ties in t it equals "nothing but that light is
// hit in [0.001, t_light]", which this occlusion query answers and which stops at the first
// occluder instead of searching for the closest one.
template <bool WIDE, typename Stack = ShortStack>
__device__ __forceinline__ bool occluded(const SceneView& s, float3 o, float3 d, float t_light, int light, int* err)
{
    Hit h;
    return trace_closest<WIDE, true, Stack>(s, o, d, 0.001f, t_light, h, err, light);
}

}  // namespace cpt
