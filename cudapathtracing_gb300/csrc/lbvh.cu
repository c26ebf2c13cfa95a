// lbvh.cu — LBVH construction on the GPU (Device::buildBVH, Device.cuh:169-195).
//
//   k_prep        centroid (FP64) + Morton code + leaf box per primitive
//                 (generateMortonCodes Device.cuh:134-142, morton3D BVH.cuh:23-41,
//                  Hittable ctors Hittable.cuh:456-462)
//   radix sort    stable LSD over the 30-bit codes, four 8-bit digits, one launch per digit: tiles
//                 take their offsets from the tiles before them while those are still running
//                 (chained scan; replaces thrust::sort_by_key Device.cuh:187-189: keys are
//                 code<<32|index, so a stable sort of codes with ascending indices is the
//                 same permutation)
//   k_tree        the Karras 2012 hierarchy with its boxes, a thread per node
//                 (generateHierarchy BVH.cuh:174-241, constructAABB BVH.cuh:243-280)
//   refit         (moved vertices, same topology) atomic-free: an internal node covers the
//                 contiguous sorted leaves [first, last], so its box is a range union, answered
//                 from a 4-ary pyramid of unions of the leaf boxes (min/max is exact, so the boxes
//                 equal the pairwise unions)
//
// All boxes are FP32 rounded outwards from the reference's FP64 boxes.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "cpt_internal.h"
#include "cpt_quant.cuh"

namespace cg = cooperative_groups;

namespace cpt {

namespace {

constexpr int RS_BITS = 8;
constexpr int RS_BINS = 1 << RS_BITS;
constexpr uint32_t RS_MASK = RS_BINS - 1;
constexpr int RS_PASSES = 4;                     // bits 0-7, 8-15, 16-23, 24-31: the whole 30-bit code
static_assert(RS_BITS * RS_PASSES >= 30 && RS_PASSES % 2 == 0, "radix digits");

__device__ __forceinline__ uint32_t expand_bits(uint32_t v)   // BVH.cuh:12-19
{
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

// morton3D (BVH.cuh:23-41) in double with explicitly rounded operations (no contraction).
__device__ __forceinline__ uint32_t morton_axis(double c, double mn, double mx)
{
    double nrm = __ddiv_rn(__dsub_rn(c, mn), __dsub_rn(mx, mn));
    double x = __dmul_rn(nrm, 1024.0);
    x = x > 0.0 ? x : 0.0;        // mMax(x, 0.0): NaN -> 0
    x = x < 1023.0 ? x : 1023.0;  // mMin(x, 1023.0)
    return (uint32_t)x;
}

__device__ __forceinline__ double dmin(double a, double b) { return a < b ? a : b; }   // mMin
__device__ __forceinline__ double dmax(double a, double b) { return a > b ? a : b; }   // mMax

template <typename VT>
__device__ __forceinline__ void load_tri(const VT* __restrict__ v, uint32_t t, double p[9])
{
#pragma unroll
    for (int k = 0; k < 9; ++k) p[k] = (double)v[9ull * t + k];
}

// Constants of the fast Morton paths for one axis: the reference's bounds, the scale
// k = 1024 / (max - min) in FP64, and min and k as FP32 (hi) and as unevaluated FP32 pairs
// (hi + lo, within 2^-48 relative of the FP64 values).
struct MortonAxis {
    double mn, mx, k64;
    float mn32, k32;      // RN32(min), RN32(k)
    float mn_lo, k_lo;    // RN32(min - mn32), RN32(k - k32)
};

// floor(x) for 0 <= x < 2^23 on the integer units, without conversion or directed-rounding
// instructions: f = x with its fractional mantissa bits cleared, and the integer from the
// significand shifted by the exponent.
__device__ __forceinline__ int floor_small(float x, float& f)
{
    const uint32_t b = __float_as_uint(x);
    const int e = (int)(b >> 23) - 127;
    if (e < 0) {
        f = 0.0f;
        return 0;
    }
    const uint32_t sh = 23u - (uint32_t)e;
    f = __uint_as_float(b & ~((1u << sh) - 1u));
    return (int)(((b & 0x7FFFFFu) | 0x800000u) >> sh);
}

// Morton cell of a triangle-centroid coordinate, equal to the reference's exactly rounded FP64
// sequence morton_axis(RN((p0 + p1 + p2) / 3), min, max) (BVH.cuh:23-33 on the centroid of
// Hittable.cuh:459-461), computed without its two FP64 divisions where that is provably safe:
//   1. FP32: x = (s * (1/3) - min) * k with s = p0 + p1 + p2.  Its distance to the reference's
//      x is below tol = 2^-20 (k (|p0| + |p1| + |p2| + |min|) + 2 |x|), four times the worst-case
//      sum of the rounding errors (two additions, the multiplications and the rounded 1/3 and
//      k, each at most 2^-24 relative).  The cell is floor(x) when x is farther than tol from
//      every cell boundary (the integers 1 .. 1023; below 1 the cell is 0, at or above 1023 it
//      is 1023).
//   2. Otherwise the same in unevaluated pairs of FP32 numbers (TwoSum and FMA-based TwoProd,
//      about 44 significant bits), with tol = 2^-40 (...): still on the FP32 units, whereas one
//      lane on an FP64 path costs its whole warp the part's low FP64 issue rate.
//   3. Otherwise the reference's own sequence with IEEE divisions, in FP64.
// Non-finite intermediates (a degenerate axis) always take step 3.
__device__ __forceinline__ int cell_of(float x, float tol)
{
    if (!(tol < 0.25f) || !(fabsf(x) < 1e30f)) return -1;   // also rejects NaN and infinities
    if (x < 1.0f - tol) return 0;
    if (x > 1023.0f + tol) return 1023;
    float f;
    const int c = floor_small(x, f);   // here 1 - tol <= x <= 1023 + tol
    return (x - f > tol && f + 1.0f - x > tol) ? c : -1;
}

// Step 3.  Out of line, with the widening inside, so that the compiler cannot evaluate any of it
// speculatively beside the FP32 steps.
template <typename VT>
__device__ __noinline__ uint32_t morton_tri_axis_fp64(VT a_, VT b_, VT c_, MortonAxis m)
{
    const double a = (double)a_, b = (double)b_, c = (double)c_;
    return morton_axis(__ddiv_rn(__dadd_rn(__dadd_rn(a, b), c), 3.0), m.mn, m.mx);
}

// Error-free transformations on FP32 (Knuth's TwoSum; the product's error from one FMA).
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e)
{
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

__device__ __forceinline__ void two_prod(float a, float b, float& p, float& e)
{
    p = __fmul_rn(a, b);
    e = __fmaf_rn(a, b, -p);
}

constexpr float THIRD_HI = 0x1.555556p-2f;    // RN32(1/3)
constexpr float THIRD_LO = -0x1.555556p-27f;  // RN32(1/3 - THIRD_HI); the rest is below 2^-50

// Step 2 (and 3 where it cannot decide).  Out of line: it runs for a fraction of a percent of the
// coordinates.
__device__ __noinline__ uint32_t morton_tri_axis_ff(float a, float b, float c, MortonAxis m)
{
    // s = a + b + c as hi + lo
    float s1, e1, s2, e2;
    two_sum(a, b, s1, e1);
    two_sum(s1, c, s2, e2);
    const float slo = __fadd_rn(e1, e2);
    // y = s / 3
    float y, ye;
    two_prod(s2, THIRD_HI, y, ye);
    ye = __fadd_rn(ye, __fadd_rn(__fmul_rn(s2, THIRD_LO), __fmul_rn(slo, THIRD_HI)));
    // z = y - min
    float z, ze;
    two_sum(y, -m.mn32, z, ze);
    ze = __fadd_rn(ze, __fsub_rn(ye, m.mn_lo));
    // x = z * k
    float x, xe;
    two_prod(z, m.k32, x, xe);
    xe = __fadd_rn(xe, __fadd_rn(__fmul_rn(z, m.k_lo), __fmul_rn(ze, m.k32)));
    const float mag = fabsf(a) + fabsf(b) + fabsf(c) + fabsf(m.mn32);
    const float tol = 0x1p-40f * (m.k32 * mag + 2.0f * fabsf(x));
    if (isfinite(x) && isfinite(xe) && isfinite(tol) && tol < 0.25f) {
        const float xs = __fadd_rn(x, xe);
        if (xs < 1.0f - tol) return 0u;
        if (xs > 1023.0f + tol) return 1023u;
        float f;
        const int cell = floor_small(fminf(fmaxf(x, 0.0f), 1024.0f), f);
        // signed distances of x + xe above floor(x) and below floor(x) + 1 (x - f and f + 1 - x are
        // exact); xe can move the sum across either integer
        const float below = __fadd_rn(__fsub_rn(x, f), xe), above = __fsub_rn(__fsub_rn(__fadd_rn(f, 1.0f), x), xe);
        if (below > tol && above > tol) return (uint32_t)min(cell, 1023);
        if (below < -tol && cell >= 1) return (uint32_t)min(cell - 1, 1023);
        if (above < -tol) return (uint32_t)min(cell + 1, 1023);
    }
    return morton_tri_axis_fp64<float>(a, b, c, m);
}

template <typename VT>
__device__ __forceinline__ uint32_t morton_tri_axis(VT a, VT b, VT c, const MortonAxis& m)
{
    const float a32 = (float)a, b32 = (float)b, c32 = (float)c;
    const float x32 = ((a32 + b32 + c32) * (1.0f / 3.0f) - m.mn32) * m.k32;
    const float mag = fabsf(a32) + fabsf(b32) + fabsf(c32) + fabsf(m.mn32);
    const float tol32 = 0x1p-20f * (m.k32 * mag + 2.0f * fabsf(x32));
    const int cell = cell_of(x32, tol32);
    if (cell >= 0) return (uint32_t)cell;
    return morton_tri_axis_ff(a32, b32, c32, m);
}

// Triangle centroid and padded box (Hittable.cuh:459-461, AABB.cuh:30-40), boxes rounded
// outwards to FP32.
__device__ __forceinline__ void tri_center_box(const double p[9], double c[3], float4& bmin, float4& bmax)
{
    double mn[3], mx[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        c[a] = __ddiv_rn(__dadd_rn(__dadd_rn(p[a], p[3 + a]), p[6 + a]), 3.0);
        mn[a] = __dsub_rn(dmin(dmin(p[a], p[3 + a]), p[6 + a]), 0.0001);
        mx[a] = __dadd_rn(dmax(dmax(p[a], p[3 + a]), p[6 + a]), 0.0001);
    }
    bmin = make_float4(__double2float_rd(mn[0]), __double2float_rd(mn[1]), __double2float_rd(mn[2]), 0.f);
    bmax = make_float4(__double2float_ru(mx[0]), __double2float_ru(mx[1]), __double2float_ru(mx[2]), 0.f);
}

// Conversions between FP32 and FP64 by bit manipulation on the integer units: on this part the
// FP64 pipe also executes the hardware conversions, and it is the scarce resource of k_prep.
// widen: exact float -> double.  narrow_rd / narrow_ru: double -> float rounded down / up.  Values
// outside the normal range of the narrower type take the hardware conversion, out of line (an
// inline conversion is evaluated for every value and then discarded by a select).
__device__ __noinline__ double widen_hw(float f) { return (double)f; }
__device__ __noinline__ float narrow_hw_rd(double d) { return __double2float_rd(d); }
__device__ __noinline__ float narrow_hw_ru(double d) { return __double2float_ru(d); }

__device__ __forceinline__ double widen(float f)
{
    const uint32_t b = __float_as_uint(f);
    const uint32_t e = (b >> 23) & 0xFFu;
    if (e == 0u || e == 0xFFu) return widen_hw(f);   // zero, subnormal, infinity, NaN
    const uint32_t hi = (b & 0x80000000u) | ((e + 896u) << 20) | ((b & 0x7FFFFFu) >> 3);
    return __hiloint2double((int)hi, (int)(b << 29));
}

template <bool UP>
__device__ __forceinline__ float narrow(double d)
{
    const uint32_t hi = (uint32_t)__double2hiint(d), lo = (uint32_t)__double2loint(d);
    const uint32_t e = (hi >> 20) & 0x7FFu;
    if (e < 897u || e > 1150u) return UP ? narrow_hw_ru(d) : narrow_hw_rd(d);
    uint32_t fb = (hi & 0x80000000u) | ((e - 896u) << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29);
    const bool inexact = (lo & 0x1FFFFFFFu) != 0u;
    const bool negative = (hi >> 31) != 0u;
    // truncation rounds the magnitude down; moving away from zero is one step up in the bits
    if (inexact && (UP ? !negative : negative)) fb += 1u;
    return __uint_as_float(fb);
}

// The reference's padding in FP64: RD32(RN64(x - 1e-4)) (UP false) or RU32(RN64(x + 1e-4)).
template <bool UP>
__device__ __noinline__ float pad_fp64(float x)
{
    return UP ? narrow<true>(__dadd_rn(widen(x), 0.0001)) : narrow<false>(__dsub_rn(widen(x), 0.0001));
}

// The same value from FP32 operations.  c = RN64(1e-4) is split as PAD_HI + PAD_LO (PAD_HI =
// RN32(c), PAD_LO = RN32(c - PAD_HI) = 2.53e-12, within 2^-62 of the exact remainder).  TwoSum
// gives x -+ PAD_HI = s + e exactly, so the exact q = x -+ c is s + r with r = e -+ PAD_LO.  For
// |s| >= 2^-10, |r| is below half the spacing of the floats next to s, so the directed rounding of
// q is s or its neighbour, by the sign of r.  It equals the rounding of RN64(q) unless RN64 moves
// q onto or across s, which needs |r| <= 2^-53 |q|.  The result is therefore certain when |r| >
// 2^-50 |s| (double rounding) + 2^-23 |r| (rounding of r) + 2^-62 (PAD_LO); otherwise, and for
// |s| outside [2^-10, 2^100) or a non-finite x, the FP64 sequence runs.  tests/test_pad_fp32.py
// restates this in numpy float32 and compares it bit for bit with the FP64 sequence on sweeps of
// float32 bit patterns; coordinates of magnitude 0.01 .. 4000 never take the fallback.
constexpr float PAD_HI = 0x1.a36e2ep-14f;
constexpr float PAD_LO = 0x1.638866p-39f;

template <bool UP>
__device__ __forceinline__ float pad_fp32(float x)
{
    const float h = UP ? PAD_HI : -PAD_HI;
    const float s = __fadd_rn(x, h);
    const float bb = __fsub_rn(s, x);
    const float e = __fadd_rn(__fsub_rn(x, __fsub_rn(s, bb)), __fsub_rn(h, bb));
    const float r = UP ? __fadd_rn(e, PAD_LO) : __fsub_rn(e, PAD_LO);
    const float as = fabsf(s);
    const float tol = 0x1p-50f * as + 0x1p-23f * fabsf(r) + 0x1p-62f;
    if (!(as >= 0x1p-10f && as < 0x1p100f) || !(fabsf(r) > tol)) return pad_fp64<UP>(x);
    const uint32_t sb = __float_as_uint(s);
    const bool away = UP ? r > 0.f : r < 0.f;   // the neighbour of s in the rounding direction
    const bool neg = (sb >> 31) != 0u;
    return away ? __uint_as_float((UP != neg) ? sb + 1u : sb - 1u) : s;
}

// Padded triangle box (AABB::pad, AABB.cuh:30-40) rounded outwards to FP32.  For FP32 vertices
// the minimum and maximum are exact in FP32; the padding is the reference's FP64 operation,
// evaluated by pad_fp32.
__device__ __forceinline__ void tri_box(const float p[9], float4& bmin, float4& bmax)
{
    float mn[3], mx[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        mn[a] = fminf(fminf(p[a], p[3 + a]), p[6 + a]);
        mx[a] = fmaxf(fmaxf(p[a], p[3 + a]), p[6 + a]);
    }
    bmin = make_float4(pad_fp32<false>(mn[0]), pad_fp32<false>(mn[1]), pad_fp32<false>(mn[2]), 0.f);
    bmax = make_float4(pad_fp32<true>(mx[0]), pad_fp32<true>(mx[1]), pad_fp32<true>(mx[2]), 0.f);
}

// Codes and boxes of all primitives, and (they do not depend on the order) the digit totals of every
// sort pass: totals[pass][digit].
constexpr int PREP_THREADS = 256;
constexpr unsigned PREP_BLOCKS = 152 * 8;   // each adds its 1,024 digit counts once
template <typename VT>
__global__ void __launch_bounds__(PREP_THREADS) k_prep(uint32_t n_extra, const double* __restrict__ extra_c, const float4* __restrict__ extra_box,
                       uint32_t n_tri, const VT* __restrict__ tri_v, MortonAxis ax, MortonAxis ay, MortonAxis az,
                       uint32_t* __restrict__ code, float4* __restrict__ box, uint32_t* __restrict__ totals)
{
    __shared__ uint32_t hist[RS_PASSES][RS_BINS];
    for (int t = threadIdx.x; t < RS_PASSES * RS_BINS; t += PREP_THREADS) (&hist[0][0])[t] = 0;
    __syncthreads();
    const uint32_t n = n_extra + n_tri;
    for (uint64_t i64 = blockIdx.x * (uint64_t)PREP_THREADS + threadIdx.x; i64 < n; i64 += gridDim.x * (uint64_t)PREP_THREADS) {
    const uint32_t i = (uint32_t)i64;
    float4 bmin, bmax;
    uint32_t xx, yy, zz;
    if (i < n_extra) {
        bmin = extra_box[2ull * i];
        bmax = extra_box[2ull * i + 1];
        xx = morton_axis(extra_c[3ull * i], ax.mn, ax.mx);
        yy = morton_axis(extra_c[3ull * i + 1], ay.mn, ay.mx);
        zz = morton_axis(extra_c[3ull * i + 2], az.mn, az.mx);
    } else if (sizeof(VT) == sizeof(float)) {
        const float* v = reinterpret_cast<const float*>(tri_v) + 9ull * (i - n_extra);
        float p[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) p[k] = __ldg(v + k);
        tri_box(p, bmin, bmax);
        xx = morton_tri_axis(p[0], p[3], p[6], ax);
        yy = morton_tri_axis(p[1], p[4], p[7], ay);
        zz = morton_tri_axis(p[2], p[5], p[8], az);
    } else {
        double p[9], c[3];
        load_tri(tri_v, i - n_extra, p);
        tri_center_box(p, c, bmin, bmax);
        xx = morton_axis(c[0], ax.mn, ax.mx);
        yy = morton_axis(c[1], ay.mn, ay.mx);
        zz = morton_axis(c[2], az.mn, az.mx);
    }
    const uint32_t c = expand_bits(xx) * 4 + expand_bits(yy) * 2 + expand_bits(zz);
    code[i] = c;
    box[2ull * i] = bmin;
    box[2ull * i + 1] = bmax;
#pragma unroll
    for (int p = 0; p < RS_PASSES; ++p) atomicAdd(&hist[p][(c >> (RS_BITS * p)) & RS_MASK], 1u);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < RS_PASSES * RS_BINS; t += PREP_THREADS) {
        const uint32_t v = (&hist[0][0])[t];
        if (v) atomicAdd(&totals[t], v);
    }
}

template <typename VT>
__global__ void k_prim_boxes(uint32_t n_extra, const float4* __restrict__ extra_box, uint32_t n_tri,
                             const VT* __restrict__ tri_v, const uint32_t* __restrict__ order,
                             float4* __restrict__ leaf_box, uint32_t n)
{
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    uint32_t i = order[k];
    float4 bmin, bmax;
    if (i < n_extra) {
        bmin = extra_box[2ull * i];
        bmax = extra_box[2ull * i + 1];
    } else if (sizeof(VT) == sizeof(float)) {
        const float* v = reinterpret_cast<const float*>(tri_v) + 9ull * (i - n_extra);
        float p[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) p[q] = __ldg(v + q);
        tri_box(p, bmin, bmax);
    } else {
        double p[9], c[3];
        load_tri(tri_v, i - n_extra, p);
        tri_center_box(p, c, bmin, bmax);
    }
    leaf_box[2ull * k] = bmin;
    leaf_box[2ull * k + 1] = bmax;
}

// ---------------------------------------------------------------- radix sort
__device__ __forceinline__ uint32_t lanemask_lt()
{
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Inclusive sum of x over the block's first RS_BINS threads (s_part: RS_BINS / 32 words; every thread
// of the block calls it; the caller synchronises before s_part is used again).
__device__ __forceinline__ uint32_t bins_scan(uint32_t x, uint32_t* s_part)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31 && w < RS_BINS / 32) s_part[w] = x;
    __syncthreads();
    for (int q = 0; q < min(w, RS_BINS / 32); ++q) x += s_part[q];
    return x;
}

// Progress of one (tile, digit) of a pass: nothing yet, the tile's own count, or the count over all
// tiles up to it.  The two top bits say which, the rest is the count, so one store publishes both.
template <typename Word>
struct Chain {
    static constexpr int SHIFT = sizeof(Word) * 8 - 2;
    static constexpr Word VALUE = ((Word)1 << SHIFT) - 1;
    static __device__ __forceinline__ Word own(uint32_t c) { return ((Word)1 << SHIFT) | c; }
    static __device__ __forceinline__ Word total(Word c) { return ((Word)2 << SHIFT) | c; }
};

// One digit of the stable LSD sort (Adinets and Merrill, "Onesweep", 2022): a block takes the next
// tile, ranks its keys by the digit (warp-ordered, lane-ordered), publishes its counts, adds up the
// counts of the tiles before it (thread d for digit d) and writes its keys to their places, staged in
// shared memory so that equal digits leave as runs.  Tiles are taken in order, so those before a tile
// are done or running; a count that is not there after CHAIN_POLLS looks is counted from the keys
// instead of waited for.
//
// The sort is bound by latency at these sizes (1.31M keys: 5 MB a buffer, in L2): one launch a digit
// in place of three, with 8-bit digits (32-key runs, 256 counters a warp) in place of 10-bit ones.
// 1.31M keys: 158 -> 91 us, 12,500: 91 -> 28 us.  Of the 158 us, 52 went to match instructions.  Tiles of
// 2,048 keys took 29 us a pass (every tile adds up the hundreds running beside it) against 23.
//
// FIRST: the values are the positions.
#ifndef CPT_CHAIN_POLLS
#define CPT_CHAIN_POLLS 4096
#endif
#ifndef CPT_CHAIN_WIDE_FROM
#define CPT_CHAIN_WIDE_FROM (1u << 30)   // primitives; at least SORT_MEDIUM + 1
#endif
constexpr int CHAIN_POLLS = CPT_CHAIN_POLLS;
constexpr int CHAIN_BATCH = 8;   // tiles a thread fetches at once

template <int THREADS, int ITEMS, typename Word>
struct SortSmem {
    uint32_t wh[THREADS / 32][RS_BINS];   // per-warp digit counts, then per-warp exclusive offsets
    uint32_t start[RS_BINS];              // tile-local start of each digit
    uint32_t gofs[RS_BINS];               // global start of each digit's run of this tile
    uint32_t keys[THREADS * ITEMS], vals[THREADS * ITEMS];
    uint32_t part0[RS_BINS / 32], part1[RS_BINS / 32];
    uint32_t tile;
    Word sum[THREADS / RS_BINS][RS_BINS];   // look-back: sums of the groups of threads, flagged when closed
};

template <int THREADS, int ITEMS, typename Word, bool FIRST>
__global__ void __launch_bounds__(THREADS, 1) k_sort_digit(const uint32_t* __restrict__ keys_in,
                                                           const uint32_t* __restrict__ vals_in,
                                                           uint32_t* __restrict__ keys_out,
                                                           uint32_t* __restrict__ vals_out, uint32_t n, int shift,
                                                           const uint32_t* __restrict__ totals, Word* state,
                                                           uint32_t* ticket)
{
    constexpr int TILE = THREADS * ITEMS, WARPS = THREADS / 32, GROUPS = THREADS / RS_BINS;
    extern __shared__ __align__(16) unsigned char sort_smem[];
    SortSmem<THREADS, ITEMS, Word>& S = *reinterpret_cast<SortSmem<THREADS, ITEMS, Word>*>(sort_smem);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, d_own = threadIdx.x;
    const bool has_digit = d_own < RS_BINS;
    if (threadIdx.x == 0) S.tile = atomicAdd(ticket, 1u);
    for (int q = threadIdx.x; q < WARPS * RS_BINS; q += THREADS) (&S.wh[0][0])[q] = 0;
    const uint32_t digit_total = has_digit ? totals[d_own] : 0u;
    __syncthreads();
    const uint32_t tile = S.tile;
    const uint32_t base = tile * TILE + w * 32 * ITEMS;
    const uint32_t lt = lanemask_lt();
    uint32_t k[ITEMS], v[ITEMS], rank[ITEMS];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const uint32_t e = base + it * 32 + lane;
        const bool valid = e < n;
        k[it] = valid ? keys_in[e] : 0u;
        v[it] = FIRST ? e : (valid ? vals_in[e] : 0u);
    }
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const bool valid = base + it * 32 + lane < n;
        const uint32_t d = (k[it] >> shift) & RS_MASK;
        // lanes with the same digit: a vote per bit (__match_any_sync takes a turn per distinct value)
        uint32_t peers = __ballot_sync(0xffffffffu, valid);
        if (!valid) peers = ~peers;
#pragma unroll
        for (int bit = 0; bit < RS_BITS; ++bit) {
            const bool one = (d >> bit) & 1u;
            const uint32_t votes = __ballot_sync(0xffffffffu, one);
            peers &= one ? votes : ~votes;
        }
        const int leader = __ffs(peers) - 1;
        uint32_t old = 0;
        if (lane == leader && valid) {
            old = S.wh[w][d];
            S.wh[w][d] = old + __popc(peers);
        }
        rank[it] = __shfl_sync(0xffffffffu, old, leader) + __popc(peers & lt);
        __syncwarp();
    }
    __syncthreads();
    // thread d: exclusive prefix of digit d over the warps (in place) and its count in the tile
    uint32_t count = 0;
    volatile Word* mine = state + (size_t)tile * RS_BINS + d_own;
    if (has_digit) {
#pragma unroll 8
        for (int q = 0; q < WARPS; ++q) {
            const uint32_t c = S.wh[q][d_own];
            S.wh[q][d_own] = count;
            count += c;
        }
        *mine = tile ? Chain<Word>::own(count) : Chain<Word>::total(count);
    }
    const uint32_t tile_start = bins_scan(count, S.part0) - count;
    const uint32_t digit_base = bins_scan(digit_total, S.part1) - digit_total;
    Word before = 0;   // keys with this digit in earlier tiles
    bool done = false;
    // Windows of GROUPS x CHAIN_BATCH tiles, nearest first: group q of 256 threads adds up its
    // CHAIN_BATCH tiles (fetched together), thread d of the first group joins the groups' sums.
    for (uint32_t p = tile; p > 0;) {
        const int q = threadIdx.x / RS_BINS, dg = threadIdx.x % RS_BINS;
        Word x[CHAIN_BATCH];
#pragma unroll
        for (int j = 0; j < CHAIN_BATCH; ++j) {
            const uint32_t back = q * CHAIN_BATCH + j + 1;
            x[j] = back <= p ? *(volatile const Word*)(state + (size_t)(p - back) * RS_BINS + dg) : Chain<Word>::total(0);
        }
        Word sum = 0;
        bool closed = false;
#pragma unroll
        for (int j = 0; j < CHAIN_BATCH; ++j) {
            const uint32_t back = q * CHAIN_BATCH + j + 1;
            Word y = x[j];
            if (!closed && !(y >> Chain<Word>::SHIFT)) {
                volatile const Word* theirs = state + (size_t)(p - back) * RS_BINS + dg;
                for (int polls = 0; !(y >> Chain<Word>::SHIFT) && polls < CHAIN_POLLS; ++polls) y = *theirs;
                if (!(y >> Chain<Word>::SHIFT)) {
                    uint32_t c = 0;
                    for (uint32_t e = (p - back) * TILE; e < (p - back + 1) * TILE; ++e)
                        c += ((keys_in[e] >> shift) & RS_MASK) == (uint32_t)dg;
                    y = Chain<Word>::own(c);
                }
            }
            if (!closed) sum += y & Chain<Word>::VALUE;
            closed = closed || (y >> Chain<Word>::SHIFT) == 2;
        }
        S.sum[q][dg] = (closed ? Chain<Word>::total(0) : Chain<Word>::own(0)) | sum;
        __syncthreads();
        bool open = false;
        if (has_digit && !done) {
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) {
                if (done) continue;
                before += S.sum[g][d_own] & Chain<Word>::VALUE;
                done = (S.sum[g][d_own] >> Chain<Word>::SHIFT) == 2;
            }
            open = !done;
        }
        if (!__syncthreads_or(open)) break;
        p -= min(p, (uint32_t)(GROUPS * CHAIN_BATCH));
    }
    if (has_digit) {
        if (tile) *mine = Chain<Word>::total(before + count);
        S.start[d_own] = tile_start;
        S.gofs[d_own] = digit_base + (uint32_t)before;
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        if (base + it * 32 + lane < n) {
            const uint32_t d = (k[it] >> shift) & RS_MASK;
            const uint32_t pos = S.start[d] + S.wh[w][d] + rank[it];
            S.keys[pos] = k[it];
            S.vals[pos] = v[it];
        }
    }
    __syncthreads();
    const uint32_t tile_n = min((uint32_t)TILE, n - tile * TILE);
    for (uint32_t p = threadIdx.x; p < tile_n; p += THREADS) {
        const uint32_t kk = S.keys[p];
        const uint32_t d = (kk >> shift) & RS_MASK;
        const uint32_t g = S.gofs[d] + (p - S.start[d]);
        keys_out[g] = kk;
        vals_out[g] = S.vals[p];
    }
}

// ---------------------------------------------------------------- range-union refit
// The box pyramid: level 0 is the sorted leaf boxes (n of them); level l + 1 holds
// ceil(size(l) / 4) boxes, box j the union of boxes 4j .. 4j + 3 of level l; the levels above
// the leaves are stored back to back (two float4 per box) down to a level of one box.
__device__ __forceinline__ void box_union(float4& mn, float4& mx, float4 a, float4 b)
{
    mn.x = fminf(mn.x, a.x); mn.y = fminf(mn.y, a.y); mn.z = fminf(mn.z, a.z);
    mx.x = fmaxf(mx.x, b.x); mx.y = fmaxf(mx.y, b.y); mx.z = fmaxf(mx.z, b.z);
}

__device__ __forceinline__ void empty_box(float4& mn, float4& mx)
{
    mn = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
    mx = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
}

__device__ __forceinline__ void shfl_union(float4& mn, float4& mx, int o)
{
    mn.x = fminf(mn.x, __shfl_xor_sync(0xffffffffu, mn.x, o));
    mn.y = fminf(mn.y, __shfl_xor_sync(0xffffffffu, mn.y, o));
    mn.z = fminf(mn.z, __shfl_xor_sync(0xffffffffu, mn.z, o));
    mx.x = fmaxf(mx.x, __shfl_xor_sync(0xffffffffu, mx.x, o));
    mx.y = fmaxf(mx.y, __shfl_xor_sync(0xffffffffu, mx.y, o));
    mx.z = fmaxf(mx.z, __shfl_xor_sync(0xffffffffu, mx.z, o));
}

__device__ __forceinline__ void store_box(float4* __restrict__ a, uint32_t j, float4 mn, float4 mx)
{
    a[2ull * j] = mn;
    a[2ull * j + 1] = mx;
}

constexpr int PYR_THREADS = 256;   // one block reduces 256 boxes: up to four levels per launch

// Writes the next `depth` (1 to 4) pyramid levels above a level of n boxes.  Thread t of block b
// holds box 256 b + t of that level (an empty box past n); `out` is the first level to write.
// Every thread of the block must call it (it shuffles and synchronises); depth is uniform.
__device__ __forceinline__ void pyramid_up(float4 mn, float4 mx, uint32_t n, float4* __restrict__ out, int depth)
{
    __shared__ float4 s_mn[PYR_THREADS / 16], s_mx[PYR_THREADS / 16];
    const uint32_t t = threadIdx.x, i = blockIdx.x * PYR_THREADS + t;
    shfl_union(mn, mx, 1);
    shfl_union(mn, mx, 2);
    const uint32_t n1 = (n + 3) / 4;
    if ((t & 3u) == 0 && (i >> 2) < n1) store_box(out, i >> 2, mn, mx);
    if (depth == 1) return;
    float4* out2 = out + 2ull * n1;
    shfl_union(mn, mx, 4);
    shfl_union(mn, mx, 8);
    const uint32_t n2 = (n1 + 3) / 4;
    if ((t & 15u) == 0 && (i >> 4) < n2) store_box(out2, i >> 4, mn, mx);
    if (depth == 2) return;
    if ((t & 15u) == 0) {
        s_mn[t >> 4] = mn;
        s_mx[t >> 4] = mx;
    }
    __syncthreads();
    if (t >= 32) return;
    // warp 0: lane L < 16 holds group L of 16 boxes
    if (t < PYR_THREADS / 16) {
        mn = s_mn[t];
        mx = s_mx[t];
    } else {
        empty_box(mn, mx);
    }
    float4* out3 = out2 + 2ull * n2;
    const uint32_t n3 = (n2 + 3) / 4;
    shfl_union(mn, mx, 1);
    shfl_union(mn, mx, 2);
    const uint32_t j3 = blockIdx.x * (PYR_THREADS / 64) + (t >> 2);
    if ((t & 3u) == 0 && t < PYR_THREADS / 16 && j3 < n3) store_box(out3, j3, mn, mx);
    if (depth == 3) return;
    float4* out4 = out3 + 2ull * n3;
    const uint32_t n4 = (n3 + 3) / 4;
    shfl_union(mn, mx, 4);
    shfl_union(mn, mx, 8);
    if (t == 0 && blockIdx.x < n4) store_box(out4, blockIdx.x, mn, mx);
}

// Pyramid levels above level `in` (n boxes), `depth` of them, starting at `out`.
__global__ void __launch_bounds__(PYR_THREADS) k_pyramid(const float4* __restrict__ in, uint32_t n,
                                                         float4* __restrict__ out, int depth)
{
    const uint32_t i = blockIdx.x * PYR_THREADS + threadIdx.x;
    float4 mn, mx;
    empty_box(mn, mx);
    if (i < n) {
        mn = in[2ull * i];
        mx = in[2ull * i + 1];
    }
    pyramid_up(mn, mx, n, out, depth);
}

// ---------------------------------------------------------------- hierarchy
// The binary LBVH and its boxes.  Between neighbouring sorted keys lies a gap, the length of their
// common prefix; the Karras hierarchy (generateHierarchy, BVH.cuh:174-241) has one internal node per
// gap, which splits there and covers the keys up to the nearest smaller gap on either side (all of its
// keys share gap[split] bits, and no two of its gaps are equal).  The node a parent that splits behind
// key s calls its left child has number s, its right child s + 1, the root 0; a node is a left child
// when the gap behind it is longer than the one before it, so its number is `last` then and `first`
// otherwise.
//
// k_tree: a block holds TREE_THREADS keys, thread t the gap behind key t.  Nearest smaller gaps come
// from a table of minima over 2^k gaps in shared memory, boxes from a 4-ary pyramid of box unions
// there.  Gaps whose node reaches beyond the block (about one in fifty) are listed in `crossing` for
// k_tree_top, which does the same from global memory: a search over the keys, and the pyramid of the
// blocks' upper levels.
//
// All of it is independent per node, with the warps' lanes in step.  Former passes: a search over the
// keys per node for range and split, leaf gather, pyramid, range unions and (NODES) the traversal nodes
// (1.31M keys: 150 us with the nodes' 35, bound by dependent loads with 14 of 32 lanes active); now 97
// us, with nodes 133.  Climbing from the leaves, the second child to arrive going on, took 82 us within
// blocks (11 of 32 lanes) and 58 us across them (fences).
constexpr int TREE_THREADS = 512;
constexpr int TREE_LEVELS = 9;   // 2^9 gaps
constexpr unsigned TOP_BLOCKS = 152 * 16;
// start of the block pyramid's level l: 512, 128, 32, 8 and 2 boxes
__host__ __device__ constexpr int tree_pyr(int l) { return l == 0 ? 0 : l == 1 ? 512 : l == 2 ? 640 : l == 3 ? 672 : 680; }
constexpr int TREE_BOXES = 682;
static_assert(TREE_THREADS == 1 << TREE_LEVELS, "gap table");

// Length of the common prefix of two keys (code << 32 | primitive; delta, BVH.cuh:120-128): the
// primitive word counts only when the codes are equal.  Keys are distinct.
__device__ __forceinline__ int prefix_len(uint32_t ca, uint32_t oa, uint32_t cb, uint32_t ob)
{
    return ca != cb ? __clz(ca ^ cb) : 32 + __clz(oa ^ ob);
}

struct Box6 {
    float v[6];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int a = 0; a < 6; ++a) v[a] = a < 3 ? INFINITY : -INFINITY;
    }
    __device__ __forceinline__ void add(const Box6& b)
    {
#pragma unroll
        for (int a = 0; a < 6; ++a) v[a] = a < 3 ? fminf(v[a], b.v[a]) : fmaxf(v[a], b.v[a]);
    }
};

__device__ __forceinline__ Box6 box6(float4 mn, float4 mx) { return Box6{{mn.x, mn.y, mn.z, mx.x, mx.y, mx.z}}; }

// Union of the block's boxes [lo, hi) from its pyramid in shared memory, as range_union.
__device__ __forceinline__ Box6 block_union(const float (&pyr)[6][TREE_BOXES], int lo, int hi)
{
    Box6 b;
    b.clear();
    auto take = [&](int k) {
#pragma unroll
        for (int a = 0; a < 6; ++a) b.v[a] = a < 3 ? fminf(b.v[a], pyr[a][k]) : fmaxf(b.v[a], pyr[a][k]);
    };
#pragma unroll
    for (int l = 0; l < 5; ++l) {
        const int up = (lo + 3) & ~3, dn = hi & ~3;
        if (l == 4 || up >= dn) {
            for (int j = lo; j < hi; ++j) take(tree_pyr(l) + j);
            break;
        }
        for (int j = lo; j < up; ++j) take(tree_pyr(l) + j);
        for (int j = dn; j < hi; ++j) take(tree_pyr(l) + j);
        lo = up >> 2;
        hi = dn >> 2;
    }
    return b;
}

// Writes the node that splits behind key s and covers [first, last]; box_of(lo, hi) is the union of
// leaf boxes lo .. hi - 1.
template <bool NODES, typename BoxOf>
__device__ __forceinline__ void store_node(int s, int first, int last, bool root, bool left, const BoxOf& box_of,
                                           int2* __restrict__ child, int2* __restrict__ range,
                                           float4* __restrict__ node_box, float4* __restrict__ nodes)
{
    const uint32_t i = root ? 0u : (uint32_t)(left ? last : first);
    const int2 c = make_int2(first == s ? ~s : s, s + 1 == last ? ~(s + 1) : s + 1);
    child[i] = c;
    range[i] = make_int2(first, last);
    Box6 u;
    if (NODES) {   // layout: k_bvh2_nodes
        u = box_of(first, s + 1);
        const Box6 r = box_of(s + 1, last + 1);
        nodes[4ull * i + 0] = make_float4(u.v[0], u.v[3], u.v[1], u.v[4]);
        nodes[4ull * i + 1] = make_float4(r.v[0], r.v[3], r.v[1], r.v[4]);
        nodes[4ull * i + 2] = make_float4(u.v[2], u.v[5], r.v[2], r.v[5]);
        nodes[4ull * i + 3] = make_float4(__int_as_float(c.x), __int_as_float(c.y), 0.f, 0.f);
        u.add(r);
    } else {
        u = box_of(first, last + 1);
    }
    node_box[2ull * i] = make_float4(u.v[0], u.v[1], u.v[2], 0.f);
    node_box[2ull * i + 1] = make_float4(u.v[3], u.v[4], u.v[5], 0.f);
}

// up: pyramid levels above the leaves by 16, 64 and 256 boxes, back to back (n2, n3, n4 boxes).
template <bool NODES>
__global__ void __launch_bounds__(TREE_THREADS) k_tree(const uint32_t* __restrict__ code,
                                                       const uint32_t* __restrict__ order, int n,
                                                       const float4* __restrict__ box_unsorted,
                                                       float4* __restrict__ leaf_box, uint64_t* __restrict__ keys,
                                                       int8_t* __restrict__ gaps, uint32_t* __restrict__ crossing,
                                                       uint32_t* n_crossing, float4* __restrict__ up,
                                                       int2* __restrict__ child, int2* __restrict__ range,
                                                       float4* __restrict__ node_box, float4* __restrict__ nodes)
{
    constexpr int T = TREE_THREADS;
    // low[k][g] = the smallest of gaps g .. g + 2^k - 1; gap g lies between keys base + g - 1 and base + g
    __shared__ int8_t low[TREE_LEVELS][T + 1];
    __shared__ float pyr[6][TREE_BOXES];
    const int t = threadIdx.x;
    const int base = blockIdx.x * T, i = base + t;
    int p = -1;   // the gap behind this thread's key
    Box6 b;
    b.clear();
    if (i < n) {
        const uint32_t c = code[i], o = order[i];
        if (i + 1 < n) p = prefix_len(c, o, code[i + 1], order[i + 1]);
        if (t == 0) low[0][0] = (int8_t)(i > 0 ? prefix_len(code[i - 1], order[i - 1], c, o) : -1);
        const float4 mn = box_unsorted[2ull * o], mx = box_unsorted[2ull * o + 1];
        leaf_box[2ull * i] = mn;
        leaf_box[2ull * i + 1] = mx;
        if (keys) keys[i] = ((uint64_t)c << 32) | o;
        b = box6(mn, mx);
        gaps[i] = (int8_t)p;
    }
    low[0][t + 1] = (int8_t)p;
#pragma unroll
    for (int a = 0; a < 6; ++a) pyr[a][t] = b.v[a];
    __syncthreads();
#pragma unroll
    for (int k = 1; k < TREE_LEVELS; ++k) {
        const int w = 1 << (k - 1);
        for (int g = t; g + 2 * w <= T + 1; g += T) low[k][g] = min(low[k - 1][g], low[k - 1][g + w]);
        if (k <= 4) {   // pyramid level k: T >> 2k boxes
            const int m = T >> (2 * k);
            if (t < m) {
                Box6 u;
                u.clear();
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int a = 0; a < 6; ++a)
                        u.v[a] = a < 3 ? fminf(u.v[a], pyr[a][tree_pyr(k - 1) + 4 * t + j])
                                       : fmaxf(u.v[a], pyr[a][tree_pyr(k - 1) + 4 * t + j]);
#pragma unroll
                for (int a = 0; a < 6; ++a) pyr[a][tree_pyr(k) + t] = u.v[a];
                if (k >= 2) {
                    const uint32_t n2 = ((uint32_t)n + 15) / 16, n3 = (n2 + 3) / 4, n4 = (n3 + 3) / 4;
                    const uint32_t at = (uint32_t)blockIdx.x * m + t, count = k == 2 ? n2 : k == 3 ? n3 : n4,
                                   from = k == 2 ? 0 : k == 3 ? n2 : n2 + n3;
                    if (at < count)
                        store_box(up, from + at, make_float4(u.v[0], u.v[1], u.v[2], 0.f),
                                  make_float4(u.v[3], u.v[4], u.v[5], 0.f));
                }
            }
        }
        __syncthreads();
    }
    if (i + 1 >= n) return;
    // nearest smaller gap on either side of gap g
    const int g = t + 1;
    int a = g, z = g;   // gaps a .. z are not smaller than p
#pragma unroll
    for (int k = TREE_LEVELS - 1; k >= 0; --k) {
        const int w = 1 << k;
        if (a - w >= 0 && low[k][a - w] >= p) a -= w;
        if (z + w <= T && low[k][z + 1] >= p) z += w;
    }
    if (a == 0 || z == T) {
        cg::coalesced_group cgp = cg::coalesced_threads();
        uint32_t at = 0;
        if (cgp.thread_rank() == 0) at = atomicAdd(n_crossing, (uint32_t)cgp.size());
        crossing[cgp.shfl(at, 0) + cgp.thread_rank()] = (uint32_t)i;
        return;
    }
    const int before = low[0][a - 1], behind = low[0][z + 1];
    store_node<NODES>(
        i, base + a - 1, base + z, before < 0 && behind < 0, behind > before,
        [&](int lo, int hi) { return block_union(pyr, lo - base, hi - base); }, child, range, node_box, nodes);
}

// Union of leaf boxes [lo, hi) from the leaves, 16 at a time, and the levels above them.
__device__ __forceinline__ Box6 wide_union(const float4* __restrict__ leaves, const float4* __restrict__ up, uint32_t n,
                                           uint32_t lo, uint32_t hi)
{
    Box6 b;
    b.clear();
    const float4* a = leaves;
    const float4* next = up;
    uint32_t na = n;
    for (uint32_t step = 16;; step = 4) {
        const uint32_t up_lo = (lo + step - 1) & ~(step - 1), dn = hi & ~(step - 1);
        if (up_lo >= dn) {
#pragma unroll 4
            for (uint32_t j = lo; j < hi; ++j) b.add(box6(a[2ull * j], a[2ull * j + 1]));
            return b;
        }
#pragma unroll 4
        for (uint32_t j = lo; j < up_lo; ++j) b.add(box6(a[2ull * j], a[2ull * j + 1]));
#pragma unroll 4
        for (uint32_t j = dn; j < hi; ++j) b.add(box6(a[2ull * j], a[2ull * j + 1]));
        lo = up_lo / step;
        hi = dn / step;
        na = (na + step - 1) / step;
        a = next;
        next += 2ull * na;
    }
}

template <bool NODES>
__global__ void __launch_bounds__(64) k_tree_top(const uint32_t* __restrict__ code, const uint32_t* __restrict__ order,
                                                 int n, const uint32_t* __restrict__ crossing,
                                                 const uint32_t* __restrict__ n_crossing,
                                                 const int8_t* __restrict__ gaps, const float4* __restrict__ leaf_box,
                                                 const float4* __restrict__ up, int2* __restrict__ child,
                                                 int2* __restrict__ range, float4* __restrict__ node_box,
                                                 float4* __restrict__ nodes)
{
    const uint32_t count = *n_crossing;
    for (uint32_t k = blockIdx.x * 64 + threadIdx.x; k < count; k += gridDim.x * 64) {
        const int s = (int)crossing[k];
        const uint32_t c = code[s], o = order[s];
        const int p = gaps[s];
        // both ends: the farthest keys that share p bits with key s, by doubling steps, then halving
        // ones; the two searches step together
        int lo = s, hi = s + 1;
        int wl = 64, wh = 64;
        bool gl = true, gh = true;   // still doubling
        while (wl || wh) {
            const int jl = lo - wl, jh = hi + wh;
            const bool il = wl && wl <= lo, ih = wh && wh < n - hi;
            const uint32_t cl = il ? code[jl] : 0u, ol = il ? order[jl] : 0u, ch = ih ? code[jh] : 0u,
                           oh = ih ? order[jh] : 0u;
            if (wl) {
                if (il && prefix_len(cl, ol, c, o) >= p) {
                    lo = jl;
                    wl = gl ? (wl < 1 << 30 ? wl * 2 : wl) : wl / 2;
                } else {
                    gl = false;
                    wl /= 2;
                }
            }
            if (wh) {
                if (ih && prefix_len(c, o, ch, oh) >= p) {
                    hi = jh;
                    wh = gh ? (wh < 1 << 30 ? wh * 2 : wh) : wh / 2;
                } else {
                    gh = false;
                    wh /= 2;
                }
            }
        }
        const int before = lo > 0 ? gaps[lo - 1] : -1, behind = gaps[hi];
        store_node<NODES>(
            s, lo, hi, before < 0 && behind < 0, behind > before,
            [&](int x, int y) { return wide_union(leaf_box, up, (uint32_t)n, (uint32_t)x, (uint32_t)y); }, child, range,
            node_box, nodes);
    }
}

// Union of leaf boxes [lo, hi) (exclusive hi) from the pyramid: at each level the partial groups
// at both ends (at most three boxes each), then up one level with the aligned middle; the last
// level visited holds at most six boxes of the range.  All loads of a level are independent, so
// a thread has up to six in flight at once.
__device__ __forceinline__ void range_union(const float4* __restrict__ leaves, const float4* __restrict__ levels,
                                            uint32_t n, int count, uint32_t lo, uint32_t hi, float4& mn, float4& mx)
{
    empty_box(mn, mx);
    const float4* a = leaves;
    const float4* next = levels;
    uint32_t na = n;
    for (int l = 0;; ++l) {
        const uint32_t lo_up = (lo + 3u) & ~3u, hi_dn = hi & ~3u;
        if (l == count || lo_up >= hi_dn) {
#pragma unroll
            for (uint32_t j = 0; j < 6; ++j)
                if (lo + j < hi) box_union(mn, mx, a[2ull * (lo + j)], a[2ull * (lo + j) + 1]);
            return;
        }
#pragma unroll
        for (uint32_t j = 0; j < 3; ++j) {
            if (lo + j < lo_up) box_union(mn, mx, a[2ull * (lo + j)], a[2ull * (lo + j) + 1]);
            if (hi_dn + j < hi) box_union(mn, mx, a[2ull * (hi_dn + j)], a[2ull * (hi_dn + j) + 1]);
        }
        lo = lo_up >> 2;
        hi = hi_dn >> 2;
        na = (na + 3) / 4;
        a = next;
        next += 2ull * na;
    }
}

// Node i's box = union of its sorted leaf range (min and max are exact, so the result equals the
// pairwise unions of the reference's bottom-up refit).
__global__ void k_node_boxes(const float4* __restrict__ leaves, const float4* __restrict__ levels, uint32_t n,
                             int count, const int2* __restrict__ range, float4* __restrict__ node_box)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int2 r = range[i];
    float4 mn, mx;
    range_union(leaves, levels, n, count, (uint32_t)r.x, (uint32_t)r.y + 1u, mn, mx);
    node_box[2ull * i] = mn;
    node_box[2ull * i + 1] = mx;
}

// ---------------------------------------------------------------- traversal layout
// BVH2 node i: (A.lo.x, A.hi.x, A.lo.y, A.hi.y), (B.lo.x, B.hi.x, B.lo.y, B.hi.y),
// (A.lo.z, A.hi.z, B.lo.z, B.hi.z), (childA, childB, 0, 0) — 64 bytes, four 16-byte loads.
__global__ void k_bvh2_nodes(const int2* __restrict__ child, const float4* __restrict__ node_box,
                             const float4* __restrict__ leaf_box, uint32_t n_internal, float4* __restrict__ nodes)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_internal) return;
    int2 c = child[i];
    const float4* ba = c.x < 0 ? leaf_box + 2ull * (uint32_t)(~c.x) : node_box + 2ull * (uint32_t)c.x;
    const float4* bb = c.y < 0 ? leaf_box + 2ull * (uint32_t)(~c.y) : node_box + 2ull * (uint32_t)c.y;
    float4 amn = ba[0], amx = ba[1], bmn = bb[0], bmx = bb[1];
    nodes[4ull * i + 0] = make_float4(amn.x, amx.x, amn.y, amx.y);
    nodes[4ull * i + 1] = make_float4(bmn.x, bmx.x, bmn.y, bmx.y);
    nodes[4ull * i + 2] = make_float4(amn.z, amx.z, bmn.z, bmx.z);
    nodes[4ull * i + 3] = make_float4(__int_as_float(c.x), __int_as_float(c.y), 0.f, 0.f);
}

// Compressed BVH2 node i (32 bytes, one memory sector per visit instead of two): both child boxes
// quantised outwards to 8 bits on a grid anchored at the node box's minimum (cpt_quant.cuh), and
// the split index of the Karras tree, whose children are always split and split + 1 (each a leaf
// or an internal node, as two flags say):
//   float4 q0: origin xyz; w = ex | ey << 8 | ez << 16 | leaf(A) << 24 | leaf(B) << 25
//   uint4  q1: x = A.lo.x | A.lo.y << 8 | A.lo.z << 16 | A.hi.x << 24
//              y = A.hi.y | A.hi.z << 8 | B.lo.x << 16 | B.lo.y << 24
//              z = B.lo.z | B.hi.x << 8 | B.hi.y << 16 | B.hi.z << 24
//              w = split
__global__ void k_bvh2_qnodes(const int2* __restrict__ child, const float4* __restrict__ node_box,
                              const float4* __restrict__ leaf_box, uint32_t n_internal, float4* __restrict__ nodes)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_internal) return;
    int2 c = child[i];
    const float4* ba = c.x < 0 ? leaf_box + 2ull * (uint32_t)(~c.x) : node_box + 2ull * (uint32_t)c.x;
    const float4* bb = c.y < 0 ? leaf_box + 2ull * (uint32_t)(~c.y) : node_box + 2ull * (uint32_t)c.y;
    const float4 amn = ba[0], amx = ba[1], bmn = bb[0], bmx = bb[1];
    const float ox = fminf(amn.x, bmn.x), oy = fminf(amn.y, bmn.y), oz = fminf(amn.z, bmn.z);
    const uint32_t ex = grid_exponent(ox, fmaxf(amx.x, bmx.x)), ey = grid_exponent(oy, fmaxf(amx.y, bmx.y)),
                   ez = grid_exponent(oz, fmaxf(amx.z, bmx.z));
    const float sx = inv_grid(ex), sy = inv_grid(ey), sz = inv_grid(ez);
    const uint32_t split = (uint32_t)(c.x < 0 ? ~c.x : c.x);
    const uint32_t flags = (c.x < 0 ? 1u : 0u) | (c.y < 0 ? 2u : 0u);
    const uint32_t w0 = q_lo(amn.x, ox, sx) | q_lo(amn.y, oy, sy) << 8 | q_lo(amn.z, oz, sz) << 16 | q_hi(amx.x, ox, sx) << 24;
    const uint32_t w1 = q_hi(amx.y, oy, sy) | q_hi(amx.z, oz, sz) << 8 | q_lo(bmn.x, ox, sx) << 16 | q_lo(bmn.y, oy, sy) << 24;
    const uint32_t w2 = q_lo(bmn.z, oz, sz) | q_hi(bmx.x, ox, sx) << 8 | q_hi(bmx.y, oy, sy) << 16 | q_hi(bmx.z, oz, sz) << 24;
    nodes[2ull * i] = make_float4(ox, oy, oz, __uint_as_float(ex | ey << 8 | ez << 16 | flags << 24));
    nodes[2ull * i + 1] = make_float4(__uint_as_float(w0), __uint_as_float(w1), __uint_as_float(w2), __uint_as_float(split));
}

// Triangle edge b - a of FP32 vertices, rounded once from the FP64 difference.  When both are
// normal and their exponents differ by at most 28, the difference of the two 24-bit significands
// spans at most 53 bits, so the FP64 subtraction is exact and one FP32 subtraction rounds the same
// exact value; so it is when either is zero.  Otherwise the FP64 sequence runs, out of line.
__device__ __noinline__ float edge64(float b, float a) { return (float)((double)b - (double)a); }

__device__ __forceinline__ float edge32(float b, float a)
{
    const int eb = (int)((__float_as_uint(b) >> 23) & 0xFFu), ea = (int)((__float_as_uint(a) >> 23) & 0xFFu);
    const bool normal = eb != 0 && eb != 0xFF && ea != 0 && ea != 0xFF;
    const bool zero = (__float_as_uint(b) << 1) == 0u || (__float_as_uint(a) << 1) == 0u;
    const bool finite = eb != 0xFF && ea != 0xFF;
    return ((normal && abs(eb - ea) <= 28) || (zero && finite)) ? __fsub_rn(b, a) : edge64(b, a);
}

// Leaf record k (48 bytes) for primitive order[k]:
//   triangle: (p0, id), (p1 - p0, TRI), (p2 - p0, 0)   edges formed in double, rounded once
//   sphere:   (centre, id), (radius, 0, 0, SPHERE), 0
//   light:    (0, 0, 0, id), (light index, 0, 0, LIGHT), 0
template <typename VT>
__global__ void k_leaf_records(const uint32_t* __restrict__ order, uint32_t n, uint32_t n_lights, uint32_t n_spheres,
                               const VT* __restrict__ tri_v, const float4* __restrict__ spheres,
                               const uint32_t* __restrict__ n_ready, float4* __restrict__ rec)
{
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n || (n_ready && k >= *n_ready)) return;
    uint32_t p = order[k];
    float4 r0, r1, r2 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p < n_lights) {
        r0 = make_float4(0.f, 0.f, 0.f, __int_as_float((int)p));
        r1 = make_float4(__int_as_float((int)p), 0.f, 0.f, __int_as_float(CPT_KIND_LIGHT));
    } else if (p < n_lights + n_spheres) {
        float4 s = spheres[p - n_lights];
        r0 = make_float4(s.x, s.y, s.z, __int_as_float((int)p));
        r1 = make_float4(s.w, 0.f, 0.f, __int_as_float(CPT_KIND_SPHERE));
    } else if (sizeof(VT) == sizeof(float)) {
        const float* v = reinterpret_cast<const float*>(tri_v) + 9ull * (p - n_lights - n_spheres);
        float q[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) q[k] = __ldg(v + k);
        r0 = make_float4(q[0], q[1], q[2], __int_as_float((int)p));
        r1 = make_float4(edge32(q[3], q[0]), edge32(q[4], q[1]), edge32(q[5], q[2]), __int_as_float(CPT_KIND_TRI));
        r2 = make_float4(edge32(q[6], q[0]), edge32(q[7], q[1]), edge32(q[8], q[2]), 0.f);
    } else {
        double q[9];
        load_tri(tri_v, p - n_lights - n_spheres, q);
        r0 = make_float4((float)q[0], (float)q[1], (float)q[2], __int_as_float((int)p));
        r1 = make_float4((float)(q[3] - q[0]), (float)(q[4] - q[1]), (float)(q[5] - q[2]), __int_as_float(CPT_KIND_TRI));
        r2 = make_float4((float)(q[6] - q[0]), (float)(q[7] - q[1]), (float)(q[8] - q[2]), 0.f);
    }
    rec[3ull * k] = r0;
    rec[3ull * k + 1] = r1;
    rec[3ull * k + 2] = r2;
}

inline unsigned blocks_for(uint64_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

// Threads of a sort block (4 or 8 keys each).  A tile adds up the counts of the tiles before it that run
// beside it, so large sorts want about as many tiles as SMs; below that, small tiles, since a pass lasts
// as long as one tile.  Whole builds (us) with blocks of 256 / 512 / 1,024 threads at every size:
//   32,768 73 / 76 / 92     196,608 104 / 105 / 115    655,360  167 / 152 / 150
//   65,536 79 / 81 / 97     262,144 112 / 109 / 120  1,048,576  221 / 190 / 180
//  131,072 89 / 95 / 107    524,288 150 / 130 / 140  1,310,720  258 / 212 / 219
// The upper line lies between the middle shape's last size and the large one's first; at 1.31M the large
// shape has 160 tiles for 152 SMs, and the last eight cost it its lead.  The lower line could be near
// 200,000 (6 % of a build between) but for cpt_lbvh_build_device_static: with tiles of 1,024 keys the
// chains of 65,536 primitives do not fit its 3 MiB.
constexpr uint32_t SORT_SMALL = 1u << 15, SORT_MEDIUM = 1u << 19;
int sort_threads(uint32_t n) { return n <= SORT_SMALL ? 256 : n <= SORT_MEDIUM ? 512 : 1024; }
uint32_t sort_tile(uint32_t n) { return (uint32_t)sort_threads(n) * (sort_threads(n) == 256 ? 4u : 8u); }
// Words of the sort's chains hold two flag bits beside a count of up to n.
size_t chain_word(uint32_t n) { return n < CPT_CHAIN_WIDE_FROM ? 4 : 8; }
static_assert(CPT_CHAIN_WIDE_FROM > SORT_MEDIUM && CPT_CHAIN_WIDE_FROM <= 1u << 30, "64-bit chains run on the largest tiles");

// Upper pyramid of a build: unions of 16, 64, 256, ... sorted leaf boxes, level after level to one box; at
// least the three levels that k_tree writes.
size_t upper_boxes(uint32_t n)
{
    size_t boxes = 0;
    uint32_t m = (uint32_t)(((uint64_t)n + 15) / 16);
    for (int l = 0;; ++l) {
        boxes += m;
        if (m <= 1 && l >= 2) return boxes;
        m = (m + 3) / 4;
    }
}

// code0 and box_unsorted live through a build.  The rest of the scratch holds one stage's arrays after
// another's: the sort's, the tree's (which keep the cleared words: n_crossing is one of them), a refit's.
struct ScratchLayout {
    size_t code0, box_unsorted, total;
    size_t totals, tickets, state, sort_clear;   // the sort's counters and chains, cleared together
    size_t code1, val1;                          // the sort's second buffers
    size_t gaps, crossing, up;                   // tree
    size_t levels;                               // refit: the box pyramid
    uint32_t num_tiles;
    int level_count;   // pyramid levels above the leaves (0 for a single leaf)
};

ScratchLayout layout_for(uint32_t n)
{
    ScratchLayout L;
    std::memset(&L, 0, sizeof L);
    const uint32_t tile = sort_tile(n);
    L.num_tiles = (uint32_t)(((uint64_t)n + tile - 1) / tile);
    size_t lv_boxes = 0;
    for (uint32_t m = n; m > 1;) {
        m = (uint32_t)(((uint64_t)m + 3) / 4);
        lv_boxes += m;
        L.level_count++;
    }
    size_t off = 0, end = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off = align_up(off + bytes, 256);
        end = std::max(end, off);
        return o;
    };
    L.code0 = take((size_t)n * 4);
    L.box_unsorted = take((size_t)n * 32);
    const size_t stages = off;
    L.totals = take(RS_PASSES * RS_BINS * 4);
    L.tickets = take(256);
    const size_t cleared = off;
    L.state = take((size_t)RS_PASSES * L.num_tiles * RS_BINS * chain_word(n));
    L.sort_clear = off - L.totals;
    L.code1 = take((size_t)n * 4);
    L.val1 = take((size_t)n * 4);
    off = cleared;
    L.gaps = take(n);
    L.crossing = take((size_t)n * 4);
    L.up = take(upper_boxes(n) * 32);
    off = stages;
    L.levels = take(lv_boxes * 32);
    L.total = end;
    return L;
}

template <int THREADS, int ITEMS, typename Word>
cpt_status sort_passes(uint32_t n, const ScratchLayout& SL, char* base, uint32_t* code0, uint32_t* code1,
                       uint32_t* val0, uint32_t* val1, cudaStream_t stream)
{
    const uint32_t* totals = (const uint32_t*)(base + SL.totals);
    uint32_t* tickets = (uint32_t*)(base + SL.tickets);
    Word* state = (Word*)(base + SL.state);
    const size_t per_pass = (size_t)SL.num_tiles * RS_BINS;
    const int smem = (int)sizeof(SortSmem<THREADS, ITEMS, Word>);
    for (int p = 0; p < RS_PASSES; ++p) {
        uint32_t *ki = p & 1 ? code1 : code0, *vi = p & 1 ? val1 : val0, *ko = p & 1 ? code0 : code1,
                 *vo = p & 1 ? val0 : val1;
        const auto k = p == 0 ? k_sort_digit<THREADS, ITEMS, Word, true> : k_sort_digit<THREADS, ITEMS, Word, false>;
        if (smem > 48 << 10) CPT_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        k<<<SL.num_tiles, THREADS, smem, stream>>>(ki, vi, ko, vo, n, RS_BITS * p, totals + p * RS_BINS,
                                                   state + p * per_pass, tickets + p);
    }
    CPT_CUDA(cudaGetLastError());
    add_launches(RS_PASSES);
    return CPT_OK;
}

// The pyramid above the sorted leaf boxes, then the node boxes.
cpt_status refit_from_leaves(uint32_t n, const ScratchLayout& SL, char* base, const int2* range, float4* node_box,
                             const float4* leaf_box, cudaStream_t stream)
{
    if (n < 2) return CPT_OK;
    float4* levels = (float4*)(base + SL.levels);
    const float4* in = leaf_box;
    float4* out = levels;
    uint32_t m = n;
    int launches = 1;
    for (int l = 0; l < SL.level_count; l += 4) {
        const int depth = std::min(4, SL.level_count - l);
        k_pyramid<<<blocks_for(m, PYR_THREADS), PYR_THREADS, 0, stream>>>(in, m, out, depth);
        launches++;
        for (int d = 0; d < depth; ++d) {
            const uint32_t up = (m + 3) / 4;
            in = out;
            out += 2ull * up;
            m = up;
        }
    }
    k_node_boxes<<<blocks_for(n - 1, 256), 256, 0, stream>>>(leaf_box, levels, n, SL.level_count, range, node_box);
    add_launches(launches);
    CPT_CUDA(cudaGetLastError());
    return CPT_OK;
}

}  // namespace

// Scratch for n primitives holds every smaller build too: where the sort's tiles grow (sort_tile) the
// chains shrink, so the largest build of each smaller tile size counts as well (32,768 primitives need
// 1,577,216 bytes, 32,769 by themselves 1,530,112).
size_t lbvh_scratch_bytes(uint32_t n)
{
    size_t bytes = layout_for(std::max(n, 1u)).total;
    for (uint32_t last : {SORT_SMALL, SORT_MEDIUM})
        if (n > last) bytes = std::max(bytes, layout_for(last).total);
    return bytes;
}

cpt_status lbvh_build(uint32_t n_extra, const double* extra_centroid, const float4* extra_box, uint32_t n_tri,
                      const float* tri_f32, const double* tri_f64, const double smin_in[3], const double smax_in[3],
                      const LbvhBuffers& out, void* scratch, size_t scratch_bytes, cudaStream_t stream,
                      const cudaEvent_t* stages)
{
    uint64_t n64 = (uint64_t)n_extra + n_tri;
    if (n64 == 0) return CPT_OK;
    if (n64 > 0x7fffffffull) return fail(CPT_ERR_INVALID_ARGUMENT, "lbvh_build: too many primitives");
    uint32_t n = (uint32_t)n64;
    if (n_tri && !tri_f32 && !tri_f64) return fail(CPT_ERR_INVALID_ARGUMENT, "lbvh_build: no triangle vertices");
    if (n_extra && (!extra_centroid || !extra_box)) return fail(CPT_ERR_INVALID_ARGUMENT, "lbvh_build: extra prims");
    if (!out.order || !out.leaf_box || (n > 1 && (!out.child || !out.node_box || !out.range)))
        return fail(CPT_ERR_INVALID_ARGUMENT, "lbvh_build: missing output buffer");
    ScratchLayout SL = layout_for(n);
    if (!scratch || scratch_bytes < SL.total || ((uintptr_t)scratch & 255u))
        return fail(CPT_ERR_INVALID_ARGUMENT, "lbvh_build: scratch too small or not 256-byte aligned");
    char* base = (char*)scratch;
    // Keys and values ping-pong between (code0, val0 = out.order) and (code1, val1); an even number
    // of passes ends where it began.
    uint32_t* code0 = (uint32_t*)(base + SL.code0);
    uint32_t* code1 = (uint32_t*)(base + SL.code1);
    uint32_t* val0 = out.order;
    uint32_t* val1 = (uint32_t*)(base + SL.val1);
    uint32_t* totals = (uint32_t*)(base + SL.totals);
    float4* box_unsorted = (float4*)(base + SL.box_unsorted);

    // Device::buildBVH: expand the mesh bounds by 1, fall back to [-20,20]^3 (Device.cuh:174-181).
    double3 smin = make_double3(smin_in[0] - 1.0, smin_in[1] - 1.0, smin_in[2] - 1.0);
    double3 smax = make_double3(smax_in[0] + 1.0, smax_in[1] + 1.0, smax_in[2] + 1.0);
    if (smin.x > smax.x) {
        smin = make_double3(-20.0, -20.0, -20.0);
        smax = make_double3(20.0, 20.0, 20.0);
    }

    if (stages) CPT_CUDA(cudaEventRecord(stages[0], stream));
    auto axis = [](double mn, double mx) {
        MortonAxis m;
        m.mn = mn;
        m.mx = mx;
        m.k64 = 1024.0 / (mx - mn);
        m.mn32 = (float)mn;
        m.k32 = (float)m.k64;
        m.mn_lo = (float)(mn - (double)m.mn32);
        m.k_lo = (float)(m.k64 - (double)m.k32);
        return m;
    };
    const MortonAxis ax = axis(smin.x, smax.x), ay = axis(smin.y, smax.y), az = axis(smin.z, smax.z);
    CPT_CUDA(cudaMemsetAsync(totals, 0, SL.sort_clear, stream));
    const unsigned prep_grid = std::min(blocks_for(n, PREP_THREADS), PREP_BLOCKS);
    if (tri_f64)
        k_prep<double><<<prep_grid, PREP_THREADS, 0, stream>>>(n_extra, extra_centroid, extra_box, n_tri, tri_f64, ax,
                                                               ay, az, code0, box_unsorted, totals);
    else
        k_prep<float><<<prep_grid, PREP_THREADS, 0, stream>>>(n_extra, extra_centroid, extra_box, n_tri, tri_f32, ax,
                                                              ay, az, code0, box_unsorted, totals);
    CPT_CUDA(cudaGetLastError());
    add_launches(1);
    if (stages) CPT_CUDA(cudaEventRecord(stages[1], stream));

    const auto sort = chain_word(n) == 8        ? sort_passes<1024, 8, unsigned long long>
                      : sort_threads(n) == 1024 ? sort_passes<1024, 8, uint32_t>
                      : sort_threads(n) == 512  ? sort_passes<512, 8, uint32_t>
                                                : sort_passes<256, 4, uint32_t>;
    const cpt_status st = sort(n, SL, base, code0, code1, val0, val1, stream);
    if (st != CPT_OK) return st;
    if (stages) CPT_CUDA(cudaEventRecord(stages[2], stream));

    // Hierarchy, leaf and node boxes.
    int8_t* gaps = (int8_t*)(base + SL.gaps);
    uint32_t* crossing = (uint32_t*)(base + SL.crossing);
    uint32_t* n_crossing = (uint32_t*)(base + SL.tickets) + RS_PASSES;
    float4* up = (float4*)(base + SL.up);
    const unsigned tree_grid = blocks_for(n, TREE_THREADS), top_grid = std::min(blocks_for(n, 64), TOP_BLOCKS);
    const auto tree = out.nodes ? k_tree<true> : k_tree<false>;
    tree<<<tree_grid, TREE_THREADS, 0, stream>>>(code0, val0, (int)n, box_unsorted, out.leaf_box, out.keys, gaps, crossing,
                                                 n_crossing, up, out.child, out.range, out.node_box, out.nodes);
    if (n > TREE_THREADS) {   // nodes reach across blocks: the rest of the pyramid, then those nodes
        const uint32_t n2 = (n + 15) / 16, n3 = (n2 + 3) / 4;
        const float4* in = up + 2ull * (n2 + n3);
        uint32_t m = (n3 + 3) / 4;
        float4* next = up + 2ull * (n2 + n3 + m);
        while (m > 1) {
            int depth = 0;
            uint32_t top = m;
            float4* after = next;
            const float4* last = in;
            while (depth < 4 && top > 1) {
                top = (top + 3) / 4;
                last = after;
                after += 2ull * top;
                depth++;
            }
            k_pyramid<<<blocks_for(m, PYR_THREADS), PYR_THREADS, 0, stream>>>(in, m, next, depth);
            add_launches(1);
            in = last;
            next = after;
            m = top;
        }
        const auto rest = out.nodes ? k_tree_top<true> : k_tree_top<false>;
        rest<<<top_grid, 64, 0, stream>>>(code0, val0, (int)n, crossing, n_crossing, gaps, out.leaf_box, up, out.child,
                                          out.range, out.node_box, out.nodes);
        add_launches(1);
    }
    CPT_CUDA(cudaGetLastError());
    add_launches(1);
    if (stages) CPT_CUDA(cudaEventRecord(stages[3], stream));
    if (stages) CPT_CUDA(cudaEventRecord(stages[4], stream));   // boxes came with the hierarchy: no refit
    return CPT_OK;
}

cpt_status lbvh_leaf_boxes(uint32_t n_extra, const float4* extra_box, uint32_t n_tri, const float* tri_f32,
                           const double* tri_f64, const uint32_t* order, float4* leaf_box, uint32_t n,
                           cudaStream_t stream)
{
    if (n == 0) return CPT_OK;
    if (tri_f64)
        k_prim_boxes<double><<<blocks_for(n, 256), 256, 0, stream>>>(n_extra, extra_box, n_tri, tri_f64, order, leaf_box, n);
    else
        k_prim_boxes<float><<<blocks_for(n, 256), 256, 0, stream>>>(n_extra, extra_box, n_tri, tri_f32, order, leaf_box, n);
    CPT_CUDA(cudaGetLastError());
    add_launches(1);
    return CPT_OK;
}

cpt_status lbvh_refit(uint32_t n, const LbvhBuffers& out, void* scratch, size_t scratch_bytes, cudaStream_t stream)
{
    ScratchLayout SL = layout_for(std::max(n, 1u));
    if (!scratch || scratch_bytes < SL.total) return fail(CPT_ERR_INVALID_ARGUMENT, "lbvh_refit: scratch too small");
    return refit_from_leaves(n, SL, (char*)scratch, out.range, out.node_box, out.leaf_box, stream);
}

cpt_status build_trace_layout(uint32_t n, uint32_t n_lights, uint32_t n_spheres, const int2* child,
                              const float4* node_box, const float4* leaf_box, const uint32_t* order,
                              const float* tri_f32, const double* tri_f64, const float4* spheres, float4* nodes,
                              float4* leaf_rec, cudaStream_t stream, bool compressed,
                              const uint32_t* n_ready)
{
    if (n == 0) return CPT_OK;
    if (n > 1 && nodes && compressed)
        k_bvh2_qnodes<<<blocks_for(n - 1, 256), 256, 0, stream>>>(child, node_box, leaf_box, n - 1, nodes);
    else if (n > 1 && nodes)
        k_bvh2_nodes<<<blocks_for(n - 1, 256), 256, 0, stream>>>(child, node_box, leaf_box, n - 1, nodes);
    if (tri_f64)
        k_leaf_records<double><<<blocks_for(n, 256), 256, 0, stream>>>(order, n, n_lights, n_spheres, tri_f64, spheres,
                                                                       n_ready, leaf_rec);
    else
        k_leaf_records<float><<<blocks_for(n, 256), 256, 0, stream>>>(order, n, n_lights, n_spheres, tri_f32, spheres,
                                                                      n_ready, leaf_rec);
    CPT_CUDA(cudaGetLastError());
    add_launches((n > 1 && nodes ? 1 : 0) + 1);
    return CPT_OK;
}

}  // namespace cpt

// ---------------------------------------------------------------- C ABI (low level)
CPT_EXPORT size_t cpt_lbvh_scratch_bytes(uint32_t num_prims) { return cpt::lbvh_scratch_bytes(num_prims); }

CPT_EXPORT cpt_status cpt_lbvh_build_device(uint32_t num_extra, const double* extra_centroids, const float* extra_boxes,
                                            uint32_t num_tri, const float* tri_vertices, const double scene_min[3],
                                            const double scene_max[3], uint64_t* out_keys, uint32_t* out_order,
                                            int32_t* out_children, int32_t* out_node_range, float* out_node_boxes,
                                            float* out_leaf_boxes, void* scratch, size_t scratch_bytes, void* stream)
{
    if (!scene_min || !scene_max) return cpt::fail(CPT_ERR_INVALID_ARGUMENT, "cpt_lbvh_build_device: bounds");
    cpt::LbvhBuffers b;
    b.keys = out_keys;
    b.order = out_order;
    b.child = (int2*)out_children;
    b.range = (int2*)out_node_range;
    b.node_box = (float4*)out_node_boxes;
    b.leaf_box = (float4*)out_leaf_boxes;
    b.nodes = nullptr;
    return cpt::lbvh_build(num_extra, extra_centroids, (const float4*)extra_boxes, num_tri, tri_vertices, nullptr,
                           scene_min, scene_max, b, scratch, scratch_bytes, (cudaStream_t)stream, nullptr);
}
