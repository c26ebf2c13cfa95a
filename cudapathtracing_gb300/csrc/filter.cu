// filter.cu — the reference's non-learned denoiser, in FP32 on device-resident images:
//
//   cpt_filter_bilateral  separable joint-bilateral filter (gaussianSeparate, Render.cu:356-398),
//                         horizontal pass then vertical pass as the REAL_TIME loop runs it
//                         (main.cu:99-103): weights exp(-i^2/2sg^2 - |c_n - c|^2/2sr^2
//                         - |n_n - n|^2/2sn^2 - (d_n - d)^2/2sd^2) over a (2R+1)-tap window with
//                         clamped borders, normalised by their sum.
//   cpt_filter_temporal   reprojection + exponential blend with the previous frame
//                         (addPrevious, Render.cu:400-420, Camera::getPrePositionInImg,
//                         Camera.cuh:103-132).
//
// Images are W*H float3 (row j = 0 at the bottom, as rendered); the G-buffer is the renderer's
// 2 float4 per pixel, (normal, depth) then (albedo, 0), depth 999999 (INF) on a miss.
//
// The reference reads the world position of the first hit from a separate buffer; this build
// reconstructs it as look_from + depth * unit(direction through the pixel centre), which differs
// from the sample's jittered hit point by less than a pixel footprint.  The reference indexes
// the previous frame at int(x * W) for x in [0, 1], which reaches W at x = 1; here the index is
// clamped to the image.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "cpt_internal.h"

namespace cpt {

namespace {

struct BilateralConsts {
    float kg, kr, kn, kd;   // 1 / (2 sigma^2) of the four terms
    int radius;
};

// One separable pass over `src`: the centre value and the neighbours come from the same image
// (in the reference the centre is read from pic, which holds the same values as the pass input).
//
// A tap costs about 20 arithmetic instructions and one expf, and the pass is bound by the multiply-add
// pipe (72 % of its cycles busy, issue slots 66 %, DRAM 15 % at 1080p); a pixel a thread was bound by
// issue slots (82 %).  So everything else is shared: a thread filters four pixels
// that follow one another along the pass and takes each neighbour once for the four, and two pixels
// share a packed multiply-add.  The horizontal pass keeps its row, one array per component, in shared
// memory (four neighbours' component in one conflict-free 16-byte load); in the vertical pass lanes
// are neighbouring columns and read the images directly.  Each pixel's taps are added in the
// window's order, with the multiply-adds that the compiler forms for a pixel a thread, so both give the
// same bits (tests/test_gpu_filter_forms.py).  Both passes, radius 16 at 1920x1080: 227 us with a pixel a
// thread, 174 us so.  Other forms of this one: scalar multiply-adds +19 us, 80 registers (three blocks an
// SM) +20, distances from converted tap numbers instead of a table +4; the exponentials are 27 us of it.
constexpr int FPX = 4;   // pixels a thread; also neighbours a step

__device__ __forceinline__ uint64_t pack2(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Colour (0-2), normal (3-5) and depth (6) of a pixel.
struct Tap {
    float v[7];
};

// Two neighbouring pixels: their negated centre values, weight and colour sums.
struct PixelPair {
    uint64_t c[7], wsum, acc[3];

    __device__ __forceinline__ void start(const Tap& a, const Tap& b)
    {
        for (int j = 0; j < 7; ++j) c[j] = pack2(-a.v[j], -b.v[j]);
        wsum = pack2(0.f, 0.f);
        for (int j = 0; j < 3; ++j) acc[j] = pack2(0.f, 0.f);
    }

    // Adds a neighbour that lies i pixels after the first pixel of the pair (i - 1 after the second);
    // ii holds both distances' squares.  CHECK: only where it is inside the window; a pixel's sums are left alone otherwise.
    template <bool CHECK>
    __device__ __forceinline__ void add(const Tap& p, int i, uint64_t ii, const BilateralConsts& k)
    {
        uint64_t pp[3], d[7];
        for (int j = 0; j < 7; ++j) {
            const uint64_t q = pack2(p.v[j], p.v[j]);
            if (j < 3) pp[j] = q;
            d[j] = add2(q, c[j]);
        }
        const uint64_t dc = fma2(d[2], d[2], fma2(d[0], d[0], mul2(d[1], d[1])));
        const uint64_t dn = fma2(d[5], d[5], fma2(d[3], d[3], mul2(d[4], d[4])));
        uint64_t e = fma2(ii, pack2(-k.kg, -k.kg), mul2(dc, pack2(-k.kr, -k.kr)));
        e = fma2(dn, pack2(-k.kn, -k.kn), e);
        e = fma2(mul2(d[6], d[6]), pack2(-k.kd, -k.kd), e);
        float e0, e1;
        unpack2(e, e0, e1);
        const uint64_t w = pack2(expf(e0), expf(e1));
        uint64_t s[4] = {add2(wsum, w), fma2(w, pp[0], acc[0]), fma2(w, pp[1], acc[1]), fma2(w, pp[2], acc[2])};
        if (CHECK) {
            const bool in0 = i >= -k.radius && i <= k.radius, in1 = i - 1 >= -k.radius && i - 1 <= k.radius;
            for (int j = 0; j < 4; ++j) {
                float n0, n1, o0, o1;
                unpack2(s[j], n0, n1);
                unpack2(j ? acc[j - 1] : wsum, o0, o1);
                s[j] = pack2(in0 ? n0 : o0, in1 ? n1 : o1);
            }
        }
        wsum = s[0];
        for (int j = 0; j < 3; ++j) acc[j] = s[j + 1];
    }

    __device__ __forceinline__ void result(float (&a)[3], float (&b)[3]) const
    {
        float w0, w1;
        unpack2(wsum, w0, w1);
        for (int j = 0; j < 3; ++j) {
            float x, y;
            unpack2(acc[j], x, y);
            a[j] = x / w0;
            b[j] = y / w1;
        }
    }
};

// The four pixels' windows span 2 * radius + 4 neighbours; steps that are inside all of them are
// not checked.
__host__ __device__ __forceinline__ int filter_steps(int radius) { return (2 * radius + 2 * FPX - 1) / FPX; }
__device__ __forceinline__ bool full_step(int base, int radius) { return base >= FPX - 1 && base + FPX - 1 <= 2 * radius; }

// Entry m holds i^2 for i = m - 2 - radius and for i - 1, a pair's distances to a neighbour.
__host__ __device__ __forceinline__ int table_size(int radius) { return FPX * filter_steps(radius) + FPX; }

__device__ __forceinline__ void fill_table(float2* table, int radius)
{
    const int size = table_size(radius);
    for (int m = threadIdx.y * 32 + threadIdx.x; m < size; m += blockDim.y * 32) {
        const int i = m - 2 - radius;
        table[m] = make_float2((float)(i * i), (float)((i - 1) * (i - 1)));
    }
    __syncthreads();
}

// Neighbours base .. base + 3, counted from the first pixel's window start, for four pixels.
template <bool CHECK>
__device__ __forceinline__ void add_step(const Tap (&t)[FPX], int base, const float2* table, PixelPair& p0, PixelPair& p1,
                                         const BilateralConsts& k)
{
    uint64_t ii[FPX + 2];
    for (int j = 0; j < FPX + 2; j += 2) {
        const float4 v = *reinterpret_cast<const float4*>(table + base + j);
        ii[j] = pack2(v.x, v.y);
        ii[j + 1] = pack2(v.z, v.w);
    }
#pragma unroll
    for (int j = 0; j < FPX; ++j) {
        const int i = base + j - k.radius;
        p0.add<CHECK>(t[j], i, ii[j + 2], k);
        p1.add<CHECK>(t[j], i - 2, ii[j], k);
    }
}

__device__ __forceinline__ Tap load_tap(const float* __restrict__ src, const float4* __restrict__ gbuf, size_t n)
{
    const float4 g = __ldg(gbuf + 2 * n);
    return {{__ldg(src + 3 * n), __ldg(src + 3 * n + 1), __ldg(src + 3 * n + 2), g.x, g.y, g.z, g.w}};
}

// A warp filters HTILE pixels of a row.
constexpr int HTILE = 32 * FPX;
__host__ __device__ __forceinline__ int h_pitch(int radius) { return HTILE - FPX + FPX * filter_steps(radius); }

__global__ void __launch_bounds__(256, 2) k_bilateral_rows(const float* __restrict__ src, const float4* __restrict__ gbuf,
                                                        float* __restrict__ out, int W, int H, BilateralConsts k)
{
    extern __shared__ float4 smem4[];
    const uint32_t tiles = ((uint32_t)W + HTILE - 1) / HTILE;   // blocks go tile by tile, then down the image
    const int lane = threadIdx.x, y = (int)(blockIdx.x / tiles * blockDim.y + threadIdx.y), x0 = (int)(blockIdx.x % tiles) * HTILE;
    float2* table = reinterpret_cast<float2*>(smem4);
    fill_table(table, k.radius);
    if (y >= H) return;   // a warp is one row; no barrier below spans warps
    const int pitch = h_pitch(k.radius);
    float* row = reinterpret_cast<float*>(table + table_size(k.radius)) + 7 * pitch * threadIdx.y;
    const size_t first = (size_t)y * W;
    for (int i = lane; i < pitch; i += 32) {
        const Tap t = load_tap(src, gbuf, first + min(max(x0 - k.radius + i, 0), W - 1));
        for (int j = 0; j < 7; ++j) row[j * pitch + i] = t.v[j];
    }
    __syncwarp();
    Tap centre[FPX];
    for (int q = 0; q < FPX; ++q)
        for (int j = 0; j < 7; ++j) centre[q].v[j] = row[j * pitch + FPX * lane + q + k.radius];
    PixelPair p0, p1;
    p0.start(centre[0], centre[1]);
    p1.start(centre[2], centre[3]);
    const int steps = filter_steps(k.radius);
    for (int s = 0; s < steps; ++s) {
        Tap t[FPX];
        for (int j = 0; j < 7; ++j) {
            const float4 v = *reinterpret_cast<const float4*>(row + j * pitch + FPX * (lane + s));
            t[0].v[j] = v.x;
            t[1].v[j] = v.y;
            t[2].v[j] = v.z;
            t[3].v[j] = v.w;
        }
        if (full_step(FPX * s, k.radius)) add_step<false>(t, FPX * s, table, p0, p1, k);
        else add_step<true>(t, FPX * s, table, p0, p1, k);
    }
    __syncwarp();   // the row is read; its space takes the results, to be written out in order
    float r[FPX][3];
    p0.result(r[0], r[1]);
    p1.result(r[2], r[3]);
    for (int q = 0; q < FPX; ++q)
        for (int j = 0; j < 3; ++j) row[3 * (FPX * lane + q) + j] = r[q][j];
    __syncwarp();
    const int n = 3 * min(HTILE, W - x0);
    for (int i = lane; i < n; i += 32) out[3 * (first + x0) + i] = row[i];
}

constexpr int VROWS = 8;   // warps a block, each FPX rows of 32 columns

__global__ void __launch_bounds__(32 * VROWS, 2) k_bilateral_columns(const float* __restrict__ src, const float4* __restrict__ gbuf,
                                                                 float* __restrict__ out, int W, int H, BilateralConsts k)
{
    const int x = blockIdx.x * 32 + threadIdx.x, y0 = (blockIdx.y * VROWS + threadIdx.y) * FPX;
    extern __shared__ float4 smem4[];
    float2* table = reinterpret_cast<float2*>(smem4);
    fill_table(table, k.radius);
    if (x >= W || y0 >= H) return;
    const auto at = [&](int y) { return load_tap(src, gbuf, (size_t)min(max(y, 0), H - 1) * W + x); };
    PixelPair p0, p1;
    p0.start(at(y0), at(y0 + 1));
    p1.start(at(y0 + 2), at(y0 + 3));
    const int steps = filter_steps(k.radius);
    for (int s = 0; s < steps; ++s) {
        Tap t[FPX];
        for (int j = 0; j < FPX; ++j) t[j] = at(y0 - k.radius + FPX * s + j);
        if (full_step(FPX * s, k.radius)) add_step<false>(t, FPX * s, table, p0, p1, k);
        else add_step<true>(t, FPX * s, table, p0, p1, k);
    }
    float r[FPX][3];
    p0.result(r[0], r[1]);
    p1.result(r[2], r[3]);
    for (int q = 0; q < FPX; ++q)
        if (y0 + q < H)
            for (int j = 0; j < 3; ++j) out[3 * ((size_t)(y0 + q) * W + x) + j] = r[q][j];
}

// A pixel a thread, for short windows: there the pass is nearer to a stream over the images, and the
// wider form's staging and unfilled steps cost more than they save (us at 1920x1080, 901x507 and
// 100x400; a pixel a thread / four: radius 4 82 / 92, 30 / 36, 16 / 18; 6 106 / 105, 37 / 39, 16 / 20;
// 8 129 / 116, 45 / 43, 19 / 20; 16 227 / 174, 69 / 61, 26 / 24).
#ifndef CPT_FILTER_SMALL_RADIUS
#define CPT_FILTER_SMALL_RADIUS 6
#endif
constexpr int SMALL_RADIUS = CPT_FILTER_SMALL_RADIUS;

template <bool HORIZONTAL>
__global__ void __launch_bounds__(256) k_bilateral_small(const float* __restrict__ src, const float4* __restrict__ gbuf,
                                                        float* __restrict__ out, int W, int H, BilateralConsts k)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const size_t off = (size_t)y * W + x;
    const float4 g = __ldg(gbuf + 2 * off);
    const float3 c = f3(__ldg(src + 3 * off), __ldg(src + 3 * off + 1), __ldg(src + 3 * off + 2));
    float3 acc = f3(0.f, 0.f, 0.f);
    float wsum = 0.f;
    for (int i = -k.radius; i <= k.radius; ++i) {
        int nx = x, ny = y;
        if (HORIZONTAL) nx = min(max(x + i, 0), W - 1);
        else ny = min(max(y + i, 0), H - 1);
        const size_t n = (size_t)ny * W + nx;
        const float3 p = f3(__ldg(src + 3 * n), __ldg(src + 3 * n + 1), __ldg(src + 3 * n + 2));
        const float4 gp = __ldg(gbuf + 2 * n);
        const float3 dc = p - c;
        const float3 dn = f3(g.x - gp.x, g.y - gp.y, g.z - gp.z);
        const float dd = g.w - gp.w;
        const float e = -(float)(i * i) * k.kg - dot3(dc, dc) * k.kr - dot3(dn, dn) * k.kn - dd * dd * k.kd;
        const float w = expf(e);
        wsum += w;
        acc = acc + w * p;
    }
    const float3 r = acc / wsum;
    out[3 * off] = r.x;
    out[3 * off + 1] = r.y;
    out[3 * off + 2] = r.z;
}

// The previous camera's frame (getPrePositionInImg) and the current camera's pixel rays.
struct Reproj {
    float3 from, right, up, fwd;   // previous camera
    float sx, sy;                  // focal / viewport width, focal / viewport height
    float3 cur_from, cur_pc, cur_dh, cur_dv;
};

__global__ void __launch_bounds__(256) k_temporal(float* __restrict__ rgb, const float* __restrict__ prev,
                                                  const float4* __restrict__ gbuf, int W, int H, Reproj r, float alpha)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const size_t off = (size_t)y * W + x;
    const float depth = __ldg(gbuf + 2 * off).w;
    size_t src = off;
    if (depth < CPT_INF_F) {
        const float3 dir = unit3(r.cur_pc + (float)x * r.cur_dh + (float)y * r.cur_dv - r.cur_from);
        const float3 pos = r.cur_from + depth * dir;
        const float3 v = unit3(pos - r.from);
        const float px = dot3(v, r.right), py = dot3(v, r.up), pz = dot3(v, r.fwd);
        const float u = 0.5f + (px / pz) * r.sx;
        const float w = 0.5f + (py / pz) * r.sy;
        if (u >= 0.f && w >= 0.f && u <= 1.f && w <= 1.f) {
            const int i = min((int)(u * (float)W), W - 1);
            const int j = min((int)(w * (float)H), H - 1);
            src = (size_t)j * W + i;
        }
    }
    for (int c = 0; c < 3; ++c) rgb[3 * off + c] = rgb[3 * off + c] * alpha + __ldg(prev + 3 * src + c) * (1.0f - alpha);
}

struct V3 {
    double x, y, z;
};
inline V3 v3(const double* a) { return {a[0], a[1], a[2]}; }
inline V3 operator-(V3 a, V3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
inline double dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
inline V3 cross(V3 a, V3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
inline V3 unit(V3 a)
{
    double l = std::sqrt(dot(a, a));
    return {a.x / l, a.y / l, a.z / l};
}
inline float3 tof(V3 a) { return make_float3((float)a.x, (float)a.y, (float)a.z); }

inline int image_height(const cpt_camera& c)
{
    double hh = c.width / c.aspect_ratio;   // Camera.cu:8-9
    return hh < 1 ? 1 : (int)hh;
}

}  // namespace

cpt_status filter_bilateral(const float* rgb, const float* gbuf, float* out, int W, int H, const cpt_filter_params& p,
                            cudaStream_t stream, cudaMemPool_t pool)
{
    if (W <= 0 || H <= 0) return CPT_OK;
    if (p.radius < 0 || p.radius > 256 || !(p.sigma_g > 0) || !(p.sigma_r > 0) || !(p.sigma_n > 0) || !(p.sigma_d > 0))
        return fail(CPT_ERR_INVALID_ARGUMENT, "bilateral filter: sigmas must be positive, radius in [0, 256]");
    if (!rgb || !gbuf || !out) return fail(CPT_ERR_INVALID_ARGUMENT, "bilateral filter: null buffer");
    if (((uintptr_t)gbuf & 15u)) return fail(CPT_ERR_INVALID_ARGUMENT, "bilateral filter: G-buffer must be 16-byte aligned");
    BilateralConsts k;
    k.kg = 1.0f / (2.0f * p.sigma_g * p.sigma_g);
    k.kr = 1.0f / (2.0f * p.sigma_r * p.sigma_r);
    k.kn = 1.0f / (2.0f * p.sigma_n * p.sigma_n);
    k.kd = 1.0f / (2.0f * p.sigma_d * p.sigma_d);
    k.radius = p.radius;
    float* tmp = nullptr;
    const size_t bytes = (size_t)W * H * 3 * sizeof(float);
    if (pool) CPT_NEED(pool_alloc((void**)&tmp, bytes, pool, stream));
    else CPT_CUDA(cudaMallocAsync((void**)&tmp, bytes, stream));
    if (p.radius <= SMALL_RADIUS) {
        dim3 block(32, 8), grid((W + 31) / 32, (H + 7) / 8);
        k_bilateral_small<true><<<grid, block, 0, stream>>>(rgb, (const float4*)gbuf, tmp, W, H, k);
        k_bilateral_small<false><<<grid, block, 0, stream>>>(tmp, (const float4*)gbuf, out, W, H, k);
    } else {
        // rows a block: as many as the default 48 KB of shared memory hold (8 up to radius 44, 2 at 256)
        const size_t table = sizeof(float2) * table_size(p.radius), row = 7 * sizeof(float) * h_pitch(p.radius);
        const int rows = (int)std::min<size_t>(8, (48 * 1024 - table) / row);
        k_bilateral_rows<<<dim3((unsigned)((W + HTILE - 1) / HTILE) * ((H + rows - 1) / rows)), dim3(32, rows), table + rows * row, stream>>>(
            rgb, (const float4*)gbuf, tmp, W, H, k);
        k_bilateral_columns<<<dim3((W + 31) / 32, (H + VROWS * FPX - 1) / (VROWS * FPX)), dim3(32, VROWS), table, stream>>>(
            tmp, (const float4*)gbuf, out, W, H, k);
    }
    add_launches(2);
    cudaError_t e = cudaGetLastError();
    cudaFreeAsync(tmp, stream);
    if (e != cudaSuccess) return cuda_fail(e, "bilateral filter launch");
    return CPT_OK;
}

cpt_status filter_temporal(float* rgb, const float* prev, const float* gbuf, const cpt_camera& cam,
                           const cpt_camera& prev_cam, float alpha, cudaStream_t stream)
{
    const int W = cam.width, H = image_height(cam);
    if (W <= 0) return CPT_OK;
    if (!rgb || !prev || !gbuf) return fail(CPT_ERR_INVALID_ARGUMENT, "temporal filter: null buffer");
    if (((uintptr_t)gbuf & 15u)) return fail(CPT_ERR_INVALID_ARGUMENT, "temporal filter: G-buffer must be 16-byte aligned");
    if (prev_cam.width != cam.width || image_height(prev_cam) != H)
        return fail(CPT_ERR_INVALID_ARGUMENT, "temporal filter: cameras differ in image size");
    if (!(alpha >= 0.f && alpha <= 1.f)) return fail(CPT_ERR_INVALID_ARGUMENT, "temporal filter: alpha in [0, 1]");
    // previous camera frame, in double (Camera.cuh:109-123)
    const V3 from = v3(prev_cam.look_from), at = v3(prev_cam.look_at), vup = {0.0, 1.0, 0.0};
    const V3 fwd = unit(at - from);
    const V3 right = unit(cross(fwd, vup));
    const V3 up = cross(right, fwd);
    const double focal = std::sqrt(dot(from - at, from - at));
    const double h = std::tan(prev_cam.vfov_deg * 3.14159265358979323846 / 180.0 / 2.0);
    const double vh = 2.0 * h * focal;
    const double vw = (double)W / H * vh;
    Reproj r;
    r.from = tof(from);
    r.right = tof(right);
    r.up = tof(up);
    r.fwd = tof(fwd);
    r.sx = (float)(focal / vw);
    r.sy = (float)(focal / vh);
    const DevCamera dc = camera_of(cam);
    r.cur_from = dc.look_from;
    r.cur_pc = dc.pixel_center;
    r.cur_dh = dc.delta_h;
    r.cur_dv = dc.delta_v;
    dim3 block(32, 8), grid((W + 31) / 32, (H + 7) / 8);
    k_temporal<<<grid, block, 0, stream>>>(rgb, prev, (const float4*)gbuf, W, H, r, alpha);
    add_launches(1);
    CPT_CUDA(cudaGetLastError());
    return CPT_OK;
}

}  // namespace cpt
