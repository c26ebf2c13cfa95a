// trace.cu — batched closest-hit queries (traverseIterative, BVH.cuh:282-332, called by the
// reference for camera, bounce, shadow and volume rays): one thread per ray.
#include <cuda_runtime.h>

#include <algorithm>

#include "cpt_internal.h"
#include "cpt_trace.cuh"

namespace cpt {

namespace {

template <bool WIDE>
__global__ void k_trace(SceneView s, const float4* __restrict__ rays, uint64_t n, float4* __restrict__ hits, int* err)
{
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 a = __ldg(rays + 2 * i), b = __ldg(rays + 2 * i + 1);
    Hit h;
    bool hit = trace_closest<WIDE>(s, f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), a.w, b.w, h, err);
    int prim = hit ? __float_as_int(ldg4(s.leaf_rec + 3 * (size_t)h.leaf).w) : -1;
    hits[i] = make_float4(hit ? h.t : -1.0f, __int_as_float(prim), h.u, h.v);
}

// Persistent variants: warps fetch rays dynamically (trace_items_walk), so lanes whose ray finished
// take new rays instead of idling until the warp's slowest ray is done.  The traversal stack's bottom
// entries are in shared memory.
template <bool WIDE>
__global__ void __launch_bounds__(128) k_trace_dyn(SceneView s, const float4* __restrict__ rays, int n,
                                                   float4* __restrict__ hits, int* err, int* fetch)
{
    const auto scene = [&](int) -> const SceneView& { return s; };
    const auto load = [&](int i, float3& o, float3& d, float& tmn, float& tmx, int&, int&) {
        float4 a = __ldg(rays + 2 * (size_t)i), b = __ldg(rays + 2 * (size_t)i + 1);
        o = f3(a.x, a.y, a.z);
        d = f3(b.x, b.y, b.z);
        tmn = a.w;
        tmx = b.w;
    };
    const auto store = [&](int i, const Hit& h, int) {
        int prim = h.leaf >= 0 ? __float_as_int(ldg4(s.leaf_rec + 3 * (size_t)h.leaf).w) : -1;
        hits[i] = make_float4(h.leaf >= 0 ? h.t : -1.0f, __int_as_float(prim), h.u, h.v);
    };
    if (WIDE) trace_items_wide_views<false, ShortStack64<CPT_WIDE_SHORT_STACK>, true>(scene, n, fetch, err, load, store);
    else trace_items_bvh2_views<false, ShortStack, true>(scene, n, fetch, err, load, store);
}

}  // namespace

constexpr unsigned TRACE_THREADS = 128;

cpt_status trace_grids(int sm_count, int resident[2])
{
    int bb = 0, bw = 0;
    CPT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bb, k_trace_dyn<false>, TRACE_THREADS,
                                                           short_stack_bytes(TRACE_THREADS)));
    CPT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bw, k_trace_dyn<true>, TRACE_THREADS,
                                                           wide_short_stack_bytes(TRACE_THREADS)));
    resident[0] = std::max(1, bb) * sm_count;
    resident[1] = std::max(1, bw) * sm_count;
    return CPT_OK;
}

cpt_status launch_trace(const SceneView& view, const cpt_ray* rays, uint64_t n, cpt_hit* hits, int* d_err,
                        cudaStream_t stream, const int resident[2])
{
    if (n == 0) return CPT_OK;
    if (((uintptr_t)rays & 15u) || ((uintptr_t)hits & 15u))
        return fail(CPT_ERR_INVALID_ARGUMENT, "cpt_trace_closest: rays and hits must be 16-byte aligned");
    const unsigned T = TRACE_THREADS;
    uint64_t blocks = (n + T - 1) / T;
    if (blocks > 0x7fffffffull) return fail(CPT_ERR_INVALID_ARGUMENT, "cpt_trace_closest: too many rays");
    if (view.n_internal > 0 && n < 0x7fffffffull) {
        int* fetch = d_err + 1;   // the scene's work counter
        CPT_CUDA(cudaMemsetAsync(fetch, 0, sizeof(int), stream));
        // a ray a warp while there are warps left, then up to 32
        const uint64_t warps = T / 32;
        const unsigned grid = (unsigned)std::min<uint64_t>((n + warps - 1) / warps, (uint64_t)resident[view.wide ? 1 : 0]);
        if (view.wide)
            k_trace_dyn<true><<<grid, T, wide_short_stack_bytes(T), stream>>>(view, (const float4*)rays, (int)n,
                                                                             (float4*)hits, d_err, fetch);
        else
            k_trace_dyn<false><<<grid, T, short_stack_bytes(T), stream>>>(view, (const float4*)rays, (int)n, (float4*)hits,
                                                                   d_err, fetch);
    } else if (view.wide)
        k_trace<true><<<(unsigned)blocks, T, short_stack_bytes(T), stream>>>(view, (const float4*)rays, n,
                                                                             (float4*)hits, d_err);
    else
        k_trace<false><<<(unsigned)blocks, T, short_stack_bytes(T), stream>>>(view, (const float4*)rays, n,
                                                                              (float4*)hits, d_err);
    CPT_CUDA(cudaGetLastError());
    add_launches(1);
    return CPT_OK;
}

}  // namespace cpt
