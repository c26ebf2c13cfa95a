// wide.cu — collapses the binary LBVH into a compressed 8-wide BVH for traversal.
//
// The collapse runs level by level from the root, one launch per level with no host round trip
// in between (the level counts and bases live on the device).  Wide nodes are numbered compactly
// in that breadth-first order: level l occupies [base_l, base_l + n_l), and the internal children of a node
// are numbered consecutively (one atomic per block of nodes reserves their numbers), so the
// reachable nodes fill [0, num_wide) with siblings side by side and the top levels packed together
// (the hot part of the tree stays within a few megabytes).  Leaves stay in sorted Morton order in the
// leaf records.  Each wide node stands for one binary node b; starting from b's two children,
// the child with the largest surface area that is an internal binary node is replaced by its two
// children until there are 8 children or only leaves remain.  Children are then placed in slots
// by direction: slot s (bits: negative x, y, z) holds the child whose centroid offset from the
// node's centre points most along (+-1, +-1, +-1)_s (greedy assignment), so that a ray of
// octant o meets the children roughly in the order of slots s ^ (7 ^ o) — the ordering scheme of
// compressed wide BVHs (Ylitie, Karras, Laine 2017), which needs no sort during traversal.
//
// Node layout (96 bytes, three 32-byte loads; i and l are the node's internal and leaf children):
//   float4 f0   origin p.xyz (node box minimum), grid step of x
//   f1          grid steps of y and z; number of the first internal child; index of the first leaf
//   f2,f3,f4    8-bit quantised child boxes: (lo slots 0-3, lo 4-7, hi 0-3, hi 4-7) for x, y, z
//   f5          x: mask of the internal slots | mask of the leaf slots << 8, slot s at bit 7 - s
// A node's internal children have consecutive numbers and its leaves consecutive leaf records, both
// in slot order, so a child's reference is the first one plus a population count.  Leaf records are
// therefore stored in this layout's own order: the leaves of a node share memory sectors, and the
// 32 bytes that eight references would take hold the grid steps, which the traversal would
// otherwise decode from exponents on every visit.
//
// Child boxes sit on a power-of-two grid anchored at p with 255 steps across the node, rounded
// outwards, so every quantised box contains the child's FP32 box.
#include <cuda_runtime.h>

#include <algorithm>

#include "cpt_internal.h"
#include "cpt_quant.cuh"

namespace cpt {

namespace {

__device__ __forceinline__ float area(float4 mn, float4 mx)
{
    float dx = mx.x - mn.x, dy = mx.y - mn.y, dz = mx.z - mn.z;
    return dx * dy + dy * dz + dz * dx;
}

__device__ __forceinline__ void ref_box(int ref, const float4* node_box, const float4* leaf_box, float4& mn, float4& mx)
{
    const float4* b = ref < 0 ? leaf_box + 2 * (size_t)(~ref) : node_box + 2 * (size_t)ref;
    mn = b[0];
    mx = b[1];
}


// Level l: the wide nodes [base, base + n) with base = level_base[l], n = level_count[l]; wide node
// w stands for binary node tasks[w].  Internal children get the next numbers in level l + 1, which
// starts at base + n.
//
// Eight lanes make a node, lane k holding candidate child k (reference, box, area): an expansion
// costs one round of loads (the two new children's boxes and their own children), the choice of the
// next one and of the next (child, slot) pair three shuffles.  A block makes COLLAPSE_NODES nodes at a
// time, reserves their children's and leaves' numbers with one atomic each and writes the nodes out
// together.  The levels are bound by the latency of that chain and, the large ones, by how many nodes
// are in flight: with a thread a node (152 registers, 12 warps an SM, two atomics a node) the 1.31M-
// primitive collapse took 390 us.
constexpr int COLLAPSE_NODES = 32;
constexpr int COLLAPSE_THREADS = 8 * COLLAPSE_NODES;
constexpr int MAX_WIDE_LEVELS = 80;

// (value, index) pair of the greatest value over the 8 lanes of a node, the lowest index on ties.
__device__ __forceinline__ void max_of_8(float& v, int& k)
{
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const float v2 = __shfl_xor_sync(0xffffffffu, v, o);
        const int k2 = __shfl_xor_sync(0xffffffffu, k, o);
        if (v2 > v || (v2 == v && k2 < k)) {
            v = v2;
            k = k2;
        }
    }
}

__global__ void __launch_bounds__(COLLAPSE_THREADS) k_collapse_level(const int2* __restrict__ child,
                                                                     const float4* __restrict__ node_box,
                                                                     const float4* __restrict__ leaf_box,
                                                                     int* __restrict__ tasks,
                                                                     int* __restrict__ level_count,
                                                                     int* __restrict__ level_base, int l,
                                                                     const uint32_t* __restrict__ order,
                                                                     uint32_t* __restrict__ wide_order,
                                                                     uint32_t* __restrict__ n_leaves,
                                                                     float4* __restrict__ wide)
{
    __shared__ float4 out[COLLAPSE_NODES][CPT_WIDE_F4];
    __shared__ int sums[2][COLLAPSE_NODES + 1];   // internal children and leaves of the nodes, then their first numbers
    const int n = level_count[l];
    const int base = level_base[l];
    if (blockIdx.x == 0 && threadIdx.x == 0) level_base[l + 1] = base + n;
    const int k = threadIdx.x & 7, node = threadIdx.x >> 3, lane = threadIdx.x & 31, lane0 = lane & ~7;
    for (int t0 = blockIdx.x * COLLAPSE_NODES; t0 < n; t0 += gridDim.x * COLLAPSE_NODES) {
        const bool valid = t0 + node < n;
        const int b = valid ? tasks[base + t0 + node] : 0;   // binary node
        const int2 c = child[b];
        float4 nmn, nmx, mn, mx;
        ref_box(b, node_box, leaf_box, nmn, nmx);
        int ref = k == 0 ? c.x : c.y;
        ref_box(ref, node_box, leaf_box, mn, mx);
        int2 own = child[max(ref, 0)];   // the candidate's children, fetched with its box
        float ar = area(mn, mx);
        int nr = 2;
        // Replace the internal child of largest area by its two children (the first such child in
        // candidate order on ties) until there are 8 children or only leaves remain.
        for (int step = 0; step < 6; ++step) {
            float best_a = k < nr && ref >= 0 && ar > -1.0f ? ar : -1.0f;
            int best = k;
            max_of_8(best_a, best);
            const int2 cc = make_int2(__shfl_sync(0xffffffffu, own.x, lane0 | best),
                                      __shfl_sync(0xffffffffu, own.y, lane0 | best));
            const bool more = valid && best_a > -1.0f;
            if (!__any_sync(0xffffffffu, more)) break;
            if (!more) continue;
            if (k == best || k == nr) {
                ref = k == best ? cc.x : cc.y;
                ref_box(ref, node_box, leaf_box, mn, mx);
                own = child[max(ref, 0)];
                ar = area(mn, mx);
            }
            ++nr;
        }
        __syncwarp();
        // greedy slot assignment by direction: each round takes the (child, slot) pair of least cost
        const float dx = 0.5f * (mn.x + mx.x) - 0.5f * (nmn.x + nmx.x), dy = 0.5f * (mn.y + mx.y) - 0.5f * (nmn.y + nmx.y),
                    dz = 0.5f * (mn.z + mx.z) - 0.5f * (nmn.z + nmx.z);
        float gain[8];   // minus the costs
#pragma unroll
        for (int s = 0; s < 8; ++s) gain[s] = (s & 1 ? -dx : dx) + (s & 2 ? -dy : dy) + (s & 4 ? -dz : dz);
        int slot = k < nr ? -1 : 8;   // 8: no child
        uint32_t used = 0;
        for (int round = 0; round < 8; ++round) {
            float best = -INFINITY;
            int bs = 8;
#pragma unroll
            for (int s = 0; s < 8; ++s)
                if (!((used >> s) & 1u) && gain[s] > best) {
                    best = gain[s];
                    bs = s;
                }
            int pair = slot < 0 ? k * 16 + bs : 255;
            if (slot >= 0) best = -INFINITY;
            max_of_8(best, pair);
            const bool open = round < nr;
            if (!__any_sync(0xffffffffu, open)) break;
            // a child whose box has no finite centre takes the lowest free slot
            if ((pair & 15) == 8) pair = (pair & ~15) | (__ffs(~used) - 1);
            if (open) {
                if (k == pair >> 4) slot = pair & 15;
                used |= 1u << (pair & 15);
            }
        }
        const bool leaf = ref < 0, has = valid && slot < 8;
        uint32_t masks = has ? (leaf ? 0x8000u : 0x80u) >> slot : 0u;   // slot s at bit 7 - s: internal | leaf << 8
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) masks |= __shfl_xor_sync(0xffffffffu, masks, o);
        const uint32_t imask = masks & 0xFFu, lmask = masks >> 8;
        // Internal children take consecutive wide numbers and leaves consecutive records, both in
        // slot order: the child in slot s is number first + (children of its kind in slots below s).
        if (k == 0) {
            sums[0][node] = __popc(imask);
            sums[1][node] = __popc(lmask);
        }
        for (int j = threadIdx.x; j < COLLAPSE_NODES * CPT_WIDE_F4; j += COLLAPSE_THREADS)
            (&out[0][0])[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        if (threadIdx.x < 64) {   // warp w: exclusive sums of kind w, and the block's share of its numbers
            const int w = threadIdx.x >> 5, own = sums[w][lane];
            int x = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            int first = 0;
            if (lane == 31 && x) first = w ? (int)atomicAdd(n_leaves, (uint32_t)x) : base + n + atomicAdd(level_count + l + 1, x);
            first = __shfl_sync(0xffffffffu, first, 31);
            sums[w][lane] = first + x - own;
        }
        __syncthreads();
        const int first_child = sums[0][node], first_leaf = sums[1][node];
        // the grid of axis a from lane a (its directed division is a long sequence)
        const uint32_t e_own = grid_exponent(k == 0 ? nmn.x : k == 1 ? nmn.y : nmn.z, k == 0 ? nmx.x : k == 1 ? nmx.y : nmx.z);
        const uint32_t ex = __shfl_sync(0xffffffffu, e_own, lane0), ey = __shfl_sync(0xffffffffu, e_own, lane0 | 1),
                       ez = __shfl_sync(0xffffffffu, e_own, lane0 | 2);
        if (has) {
            const uint32_t below = 8 - slot;
            if (leaf) wide_order[first_leaf + __popc(lmask >> below)] = order[~ref];
            else tasks[first_child + __popc(imask >> below)] = ref;
            const float isx = inv_grid(ex), isy = inv_grid(ey), isz = inv_grid(ez);
            uint8_t* q = reinterpret_cast<uint8_t*>(&out[node][2]) + slot;
            q[0] = (uint8_t)q_lo(mn.x, nmn.x, isx);
            q[8] = (uint8_t)q_hi(mx.x, nmn.x, isx);
            q[16] = (uint8_t)q_lo(mn.y, nmn.y, isy);
            q[24] = (uint8_t)q_hi(mx.y, nmn.y, isy);
            q[32] = (uint8_t)q_lo(mn.z, nmn.z, isz);
            q[40] = (uint8_t)q_hi(mx.z, nmn.z, isz);
        }
        if (valid && k == 0) {
            out[node][0] = make_float4(nmn.x, nmn.y, nmn.z, __uint_as_float(ex << 23));
            out[node][1] = make_float4(__uint_as_float(ey << 23), __uint_as_float(ez << 23), __int_as_float(first_child),
                                       __int_as_float(first_leaf));
            out[node][5] = make_float4(__uint_as_float(masks), 0.f, 0.f, 0.f);
        }
        __syncthreads();
        float4* dst = wide + CPT_WIDE_F4 * (size_t)(base + t0);
        const int words = min(COLLAPSE_NODES, n - t0) * CPT_WIDE_F4;
        for (int j = threadIdx.x; j < words; j += COLLAPSE_THREADS) dst[j] = (&out[0][0])[j];
        __syncthreads();
    }
}

__global__ void k_collapse_init(int* tasks, int* level_count, int* level_base, uint32_t* n_leaves)
{
    for (int i = threadIdx.x; i < MAX_WIDE_LEVELS; i += blockDim.x) {
        level_count[i] = i == 0 ? 1 : 0;   // level 0: the root
        level_base[i] = 0;
    }
    if (threadIdx.x == 0) {
        tasks[0] = 0;   // wide node 0 stands for the binary root
        *n_leaves = 0;
    }
}

}  // namespace

size_t wide_scratch_bytes(uint32_t n)
{
    // the binary node of every wide node (at most n - 1 of them), the leaves' primitives in the
    // wide layout's order, and the level counts and bases and the leaf count
    return 2 * align_up((size_t)n * 4, 256) + align_up((2 * MAX_WIDE_LEVELS + 1) * 4, 256);
}

cpt_status build_wide(uint32_t n, const int2* child, const float4* node_box, const float4* leaf_box,
                      const uint32_t* order, float4* wide, void* scratch, size_t scratch_bytes, cudaStream_t stream,
                      uint32_t* num_wide, int* host_words, const LeafRecords& leaf_records)
{
    if (n < 2) {
        if (num_wide) *num_wide = 0;
        return CPT_OK;
    }
    if (scratch_bytes < wide_scratch_bytes(n)) return fail(CPT_ERR_INVALID_ARGUMENT, "build_wide: scratch too small");
    char* p = (char*)scratch;
    int* tasks = (int*)p;
    p += align_up((size_t)n * 4, 256);
    uint32_t* prims = (uint32_t*)p;
    p += align_up((size_t)n * 4, 256);
    int* level_count = (int*)p;
    int* level_base = level_count + MAX_WIDE_LEVELS;
    uint32_t* n_leaves = (uint32_t*)(level_base + MAX_WIDE_LEVELS);
    k_collapse_init<<<1, 128, 0, stream>>>(tasks, level_count, level_base, n_leaves);
    add_launches(1);
    // A grid that is resident at once; each block takes nodes of its level in turn.  The host looks at
    // the level counts after a batch of levels (first log8(n) + 5, which meshes need: 9 of 81,920
    // primitives, 11 of 1.31M; then 8 at a time; a level whose count is zero returns at once but costs
    // its launch, 2.5 us), after queueing the leaf records of the leaves found so far, so that nothing
    // waits for its look.
    // per device (the first 64 ordinals; others are queried on every call)
    static int resident_of[64] = {};
    int dev = 0;
    CPT_CUDA(cudaGetDevice(&dev));
    int resident = (dev >= 0 && dev < 64) ? resident_of[dev] : 0;
    if (resident == 0) {
        int sms = 0, per_sm = 0;
        CPT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        CPT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_collapse_level, COLLAPSE_THREADS, 0));
        resident = std::max(1, sms * std::max(1, per_sm));
        if (dev >= 0 && dev < 64) resident_of[dev] = resident;
    }
    int l = 0, batch = 5;
    for (uint64_t m = 1; m < n; m *= 8) ++batch;
    for (;; batch = 8) {
        const int first = l, stop = std::min(l + batch, MAX_WIDE_LEVELS - 1);
        for (; l < stop; ++l) {
            // level l has at most 8^l nodes, and no more than there are binary nodes
            const uint64_t most = std::min<uint64_t>(l < 10 ? 1ull << (3 * l) : n, n);
            const unsigned grid = (unsigned)std::min<uint64_t>((most + COLLAPSE_NODES - 1) / COLLAPSE_NODES, (uint64_t)resident);
            k_collapse_level<<<grid, COLLAPSE_THREADS, 0, stream>>>(child, node_box, leaf_box, tasks, level_count,
                                                                    level_base, l, order, prims, n_leaves, wide);
        }
        add_launches(stop - first);
        CPT_CUDA(cudaGetLastError());
        cpt_status st = leaf_records(prims, n_leaves);
        if (st != CPT_OK) return st;
        // level l: its count (wide nodes still to collapse) and base (= wide nodes written)
        CPT_CUDA(cudaMemcpyAsync(host_words, level_count, 2 * MAX_WIDE_LEVELS * sizeof(int), cudaMemcpyDeviceToHost, stream));
        CPT_CUDA(cudaStreamSynchronize(stream));
        if (host_words[l] == 0 || l >= MAX_WIDE_LEVELS - 1) break;
    }
    if (host_words[l] != 0) return fail(CPT_ERR_STACK_OVERFLOW, "build_wide: collapse did not finish");
    if (num_wide) *num_wide = (uint32_t)host_words[MAX_WIDE_LEVELS + l];
    return CPT_OK;
}

}  // namespace cpt
