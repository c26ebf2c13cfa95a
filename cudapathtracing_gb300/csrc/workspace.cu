// workspace.cu — device memory: the workspace pool of each device, and allocation that gives idle
// workspace back before it fails.
//
// Workspaces of the calls (path slots, filter and host-image buffers) come from one pool per device, which
// its contexts share and which goes with the last of them.  It keeps up to 1/40 of the device's memory
// between calls (7 GB of 284): the device's default pool gives everything back to the system whenever a
// stream is waited for, and every call waits (0.33 ms per call for a 256 x 256 preview's slots, 0.2 ms for
// a 1080p filter).  One pool, not one per context: a program with a context per lane keeps the same bound.
//
// Idle workspace never makes a call fail: an allocation that does not fit waits for its stream, trims the
// pool and tries once more, and pool_trim (cpt_context_trim) does the same for a program's other users of
// the device.
#include <cuda_runtime.h>

#include <cstring>
#include <map>
#include <mutex>

#include "cpt_internal.h"

namespace cpt {

namespace {

struct DevicePool {
    cudaMemPool_t pool;
    int users;
};
std::mutex g_mu;
std::map<int, DevicePool> g_pools;   // by device ordinal

// Gives the idle memory of the device's pool back, if it has one.
cudaError_t trim(int device)
{
    std::lock_guard<std::mutex> lock(g_mu);
    const auto it = g_pools.find(device);
    return it == g_pools.end() ? cudaSuccess : cudaMemPoolTrimTo(it->second.pool, 0);
}

cudaError_t trim_current()
{
    int device = 0;
    const cudaError_t e = cudaGetDevice(&device);
    return e == cudaSuccess ? trim(device) : e;
}

// Retries a failed allocation once, after `room` has made room; a failure leaves no error behind that a
// later launch would be blamed for.
template <typename Alloc, typename Room>
cpt_status with_room(Alloc alloc, Room room, const char* what)
{
    cudaError_t e = alloc();
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        if (room() == cudaSuccess) e = alloc();
    }
    if (e == cudaSuccess) return CPT_OK;
    cudaGetLastError();
    return cuda_fail(e, what);
}

}  // namespace

cpt_status pool_acquire(int device, cudaMemPool_t* out)
{
    std::lock_guard<std::mutex> lock(g_mu);
    const auto it = g_pools.find(device);
    if (it != g_pools.end()) {
        it->second.users++;
        *out = it->second.pool;
        return CPT_OK;
    }
    cudaMemPoolProps props;
    std::memset(&props, 0, sizeof props);
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    size_t free_bytes = 0, total_bytes = 0;
    CPT_CUDA(cudaMemGetInfo(&free_bytes, &total_bytes));
    uint64_t keep = total_bytes / 40;
    cudaMemPool_t pool = nullptr;
    CPT_CUDA(cudaMemPoolCreate(&pool, &props));
    const cudaError_t e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
        cudaMemPoolDestroy(pool);
        return cuda_fail(e, "workspace pool");
    }
    g_pools[device] = {pool, 1};
    *out = pool;
    return CPT_OK;
}

void pool_release(int device)
{
    std::lock_guard<std::mutex> lock(g_mu);
    const auto it = g_pools.find(device);
    if (it == g_pools.end() || --it->second.users > 0) return;
    cudaMemPoolDestroy(it->second.pool);   // memory of work in flight goes when that is done
    g_pools.erase(it);
}

cpt_status pool_trim(int device)
{
    CPT_CUDA(trim(device));
    return CPT_OK;
}

cpt_status pool_alloc(void** p, size_t bytes, cudaMemPool_t pool, cudaStream_t stream)
{
    return with_room([&] { return cudaMallocFromPoolAsync(p, bytes, pool, stream); },
                     [&] {
                         const cudaError_t e = cudaStreamSynchronize(stream);
                         return e == cudaSuccess ? trim_current() : e;
                     },
                     "workspace allocation");
}

cpt_status device_alloc(void** p, size_t bytes)
{
    return with_room([&] { return cudaMalloc(p, bytes); }, trim_current, "device allocation");
}

}  // namespace cpt
