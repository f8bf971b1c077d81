// pool.cpp — the library's device memory pool.
//
// Plans and host-pointer calls allocate and free device memory in stream
// order, many times over in programs that use a matrix once.  The device's
// default pool returns its memory to the system at every synchronisation, so
// each such call mapped and unmapped its buffers again: csr5_kernel on 14M nnz
// took 2.6 to 10 ms a call for 0.25 ms of kernels.  The library therefore has
// a pool of its own on each device, which keeps at most 1/32 of the device's
// memory while nothing uses it, gives all of that back when an allocation of
// the library does not fit or the program asks for the free memory
// (get_gpu_availble_mem), and leaves the default pool and its settings to
// the program.  A pool gives back what it holds above its bound at the next
// synchronisation, so what frees large buffers ends with pool_settle, which
// synchronises once more if more than the bound is unused (each time would cost a
// one-off product 4 us of 107, and a batch of 512 matrices that follows another
// 130 ms of 540 for memory mapped anew).  Stream order makes the pool safe for several streams;
// the driver makes it safe for several threads.
#include <cuda.h>  // driver types only; the entry points are fetched at run time
#include <cuda_runtime.h>

#include <mutex>

#include "../sbb_internal.h"
#include "context_table.h"

namespace sbb {

unsigned long long current_context_id()
{
    using GetCurrent = CUresult (*)(CUcontext *);
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult q;
        void *f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<GetCurrent>(f);
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<GetId>(f);
    });
    if (!get_current || !get_id) return 0;
    CUcontext c = nullptr;
    if (get_current(&c) != CUDA_SUCCESS || !c) return 0;
    unsigned long long id = 0;
    return get_id(c, &id) == CUDA_SUCCESS ? id : 0;
}

namespace {

// The pool of the current device's current context, made the first time; null
// when there is none to be had, and the default pool serves, or with make ==
// false when there is none yet.  (After cudaDeviceReset the context is another.)
cudaMemPool_t device_pool(bool make = true)
{
    static std::mutex mu;
    static auto &pools = *new ContextTable<cudaMemPool_t>;  // outlives static destructors
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    unsigned long long ctx = current_context_id();
    if (ctx != 0)
        if (cudaMemPool_t *known = pools.find(dev, ctx)) return *known;
    if (!make) return nullptr;
    size_t free_b = 0, total_b = 0;  // also makes the device's context current
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return nullptr;
    ctx = current_context_id();
    if (ctx == 0) return nullptr;
    if (cudaMemPool_t *known = pools.find(dev, ctx)) return *known;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    unsigned long long keep = total_b / 32;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    pools.add(dev, ctx, pool);
    return pool;
}

}  // namespace

static bool pool_bytes(cudaMemPool_t pool, unsigned long long *reserved, unsigned long long *used)
{
    return pool &&
           cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, reserved) == cudaSuccess &&
           cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, used) == cudaSuccess;
}

size_t pool_idle_bytes()
{
    unsigned long long reserved = 0, used = 0;
    if (!pool_bytes(device_pool(), &reserved, &used)) return 0;
    return reserved > used ? (size_t)(reserved - used) : 0;
}

void pool_settle(cudaStream_t s)
{
    cudaMemPool_t pool = device_pool(false);
    unsigned long long reserved = 0, used = 0, keep = 0;
    if (pool_bytes(pool, &reserved, &used) && reserved > used &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess &&
        reserved - used > keep)
        cudaStreamSynchronize(s);
}

size_t pool_trim()
{
    cudaMemPool_t pool = device_pool(false);
    unsigned long long reserved = 0, used = 0;
    if (!pool) return 0;
    cudaMemPoolTrimTo(pool, 0);
    return pool_bytes(pool, &reserved, &used) && reserved > used ? (size_t)(reserved - used) : 0;
}

cudaError_t pool_malloc_async(void **p, size_t bytes, cudaStream_t s)
{
    // In a stream capture the allocation becomes a node of the graph, from the
    // default pool; making a pool is not allowed there.
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &capturing) != cudaSuccess) cudaGetLastError();
    cudaMemPool_t pool = capturing == cudaStreamCaptureStatusNone ? device_pool() : nullptr;
    cudaError_t e = pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s);
    if (pool && e == cudaErrorMemoryAllocation) {
        cudaMemPoolTrimTo(pool, 0);
        cudaGetLastError();
        e = cudaMallocFromPoolAsync(p, bytes, pool, s);
    }
    // The caller gets the code and may go on without this memory: it must not
    // meet the same error again behind its next launch.
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();
    return e;
}

}  // namespace sbb
