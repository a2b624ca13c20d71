// The device memory pool (pool.cuh).
#include "pool.cuh"

#include <cstdint>
#include <map>
#include <mutex>
#include <vector>

#include "../../include/decon_b200.h"

namespace dk {

int fail(int code, const char* fmt, ...);

constexpr uint64_t kPoolKeep = uint64_t(2) << 30;

cudaStream_t setup_stream() {
    static std::mutex mu;
    static std::map<int, cudaStream_t> streams;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    auto it = streams.find(dev);
    if (it != streams.end()) return it->second;
    cudaStream_t s = nullptr;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    streams[dev] = s;
    return s;
}

int device_pool(cudaMemPool_t* out) {
    static std::mutex mu;
    static std::map<int, cudaMemPool_t> pools;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    auto it = pools.find(dev);
    if (e == cudaSuccess && it == pools.end()) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool;
        uint64_t keep = kPoolKeep;
        e = cudaMemPoolCreate(&pool, &props);
        if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e == cudaSuccess) it = pools.emplace(dev, pool).first;
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(DECON_ERR_CUDA, "device memory pool: %s", cudaGetErrorString(e));
    }
    *out = it->second;
    return DECON_OK;
}

// Memory that is to be freed but that work may still be using, per device.
static std::mutex g_held_mu;
static std::map<int, std::vector<void*>> g_held;

// Everything queued on the current device, waited for.  cudaDeviceSynchronize
// is refused while any thread captures a stream, in whatever mode, and it ends
// that capture with an error; cudaFree of a plain allocation waits for every
// stream too and is legal then (3 us on an idle device, 1.6 the former).
static bool wait_for_device() {
    void* block = nullptr;
    if (cudaMalloc(&block, 256) == cudaSuccess && cudaFree(block) == cudaSuccess) return true;
    cudaGetLastError();
    if (cudaDeviceSynchronize() == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

// Frees `ptrs` and what was held for `dev`, the current device, or holds them.
static void release(int dev, std::vector<void*> ptrs) {
    {
        std::lock_guard<std::mutex> lock(g_held_mu);
        std::vector<void*>& held = g_held[dev];
        ptrs.insert(ptrs.end(), held.begin(), held.end());
        held.clear();
    }
    // memory of a capturing thread's own objects too: nothing here is captured
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    const cudaStream_t s = setup_stream();
    if (!s || !wait_for_device()) {
        std::lock_guard<std::mutex> lock(g_held_mu);
        std::vector<void*>& held = g_held[dev];
        held.insert(held.end(), ptrs.begin(), ptrs.end());
    } else {
        for (void* p : ptrs) cudaFreeAsync(p, s);
        // what the pool does not keep goes back here, and only then do allocations
        // outside of the pool find the rest: a cudaMalloc that would fail takes the
        // unused memory of pools, but not what is still queued to be freed
        cudaStreamSynchronize(s);
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    cudaGetLastError();
}

int pool_alloc(void** p, size_t bytes, const char* what) {
    *p = nullptr;
    cudaMemPool_t pool;
    const int st = device_pool(&pool);
    if (st != DECON_OK) return st;
    const cudaStream_t s = setup_stream();
    if (!s) return fail(DECON_ERR_CUDA, "set-up stream creation failed");
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool, s);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        int dev = 0;
        cudaGetDevice(&dev);
        release(dev, {});
        cudaMemPoolTrimTo(pool, 0);
        e = cudaMallocFromPoolAsync(p, bytes, pool, s);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        return fail(e == cudaErrorMemoryAllocation ? DECON_ERR_OOM : DECON_ERR_CUDA,
                    "cudaMalloc of %zu bytes for %s failed: %s", bytes, what, cudaGetErrorString(e));
    }
    return DECON_OK;
}

void pool_free(void* const* ptrs, size_t n) {
    std::vector<void*> list;
    for (size_t i = 0; i < n; ++i)
        if (ptrs[i]) list.push_back(ptrs[i]);
    if (list.empty()) return;
    // the pool and its stream belong to the device of the memory
    int cur = 0;
    cudaGetDevice(&cur);
    cudaPointerAttributes at{};
    const bool other = cudaPointerGetAttributes(&at, list[0]) == cudaSuccess && at.device != cur;
    if (other) cudaSetDevice(at.device);
    release(other ? at.device : cur, std::move(list));
    if (other) cudaSetDevice(cur);
    cudaGetLastError();
}

}  // namespace dk
