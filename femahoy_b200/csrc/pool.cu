// The device memory pool of the setup paths (common.cuh, PoolScope).
#include <mutex>

#include "common.cuh"

namespace femgpu {
namespace {

constexpr int MAX_DEVICES = 64;
// What each device's pool keeps when its buffers are freed; more goes back to the device at the
// next synchronization.
constexpr uint64_t KEPT_BYTES = (uint64_t)2 << 30;

std::mutex g_mutex;
cudaMemPool_t g_pool[MAX_DEVICES] = {};
bool g_tried[MAX_DEVICES] = {};

// The pool of `device`, made on first use; null where the device has no pools.
cudaMemPool_t pool_of(int device) {
    if (device < 0 || device >= MAX_DEVICES) return nullptr;
    std::lock_guard<std::mutex> g(g_mutex);
    if (!g_tried[device]) {
        g_tried[device] = true;
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t p = nullptr;
        uint64_t kept = KEPT_BYTES;
        if (cudaMemPoolCreate(&p, &props) == cudaSuccess) {
            if (cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &kept) == cudaSuccess)
                g_pool[device] = p;
            else
                cudaMemPoolDestroy(p);
        }
        cudaGetLastError();
    }
    return g_pool[device];
}

}  // namespace

void pool_trim() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= MAX_DEVICES) return;
    cudaMemPool_t p;
    {
        std::lock_guard<std::mutex> g(g_mutex);
        p = g_pool[device];
    }
    if (p) cudaMemPoolTrimTo(p, 0);
}

cudaError_t device_alloc(void** p, size_t bytes, bool* pooled) {
    *pooled = false;
    if (PoolScope::current()) {
        int device = 0;
        cudaError_t e = cudaGetDevice(&device);
        if (e != cudaSuccess) return e;
        if (cudaMemPool_t pool = pool_of(device)) {
            const cudaStream_t s = PoolScope::current()->stream();
            e = cudaMallocFromPoolAsync(p, bytes, pool, s);
            if (e == cudaErrorMemoryAllocation) {
                // Free blocks that other streams' order holds back, or that do not fit together.
                cudaGetLastError();
                cudaStreamSynchronize(s);
                cudaMemPoolTrimTo(pool, 0);
                e = cudaMallocFromPoolAsync(p, bytes, pool, s);
            }
            *pooled = e == cudaSuccess;
            return e;
        }
    }
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        pool_trim();
        e = cudaMalloc(p, bytes);
    }
    return e;
}

void device_free(void* p, bool pooled) {
    if (pooled && PoolScope::current())
        cudaFreeAsync(p, PoolScope::current()->stream());
    else
        cudaFree(p);
}

}  // namespace femgpu
