// The device memory pool of the setup paths (common.cuh, PoolScope).
#include <mutex>

#include "common.cuh"

namespace femgpu {
namespace {

constexpr int MAX_DEVICES = 64;
// What each device's pool keeps free outside scopes.
constexpr uint64_t KEPT_BYTES = (uint64_t)2 << 30;

struct Pool {
    cudaMemPool_t p = nullptr;
    bool tried = false;
    int scopes = 0;     // open on any thread
    uint64_t used = 0;  // bytes of its buffers (the runtime's figure does not fall at a cudaFree)
};
std::mutex g_mutex;
Pool g_pool[MAX_DEVICES];

void set_threshold(cudaMemPool_t p, uint64_t bytes) {
    cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &bytes);
}

// Bounds what the pool keeps free. The release threshold counts the buffers in use too: fixed at
// 2 GiB, the pool of a larger solver gave back every free block at each synchronization and mapped
// it again for the next buffer. Setup of the 128^3 heat solver 90 -> 62 ms, of the 256 x 32 x 32
// box-cell solver 75 -> 60, of the 200 x 20 x 20 P2 beam's 190 -> 153.
void settle(const Pool& pool) {
    if (!pool.p || pool.scopes > 0) return;
    const uint64_t keep = pool.used + KEPT_BYTES;
    set_threshold(pool.p, keep);
    uint64_t reserved = 0;
    cudaMemPoolGetAttribute(pool.p, cudaMemPoolAttrReservedMemCurrent, &reserved);
    if (reserved > keep) cudaMemPoolTrimTo(pool.p, keep);
}

// The entry of a device, or null.
Pool* entry(int device) {
    return device >= 0 && device < MAX_DEVICES ? &g_pool[device] : nullptr;
}

// The pool of `device`, made on first use; null where the device has no pools.
cudaMemPool_t pool_of(int device) {
    Pool* e = entry(device);
    if (!e) return nullptr;
    std::lock_guard<std::mutex> g(g_mutex);
    if (!e->tried) {
        e->tried = true;
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t p = nullptr;
        if (cudaMemPoolCreate(&p, &props) == cudaSuccess) {
            e->p = p;
            set_threshold(p, e->scopes > 0 ? UINT64_MAX : KEPT_BYTES);
        }
        cudaGetLastError();
    }
    return e->p;
}

}  // namespace

PoolScope::PoolScope(cudaStream_t s, bool setup) : s_(s), outer_(current_) {
    current_ = this;
    if (!setup) return;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return;
    Pool* e = entry(device);
    if (!e) return;
    device_ = device;
    std::lock_guard<std::mutex> g(g_mutex);
    if (e->scopes++ == 0 && e->p) set_threshold(e->p, UINT64_MAX);
}

PoolScope::~PoolScope() {
    current_ = outer_;
    Pool* e = entry(device_);
    if (!e) return;
    std::lock_guard<std::mutex> g(g_mutex);
    if (--e->scopes == 0) settle(*e);
}

void pool_trim() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return;
    Pool* e = entry(device);
    if (!e) return;
    std::lock_guard<std::mutex> g(g_mutex);
    if (e->p) cudaMemPoolTrimTo(e->p, 0);
}

cudaError_t device_alloc(void** p, size_t bytes, int* pool) {
    *pool = -1;
    if (PoolScope::current()) {
        int device = 0;
        cudaError_t e = cudaGetDevice(&device);
        if (e != cudaSuccess) return e;
        if (cudaMemPool_t from = pool_of(device)) {
            const cudaStream_t s = PoolScope::current()->stream();
            e = cudaMallocFromPoolAsync(p, bytes, from, s);
            if (e == cudaErrorMemoryAllocation) {
                // Free blocks that other streams' order holds back, or that do not fit together.
                cudaGetLastError();
                cudaStreamSynchronize(s);
                cudaMemPoolTrimTo(from, 0);
                e = cudaMallocFromPoolAsync(p, bytes, from, s);
            }
            if (e == cudaSuccess) {
                *pool = device;
                std::lock_guard<std::mutex> g(g_mutex);
                g_pool[device].used += bytes;
            }
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

void device_free(void* p, size_t bytes, int pool) {
    if (pool >= 0) {
        Pool& of = g_pool[pool];
        std::lock_guard<std::mutex> g(g_mutex);
        of.used -= bytes;
        if (!PoolScope::current()) settle(of);
    }
    if (pool >= 0 && PoolScope::current())
        cudaFreeAsync(p, PoolScope::current()->stream());
    else
        cudaFree(p);
}

}  // namespace femgpu
