// Shared definitions of the femgpu CUDA library: status codes, error state, device buffers and
// the launch geometry of the B200 (148 SMs).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "femgpu.h"

namespace femgpu {

// A failure carrying a status code of femgpu.h and the reference's error text.
struct Failure : std::runtime_error {
    int code;
    Failure(int c, const std::string& s) : std::runtime_error(s), code(c) {}
};

void set_last_error(const std::string& s);

// The runtime keeps a failed call's error for the next cudaGetLastError, which would then blame a
// later launch that is fine: it is taken out here.
#define FG_CUDA(call)                                                                  \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess) {                                                       \
            cudaGetLastError();                                                        \
            throw ::femgpu::Failure(FEMGPU_ERR_CUDA, std::string("CUDA error: ") +    \
                                                         cudaGetErrorString(e_) +     \
                                                         " at " __FILE__ ":" +        \
                                                         std::to_string(__LINE__));   \
        }                                                                              \
    } while (0)

#define FG_CHECK_LAUNCH() FG_CUDA(cudaGetLastError())

constexpr int NUM_SMS = 148;

inline int blocks_for(int64_t n, int threads, int cap = NUM_SMS * 16) {
    int64_t b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > cap) b = cap;
    return (int)b;
}

// Device memory for the buffers below. While a PoolScope is open on a host thread, the buffers
// that the thread makes come from a pool of the device (pool.cu) in the order of the scope's
// stream, and the ones it frees go back in that order; without a scope a buffer is a cudaMalloc
// of its own and its cudaFree waits for the device.
//
// What it is for: a model's way from the mesh to the solution makes and frees about 190 buffers,
// each cudaMalloc and cudaFree mapping or unmapping memory (0.15 ms each, more when other
// processes of the machine do the same). With every buffer a cudaMalloc of its own a 64^3 heat
// model takes 88 ms on B200 and a 60 x 8 x 8 P2 beam 55 (medians, quiet machine); with the pool 34
// and 25.
//
// The rules that keep it safe. A scope is opened only around code whose buffers are used on the
// scope's stream alone until it has been synchronized, and every buffer that outlives the scope
// is handed on after that. A pooled buffer freed with no scope open is returned at once: its
// owner has then synchronized the streams that used it (the solver's destructor its own stream;
// every call on a matrix synchronizes before it returns, on errors too). Outside scopes the pool
// keeps 2 GiB of free memory at most (while one is open, all that it has: a setup frees and asks
// again and again), gives them back when an allocation does not fit, when a server makes room or
// when the caller asks (femgpu_trim), and its order across streams and threads is the CUDA
// runtime's own.
class PoolScope {
   public:
    // `setup` false: a run of a handle, whose buffers are few and alike from call to call, so that
    // what the pool keeps need not be touched.
    explicit PoolScope(cudaStream_t s, bool setup = true);
    ~PoolScope();
    PoolScope(const PoolScope&) = delete;
    PoolScope& operator=(const PoolScope&) = delete;
    cudaStream_t stream() const { return s_; }
    static const PoolScope* current() { return current_; }

   private:
    cudaStream_t s_;
    int device_ = -1;
    const PoolScope* outer_;
    static inline thread_local const PoolScope* current_ = nullptr;
};

// `pool` tells device_free where the memory came from: the device whose pool it was, or -1.
cudaError_t device_alloc(void** p, size_t bytes, int* pool);
void device_free(void* p, size_t bytes, int pool);
// Gives what the current device's pool keeps free back to the device.
void pool_trim();

// An owned device allocation of `count` elements of T.
template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t count = 0;
    int pool = -1;  // of the device whose pool p is from
    DevBuf() = default;
    explicit DevBuf(size_t n) { alloc(n); }
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    DevBuf(DevBuf&& o) noexcept : p(o.p), count(o.count), pool(o.pool) {
        o.p = nullptr;
        o.count = 0;
    }
    DevBuf& operator=(DevBuf&& o) noexcept {
        if (this != &o) {
            release();
            p = o.p;
            count = o.count;
            pool = o.pool;
            o.p = nullptr;
            o.count = 0;
        }
        return *this;
    }
    ~DevBuf() { release(); }
    void alloc(size_t n) {
        release();
        count = n;
        if (n) FG_CUDA(device_alloc((void**)&p, n * sizeof(T), &pool));
    }
    void release() {
        if (p) device_free(p, count * sizeof(T), pool);
        p = nullptr;
        count = 0;
    }
    size_t bytes() const { return count * sizeof(T); }
    void upload(const T* h, size_t n, cudaStream_t s) {
        if (n > count) alloc(n);
        if (n) FG_CUDA(cudaMemcpyAsync(p, h, n * sizeof(T), cudaMemcpyHostToDevice, s));
    }
    void download(T* h, size_t n, cudaStream_t s) const {
        if (n) FG_CUDA(cudaMemcpyAsync(h, p, n * sizeof(T), cudaMemcpyDeviceToHost, s));
    }
    std::vector<T> to_host(cudaStream_t s) const {
        std::vector<T> v(count);
        download(v.data(), count, s);
        FG_CUDA(cudaStreamSynchronize(s));
        return v;
    }
    void zero(cudaStream_t s) {
        if (count) FG_CUDA(cudaMemsetAsync(p, 0, bytes(), s));
    }
};

// A device CSR matrix with both triangles, sorted columns (sparse.rs:12-17).
struct DevCsr {
    int64_t n = 0;
    int64_t nnz = 0;
    DevBuf<int64_t> ptr;
    DevBuf<uint32_t> idx;
    DevBuf<double> val;
};

// Exclusive prefix sum of `n` counts into `out` (n + 1 values; out[n] = total), on `s`.
void exclusive_scan(const int64_t* in, int64_t* out, int64_t n, cudaStream_t s);
void exclusive_scan32(const uint32_t* in, int64_t* out, int64_t n, cudaStream_t s);

// Programmatic dependent launch. The kernels of a PCG iteration are launched so that each may
// start while the one before it drains; every such kernel first waits (griddepcontrol.wait) for
// the completion and the memory of the kernel before it, so it reads what it would have read
// without the attribute. On the short kernels of the coarse levels the launch latency this
// hides is most of their time.
// (An explicit early trigger in the PCG kernels, whose inputs nothing can load ahead, measured no
// better on the 128^3 heat solve and worse on a transient run, 6.47 -> 6.64 ms, and a batch, 22.0
// -> 23.1 ms: those blocks trigger when they exit. The sparse solves trigger early.)
// Lets the blocks of the kernel after this one start once every block of this one has called it
// (or exited). For kernels that load much before their pdl_wait, and whose inputs the next kernel
// reads by plain loads: the read-only path is for data that nothing writes while a kernel exists.
__device__ __forceinline__ void pdl_trigger() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
static void launch(bool pdl, void (*kernel)(KArgs...), int grid, int block, cudaStream_t s,
                   Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = pdl ? &attr : nullptr;
    cfg.numAttrs = pdl ? 1 : 0;
    FG_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
}

// The same with `smem` bytes of dynamic shared memory.
template <typename... KArgs, typename... Args>
static void launch_smem(bool pdl, void (*kernel)(KArgs...), int grid, int block, size_t smem,
                        cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = pdl ? &attr : nullptr;
    cfg.numAttrs = pdl ? 1 : 0;
    FG_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
}

// A scalar from device memory.
template <class T>
T fetch(const T* d, cudaStream_t s) {
    T h;
    FG_CUDA(cudaMemcpyAsync(&h, d, sizeof(T), cudaMemcpyDeviceToHost, s));
    FG_CUDA(cudaStreamSynchronize(s));
    return h;
}

}  // namespace femgpu
