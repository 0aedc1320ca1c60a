// mem.cu -- device memory of the library's buffers (DBuf).
//
// cudaMalloc and cudaFree cost about 0.25 ms each here, cudaFree stops the
// device, and a set-up makes a thousand of each (550 of the 890 ms of a
// 250k-node hierarchy's set-up).  Buffers therefore come from a memory pool
// per device, in stream order: an API call names the stream that its work
// runs on (alloc_stream), allocations and frees are enqueued there, and a
// buffer is reused only after the work before its free.  Where no stream is
// named (objects being destroyed, after their stream was synchronised) a
// stream of the pool's own is used.
//
// What the pool keeps beyond the buffers in use is bounded by kIdleBytes (and
// kTrimEvery for each further thread) when a call returns, whether it succeeded
// or not: trim_memory, at the end of every entry point, gives back what is above
// once its thread has freed kTrimEvery since the last time (a trim is a
// synchronisation and two calls of the driver).  When an allocation fails all
// of it is given back and the allocation tried again.
#include <mutex>

#include "mgm_internal.cuh"

namespace mgm {

namespace {

constexpr size_t kIdleBytes = size_t(2) << 30, kTrimEvery = size_t(64) << 20;
constexpr int kMaxDevices = 64;

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t idle = nullptr;
};
std::mutex g_mutex;
DevicePool g_pools[kMaxDevices];
thread_local cudaStream_t t_stream = nullptr;
thread_local size_t t_freed = 0;  // bytes since this thread's last trim

void check(cudaError_t e, const char *what)
{
    if (e != cudaSuccess) {
        cudaGetLastError();
        throw Error{e == cudaErrorMemoryAllocation ? 5 : 1, std::string(what) + ": " + cudaGetErrorString(e)};
    }
}

DevicePool &device_pool(int dev)
{
    if (dev < 0 || dev >= kMaxDevices) throw Error{1, "device memory: device number out of range"};
    std::lock_guard<std::mutex> lock(g_mutex);
    DevicePool &p = g_pools[dev];
    if (!p.pool) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        check(cudaMemPoolCreate(&pool, &props), "cudaMemPoolCreate");
        unsigned long long keep = ~0ull;  // trim_memory gives memory back
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        check(cudaStreamCreateWithFlags(&p.idle, cudaStreamNonBlocking), "cudaStreamCreate");
        p.pool = pool;
    }
    return p;
}

}  // namespace

void alloc_stream(cudaStream_t s) { t_stream = s; }
cudaStream_t alloc_stream() { return t_stream; }

void *dev_alloc(size_t bytes)
{
    int dev = 0;
    check(cudaGetDevice(&dev), "cudaGetDevice");
    DevicePool &p = device_pool(dev);
    const cudaStream_t s = t_stream ? t_stream : p.idle;
    void *ptr = nullptr;
    cudaError_t e = cudaMallocFromPoolAsync(&ptr, bytes, p.pool, s);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        cudaStreamSynchronize(s);
        cudaMemPoolTrimTo(p.pool, 0);
        e = cudaMallocFromPoolAsync(&ptr, bytes, p.pool, s);
    }
    check(e, "device allocation");
    if (s == p.idle) check(cudaStreamSynchronize(s), "device allocation");
    return ptr;
}

void dev_free(void *ptr, size_t bytes) noexcept
{
    if (!ptr) return;
    t_freed += bytes;
    cudaStream_t s = t_stream;
    if (!s) {
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, ptr) != cudaSuccess || at.device < 0 || at.device >= kMaxDevices) {
            cudaGetLastError();
            return;
        }
        s = g_pools[at.device].idle;
    }
    if (cudaFreeAsync(ptr, s) != cudaSuccess) cudaGetLastError();
}

void trim_memory() noexcept
{
    if (t_freed < kTrimEvery) return;
    t_freed = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return;
    cudaMemPool_t pool;
    cudaStream_t s;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        pool = g_pools[dev].pool;
        if (!pool) return;
        s = t_stream ? t_stream : g_pools[dev].idle;
    }
    cudaStreamSynchronize(s);  // memory is given back once the work before its free is done
    unsigned long long used = 0;
    if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess)
        cudaMemPoolTrimTo(pool, (size_t)used + kIdleBytes - kTrimEvery);
    cudaGetLastError();
}

}  // namespace mgm
