// pool.cu -- device memory of the library's buffers (DevBuf), from one CUDA
// memory pool per device.
//
// Building a graph and a run's first call make dozens of buffers, and
// cudaMalloc / cudaFree map and unmap device memory each time: loading a
// 2^20 / 2^24 edge list and one SSSP on it spent more than half of its
// 28.3 ms there.  The pool keeps at most 1/16 of the device's memory mapped
// between uses, no more than kPoolSpare of it unused once a graph or a batch is
// destroyed (so that other allocators of the process find the rest), and gives
// all of it back when the last context of the device is destroyed.  Buffers above kPoolMax come from cudaMalloc: past the kept
// size the pool unmaps at every wait, and mapping anew there is slower (a
// 2^24 / 2^28 graph with every buffer from the pool: built in 739 ms against
// 223 ms).  So do buffers whose addresses callers get (pool_detach): memory of
// a pool can neither be opened by another process (cudaIpcGetMemHandle) nor
// reached from a peer GPU by cudaDeviceEnablePeerAccess.
//
// Ordering.  Callers rely on what cudaMalloc and cudaFree give them: memory
// usable on every stream at once, and no use in flight when it is handed on.
// So an allocation waits for the pool's own stream, and a release first waits
// for the calling context's stream, on which all work of its buffers runs or
// joins (the whole device when no context is current).
#include <mutex>
#include <unordered_set>
#include "mb_internal.cuh"

namespace mb {
namespace {

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    int contexts = 0;
    std::unordered_set<void *> live, plain;  // pool allocations; cudaMalloc'ed ones (no pool to be had)
};

std::mutex g_mutex;
constexpr int kMaxDevices = 64;
constexpr size_t kPoolMax = (size_t)256 << 20;
// What building a graph of pooled arrays and one SSSP on it take at most: a
// dozen buffers of kPoolMax.  With 2 GB a graph of 2^20 / 6.3 10^7 was built in 12.2 ms
// and destroyed in 5.2, with this in 7.1 and 0.1.
constexpr uint64_t kPoolSpare = (uint64_t)3 << 30;
DevicePool g_pools[kMaxDevices];

void drop_pool(DevicePool &d) {
    if (d.pool) cudaMemPoolDestroy(d.pool);
    if (d.stream) cudaStreamDestroy(d.stream);
    d.pool = nullptr;
    d.stream = nullptr;
    cudaGetLastError();
}

bool make_pool(DevicePool &d, int device) {
    if (d.pool) return true;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    size_t free_b = 0, total = 0;
    if (cudaMemGetInfo(&free_b, &total) != cudaSuccess || cudaMemPoolCreate(&d.pool, &props) != cudaSuccess) {
        d.pool = nullptr;
        cudaGetLastError();
        return false;
    }
    uint64_t keep = total / 16;
    if (cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
        cudaStreamCreateWithFlags(&d.stream, cudaStreamNonBlocking) != cudaSuccess) {
        drop_pool(d);
        return false;
    }
    return true;
}

cudaError_t pool_try(DevicePool &d, size_t n, void **p) {
    cudaError_t e = cudaMallocFromPoolAsync(p, n, d.pool, d.stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(d.stream);
    return e;
}

thread_local cudaStream_t t_stream = nullptr;
thread_local bool t_idle = false;

}  // namespace

void *pool_alloc(size_t n) {
    int device = 0;
    MB_CUDA(cudaGetDevice(&device));
    std::lock_guard<std::mutex> lock(g_mutex);
    void *p = nullptr;
    if (device < kMaxDevices) {
        DevicePool &d = g_pools[device];
        for (int attempt = 0; attempt < 2 && n <= kPoolMax && make_pool(d, device); attempt++) {
            const cudaError_t e = pool_try(d, n, &p);
            if (e == cudaSuccess) {
                d.live.insert(p);
                return p;
            }
            cudaGetLastError();
            if (e == cudaErrorMemoryAllocation) cudaMemPoolTrimTo(d.pool, 0);
            else drop_pool(d);  // the device was reset under it
            cudaGetLastError();
        }
        cudaError_t e = cudaMalloc(&p, n);
        if (e == cudaErrorMemoryAllocation && d.pool) {  // what the pool keeps may be enough
            cudaGetLastError();
            cudaMemPoolTrimTo(d.pool, 0);
            e = cudaMalloc(&p, n);
        }
        MB_CUDA(e);
        d.plain.insert(p);
        return p;
    }
    MB_CUDA(cudaMalloc(&p, n));
    return p;
}

void pool_free(void *p) {
    if (!p) return;
    if (!t_idle) {
        if (t_stream) cudaStreamSynchronize(t_stream);
        else cudaDeviceSynchronize();
    }
    std::lock_guard<std::mutex> lock(g_mutex);
    for (DevicePool &d : g_pools) {
        if (d.live.erase(p)) {
            if (d.stream) cudaFreeAsync(p, d.stream);
            if (d.contexts == 0 && d.live.empty()) drop_pool(d);
            cudaGetLastError();
            return;
        }
        if (d.plain.erase(p)) break;
    }
    cudaFree(p);
    cudaGetLastError();
}

void pool_detach(DevBuf &b) {
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        bool pooled = false;
        for (DevicePool &d : g_pools) pooled = pooled || d.live.count(b.p);
        if (!pooled) return;
    }
    void *p = nullptr;
    if (cudaMalloc(&p, b.bytes) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaMemcpy(p, b.p, b.bytes, cudaMemcpyDeviceToDevice);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        cudaFree(p);
        MB_CUDA(e);
    }
    pool_free(b.p);
    b.p = p;
    std::lock_guard<std::mutex> lock(g_mutex);
    if (device < kMaxDevices) g_pools[device].plain.insert(p);
}

void pool_use_stream(cudaStream_t s) { t_stream = s; }

void pool_trim(int device) {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (device < 0 || device >= kMaxDevices) return;
    DevicePool &d = g_pools[device];
    uint64_t used = 0, reserved = 0;
    if (d.pool && cudaStreamSynchronize(d.stream) == cudaSuccess &&
        cudaMemPoolGetAttribute(d.pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess &&
        cudaMemPoolGetAttribute(d.pool, cudaMemPoolAttrReservedMemCurrent, &reserved) == cudaSuccess &&
        reserved > used + kPoolSpare)
        cudaMemPoolTrimTo(d.pool, used + kPoolSpare);
    cudaGetLastError();
}

void pool_context(int device, int delta) {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (device < 0 || device >= kMaxDevices) return;
    DevicePool &d = g_pools[device];
    d.contexts += delta;
    if (d.contexts > 0 || !d.pool) return;
    cudaStreamSynchronize(d.stream);
    if (d.live.empty()) drop_pool(d);
    else cudaMemPoolTrimTo(d.pool, 0);
    cudaGetLastError();
}

PoolIdle::PoolIdle() : was(t_idle) { t_idle = true; }
PoolIdle::~PoolIdle() { t_idle = was; }

}  // namespace mb
