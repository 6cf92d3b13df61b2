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
// Small buffers (kSmallMax) that are released stay with the library, by powers
// of two and up to kSmallSpare in all, and go to the next one that asks: a
// first PageRank on a graph of some thousand vertices makes and drops some
// forty of them, at 5 us each through CUDA (0.60 ms where cudaMalloc's own small
// blocks took 0.43; 0.50 with this alone).
//
// Ordering.  Callers rely on what cudaMalloc and cudaFree give them: memory
// usable on every stream at once, and no use in flight when it is handed on.
// So an allocation waits for the pool's own stream, and a release first waits
// for the calling context's stream, on which all work of its buffers runs or
// joins (the whole device when no context is current).
#include <mutex>
#include <unordered_map>
#include <unordered_set>
#include "mb_internal.cuh"

namespace mb {
namespace {

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    int contexts = 0;
    std::unordered_map<void *, size_t> live;  // pool allocations
    std::unordered_set<void *> plain;         // cudaMalloc'ed ones (large, detached, or no pool to be had)
    std::vector<void *> spare[32];            // released ones of 2^k bytes
    size_t spare_bytes = 0;
};

std::mutex g_mutex;
constexpr int kMaxDevices = 64;
constexpr size_t kPoolMax = (size_t)256 << 20;
constexpr size_t kSmallMax = (size_t)1 << 20, kSmallSpare = (size_t)32 << 20;
// What building a graph of pooled arrays and one SSSP on it take at most: a
// dozen buffers of kPoolMax.  With 2 GB a graph of 2^20 / 6.3 10^7 was built in 12.2 ms
// and destroyed in 5.2, with this in 7.1 and 0.1.
constexpr uint64_t kPoolSpare = (uint64_t)3 << 30;
DevicePool g_pools[kMaxDevices];

int small_class(size_t n) {
    int k = 8;
    while (((size_t)1 << k) < n) k++;
    return k;
}

void drop_spare(DevicePool &d) {
    for (auto &list : d.spare) {
        for (void *p : list) cudaFreeAsync(p, d.stream);
        list.clear();
    }
    d.spare_bytes = 0;
}

void drop_pool(DevicePool &d) {
    if (d.pool && d.stream) {
        drop_spare(d);
        cudaStreamSynchronize(d.stream);
    }
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
        if (n <= kSmallMax) {
            const int k = small_class(n);
            n = (size_t)1 << k;
            if (!d.spare[k].empty() && cudaStreamQuery(d.stream) != cudaSuccess) {  // the device was reset under it
                cudaGetLastError();
                for (auto &list : d.spare) list.clear();
                d.spare_bytes = 0;
            }
            if (!d.spare[k].empty()) {
                p = d.spare[k].back();
                d.spare[k].pop_back();
                d.spare_bytes -= n;
                d.live.emplace(p, n);
                return p;
            }
        }
        for (int attempt = 0; attempt < 2 && n <= kPoolMax && make_pool(d, device); attempt++) {
            const cudaError_t e = pool_try(d, n, &p);
            if (e == cudaSuccess) {
                d.live.emplace(p, n);
                return p;
            }
            cudaGetLastError();
            drop_spare(d);
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
        const auto it = d.live.find(p);
        if (it != d.live.end()) {
            const size_t n = it->second;
            d.live.erase(it);
            if (d.contexts > 0 && n <= kSmallMax && d.spare_bytes + n <= kSmallSpare) {
                d.spare[small_class(n)].push_back(p);
                d.spare_bytes += n;
                return;
            }
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
    drop_spare(d);
    cudaStreamSynchronize(d.stream);
    if (d.live.empty()) drop_pool(d);
    else cudaMemPoolTrimTo(d.pool, 0);
    cudaGetLastError();
}

PoolIdle::PoolIdle() : was(t_idle) { t_idle = true; }
PoolIdle::~PoolIdle() { t_idle = was; }

}  // namespace mb
