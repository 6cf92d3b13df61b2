// prim.cu -- device-wide primitives used to build graph storage on the GPU:
// an exclusive prefix sum and a stable LSD radix sort of (key, value) pairs.
//
// These replace the reference's serial host loops that build the CSR and the
// per-destination message slots (SSSP/EdgeDataType.cu:138-186,
// SSSP/VertexDataType.cu:64-85): a stable sort by source gives the CSR, a
// stable sort of the CSR by destination gives the reverse CSR and, through
// its permutation, the reference's msgDstID.
#include "mb_internal.cuh"

namespace mb {
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// Block-wide exclusive scan of one value per thread; returns the block total
// in *total (all threads).
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t x, uint32_t *total) {
    __shared__ uint32_t warp_tot[kScanThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t inc = warp_incl_scan(x);
    if (lane == 31) warp_tot[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        constexpr int kW = kScanThreads / 32;
        uint32_t t = lane < kW ? warp_tot[lane] : 0;
        uint32_t ti = warp_incl_scan(t);
        if (lane < kW) warp_tot[lane] = ti - t;  // exclusive prefix of warp totals
        if (lane == kW - 1) *total = ti;
    }
    __syncthreads();
    uint32_t r = warp_tot[wid] + inc - x;
    __syncthreads();
    return r;
}

__global__ void k_scan_reduce(const uint32_t *__restrict__ in, int64_t n,
                              uint32_t *__restrict__ partial) {
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        int64_t j = base + i * kScanThreads + threadIdx.x;
        if (j < n) s += in[j];
    }
    __shared__ uint32_t tot;
    (void)block_excl_scan(s, &tot);
    if (threadIdx.x == 0) partial[blockIdx.x] = tot;
}

__global__ void k_scan_apply(const uint32_t *__restrict__ in, uint32_t *__restrict__ out,
                             int64_t n, const uint32_t *__restrict__ partial,
                             uint32_t *__restrict__ total_dev) {
    __shared__ uint32_t sm[kScanTile + kScanTile / 32];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    // striped, coalesced load into padded shared memory
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        int idx = i * kScanThreads + threadIdx.x;
        int64_t j = base + idx;
        sm[idx + (idx >> 5)] = j < n ? in[j] : 0u;
    }
    __syncthreads();
    uint32_t v[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        int idx = threadIdx.x * kScanItems + i;
        v[i] = sm[idx + (idx >> 5)];
        s += v[i];
    }
    __shared__ uint32_t tot;
    uint32_t run = block_excl_scan(s, &tot) + (partial ? partial[blockIdx.x] : 0u);
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        int idx = threadIdx.x * kScanItems + i;
        sm[idx + (idx >> 5)] = run;
        run += v[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
        int idx = i * kScanThreads + threadIdx.x;
        int64_t j = base + idx;
        if (j < n) out[j] = sm[idx + (idx >> 5)];
    }
    if (total_dev && blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanThreads - 1)
        *total_dev = run;  // exclusive prefix of the last thread + its items
}

// ---------------------------------------------------------------------------
// radix sort: least significant digit first, digits of at most 8 bits.  A pass
// counts each tile's digits, scans the counts digit-major, and scatters.  The
// scatter is bound by its stores: a tile's elements are first put in digit
// order in shared memory, so that each digit's run goes out as one coalesced
// piece (kSortTile / 256 elements on average), and the values ride along
// with their keys, instead of a permutation that a random gather applies
// afterwards.

constexpr int kSortThreads = 512;
constexpr int kSortRounds = 8;
constexpr int kSortTile = kSortThreads * kSortRounds;  // 4096 keys per tile
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kRadix = 256;
constexpr int kMaxPay = 3;

struct SortPass {
    const uint32_t *key_in, *pay_in[kMaxPay];
    uint32_t *key_out, *pay_out[kMaxPay];
    uint32_t *slot_out;  // the last payload's inverse: slot_out[value] = position
    int64_t n, ntiles;
    int shift;
    uint32_t mask;
    bool reverse;        // element j is input n - 1 - j
    bool iota;           // the last payload is j itself
    const uint32_t *offsets;  // exclusive scan of the digit counts, [digit][tile]
};

__global__ void __launch_bounds__(kSortThreads) k_radix_hist(SortPass a, uint32_t *hist) {
    __shared__ uint32_t h[4][kRadix];
    for (int i = threadIdx.x; i < 4 * kRadix; i += kSortThreads) h[i / kRadix][i % kRadix] = 0;
    __syncthreads();
    uint32_t *my = h[(threadIdx.x >> 5) & 3];
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
    uint32_t key[kSortRounds];
#pragma unroll
    for (int r = 0; r < kSortRounds; r++) {
        const int64_t j = base + r * kSortThreads + threadIdx.x;
        key[r] = j < a.n ? __ldg(&a.key_in[a.reverse ? a.n - 1 - j : j]) : 0u;
    }
#pragma unroll
    for (int r = 0; r < kSortRounds; r++) {
        const int64_t j = base + r * kSortThreads + threadIdx.x;
        if (j < a.n) atomicAdd(&my[(key[r] >> a.shift) & a.mask], 1u);
    }
    __syncthreads();
    if (threadIdx.x <= a.mask)
        hist[(int64_t)threadIdx.x * a.ntiles + blockIdx.x] =
            h[0][threadIdx.x] + h[1][threadIdx.x] + h[2][threadIdx.x] + h[3][threadIdx.x];
}

template <int kPay>
__global__ void __launch_bounds__(kSortThreads, 2) k_radix_scatter(SortPass a) {
    __shared__ uint16_t wcnt[kSortWarps][kRadix];  // at most kSortTile
    __shared__ uint32_t skey[kSortTile], sbuf[kSortTile];
    __shared__ uint32_t dstart[kRadix], gbase[kRadix], wtot[kRadix / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
    const uint32_t cnt = (uint32_t)min((int64_t)kSortTile, a.n - base);
    for (int i = threadIdx.x; i < kSortWarps * kRadix; i += kSortThreads) wcnt[i / kRadix][i % kRadix] = 0;
    // a warp's elements are consecutive: its rounds keep the input's order
    uint32_t key[kSortRounds], pay[kPay > 0 ? kPay : 1][kSortRounds], lpos[kSortRounds];
#pragma unroll
    for (int r = 0; r < kSortRounds; r++) {
        const int64_t j = base + wid * (32 * kSortRounds) + r * 32 + lane;
        const int64_t i = a.reverse ? a.n - 1 - j : j;
        const bool in = j < a.n;
        key[r] = in ? __ldg(&a.key_in[i]) : 0u;
#pragma unroll
        for (int p = 0; p < kPay; p++)
            pay[p][r] = p == kPay - 1 && a.iota ? (uint32_t)j : in ? __ldg(&a.pay_in[p][i]) : 0u;
    }
    __syncthreads();
    // rank within the warp's elements of the same digit
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < kSortRounds; r++) {
        const bool in = (uint32_t)(wid * (32 * kSortRounds) + r * 32 + lane) < cnt;
        const uint32_t d = (key[r] >> a.shift) & a.mask;
        const unsigned peers = __match_any_sync(0xffffffffu, in ? d : 0x100u);
        const unsigned before = __popc(peers & lt);
        lpos[r] = in ? wcnt[wid][d] + before : 0u;
        __syncwarp();
        if (in && before == 0) wcnt[wid][d] = (uint16_t)(wcnt[wid][d] + __popc(peers));
        __syncwarp();
    }
    __syncthreads();
    // where each digit, and each warp's part of it, starts in the tile
    uint32_t tot = 0, incl = 0;
    if (threadIdx.x < kRadix) {
#pragma unroll
        for (int w = 0; w < kSortWarps; w++) {
            const uint32_t c = wcnt[w][threadIdx.x];
            wcnt[w][threadIdx.x] = (uint16_t)tot;
            tot += c;
        }
        incl = warp_incl_scan(tot);
        if (lane == 31) wtot[wid] = incl;
    }
    __syncthreads();
    if (threadIdx.x < kRadix) {
        uint32_t s = incl - tot;
        for (int w = 0; w < wid; w++) s += wtot[w];
        dstart[threadIdx.x] = s;
        gbase[threadIdx.x] =
            threadIdx.x <= a.mask ? a.offsets[(int64_t)threadIdx.x * a.ntiles + blockIdx.x] - s : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortRounds; r++) {
        const bool in = (uint32_t)(wid * (32 * kSortRounds) + r * 32 + lane) < cnt;
        const uint32_t d = (key[r] >> a.shift) & a.mask;
        lpos[r] = in ? lpos[r] + dstart[d] + wcnt[wid][d] : kSortTile;
        if (in) skey[lpos[r]] = key[r];
    }
    __syncthreads();
    uint32_t gpos[kSortRounds];
#pragma unroll
    for (int r = 0; r < kSortRounds; r++) {
        const uint32_t i = r * kSortThreads + threadIdx.x;
        gpos[r] = 0;
        if (i < cnt) {
            const uint32_t k = skey[i];
            gpos[r] = gbase[(k >> a.shift) & a.mask] + i;
            if (a.key_out) a.key_out[gpos[r]] = k;
        }
    }
#pragma unroll
    for (int p = 0; p < kPay; p++) {
        uint32_t *buf = p & 1 ? skey : sbuf;  // skey is free after the first payload's barrier
#pragma unroll
        for (int r = 0; r < kSortRounds; r++)
            if (lpos[r] < kSortTile) buf[lpos[r]] = pay[p][r];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSortRounds; r++) {
            const uint32_t i = r * kSortThreads + threadIdx.x;
            if (i < cnt) {
                if (p == kPay - 1 && a.slot_out) a.slot_out[buf[i]] = gpos[r];
                else a.pay_out[p][gpos[r]] = buf[i];
            }
        }
    }
}

// First position of each key in the sorted sequence: out[v] for v in [0, V],
// out[V] = n.  From the boundaries between different keys; a long gap (keys
// without elements) is filled by the whole warp.
__global__ void k_key_offsets(const uint32_t *key, int64_t n, uint32_t V, uint32_t *out) {
    const int lane = threadIdx.x & 31;
    for (int64_t b = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~31ll; b <= n;
         b += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = b + lane;
        uint32_t from = 1, to = 0;  // keys (from - 1, to] start at i
        if (i <= n) {
            from = i > 0 ? key[i - 1] + 1u : 0u;
            to = i < n ? key[i] : V;
        }
        const bool any = i <= n && from <= to;
        const bool wide = any && to - from >= 64u;
        if (any && !wide)
            for (uint32_t v = from; v <= to; v++) out[v] = (uint32_t)i;
        unsigned m = __ballot_sync(0xffffffffu, wide);
        while (m) {
            const int l = __ffs(m) - 1;
            m &= m - 1;
            const uint32_t f = __shfl_sync(0xffffffffu, from, l), t = __shfl_sync(0xffffffffu, to, l);
            for (uint64_t v = (uint64_t)f + lane; v <= t; v += 32) out[v] = (uint32_t)(b + l);
        }
    }
}

}  // namespace

void scan_exclusive_u32(Context &ctx, const uint32_t *in, uint32_t *out, int64_t n,
                        uint32_t *total_dev, cudaStream_t s) {
    if (n <= 0) {
        if (total_dev) MB_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(uint32_t), s));
        return;
    }
    int64_t nb = (n + kScanTile - 1) / kScanTile;
    if (nb == 1) {
        k_scan_apply<<<1, kScanThreads, 0, s>>>(in, out, n, nullptr, total_dev);
        MB_CHECK_LAUNCH();
        return;
    }
    // partial sums of the tiles live in their own allocation (recursion-safe)
    DevBuf partial;
    partial.reserve(sizeof(uint32_t) * (size_t)nb);
    try {
        k_scan_reduce<<<(unsigned)nb, kScanThreads, 0, s>>>(in, n, partial.as<uint32_t>());
        MB_CHECK_LAUNCH();
        scan_exclusive_u32(ctx, partial.as<uint32_t>(), partial.as<uint32_t>(), nb, nullptr, s);
        k_scan_apply<<<(unsigned)nb, kScanThreads, 0, s>>>(in, out, n, partial.as<uint32_t>(),
                                                           total_dev);
        MB_CHECK_LAUNCH();
        MB_CUDA(cudaStreamSynchronize(s));  // partial is freed on return
    } catch (...) {
        partial.release();
        throw;
    }
    partial.release();
}

namespace {

void sort_pass(Context &ctx, SortPass &a, int npay, DevBuf &hist, cudaStream_t s) {
    const unsigned tiles = (unsigned)a.ntiles;
    k_radix_hist<<<tiles, kSortThreads, 0, s>>>(a, hist.as<uint32_t>());
    MB_CHECK_LAUNCH();
    scan_exclusive_u32(ctx, hist.as<uint32_t>(), hist.as<uint32_t>(), ((int64_t)a.mask + 1) * a.ntiles, nullptr, s);
    a.offsets = hist.as<uint32_t>();
    switch (npay) {
        case 0: k_radix_scatter<0><<<tiles, kSortThreads, 0, s>>>(a); break;
        case 1: k_radix_scatter<1><<<tiles, kSortThreads, 0, s>>>(a); break;
        case 2: k_radix_scatter<2><<<tiles, kSortThreads, 0, s>>>(a); break;
        default: k_radix_scatter<3><<<tiles, kSortThreads, 0, s>>>(a); break;
    }
    MB_CHECK_LAUNCH();
}

}  // namespace

void radix_sort(Context &ctx, const SortJob &job, int64_t n, int bits, cudaStream_t s) {
    if (n <= 0) return;
    if (job.npay < 0 || job.npay > kMaxPay) fail(MB_ERR_INVALID, "radix sort: payload count");
    const int passes = bits > 0 ? (bits + 7) / 8 : 1;
    const int digit = (std::max(bits, 0) + passes - 1) / passes;  // even digits: longer runs in each pass
    DevBuf hist, tmp[1 + kMaxPay], last, key_end;
    auto drop = [&] {
        hist.release();
        last.release();
        key_end.release();
        for (DevBuf &b : tmp) b.release();
    };
    try {
        SortPass a{};
        a.n = n;
        a.ntiles = (n + kSortTile - 1) / kSortTile;
        hist.reserve(sizeof(uint32_t) * (size_t)(kRadix * a.ntiles));
        const size_t bytes = sizeof(uint32_t) * (size_t)n;
        // pass k of p writes the output where p - 1 - k is even, else the
        // temporaries (the inputs are never written)
        if (passes > 1)
            for (int p = 0; p <= job.npay; p++) tmp[p].reserve(bytes);
        if (passes > 2 && job.slot_out) last.reserve(bytes);
        uint32_t *key_out = job.key_out;
        if (!key_out && passes > 2) key_out = (uint32_t *)key_end.reserve(bytes);
        for (int k = 0; k < passes; k++) {
            const bool fin = k == passes - 1, to_out = (passes - 1 - k) % 2 == 0;
            a.shift = k * digit;
            a.mask = (1u << std::min(digit, std::max(bits - a.shift, 0))) - 1u;
            a.key_out = fin ? job.key_out : to_out ? key_out : tmp[0].as<uint32_t>();
            a.slot_out = fin ? job.slot_out : nullptr;
            a.reverse = k == 0 && job.reverse;
            a.iota = k == 0 && job.iota;
            if (k == 0) {
                a.key_in = job.key_in;
                for (int p = 0; p < job.npay; p++) a.pay_in[p] = job.pay_in[p];
            }
            for (int p = 0; p < job.npay; p++)
                a.pay_out[p] = !to_out ? tmp[1 + p].as<uint32_t>()
                               : job.slot_out && p == job.npay - 1 ? last.as<uint32_t>() : job.pay_out[p];
            sort_pass(ctx, a, job.npay, hist, s);
            a.key_in = a.key_out;
            for (int p = 0; p < job.npay; p++) a.pay_in[p] = a.pay_out[p];
        }
        MB_CUDA(cudaStreamSynchronize(s));
    } catch (...) {
        drop();
        throw;
    }
    drop();
}

void radix_sort_pairs(Context &ctx, uint32_t *keys, uint32_t *vals, int64_t n, int bits,
                      cudaStream_t s) {
    if (n <= 1 || bits <= 0) return;
    const int passes = (bits + 7) / 8, digit = (bits + passes - 1) / passes;
    DevBuf kb, vb, hist;
    try {
        SortPass a{};
        a.n = n;
        a.ntiles = (n + kSortTile - 1) / kSortTile;
        kb.reserve(sizeof(uint32_t) * (size_t)n);
        vb.reserve(sizeof(uint32_t) * (size_t)n);
        hist.reserve(sizeof(uint32_t) * (size_t)(kRadix * a.ntiles));
        uint32_t *ki = keys, *vi = vals, *ko = kb.as<uint32_t>(), *vo = vb.as<uint32_t>();
        for (int k = 0; k < passes; k++) {
            a.shift = k * digit;
            a.mask = (1u << std::min(digit, bits - a.shift)) - 1u;
            a.key_in = ki;
            a.pay_in[0] = vi;
            a.key_out = ko;
            a.pay_out[0] = vo;
            sort_pass(ctx, a, 1, hist, s);
            std::swap(ki, ko);
            std::swap(vi, vo);
        }
        if (ki != keys) {
            MB_CUDA(cudaMemcpyAsync(keys, ki, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s));
            MB_CUDA(cudaMemcpyAsync(vals, vi, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s));
        }
        MB_CUDA(cudaStreamSynchronize(s));
    } catch (...) {
        kb.release(); vb.release(); hist.release();
        throw;
    }
    kb.release(); vb.release(); hist.release();
}

void key_offsets(Context &ctx, const uint32_t *key, int64_t n, int32_t V, uint32_t *out, cudaStream_t s) {
    k_key_offsets<<<grid_for(n + 1, 256, ctx.num_sms * 16), 256, 0, s>>>(key, n, (uint32_t)V, out);
    MB_CHECK_LAUNCH();
}

}  // namespace mb
