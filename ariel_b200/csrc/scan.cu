// scan.cu -- exclusive prefix sum of uint32 counts (cell histograms, FLUID-cell compaction).
//
// Passes over tiles of 4096 values: per-tile sums, with many tiles one block scanning the tile
// sums, per-tile scan plus offset.  Integer arithmetic, so the result does not depend on the order
// in which blocks run.
#include <atomic>

#include "state.cuh"

namespace ariel {

namespace {
constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kTile = kScanThreads * kScanItems;
// Tiles (4 M values) up to which every block adds the earlier tiles' sums itself, a launch less: a
// step's sort 41.0 -> 39.3 us at 64 tiles, 177.5 -> 176.2 at 512, 332 -> 328 at 1,000; above the line
// 564 -> 560 at 1,728 and 1,310 -> 1,304 at 4,096.  The line does not lie where that stops to pay; it bounds
// the work, which grows with the square of the tiles.
constexpr long long kOwnPrefix = 1024;

template <class T>
__device__ __forceinline__ T warp_incl_scan(T v) {
    const unsigned lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (unsigned)o) v += t;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread; returns the exclusive prefix and the
// block total through *total.
template <class T>
__device__ __forceinline__ T block_excl_scan(T v, T* total) {
    __shared__ T warp_sums[kScanThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    T inc = warp_incl_scan(v);
    if (lane == 31) warp_sums[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        constexpr int kWarps = kScanThreads / 32;
        T w = lane < kWarps ? warp_sums[lane] : 0;
        __syncwarp();
        T wi = warp_incl_scan(w);
        if (lane < kWarps) warp_sums[lane] = wi - w;
        if (lane == kWarps - 1) *total = wi;
    }
    __syncthreads();
    T r = warp_sums[wid] + inc - v;
    __syncthreads();
    return r;
}

// What is summed for one count: the count itself, or with it, in the upper half of 64 bits, the
// pairs that hold it (the sort's scan: both prefixes in one pass over the counts).
__device__ __forceinline__ void widen(uint32_t v, uint32_t& t) { t = v; }
__device__ __forceinline__ void widen(uint32_t v, unsigned long long& t) {
    t = (unsigned long long)((v + 1u) >> 1) << 32 | v;
}
__device__ __forceinline__ void put(uint32_t* out, uint32_t*, long long i, uint32_t t) { out[i] = t; }
__device__ __forceinline__ void put(uint32_t* out, uint32_t* pairs, long long i, unsigned long long t) {
    out[i] = (uint32_t)t;
    pairs[i] = (uint32_t)(t >> 32);
}

template <class T>
__global__ void k_tile_sums(const uint32_t* in, long long n, T* sums) {
    kernel_begin();
    long long base = (long long)blockIdx.x * kTile;
    T acc = 0;
#pragma unroll
    for (int it = 0; it < kScanItems; ++it) {
        long long i = base + (long long)it * kScanThreads + threadIdx.x;
        T t = 0;
        if (i < n) widen(in[i], t);
        acc += t;
    }
    __shared__ T tot;
    block_excl_scan(acc, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

template <class T>
__global__ void k_scan_sums(T* sums, long long nt) {
    kernel_begin();
    __shared__ T carry_s;
    if (threadIdx.x == 0) carry_s = 0;
    __syncthreads();
    for (long long b = 0; b < nt; b += kScanThreads) {
        long long i = b + threadIdx.x;
        T v = i < nt ? sums[i] : 0;
        __shared__ T tot;
        T ex = block_excl_scan(v, &tot);
        T carry = carry_s;
        if (i < nt) sums[i] = carry + ex;
        __syncthreads();
        if (threadIdx.x == 0) carry_s = carry + tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[nt] = carry_s;
}

// SUMMED: `sums` holds the exclusive prefixes of the tiles (k_scan_sums); else the tiles' own sums,
// and each block adds those before it itself, which spares a launch while the tiles are few.
template <class T, bool SUMMED>
__global__ void k_tile_scan(const uint32_t* in, uint32_t* out, uint32_t* pairs,
                            long long n, const T* sums, long long nt) {
    kernel_begin();
    long long base = (long long)blockIdx.x * kTile + (long long)threadIdx.x * kScanItems;
    T vals[kScanItems];
    T acc = 0;
#pragma unroll
    for (int it = 0; it < kScanItems; ++it) {
        long long i = base + it;
        vals[it] = 0;
        if (i < n) widen(in[i], vals[it]);
        acc += vals[it];
    }
    __shared__ T tot, before_s;
    T before;
    if (SUMMED) {
        before = sums[blockIdx.x];
    } else {
        T b = 0;
        for (long long i = threadIdx.x; i < (long long)blockIdx.x; i += kScanThreads) b += sums[i];
        block_excl_scan(b, &before_s);
        before = before_s;
    }
    T ex = block_excl_scan(acc, &tot) + before;
#pragma unroll
    for (int it = 0; it < kScanItems; ++it) {
        long long i = base + it;
        if (i < n) put(out, pairs, i, ex);
        ex += vals[it];
    }
    if ((long long)blockIdx.x == nt - 1 && threadIdx.x == 0) put(out, pairs, n, before + tot);
}

template <class T>
cudaError_t scan(const uint32_t* in, uint32_t* out, uint32_t* pairs, long long n, void* tmp, cudaStream_t st) {
    long long nt = (n + kTile - 1) / kTile;
    T* sums = (T*)tmp;
    if (nt == 0) {
        cudaMemsetAsync(out, 0, sizeof(uint32_t), st);
        if (pairs) cudaMemsetAsync(pairs, 0, sizeof(uint32_t), st);
        return cudaGetLastError();
    }
    launch_k(k_tile_sums<T>, nt, kScanThreads, st, in, n, sums);
    if (nt <= kOwnPrefix) {
        launch_k(k_tile_scan<T, false>, nt, kScanThreads, st, in, out, pairs, n, sums, nt);
        count_launch(2);
    } else {
        launch_k(k_scan_sums<T>, 1, kScanThreads, st, sums, nt);
        launch_k(k_tile_scan<T, true>, nt, kScanThreads, st, in, out, pairs, n, sums, nt);
        count_launch(3);
    }
    return cudaGetLastError();
}

std::atomic<long long> g_launches{0};
}  // namespace

void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long long launch_count() { return g_launches.load(std::memory_order_relaxed); }

size_t scan_tmp_bytes(long long n) { return sizeof(uint64_t) * (size_t)((n + kTile - 1) / kTile + 2); }

cudaError_t launch_scan_u32(const uint32_t* in, uint32_t* out, long long n, void* tmp, cudaStream_t st) {
    return scan<uint32_t>(in, out, nullptr, n, tmp, st);
}

cudaError_t launch_scan_pairs(const uint32_t* in, uint32_t* out, uint32_t* pairs, long long n, void* tmp,
                              cudaStream_t st) {
    return scan<unsigned long long>(in, out, pairs, n, tmp, st);
}

}  // namespace ariel
