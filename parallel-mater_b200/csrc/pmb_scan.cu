// SPDX-License-Identifier: MIT
// Device-wide exclusive prefix sums whose length is read from device memory,
// so compaction stages (candidate pairs, contacts) need no host round trip.
//
// A tick makes nine of them, most over a few thousand elements, where the
// launches are the cost (about 2 us each, against 0.1 us of memory time for
// 32,768 words). So a scan whose capacity fits one block's few rounds is one
// launch (k_scan_block); a longer one is two: per-tile totals, then every
// tile's block adds up the totals before its own (at most a few thousand
// words, read by 256 threads at once) instead of waiting for a pass over them.
#include "pmb_world.cuh"

namespace pmb {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr uint32_t kScanTile = kScanThreads * kScanItems;
constexpr int kScanBlockThreads = 1024;
// Longest capacity scanned by one block: four rounds of 8,192 elements.
constexpr uint32_t kScanBlockMost = 4u * kScanBlockThreads * kScanItems;

template <class T, int kThreads> __device__ T block_exclusive_scan(T v, T* total) {
    __shared__ T warp_sums[kThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    T inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) warp_sums[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        T s = lane < kThreads / 32 ? warp_sums[lane] : T(0);
        T si = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(0xffffffffu, si, o);
            if (lane >= o) si += y;
        }
        if (lane < kThreads / 32) warp_sums[lane] = si - s;
        if (lane == kThreads / 32 - 1 && total) *total = si;
    }
    __syncthreads();
    T r = inc - v + warp_sums[wid];
    __syncthreads();
    return r;
}

// This thread's kScanItems elements from `first` on (zeros past `count`).
template <class T> __device__ __forceinline__ T load_items(const T* in, uint32_t first, uint32_t count, T* vals) {
    T s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        vals[k] = first + k < count ? in[first + k] : T(0);
        s += vals[k];
    }
    return s;
}
template <class T>
__device__ __forceinline__ void store_items(T* out, uint32_t first, uint32_t count, const T* vals, T off) {
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (first + k < count) out[first + k] = off;
        off += vals[k];
    }
}

// One scan of a launch (blockIdx.y picks it; scans of one length can share
// their launches).
template <class T> struct ScanJob {
    const T* in;
    T* out;
    T* total;  // may be null
    T* tiles;  // tile totals (long scans)
};
template <class T> struct ScanJobs {
    ScanJob<T> job[2];
};

template <class T>
__global__ void __launch_bounds__(kScanBlockThreads)
    k_scan_block(ScanJobs<T> jobs, const uint32_t* count_ptr, uint32_t capacity, uint32_t total_cap) {
    tick_begin();
    const T* in = jobs.job[blockIdx.y].in;
    T* out = jobs.job[blockIdx.y].out;
    T* total = jobs.job[blockIdx.y].total;
    const uint32_t count = count_ptr ? min(*count_ptr, capacity) : capacity;
    __shared__ T chunk;
    T carry = 0;
    for (uint32_t base = 0; base < count; base += kScanBlockThreads * kScanItems) {
        const uint32_t first = base + threadIdx.x * kScanItems;
        T vals[kScanItems];
        const T s = load_items(in, first, count, vals);
        const T off = block_exclusive_scan<T, kScanBlockThreads>(s, &chunk) + carry;
        store_items(out, first, count, vals, off);
        carry += chunk;
    }
    if (threadIdx.x == 0) {
        out[count] = carry;
        if (total) *total = carry < T(total_cap) ? carry : T(total_cap);
    }
}

template <class T>
__global__ void k_tile_sums(ScanJobs<T> jobs, const uint32_t* count_ptr, uint32_t capacity) {
    tick_begin();
    const T* in = jobs.job[blockIdx.y].in;
    T* tile_sums = jobs.job[blockIdx.y].tiles;
    const uint32_t count = count_ptr ? min(*count_ptr, capacity) : capacity;
    const uint32_t base = blockIdx.x * kScanTile;
    if (base >= count) return;  // totals past the end are never read
    T vals[kScanItems];
    const T s = load_items(in, base + threadIdx.x * kScanItems, count, vals);
    __shared__ T total;
    block_exclusive_scan<T, kScanThreads>(s, &total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

template <class T>
__global__ void k_scan_apply(ScanJobs<T> jobs, const uint32_t* count_ptr, uint32_t capacity, uint32_t total_cap) {
    tick_begin();
    const T* in = jobs.job[blockIdx.y].in;
    T* out = jobs.job[blockIdx.y].out;
    T* total = jobs.job[blockIdx.y].total;
    const T* tile_sums = jobs.job[blockIdx.y].tiles;
    const uint32_t count = count_ptr ? min(*count_ptr, capacity) : capacity;
    const uint32_t base = blockIdx.x * kScanTile;
    if (base >= count && !(blockIdx.x == 0 && count == 0)) return;
    T before = 0;
    for (uint32_t k = threadIdx.x; k < blockIdx.x; k += kScanThreads) before += tile_sums[k];
    __shared__ T start, tile;
    block_exclusive_scan<T, kScanThreads>(before, &start);
    const T carry = start;
    const uint32_t first = base + threadIdx.x * kScanItems;
    T vals[kScanItems];
    const T s = load_items(in, first, count, vals);
    const T off = block_exclusive_scan<T, kScanThreads>(s, &tile) + carry;
    store_items(out, first, count, vals, off);
    if (threadIdx.x == 0 && count - base <= kScanTile) {  // the last tile
        const T all = carry + tile;
        out[count] = all;
        if (total) *total = all < T(total_cap) ? all : T(total_cap);
    }
}

// out holds capacity + 1 entries; out[count] receives the total and, when
// `total` is non-null, *total the total or `total_cap` if that is less.
template <class T>
static void scan_impl(const ScanJobs<T>& jobs, uint32_t njobs, const uint32_t* count_ptr, uint32_t capacity,
                      uint32_t total_cap, cudaStream_t s) {
    if (capacity <= kScanBlockMost) {
        launch(k_scan_block<T>, dim3(1, njobs), kScanBlockThreads, s, jobs, count_ptr, capacity, total_cap);
        return;
    }
    const uint32_t tiles = (capacity + kScanTile - 1) / kScanTile;
    launch(k_tile_sums<T>, dim3(tiles, njobs), kScanThreads, s, jobs, count_ptr, capacity);
    launch(k_scan_apply<T>, dim3(tiles, njobs), kScanThreads, s, jobs, count_ptr, capacity, total_cap);
}

void scan_u32(const uint32_t* in, uint32_t* out, const uint32_t* count_ptr, uint32_t capacity, uint32_t* total,
              uint32_t total_cap, uint32_t* tmp, cudaStream_t s) {
    scan_impl<uint32_t>({{{in, out, total, tmp}, {}}}, 1, count_ptr, capacity, total_cap, s);
}

void scan_u32_pair(const uint32_t* in0, uint32_t* out0, uint32_t* total0, const uint32_t* in1, uint32_t* out1,
                   uint32_t* total1, const uint32_t* count_ptr, uint32_t capacity, uint32_t* tmp, cudaStream_t s) {
    const uint32_t tiles = (capacity + kScanTile - 1) / kScanTile;
    scan_impl<uint32_t>({{{in0, out0, total0, tmp}, {in1, out1, total1, tmp + tiles}}}, 2, count_ptr, capacity,
                        0xffffffffu, s);
}

void scan_u64(const uint64_t* in, uint64_t* out, const uint32_t* count_ptr, uint32_t capacity, uint64_t* tmp,
              cudaStream_t s) {
    scan_impl<uint64_t>({{{in, out, nullptr, tmp}, {}}}, 1, count_ptr, capacity, 0u, s);
}

}  // namespace pmb
