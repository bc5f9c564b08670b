// SPDX-License-Identifier: MIT
// Mesh BVH build on the GPU: the same tree as the host builder the reference
// runs at mesh upload (src/simulation/runtime_deformables.cu.inc:136-210,
// restated in pmb_mesh.cpp) -- median split, split axis = longest extent of
// the node's triangle bounds, triangles ordered by the centroid coordinate
// on that axis (ties by triangle index), leaves of at most four triangles,
// nodes in pre-order -- for meshes too large to prepare on the host.
//
// A node's triangles in the order of any axis are a subsequence of all
// triangles in that order, so the triangles are sorted once per axis (a
// stable 8-bit LSD radix sort, three axes at a time) and every split only
// partitions the three lists, keeping their order: O(n) a level, no sort.
// The shape of the tree depends on the triangle count alone -- at every
// level the nodes have one of two sizes -- so a node's range and pre-order
// index follow from its path, and nothing is laid out on the host.
//
// Nodes of more than kLocal triangles go level by level across the grid;
// a block then builds each remaining subtree in shared memory. What bounds
// it: launches (4 radix passes of 4, then six a top level, 2-4 us each) and
// the latency of the shared-memory levels (27 us); the memory time of 200,000
// triangles is a few microseconds. Sorting every node of every level anew, with one
// thread per 256-key tile, took 56 ms for 200,000 triangles.
#include <algorithm>
#include <mutex>

#include "../../include/pmb200_core.h"
#include "pmb_world.cuh"

namespace pmb {
namespace {

constexpr uint32_t kLeaf = 4;        // triangles of a leaf at most
constexpr uint32_t kLocal = 512;     // largest subtree built by one block
constexpr uint32_t kLocalThreads = 256;
constexpr uint32_t kRadixTile = 2048;  // keys per block of a radix pass
constexpr uint32_t kRadixThreads = 256;
constexpr uint32_t kRadixWarps = kRadixThreads / 32;
constexpr uint32_t kRadixRounds = kRadixTile / kRadixThreads;

__device__ __forceinline__ V3 vertex(const float* v, uint32_t k) {
    return {v[3 * size_t(k)], v[3 * size_t(k) + 1], v[3 * size_t(k) + 2]};
}

// An order-preserving unsigned image of a float (-0 taken as +0, so the two
// compare equal as the host's `<` does).
__device__ __forceinline__ uint32_t float_key(float f) {
    uint32_t u = f == 0.0f ? 0u : __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// The same with -0 below +0 (as fminf and fmaxf order them), and its inverse.
__device__ __forceinline__ uint32_t bound_key(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_bound(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Nodes of a subtree over c triangles. Its levels hold x nodes of f triangles
// and y of f + 1.
__host__ __device__ inline uint32_t node_total(uint32_t c) {
    uint32_t total = 0, x = 1, y = 0, f = c;
    for (;;) {
        total += x + y;
        if (f < kLeaf) return total;
        if (f == kLeaf) return total + 2u * y;
        if (f & 1u) {  // f -> (h, h + 1), f + 1 -> (h + 1, h + 1)
            y = x + 2u * y;
        } else {  // f -> (h, h), f + 1 -> (h, h + 1)
            x = 2u * x + y;
        }
        f >>= 1;
    }
}

struct Seg {  // a node: its triangles [b, e) and pre-order index
    uint32_t b, e, node;
};
__device__ __forceinline__ Seg child(const Seg& s, bool right) {
    const uint32_t mid = s.b + (s.e - s.b) / 2;
    return right ? Seg{mid, s.e, s.node + 1u + node_total(mid - s.b)} : Seg{s.b, mid, s.node + 1u};
}
// The node of the top `level` that holds position p of n (every node above
// it splits), and its slot among the level's nodes.
__device__ __forceinline__ Seg seg_at(uint32_t n, uint32_t level, uint32_t p, uint32_t& slot) {
    Seg s{0u, n, 0u};
    slot = 0;
    for (uint32_t l = 0; l < level; ++l) {
        const bool right = p >= s.b + (s.e - s.b) / 2;
        s = child(s, right);
        slot = 2u * slot + (right ? 1u : 0u);
    }
    return s;
}
__device__ __forceinline__ Seg seg_of_slot(uint32_t n, uint32_t level, uint32_t slot) {
    Seg s{0u, n, 0u};
    for (uint32_t l = level; l-- > 0;) s = child(s, (slot >> l) & 1u);
    return s;
}

__device__ __forceinline__ uint32_t split_axis(const float lo[3], const float hi[3]) {
    const float ex = hi[0] - lo[0], ey = hi[1] - lo[1], ez = hi[2] - lo[2];
    return ex >= ey && ex >= ez ? 0u : (ey >= ez ? 1u : 2u);
}
__device__ __forceinline__ void write_node(float* nodes, const Seg& s, const float lo[3], const float hi[3]) {
    float* o = nodes + 10 * size_t(s.node);
    const uint32_t c = s.e - s.b;
    const bool leaf = c <= kLeaf;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        o[k] = lo[k];
        o[3 + k] = hi[k];
    }
    o[6] = __uint_as_float(leaf ? s.b : 0u);
    o[7] = __uint_as_float(leaf ? c : 0u);
    o[8] = __uint_as_float(leaf ? 0u : s.node + 1u);
    o[9] = __uint_as_float(leaf ? 0u : s.node + 1u + node_total(c / 2));
}

// Any index at or past the vertex count sets *bad (checked before use).
__global__ void k_bvh_check(const uint32_t* idx, uint32_t count, uint32_t vertices, uint32_t* bad) {
    for (uint32_t i = grid_stride_begin(); i < count; i += grid_stride())
        if (idx[i] >= vertices) atomicOr(bad, 1u);
}

// Per triangle: its bounds, and its centroid's key on every axis.
__global__ void k_bvh_triangles(const float* v, const uint32_t* idx, uint32_t n, float4* lo, float4* hi,
                                uint32_t* key, uint32_t* val) {
    for (uint32_t t = grid_stride_begin(); t < n; t += grid_stride()) {
        const V3 a = vertex(v, idx[3 * size_t(t)]), b = vertex(v, idx[3 * size_t(t) + 1]),
                 c = vertex(v, idx[3 * size_t(t) + 2]);
        const V3 top{kFltMax, kFltMax, kFltMax}, low{-kFltMax, -kFltMax, -kFltMax};
        lo[t] = f4(vmin(vmin(vmin(top, a), b), c));
        hi[t] = f4(vmax(vmax(vmax(low, a), b), c));
        const V3 m = mul(add(add(a, b), c), 1.0f / 3.0f);
#pragma unroll
        for (unsigned axis = 0; axis < 3; ++axis) {
            key[axis * size_t(n) + t] = float_key(comp(m, axis));
            val[axis * size_t(n) + t] = t;
        }
    }
}

// Radix pass over the 8-bit digit at `shift`, blockIdx.y the axis: per-tile
// digit counts ordered (axis, digit, tile), so their exclusive scan gives
// every tile's first slot per digit in its axis's list; then a stable
// scatter. A warp takes 256 consecutive keys, 32 a round: a key's rank is
// the warp's count of its digit so far plus the equal digits in lower lanes.
__global__ void __launch_bounds__(kRadixThreads)
    k_bvh_hist(const uint32_t* key, uint32_t shift, uint32_t n, uint32_t tiles, uint32_t* hist) {
    __shared__ uint32_t count[256];
    count[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t* k = key + blockIdx.y * size_t(n);
    const uint32_t end = min(n, (blockIdx.x + 1) * kRadixTile);
    for (uint32_t i = blockIdx.x * kRadixTile + threadIdx.x; i < end; i += kRadixThreads)
        atomicAdd(&count[(k[i] >> shift) & 255u], 1u);
    __syncthreads();
    hist[(size_t(blockIdx.y) * 256 + threadIdx.x) * tiles + blockIdx.x] = count[threadIdx.x];
}
__global__ void __launch_bounds__(kRadixThreads)
    k_bvh_scatter(const uint32_t* key, const uint32_t* val, uint32_t shift, uint32_t n, uint32_t tiles,
                  const uint32_t* offs, uint32_t* key2, uint32_t* val2) {
    __shared__ uint32_t count[kRadixWarps][256];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t w = 0; w < kRadixWarps; ++w) count[w][threadIdx.x] = 0;
    __syncthreads();
    const uint32_t base = blockIdx.x * kRadixTile + warp * (32u * kRadixRounds);
    const uint32_t* k = key + blockIdx.y * size_t(n);
    const uint32_t* v = val + blockIdx.y * size_t(n);
    uint32_t kk[kRadixRounds], vv[kRadixRounds], rank[kRadixRounds];
#pragma unroll
    for (uint32_t r = 0; r < kRadixRounds; ++r) {
        const uint32_t i = base + 32u * r + lane;
        kk[r] = i < n ? k[i] : 0u;
        vv[r] = i < n ? v[i] : 0u;
    }
#pragma unroll
    for (uint32_t r = 0; r < kRadixRounds; ++r) {
        const bool in = base + 32u * r + lane < n;
        const uint32_t digit = in ? (kk[r] >> shift) & 255u : 256u;
        const uint32_t same = __match_any_sync(0xffffffffu, digit);
        const uint32_t before = __popc(same & ((1u << lane) - 1u));
        const uint32_t so_far = in ? count[warp][digit] : 0u;
        rank[r] = so_far + before;
        __syncwarp();
        if (in && before == 0) count[warp][digit] = so_far + __popc(same);
        __syncwarp();
    }
    __syncthreads();
    {
        // Each digit's warps in order, from the tile's first slot.
        uint32_t run = offs[(size_t(blockIdx.y) * 256 + threadIdx.x) * tiles + blockIdx.x];
        for (uint32_t w = 0; w < kRadixWarps; ++w) {
            const uint32_t c = count[w][threadIdx.x];
            count[w][threadIdx.x] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < kRadixRounds; ++r)
        if (base + 32u * r + lane < n) {
            const uint32_t o = count[warp][(kk[r] >> shift) & 255u] + rank[r];
            key2[o] = kk[r];
            val2[o] = vv[r];
        }
}

// ---- top levels (every node of the level splits)
constexpr uint32_t kBoundsPerWarp = 256;  // positions a warp reduces before its atomics

// Bounds of the level's nodes, as keys: acc[slot] = lo x, y, z, hi x, y, z.
__global__ void k_bvh_top_bounds(uint32_t n, uint32_t level, const uint32_t* list, const float4* lo, const float4* hi,
                                 uint32_t* acc) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t first = warp * kBoundsPerWarp;
    uint32_t held = kInvalid;
    uint32_t k[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    auto flush = [&] {  // by the whole warp
        uint32_t* a = acc + 6 * size_t(held);
        if (__match_any_sync(0xffffffffu, held) == 0xffffffffu) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                k[c] = __reduce_min_sync(0xffffffffu, k[c]);
                k[3 + c] = __reduce_max_sync(0xffffffffu, k[3 + c]);
            }
            if (lane != 0) return;
        }
        if (held == kInvalid) return;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            atomicMin(a + c, k[c]);
            atomicMax(a + 3 + c, k[3 + c]);
        }
    };
    for (uint32_t r = 0; r < kBoundsPerWarp; r += 32u) {
        const uint32_t p = first + r + lane;
        uint32_t slot = kInvalid;
        if (p < n) seg_at(n, level, p, slot);
        // A new node anywhere in the warp: hand over what the warp holds.
        if (__any_sync(0xffffffffu, slot != held)) {
            if (r != 0) flush();
            __syncwarp();
            held = slot;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                k[c] = 0xffffffffu;
                k[3 + c] = 0u;
            }
        }
        if (p < n) {
            const uint32_t t = list[p];
            const float4 l = lo[t], h = hi[t];
            k[0] = min(k[0], bound_key(l.x));
            k[1] = min(k[1], bound_key(l.y));
            k[2] = min(k[2], bound_key(l.z));
            k[3] = max(k[3], bound_key(h.x));
            k[4] = max(k[4], bound_key(h.y));
            k[5] = max(k[5], bound_key(h.z));
        }
    }
    flush();
}

// The level's node records, and every triangle's side of its node's split.
__global__ void k_bvh_top_sides(uint32_t n, uint32_t level, const uint32_t* list, const uint32_t* acc, float* nodes,
                                uint8_t* side) {
    for (uint32_t p = grid_stride_begin(); p < n; p += grid_stride()) {
        uint32_t slot;
        const Seg s = seg_at(n, level, p, slot);
        float lo[3], hi[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c] = key_bound(acc[6 * size_t(slot) + c]);
            hi[c] = key_bound(acc[6 * size_t(slot) + 3 + c]);
        }
        if (p == s.b) write_node(nodes, s, lo, hi);
        const uint32_t t = list[split_axis(lo, hi) * size_t(n) + p];
        side[t] = p >= s.b + (s.e - s.b) / 2 ? 1u : 0u;
    }
}
__global__ void k_bvh_top_flags(uint32_t n, const uint32_t* list, const uint8_t* side, uint32_t* left) {
    for (uint32_t i = grid_stride_begin(); i < 3u * n; i += grid_stride()) left[i] = side[list[i]] ? 0u : 1u;
}
// Stable partition of every node's part of the three lists (pre: exclusive
// scan of the left flags over all of them). Also the next level's bounds.
__global__ void k_bvh_top_split(uint32_t n, uint32_t level, const uint32_t* list, const uint32_t* left,
                                const uint32_t* pre, uint32_t* list2, uint32_t* acc) {
    for (uint32_t i = grid_stride_begin(); i < 3u * n; i += grid_stride()) {
        const uint32_t axis = i / n, p = i - axis * n;
        uint32_t slot;
        const Seg s = seg_at(n, level, p, slot);
        const uint32_t lefts = pre[i] - pre[axis * n + s.b];
        const uint32_t o = left[i] ? s.b + lefts : s.b + (s.e - s.b) / 2 + (p - s.b - lefts);
        list2[axis * size_t(n) + o] = list[i];
        if (i < 6u * (2u << level)) acc[i] = i % 6u < 3u ? 0xffffffffu : 0u;
    }
}

// ---- the remaining subtrees, one block each
__global__ void __launch_bounds__(kLocalThreads)
    k_bvh_local(uint32_t n, uint32_t level, const uint32_t* list, const float4* lo, const float4* hi, uint32_t* local,
                float* nodes, uint32_t* order) {
    constexpr uint32_t kSlots = kLocal / kLeaf;  // nodes of a level at most
    __shared__ uint32_t tri[kLocal];
    __shared__ float blo[kLocal][3], bhi[kLocal][3];
    __shared__ uint16_t lists[2][3][kLocal];
    __shared__ uint16_t pos_slot[kLocal];  // node of each position (0xffff: in a finished leaf)
    __shared__ uint8_t side[kLocal];
    __shared__ uint32_t pre[kLocal + 1];  // lefts before each position, 10 bits per list
    __shared__ Seg segs[2][kSlots];
    __shared__ uint8_t axes[kSlots];
    __shared__ uint32_t warp_sum[kLocalThreads / 32];
    const Seg root = seg_of_slot(n, level, blockIdx.x);
    const uint32_t m = root.e - root.b, tid = threadIdx.x, lane = tid & 31u;
    for (uint32_t p = tid; p < m; p += kLocalThreads) {
        const uint32_t t = list[root.b + p];
        tri[p] = t;
        local[t] = p;
        const float4 l = lo[t], h = hi[t];
        blo[p][0] = l.x;
        blo[p][1] = l.y;
        blo[p][2] = l.z;
        bhi[p][0] = h.x;
        bhi[p][1] = h.y;
        bhi[p][2] = h.z;
        lists[0][0][p] = uint16_t(p);
        pos_slot[p] = 0;
    }
    if (tid == 0) segs[0][0] = Seg{0u, m, root.node};
    __syncthreads();
    for (uint32_t p = tid; p < m; p += kLocalThreads)
#pragma unroll
        for (uint32_t a = 1; a < 3; ++a) lists[0][a][p] = uint16_t(local[list[a * size_t(n) + root.b + p]]);
    if (m <= kLeaf)  // a mesh of at most four triangles: its root is a leaf, in the given order
        for (uint32_t p = tid; p < m; p += kLocalThreads) order[p] = p;
    __syncthreads();
    uint32_t cur = 0, slots = 1, largest = m;
    for (;;) {
        // Bounds and axis of every node: a warp per node, or eight lanes once
        // the nodes are small.
        const uint32_t width = largest > 16u ? 32u : 8u;
        const uint32_t gl = tid % width, gmask = (width == 32u ? 0xffffffffu : 0xffu << (lane & ~7u));
        for (uint32_t k = tid / width; k < slots; k += kLocalThreads / width) {
            const Seg s = segs[cur][k];
            if (s.b == s.e) continue;  // absent: an ancestor is a leaf
            float l[3] = {kFltMax, kFltMax, kFltMax}, h[3] = {-kFltMax, -kFltMax, -kFltMax};
            for (uint32_t p = s.b + gl; p < s.e; p += width) {
                const uint32_t i = lists[cur][0][p];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    l[c] = fminf(l[c], blo[i][c]);
                    h[c] = fmaxf(h[c], bhi[i][c]);
                }
            }
            for (uint32_t o = width / 2; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    l[c] = fminf(l[c], __shfl_xor_sync(gmask, l[c], o));
                    h[c] = fmaxf(h[c], __shfl_xor_sync(gmask, h[c], o));
                }
            if (gl == 0) {
                write_node(nodes, Seg{root.b + s.b, root.b + s.e, s.node}, l, h);
                axes[k] = uint8_t(split_axis(l, h));
            }
        }
        if (largest <= kLeaf) break;
        __syncthreads();
        for (uint32_t p = tid; p < m; p += kLocalThreads) {
            const uint32_t k = pos_slot[p];
            if (k == 0xffffu) continue;
            const Seg s = segs[cur][k];
            const uint32_t i = lists[cur][axes[k]][p];
            const uint32_t mid = s.b + (s.e - s.b) / 2;
            side[i] = p >= mid ? 1u : 0u;
            // A child that is a leaf keeps this axis's order.
            if ((p >= mid ? s.e - mid : mid - s.b) <= kLeaf) order[root.b + p] = tri[i];
        }
        __syncthreads();
        // Exclusive scan of the left flags of the three lists at once (at
        // most 512 each, ten bits), two positions a thread.
        {
            static_assert(kLocal == 2 * kLocalThreads, "two positions a thread");
            uint32_t f[2];
#pragma unroll
            for (uint32_t q = 0; q < 2; ++q) {
                const uint32_t p = 2u * tid + q;
                f[q] = 0;
                if (p < m && pos_slot[p] != 0xffffu)
#pragma unroll
                    for (uint32_t a = 0; a < 3; ++a) f[q] += (side[lists[cur][a][p]] ? 0u : 1u) << (10u * a);
            }
            uint32_t x = f[0] + f[1];
            for (uint32_t o = 1; o < 32u; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31u) warp_sum[tid >> 5] = x;
            __syncthreads();
            uint32_t before = 0;
            for (uint32_t w = 0; w < (tid >> 5); ++w) before += warp_sum[w];
            x += before;
            pre[2u * tid] = x - f[0] - f[1];
            pre[2u * tid + 1u] = x - f[1];
        }
        __syncthreads();
        const uint32_t next = cur ^ 1u;
        for (uint32_t p = tid; p < m; p += kLocalThreads) {
            const uint32_t k = pos_slot[p];
            if (k == 0xffffu) continue;
            const Seg s = segs[cur][k];
            const uint32_t mid = s.b + (s.e - s.b) / 2;
#pragma unroll
            for (uint32_t a = 0; a < 3; ++a) {
                const uint32_t i = lists[cur][a][p];
                const uint32_t lefts = ((pre[p] >> (10u * a)) & 1023u) - ((pre[s.b] >> (10u * a)) & 1023u);
                lists[next][a][side[i] ? mid + (p - s.b - lefts) : s.b + lefts] = uint16_t(i);
            }
            const bool right = p >= mid;
            const uint32_t size = right ? s.e - mid : mid - s.b;
            pos_slot[p] = uint16_t(size <= kLeaf ? 0xffffu : 2u * k + (right ? 1u : 0u));
        }
        for (uint32_t k = tid; k < slots; k += kLocalThreads) {
            const Seg s = segs[cur][k];
            const bool splits = s.e - s.b > kLeaf;
            segs[next][2u * k] = splits ? child(s, false) : Seg{0u, 0u, 0u};
            segs[next][2u * k + 1u] = splits ? child(s, true) : Seg{0u, 0u, 0u};
        }
        __syncthreads();
        // (A new leaf's positions were just written to the next lists, where
        // its bounds read them; nothing reads or moves them after that.)
        cur = next;
        slots *= 2u;
        largest = (largest + 1u) / 2u;
    }
}

}  // namespace
}  // namespace pmb

using namespace pmb;

namespace {
// Scratch of the builds, one pool per device: cudaMalloc and cudaFree took
// 650 us of a 1,310 us call for 200,000 triangles. The pool keeps at most
// kPoolKept bytes between calls (more is given back when a call's stream
// synchronises) and is emptied when a world of its device is destroyed or by
// pmb_mesh_bvh_release; its allocations are ordered on the caller's stream,
// from any thread.
constexpr uint64_t kPoolKept = uint64_t(64) << 20;
constexpr int kPoolDevices = 64;
std::mutex g_pool_lock;
cudaMemPool_t g_pools[kPoolDevices];

cudaMemPool_t scratch_pool(int device) {
    if (device < 0 || device >= kPoolDevices) return nullptr;
    std::lock_guard<std::mutex> hold(g_pool_lock);
    if (!g_pools[device]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) return nullptr;
        uint64_t kept = kPoolKept;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &kept);
        g_pools[device] = pool;
    }
    return g_pools[device];
}
}  // namespace

namespace pmb {
void release_bvh_scratch(int device) {
    if (device < 0 || device >= kPoolDevices) return;
    std::lock_guard<std::mutex> hold(g_pool_lock);
    if (g_pools[device]) cudaMemPoolTrimTo(g_pools[device], 0);
}
}  // namespace pmb

extern "C" int pmb_mesh_bvh_release(int32_t device) {
    if (device < 0 || device >= kPoolDevices) return PMB_ERROR_INVALID_ARGUMENT;
    release_bvh_scratch(device);
    return PMB_SUCCESS;
}

extern "C" int pmb_mesh_bvh_build(const float* vertices, uint32_t vertex_count, const uint32_t* indices,
                                  uint32_t index_count, uint32_t* order, float* nodes, uint32_t node_capacity,
                                  uint32_t* node_count, void* stream) {
    if (!vertices || !indices || !order || !nodes || !node_count || vertex_count == 0 || index_count == 0 ||
        index_count % 3)
        return PMB_ERROR_INVALID_ARGUMENT;
    const uint32_t n = index_count / 3;
    const uint32_t count = node_total(n);
    *node_count = count;
    if (count > node_capacity) return PMB_ERROR_CAPACITY_EXCEEDED;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // Top levels: until no node has more than kLocal triangles.
    uint32_t top = 0;
    while (((n - 1u) >> top) + 1u > kLocal) ++top;
    // One allocation, carved (256-byte parts).
    const uint32_t tiles = (n + kRadixTile - 1) / kRadixTile;
    const size_t hist_count = size_t(3) * 256 * tiles, lists3 = size_t(3) * n;
    size_t used = 0;
    auto part = [&](size_t bytes) {
        const size_t at = used;
        used += (bytes + 255) & ~size_t(255);
        return at;
    };
    const size_t scan_most = std::max(hist_count, lists3);
    const size_t o_bad = part(4), o_lo = part(16 * size_t(n)), o_hi = part(16 * size_t(n)), o_key0 = part(4 * lists3),
                 o_key1 = part(4 * lists3), o_val0 = part(4 * lists3), o_val1 = part(4 * lists3),
                 o_hist = part(4 * (scan_most + 1)), o_offs = part(4 * (scan_most + 1)),
                 o_scan = part(4 * (scan_most / 2048 + 2)), o_side = part(n),
                 o_acc = part(4 * 6 * (size_t(2) << top));
    int device = 0;
    cudaGetDevice(&device);
    const cudaMemPool_t pool = scratch_pool(device);
    char* mem = nullptr;
    if (!pool || cudaMallocFromPoolAsync(reinterpret_cast<void**>(&mem), used, pool, s) != cudaSuccess) {
        cudaGetLastError();
        return PMB_ERROR_OUT_OF_DEVICE_MEMORY;
    }
    struct Freed {  // back to the pool once the stream is done with it
        void* p;
        cudaStream_t s;
        ~Freed() {
            cudaFreeAsync(p, s);
            cudaStreamSynchronize(s);
        }
    } freed{mem, s};
    auto words = [&](size_t at) { return reinterpret_cast<uint32_t*>(mem + at); };
    uint32_t* bad = words(o_bad);
    uint32_t bad_host = 0;
    cudaMemsetAsync(bad, 0, 4, s);
    k_bvh_check<<<cap_blocks(index_count, kBlock), kBlock, 0, s>>>(indices, index_count, vertex_count, bad);
    note_launch(cap_blocks(index_count, kBlock));
    if (cudaMemcpyAsync(&bad_host, bad, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess || bad_host)
        return PMB_ERROR_INVALID_ARGUMENT;
    float4 *lo = reinterpret_cast<float4*>(mem + o_lo), *hi = reinterpret_cast<float4*>(mem + o_hi);
    uint32_t* key[2] = {words(o_key0), words(o_key1)};
    uint32_t* val[2] = {words(o_val0), words(o_val1)};
    uint32_t *hist = words(o_hist), *offs = words(o_offs), *acc = words(o_acc);
    uint8_t* side = reinterpret_cast<uint8_t*>(mem + o_side);
    const uint32_t grid1 = cap_blocks(n, kBlock), grid3 = cap_blocks(lists3, kBlock);
    k_bvh_triangles<<<grid1, kBlock, 0, s>>>(vertices, indices, n, lo, hi, key[0], val[0]);
    note_launch(grid1);
    for (uint32_t shift = 0; shift < 32; shift += 8) {
        k_bvh_hist<<<dim3(tiles, 3), kRadixThreads, 0, s>>>(key[0], shift, n, tiles, hist);
        note_launch(3ull * tiles);
        scan_u32(hist, offs, nullptr, uint32_t(hist_count), nullptr, 0u, words(o_scan), s);
        k_bvh_scatter<<<dim3(tiles, 3), kRadixThreads, 0, s>>>(key[0], val[0], shift, n, tiles, offs, key[1], val[1]);
        note_launch(3ull * tiles);
        std::swap(key[0], key[1]);
        std::swap(val[0], val[1]);
    }
    if (top) {
        // The root's accumulator; the others are set by the level before.
        cudaMemsetAsync(acc, 0xff, 12, s);
        cudaMemsetAsync(acc + 3, 0, 12, s);
    }
    for (uint32_t level = 0; level < top; ++level) {
        const uint32_t bounds_grid = (n + kBoundsPerWarp * (kBlock / 32) - 1) / (kBoundsPerWarp * (kBlock / 32));
        k_bvh_top_bounds<<<bounds_grid, kBlock, 0, s>>>(n, level, val[0], lo, hi, acc);
        note_launch(bounds_grid);
        k_bvh_top_sides<<<grid1, kBlock, 0, s>>>(n, level, val[0], acc, nodes, side);
        note_launch(grid1);
        k_bvh_top_flags<<<grid3, kBlock, 0, s>>>(n, val[0], side, hist);
        note_launch(grid3);
        scan_u32(hist, offs, nullptr, uint32_t(lists3), nullptr, 0u, words(o_scan), s);
        k_bvh_top_split<<<grid3, kBlock, 0, s>>>(n, level, val[0], hist, offs, val[1], acc);
        note_launch(grid3);
        std::swap(val[0], val[1]);
    }
    k_bvh_local<<<1u << top, kLocalThreads, 0, s>>>(n, top, val[0], lo, hi, key[0], nodes, order);
    note_launch(1ull << top);
    const cudaError_t e = cudaStreamSynchronize(s);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? PMB_SUCCESS : PMB_ERROR_INVALID_ARGUMENT;
}
