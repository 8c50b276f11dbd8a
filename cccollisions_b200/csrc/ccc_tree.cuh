// ccc_tree.cuh — trees of the reference-format calls: the build into the exported tensors,
// and the import of caller tensors for the walk.
//
// Tensor layout per mesh of n triangles (src/build_bvh.cu:309-378): rows 0..n-2 internal
// nodes, rows n-1..2n-2 leaves in position order, bboxes row = (min xyz, max xyz), tree row =
// (parent, left, right, triangle id), -1 for "none".
//
// The reference's scene box is reduced from AABB() = (-MAX, +MAX) (aabb.cu:25-34,
// build_bvh.cu:243-244), which makes every Morton code 0; with all keys equal the stable
// sort keeps the input order, so leaf position p holds triangle p and the tree is the radix
// tree of the positions themselves (LongestCommonPrefix, bvh.cu:65-89, with equal keys).
// That tree has a closed form: at level t the positions form aligned blocks of 2^t, a block
// cut off at n is a node when its right half is not empty, and a node over [lo, hi] has the
// index that BuildRadixTree (build_bvh.cu:74-143) gives its range.
#pragma once

#include "ccc_kernels.cuh"
#include "ccc_walk.cuh"

namespace ccc {

// row of the (leaf or internal) node over the aligned block of 2^t positions from lo, cut at n
// (a left child ends at its index, a right child starts at it, the root is 0)
__device__ __forceinline__ int radix_row(int lo, int t, int n) {
    const int hi = (int)min((long long)lo + (1LL << t) - 1, (long long)n - 1);
    if (lo == hi) return n - 1 + lo;
    if (hi == n - 1) return lo;
    return ((lo >> t) & 1) ? lo : hi;
}

// parent of that node: -1 for the root
__device__ __forceinline__ int radix_parent(int lo, int t, int n) {
    // a left block without a right neighbour is the same node as the block above it
    while (!((lo >> t) & 1) && (long long)lo + (1LL << t) > n - 1) {
        if (lo == 0) return -1;
        ++t;
    }
    return radix_row((lo >> (t + 1)) << (t + 1), t + 1, n);
}

// first and last position of internal node k
__device__ __forceinline__ int2 radix_range(int k, int n) {
    if (k == 0) return make_int2(0, n - 1);
    if (k & 1) return make_int2(k + 1 - (1 << (__ffs(k + 1) - 1)), k);
    return make_int2(k, (int)min((long long)k + (1LL << (__ffs(k) - 1)) - 1, (long long)n - 1));
}

// rows of the children of the node over r, whose halves are blocks of 2^level positions
__device__ __forceinline__ int2 radix_children(int2 r, int level, int n) {
    const int mid = (r.y >> level) << level;
    return make_int2(radix_row(r.x, level, n), radix_row(mid, level, n));
}

template <class T> __device__ __forceinline__ Box<T> shfl_down_box(const Box<T>& b, int o) {
    const unsigned FULL = 0xffffffffu;
    Box<T> r;
    r.lo = mk<T>(__shfl_down_sync(FULL, b.lo.x, o), __shfl_down_sync(FULL, b.lo.y, o), __shfl_down_sync(FULL, b.lo.z, o));
    r.hi = mk<T>(__shfl_down_sync(FULL, b.hi.x, o), __shfl_down_sync(FULL, b.hi.y, o), __shfl_down_sync(FULL, b.hi.z, o));
    return r;
}

// The build: one thread a block of 2^level positions (level 0: the leaves, whose boxes, swept
// over both ends for motion, come from the triangles; above, the boxes that the launch below
// left in bboxes), LOG_THREADS levels a launch: up to five by shuffles, the rest over the
// warps' boxes in shared memory.  An internal node unites its children in the order left,
// right (CreateHierarchy, build_bvh.cu:145-209).
//
// The levels are known in advance, so no thread climbs with arrival counters (a device-wide
// fence, an atomic and two dependent reads through L2 a level), and the topology needs no
// search.  Measured against leaf rows, split search and climbs in three launches: 968
// triangles (fp64) 24.7 -> 7.8 us, 52,738 41 -> 14.5 us, 130,050 52 -> 22.7 us; what is left is
// launch latency and, at the large sizes, the row-wise stores.
template <class T, int LOG_THREADS>
__global__ void __launch_bounds__(1 << LOG_THREADS)
k_bvh_levels(const T* __restrict__ x0, const T* __restrict__ x1, int n, int chunks, int level, T* bboxes,
             long long* __restrict__ tree, WsHeader* hdr, int* __restrict__ mesh_cnt) {
    constexpr int THREADS = 1 << LOG_THREADS;
    __shared__ T wbox[6][THREADS / 32];
    const int m = blockIdx.x / chunks, t = threadIdx.x, lane = t & 31;
    const long long lo64 = ((long long)(blockIdx.x - m * chunks) * THREADS + t) << level;
    const long long base = (long long)m * (2LL * n - 1);
    T* bb = bboxes + base * 6;
    long long* tr = tree + base * 4;
    const bool live = lo64 < n;
    const int lo = live ? (int)lo64 : 0;
    if (level == 0) {
        // the workspace's status and counters, which no part of the build can raise
        if (blockIdx.x == 0 && t < (int)(sizeof(WsHeader) / sizeof(int))) reinterpret_cast<int*>(hdr)[t] = 0;
        if (lo64 == 0) mesh_cnt[m] = 0;
    }
    Box<T> b;
    b.lo = b.hi = mk<T>(T(0), T(0), T(0));
    if (live) {
        if (level == 0) {
            const long long g = (long long)m * n + lo;
            b = tri_box(load_tri(x0, g));
            if (x1) b = merge(b, tri_box(load_tri(x1, g)));      // MergeTriBoundingBoxes (452-460)
            store_box(bb + (n - 1LL + lo) * 6, b);
            // the tree rows of leaf lo and of internal node lo, both by closed form
            long long* row = tr + (n - 1LL + lo) * 4;
            row[0] = radix_parent(lo, 0, n);
            row[1] = row[2] = -1;
            row[3] = lo;
            if (lo < n - 1) {
                const int2 r = radix_range(lo, n);
                const int top = 31 - __clz(r.x ^ r.y);          // the level of its children
                const int2 c = radix_children(r, top, n);
                row = tr + lo * 4LL;
                row[0] = lo == 0 ? -1 : radix_parent(r.x, __ffs((lo & 1) ? lo + 1 : lo) - 1, n);
                row[1] = c.x;
                row[2] = c.y;
                row[3] = -1;
            }
        } else {
            b = load_box(bb + (long long)radix_row(lo, level, n) * 6);
        }
    }
    // the node over [lo, lo + 2^up) unites b and r
    auto node = [&](const Box<T>& r, int up) {
        b = merge(b, r);
        store_box(bb + (long long)radix_row(lo, up, n) * 6, b);
    };
    // (the launch that holds the root stops there)
    const int last = min(LOG_THREADS, 32 - __clz(n - 1) - level);
#pragma unroll
    for (int s = 1; s <= 5; ++s) {
        if (s > last) break;
        const Box<T> r = shfl_down_box(b, 1 << (s - 1));
        if (live && !(t & ((1 << s) - 1)) && lo64 + (1LL << (level + s - 1)) < n) node(r, level + s);
    }
    if (lane == 0) {
        const int w = t >> 5;
        wbox[0][w] = b.lo.x; wbox[1][w] = b.lo.y; wbox[2][w] = b.lo.z;
        wbox[3][w] = b.hi.x; wbox[4][w] = b.hi.y; wbox[5][w] = b.hi.z;
    }
#pragma unroll 1
    for (int s = 6; s <= last; ++s) {
        __syncthreads();
        if (live && !(t & ((1 << s) - 1)) && lo64 + (1LL << (level + s - 1)) < n) {
            const int w = (t >> 5) + (1 << (s - 6));
            Box<T> r;
            r.lo = mk<T>(wbox[0][w], wbox[1][w], wbox[2][w]);
            r.hi = mk<T>(wbox[3][w], wbox[4][w], wbox[5][w]);
            node(r, level + s);
            const int u = t >> 5;
            wbox[0][u] = b.lo.x; wbox[1][u] = b.lo.y; wbox[2][u] = b.lo.z;
            wbox[3][u] = b.hi.x; wbox[4][u] = b.hi.y; wbox[5][u] = b.hi.z;
        }
    }
}

}  // namespace ccc
