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
// A mesh takes 2^log_mesh threads of a block (with more blocks of positions than a block of
// threads, `chunks` whole ones): a block for every mesh leaves most threads idle on large batches
// of tiny meshes (bvh of 1,000,000 meshes of two triangles, fp32: 1,301 -> 119 us; 30,000 of 300
// triangles 546 -> 388 us).
//
// The levels are known in advance, so no thread climbs with arrival counters (a device-wide
// fence, an atomic and two dependent reads through L2 a level), and the topology needs no
// search.  Measured against leaf rows, split search and climbs in three launches: 968
// triangles (fp64) 24.7 -> 7.8 us, 52,738 41 -> 14.5 us, 130,050 52 -> 22.7 us; what is left is
// launch latency and, at the large sizes, the row-wise stores.
template <class T, int LOG_THREADS>
__global__ void __launch_bounds__(1 << LOG_THREADS)
k_bvh_levels(const T* __restrict__ x0, const T* __restrict__ x1, int meshes, int n, int chunks, int log_mesh, int level,
             T* bboxes, long long* __restrict__ tree, WsHeader* hdr, int* __restrict__ mesh_cnt) {
    chain_begin();
    constexpr int THREADS = 1 << LOG_THREADS;
    __shared__ T wbox[6][THREADS / 32];
    const int t = threadIdx.x, lane = t & 31, group = blockIdx.x / chunks;
    const int m = (group << (LOG_THREADS - log_mesh)) + (t >> log_mesh);
    const long long lo64 = ((long long)(blockIdx.x - group * chunks) * THREADS + (t & ((1 << log_mesh) - 1))) << level;
    const long long base = (long long)m * (2LL * n - 1);
    T* bb = bboxes + base * 6;
    long long* tr = tree + base * 4;
    const bool live = m < meshes && lo64 < n;
    const int lo = live ? (int)lo64 : 0;
    if (level == 0) {
        // the workspace's status and counters, which no part of the build can raise
        if (blockIdx.x == 0 && t < (int)(sizeof(WsHeader) / sizeof(int))) reinterpret_cast<int*>(hdr)[t] = 0;
        if (live && lo64 == 0) mesh_cnt[m] = 0;
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

// ---------------------------------------------------------------------------------------
// Import of caller tensors for the walk (build_bvh_from_array_tree, build_bvh.cu:667-705, and
// set_rightmost_nodes, 707-743): every internal node's QNode, its children with the internal
// ones replaced by their own children.  A replaced child is not visited itself, so each of
// its two slots holds the intersection of its box with the child's: the query meets both, as
// it would have to one level at a time, and for boxes that contain their children's (every
// tree built from them) the intersection is the slot's own box.
//
// The rightmost leaf position below a node, which the order rule needs, is known without a
// climb when the tree is the radix tree of the positions (bvh and bvh_motion, the reference's
// too); one with any other child, or with a child that names another parent, raises
// hdr->general, and k_import_rightmost_wide then climbs for all of them and reports a parent
// column that does not lead to the root.  Measured for a bvh_motion tree of 52,738
// triangles (fp64): binary nodes and climbs 34 us, four-wide nodes and no climb 10 us.
template <class T> __device__ __forceinline__ void box_outward(const T* p, float lo[3], float hi[3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        if (sizeof(T) == 4) {
            lo[c] = (float)__ldg(p + c);
            hi[c] = (float)__ldg(p + 3 + c);
        } else {
            lo[c] = __double2float_rd((double)__ldg(p + c));
            hi[c] = __double2float_ru((double)__ldg(p + 3 + c));
        }
    }
}

// the larger (smaller) of a and b, NaN when either is: a NaN box meets nothing
__device__ __forceinline__ float max_nan(float a, float b) { return a != a || a > b ? a : b; }
__device__ __forceinline__ float min_nan(float a, float b) { return a != a || a < b ? a : b; }

template <class T>
__global__ void k_import_wide(int n, int meshes, const T* __restrict__ bboxes, const long long* __restrict__ tree,
                              QNode* __restrict__ qnodes, int* __restrict__ visits, int* __restrict__ rmk,
                              int* __restrict__ table, int* __restrict__ moff, WsHeader* hdr) {
    chain_begin();
    const int gi = blockIdx.x * blockDim.x + threadIdx.x;
    const int internal = meshes * (n - 1);
    // the packed mesh table (Forest): count, offsets, data offsets, slot ids
    for (int i = gi; i <= meshes; i += gridDim.x * blockDim.x) {
        moff[i] = i * n;
        if (i < meshes) {
            table[4 + i] = i * n;
            table[4 + meshes + i] = i;
        }
        if (i == 0) table[0] = meshes;
    }
    if (gi >= internal) return;
    const int m = gi / (n - 1), k = gi - m * (n - 1);
    const long long base = (long long)m * (2LL * n - 1);
    const long long* tr = tree + base * 4;
    const T* bb = bboxes + base * 6;
    visits[gi] = 0;
    rmk[gi] = -1;
    const int2 r = radix_range(k, n);
    const int2 regular = radix_children(r, 31 - __clz(r.x ^ r.y), n);
    bool bad = false;
    auto child = [&](int node, int side) {
        long long c = __ldg(tr + node * 4LL + 1 + side);
        if (c <= 0 || c >= 2LL * n - 1) {
            bad = true;
            c = 2LL * n - 2;                 // keep the record pointing at a valid leaf
        }
        return (int)c;
    };
    const float inf = __int_as_float(0x7f800000);
    float lo[3][4], hi[3][4];
    int ref[4], aux[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        ref[s] = Q_EMPTY;
        aux[s] = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c][s] = inf;
            hi[c][s] = -inf;
        }
    }
    // slot s (a constant) from row c, within the box above it when there is one
    auto slot = [&](int s, int c, bool within, const float* alo, const float* ahi) {
        float l[3], h[3];
        box_outward<T>(bb + c * 6LL, l, h);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            lo[d][s] = within ? max_nan(l[d], alo[d]) : l[d];
            hi[d][s] = within ? min_nan(h[d], ahi[d]) : h[d];
        }
        if (c >= n - 1) {
            const long long id = __ldg(tr + c * 4LL + 3);
            if (id < 0 || id >= n) bad = true;
            ref[s] = ~(c - (n - 1));
            aux[s] = id < 0 || id >= n ? 0 : (int)id;
        } else {
            ref[s] = c;
            aux[s] = radix_range(c, n).y;    // (of a regular tree)
        }
    };
    const int c0 = child(k, 0), c1 = child(k, 1);
    // (the parents too: a wrong one is for the climbs to find)
    if (c0 != regular.x || c1 != regular.y || __ldg(tr + c0 * 4LL) != k || __ldg(tr + c1 * 4LL) != k) hdr->general = 1;
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        const int c = side ? c1 : c0;
        if (c >= n - 1) {
            slot(2 * side, c, false, nullptr, nullptr);
        } else {
            float alo[3], ahi[3];
            box_outward<T>(bb + c * 6LL, alo, ahi);
            slot(2 * side, child(c, 0), true, alo, ahi);
            slot(2 * side + 1, child(c, 1), true, alo, ahi);
        }
    }
    if (bad) atomicOr(&hdr->status, ST_MALFORMED_TREE);
    QNode q;
    q.lox = make_float4(lo[0][0], lo[0][1], lo[0][2], lo[0][3]);
    q.loy = make_float4(lo[1][0], lo[1][1], lo[1][2], lo[1][3]);
    q.loz = make_float4(lo[2][0], lo[2][1], lo[2][2], lo[2][3]);
    q.hix = make_float4(hi[0][0], hi[0][1], hi[0][2], hi[0][3]);
    q.hiy = make_float4(hi[1][0], hi[1][1], hi[1][2], hi[1][3]);
    q.hiz = make_float4(hi[2][0], hi[2][1], hi[2][2], hi[2][3]);
    q.ref = make_int4(ref[0], ref[1], ref[2], ref[3]);
    q.aux = make_int4(aux[0], aux[1], aux[2], aux[3]);
    qnodes[(long long)m * n + k] = q;        // mesh m's nodes start at its first triangle slot
}

// the rightmost leaf position below every internal node of a general tree, by climbs
static __global__ void k_import_rightmost_wide(int n, int total, const long long* __restrict__ tree,
                                               int* __restrict__ visits, int* __restrict__ rmk, WsHeader* hdr) {
    chain_begin();
    if (!*(volatile int*)&hdr->general) return;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    const int m = g / n, ioff = m * (n - 1);
    const long long* tr = tree + (long long)m * (2LL * n - 1) * 4;
    long long node = tr[(n - 1LL + (g - (long long)m * n)) * 4];
    for (int guard = 0; guard < n; ++guard) {
        if (node < 0 || node >= n - 1) { atomicOr(&hdr->status, ST_MALFORMED_TREE); return; }
        __threadfence();
        if (atomicAdd(visits + ioff + node, 1) == 0) return;
        int r = 0;
        for (int side = 0; side < 2; ++side) {
            long long c = tr[node * 4 + 1 + side];
            if (c <= 0 || c >= 2LL * n - 1) c = 2LL * n - 2;
            r = max(r, c >= n - 1 ? (int)(c - (n - 1)) : __ldcg(rmk + ioff + c));
        }
        rmk[ioff + node] = r;
        if (node == 0) return;
        node = tr[node * 4];
    }
    atomicOr(&hdr->status, ST_MALFORMED_TREE);
}

// The walk over imported trees (traverseBVH, collisions_static.cu:10-103; traverseBVHPartial,
// collisions_continuous.cu:127-230): fp32 boxes with outward rounding in the nodes, then the
// exact reference-precision test of every leaf hit (EXACT_F32: the fp32 boxes are exact and
// the threshold is 0, so there is nothing to test again).  MASKED: only the marked leaves
// query, against every leaf, and of two marked triangles the smaller reports the pair.
// Measured against one query a thread on binary nodes (which a workspace too small for the
// four-wide ones still takes): 968 triangles 49 -> 10 us, 7,938 (fp32) 41 -> 17 us, 52,738
// 124 -> 48 us, 130,050 260 -> 112 us, 40,800 (fp32) with 30 % marked 280 -> 42 us.
template <class T, bool MASKED, bool EXACT_F32> struct TensorWalk {
    const T* bboxes;
    const long long* tree;
    const uint8_t* mask;
    const int* rmk;          // of a general tree
    T th;
    int n, general;
    static constexpr bool ORDERED = !MASKED;
    __device__ __forceinline__ long long row(int base, int pos) const {
        return 2LL * base - base / n + (n - 1) + pos;     // mesh m's rows start at m (2 n - 1)
    }
    __device__ __forceinline__ bool query(const Forest&, int, int v, WsHeader* hdr, WalkQuery& q) const {
        const int m = v / n;
        q.base = m * n;
        q.n = n;
        q.pos = v - q.base;
        if (MASKED && !mask[v]) return false;
        const long long at = row(q.base, q.pos);
        const long long id = __ldg(tree + at * 4 + 3);
        if (id < 0 || id >= n) {
            atomicOr(&hdr->status, ST_MALFORMED_TREE);
            return false;
        }
        q.id = (int)id;
        const T* b = bboxes + at * 6;
        // conservative fp32 query box: threshold folded in, rounded outward, nudged one more ulp
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (EXACT_F32) {
                q.lo[c] = (float)__ldg(b + c);
                q.hi[c] = (float)__ldg(b + 3 + c);
            } else {
                q.lo[c] = nudge_down(__double2float_rd((double)__ldg(b + c) - (double)th));
                q.hi[c] = nudge_up(__double2float_ru((double)__ldg(b + 3 + c) + (double)th));
            }
        }
        return true;
    }
    __device__ __forceinline__ int rightmost(int base, int ref, int aux) const {
        return general ? __ldg(rmk + (base - base / n) + ref) : aux;
    }
    __device__ __forceinline__ bool keep(int base, int, int pos, int id, int cpos, int cid) const {
        if (MASKED && mask[base + cid] && !(id < cid)) return false;
        return EXACT_F32 || overlap(load_box(bboxes + row(base, pos) * 6), load_box(bboxes + row(base, cpos) * 6), th);
    }
};

template <class T, bool MASKED, bool EXACT_F32>
__global__ void __launch_bounds__(WALK_THREADS, 8)
k_walk_tensors(const QNode* __restrict__ qnodes, const T* __restrict__ bboxes, const long long* __restrict__ tree,
               const uint8_t* __restrict__ mask, const int* __restrict__ rmk, int n, Forest F, T th,
               int2* __restrict__ cand, int cand_cap, WsHeader* hdr) {
    chain_begin();
    __shared__ WalkWarp S[WALK_WARPS];
    const TensorWalk<T, MASKED, EXACT_F32> pol{bboxes, tree, mask, rmk, th, n, *(volatile int*)&hdr->general};
    walk_forest(pol, qnodes, F, cand, cand_cap, hdr, S[threadIdx.x >> 5]);
}

}  // namespace ccc
