// ccc_kernels.cuh — sm_100a kernels of the collision pipeline.
//
// Meshes are processed as a "forest": M meshes concatenated, mesh m owning triangles
// [moff[m], moff[m+1]).  The exported tree tensors use the reference layout per mesh
// (src/build_bvh.cu:309-378): rows 0..F-2 internal nodes, rows F-1..2F-2 leaves in sorted
// position order, bboxes row = (min xyz, max xyz), tree row = (parent, left, right, tri id),
// -1 for "none".  Mesh m's rows start at 2*moff[m] - m.
//
// Traversal works on copies of the internal nodes with their child boxes rounded outward to fp32
// and child references: four-wide QNodes (ccc_walk.cuh), or binary TNodes (64 B, four 16-byte
// loads a visit) in workspaces without room for those.
#pragma once

#include <atomic>

#include <cooperative_groups.h>
#include <cooperative_groups/reduce.h>
#include <cooperative_groups/scan.h>
#include "ccc_geom.cuh"

namespace cg = cooperative_groups;

namespace ccc {

// Every kernel that launch_chain launches begins with this: the launch lets it start as the
// blocks of the kernel before it in the stream end, which hides most of a launch's latency (968
// triangles' impulses, ten kernels, 113 -> 103 us; building and stepping 12 meshes, 45 kernels,
// 1,282 -> 1,204 us); here it waits until that kernel is complete and its writes are visible.
// (Letting the next kernel start as soon as this one's last block runs, by an explicit trigger,
// made the kernels that fill the GPU share it with blocks that only wait: the 256 x 256 fold
// 1,148 -> 1,254 us, the 64-mesh step 10.69 -> 11.62 ms.)
__device__ __forceinline__ void chain_begin() { cudaGridDependencySynchronize(); }

enum StatusBits {
    ST_CAND_OVERFLOW = 1,     // more candidate pairs than max_candidates_per_triangle * F
    ST_OUT_OVERFLOW = 2,      // more result rows than the output tensor holds
    ST_STACK_OVERFLOW = 4,    // traversal deeper than its stack (one query a thread: 64 entries; walk: WALK_STACK)
    ST_MALFORMED_TREE = 8,    // child / parent index out of range or a cycle in the tree
};

// per-mesh state flags of the resident engine's impulse loop
enum MeshFlags {
    MF_DONE = 1,         // the impulse loop has stopped for this mesh
    MF_CONVERGED = 2,    // ... because a collision check found no contact
};

// Workspace header (int32 words) shared by all operations.
struct WsHeader {
    int status;
    int cand_count;
    int subtests;      // continuous sub-tests (pair, type) whose swept sub-boxes overlap
    int roots;         // roots in [0, 1] put to the filter
    int front;         // engine refit: climbs handed from the block pass to the global pass
    int solved;        // sub-tests solved (fewer than subtests when repeated ones are shared)
    int fan_cursor;    // engine corner classes: member list slots handed out
    int live_count;    // engine staging: pairs with sub-tests to solve (Weld.live)
    int pending_count; // engine staging: pairs left with vertex-face sub-tests to place
    int expand_count;  // engine narrow phase: records for k_ccd_expand (Weld.expand)
    int general;       // imported tree: not the radix tree of the positions
    int walk_next;     // groups of queries that the walk's warps took after their first
    int pad[4];
};

struct __align__(16) TNode {
    float4 a;   // left  lo.x lo.y lo.z hi.x
    float4 b;   // left  hi.y hi.z | right lo.x lo.y
    float4 c;   // right lo.z hi.x hi.y hi.z
    int4 d;     // left ref, right ref, left aux, right aux
};
// ref >= 0: internal node (mesh-local index); ref < 0: leaf at position ~ref.
// aux: internal child -> rightmost leaf position of its subtree; leaf child -> triangle id.

static constexpr int TRAV_THREADS = 128;
static constexpr int STACK_DEPTH = 64;        // STACK_SIZE (flags.h:26-29)
static constexpr int NARROW_THREADS = 128;
// resident blocks per SM of the static and proximity narrow phases
static constexpr int NARROW_MIN_BLOCKS = 4;

// mesh containing element g where base(m) = off[m] - m * shift (shift 0: triangles,
// shift 1: internal nodes); off has M + 1 entries
__device__ __forceinline__ int find_mesh(const int* __restrict__ off, int M, long long g, int shift) {
    int lo = 0, hi = M - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        long long b = (long long)__ldg(off + mid) - (long long)mid * shift;
        if (b <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Mesh table of the traversal and narrow-phase kernels.  Mesh m (0 <= m < *nm) owns the
// work items [voff[m], voff[m+1]) (a dense prefix that assigns threads to meshes) and the
// data slots [poff[m], poff[m] + F_m) of the triangle, node, leaf and per-triangle output
// arrays (ascending and non-overlapping; poff = voff for a packed batch).  sid[m] is the
// mesh's stable slot id, which indexes its per-mesh counters and state.  All four live in
// device memory, so a captured launch sequence serves whatever table is current.
struct Forest {
    const int* nm;
    const int* voff;
    const int* poff;
    const int* sid;
};

__device__ __forceinline__ int forest_size(const Forest& f) { return __ldg(f.nm); }

// mesh owning data slot g (the last m with poff[m] <= g)
__device__ __forceinline__ int forest_slot_mesh(const Forest& f, int M, long long g) {
    return find_mesh(f.poff, M, g, 0);
}

// ---------------------------------------------------------------------------------------
// packed mesh table for the reference API (B meshes of F triangles): nm = B,
// voff[i] = poff[i] = i * F, sid[i] = i
static __global__ void k_uniform_offsets(int* nm, int* voff, int* poff, int* sid, int M, int F) {
    chain_begin();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *nm = M;
    if (i <= M) voff[i] = i * F;
    if (i < M) {
        poff[i] = i * F;
        sid[i] = i;
    }
}

// ---------------------------------------------------------------------------------------
// Up to three arrays of 4-byte words filled with 8-byte patterns (lo, hi), 16 bytes a store
// where an array is aligned for it.
struct FillJob {
    uint32_t* p;
    long long words;
    uint32_t lo, hi;
};
static __global__ void k_fill(FillJob a, FillJob b, FillJob c) {
    chain_begin();
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
    auto fill = [&](const FillJob& j) {
        const long long quads = ((uintptr_t)j.p & 15) == 0 ? j.words / 4 : 0;
        const uint4 v = make_uint4(j.lo, j.hi, j.lo, j.hi);
        for (long long i = t; i < quads; i += stride) reinterpret_cast<uint4*>(j.p)[i] = v;
        for (long long i = 4 * quads + t; i < j.words; i += stride) j.p[i] = i & 1 ? j.hi : j.lo;
    };
    fill(a);
    fill(b);
    fill(c);
}

// ---------------------------------------------------------------------------------------
// Import of exported tensors into traversal nodes (build_bvh_from_array_tree 667-705 and
// set_rightmost_nodes 707-743).

template <class T> __device__ __forceinline__ void box_to_f32(const T* p, float lo[3], float hi[3]) {
    if (sizeof(T) == 4) {
        for (int c = 0; c < 3; ++c) { lo[c] = (float)p[c]; hi[c] = (float)p[3 + c]; }
    } else {
        for (int c = 0; c < 3; ++c) {
            lo[c] = __double2float_rd((double)p[c]);
            hi[c] = __double2float_ru((double)p[3 + c]);
        }
    }
}

template <class T>
__global__ void k_import_nodes(const int* __restrict__ moff, int M, int total_internal, const T* __restrict__ bboxes,
                               const long long* __restrict__ tree, TNode* __restrict__ nodes, int* status) {
    chain_begin();
    int gi = blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= total_internal) return;
    int m = find_mesh(moff, M, gi, 1);
    int n = moff[m + 1] - moff[m];
    int k = gi - (moff[m] - m);
    long long base = 2LL * moff[m] - m;
    long long ch[2] = {tree[(base + k) * 4 + 1], tree[(base + k) * 4 + 2]};
    float lo[2][3], hi[2][3];
    int ref[2], aux[2];
    for (int s = 0; s < 2; ++s) {
        long long c = ch[s];
        if (c <= 0 || c >= 2LL * n - 1) {
            atomicOr(status, ST_MALFORMED_TREE);
            c = 2LL * n - 2;     // keep the record pointing at a valid leaf
        }
        box_to_f32<T>(bboxes + (base + c) * 6, lo[s], hi[s]);
        if (c >= n - 1) {
            ref[s] = ~(int)(c - (n - 1));
            long long id = tree[(base + c) * 4 + 3];
            if (id < 0 || id >= n) {
                atomicOr(status, ST_MALFORMED_TREE);
                id = 0;
            }
            aux[s] = (int)id;
        } else {
            ref[s] = (int)c;
            aux[s] = -1;
        }
    }
    TNode t;
    t.a = make_float4(lo[0][0], lo[0][1], lo[0][2], hi[0][0]);
    t.b = make_float4(hi[0][1], hi[0][2], lo[1][0], lo[1][1]);
    t.c = make_float4(lo[1][2], hi[1][0], hi[1][1], hi[1][2]);
    t.d = make_int4(ref[0], ref[1], aux[0], aux[1]);
    nodes[moff[m] + k] = t;      // mesh m's nodes start at its first triangle slot
}

// rightmost leaf position of every internal subtree, written into the parent's aux slot
static __global__ void k_import_rightmost(const int* __restrict__ moff, int M, int total, const long long* __restrict__ tree,
                                   TNode* nodes, int* __restrict__ visits, int* __restrict__ rmk, int* status) {
    chain_begin();
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    int m = find_mesh(moff, M, g, 0);
    int n = moff[m + 1] - moff[m];
    if (n < 2) return;
    int p = g - moff[m];
    long long base = 2LL * moff[m] - m;
    int ioff = moff[m] - m;
    TNode* nd = nodes + moff[m];
    long long node = tree[(base + n - 1 + p) * 4 + 0];
    for (int guard = 0; guard < n; ++guard) {
        if (node < 0 || node >= n - 1) { atomicOr(status, ST_MALFORMED_TREE); return; }
        __threadfence();
        if (atomicAdd(visits + ioff + node, 1) == 0) return;
        int4 d = nd[node].d;
        int rl = d.x < 0 ? ~d.x : __ldcg(rmk + ioff + d.x);
        int rr = d.y < 0 ? ~d.y : __ldcg(rmk + ioff + d.y);
        int r = max(rl, rr);
        rmk[ioff + node] = r;
        long long par = tree[(base + node) * 4 + 0];
        if (par >= 0 && par < n - 1) {
            int4 pd = nd[par].d;
            if (pd.x == (int)node) nd[par].d.z = r;
            else nd[par].d.w = r;
        }
        if (node == 0) return;
        node = par;
    }
    atomicOr(status, ST_MALFORMED_TREE);
}

// ---------------------------------------------------------------------------------------
// Traversal (traverseBVH, collisions_static.cu:10-103; traverseBVHPartial,
// collisions_continuous.cu:127-230).  One thread per query leaf, an explicit stack in
// shared memory, fp32 child-box tests with outward rounding, then the exact
// reference-precision leaf test for every fp32 hit.  Emits global triangle indices.

__device__ __forceinline__ float nudge_down(float x) { return nextafterf(x, -INFINITY); }
__device__ __forceinline__ float nudge_up(float x) { return nextafterf(x, INFINITY); }

// Where traversal finds the leaves of mesh m (n triangles) in the reference's exported
// tensors (mesh m's rows start at 2 voff[m] - m): the query's exact box and triangle id, and
// the exact box of a hit leaf, by sorted leaf position.
template <class T> struct TensorLeaves {
    const T* bboxes;
    const long long* tree;
    __device__ __forceinline__ long long row(int m, int vo, int n, int pos) const {
        return 2LL * vo - m + (n - 1) + pos;
    }
    __device__ __forceinline__ Box<T> box(int m, int vo, int po, int n, int pos) const {
        return load_box(bboxes + row(m, vo, n, pos) * 6);
    }
    __device__ __forceinline__ long long id(int m, int vo, int po, int n, int pos) const {
        return tree[row(m, vo, n, pos) * 4 + 3];
    }
};

// Traversal kernels pass candidates through a per-thread buffer of TRAV_BUF pairs and
// reserve TRAV_BUF slots per thread of a coalesced group with one atomic on the shared
// counter, which every SM contends for.
static constexpr int TRAV_BUF = 16;

// the first n buffered pairs of thread tid to cand[base ..]; pairs past the capacity are
// dropped and reported
__device__ __forceinline__ void flush_candidates(int2 (*cbuf)[TRAV_THREADS], int tid, int n, int base,
                                                 int2* __restrict__ cand, int cand_cap, WsHeader* hdr) {
    for (int i = 0; i < n; ++i) {
        const long long slot = (long long)base + i;
        if (base >= 0 && slot < cand_cap) cand[slot] = cbuf[i][tid];
        else atomicOr(&hdr->status, ST_CAND_OVERFLOW);
    }
}

// the remaining buffered pairs of every thread of the calling coalesced group, with one
// atomic for the group (exclusive scan of the counts)
__device__ __forceinline__ void flush_rest(int2 (*cbuf)[TRAV_THREADS], int tid, int n, int2* __restrict__ cand,
                                           int cand_cap, WsHeader* hdr) {
    cg::coalesced_group grp = cg::coalesced_threads();
    int incl = n;
    for (int o = 1; o < (int)grp.size(); o <<= 1) {
        int y = grp.shfl_up(incl, o);
        if ((int)grp.thread_rank() >= o) incl += y;
    }
    int total = grp.shfl(incl, grp.size() - 1);
    int base = 0;
    if (grp.thread_rank() == 0) base = atomicAdd(&hdr->cand_count, total);
    base = grp.shfl(base, 0) + incl - n;
    flush_candidates(cbuf, tid, n, base, cand, cand_cap, hdr);
}

template <class T, bool MASKED, bool EXACT_F32, class Leaves>
__global__ void __launch_bounds__(TRAV_THREADS)
k_traverse(const TNode* __restrict__ nodes, Leaves leaves, Forest F, const uint8_t* __restrict__ mask, T th,
           int2* __restrict__ cand, int cand_cap, WsHeader* hdr, const int* __restrict__ mflags) {
    chain_begin();
    int stack[STACK_DEPTH];          // per-thread, in local memory (L1): shared memory holds the buffer
    __shared__ int2 cbuf[TRAV_BUF][TRAV_THREADS];
    int nbuf = 0;
    const int tid = threadIdx.x;
    const int M = forest_size(F);
    const int total = __ldg(F.voff + M);
    for (int v = blockIdx.x * blockDim.x + tid; v < total; v += gridDim.x * blockDim.x) {
        int m = find_mesh(F.voff, M, v, 0);
        int vo = __ldg(F.voff + m), po = __ldg(F.poff + m);
        int n = __ldg(F.voff + m + 1) - vo;
        int p = v - vo;
        if (n < 2) continue;
        if (MASKED && !mask[po + p]) continue;
        if (mflags && (__ldg(mflags + __ldg(F.sid + m)) & MF_DONE)) continue;
        const TNode* nd = nodes + po;
        long long qid64 = leaves.id(m, vo, po, n, p);
        if (qid64 < 0 || qid64 >= n) {
            atomicOr(&hdr->status, ST_MALFORMED_TREE);
            continue;
        }
        int qid = (int)qid64;
        // conservative fp32 query box: threshold folded in, rounded outward, nudged one more ulp
        float qlo[3], qhi[3];
        Box<T> q = leaves.box(m, vo, po, n, p);
        {
            T lo[3] = {q.lo.x, q.lo.y, q.lo.z}, hi[3] = {q.hi.x, q.hi.y, q.hi.z};
            for (int c = 0; c < 3; ++c) {
                if (EXACT_F32) {
                    qlo[c] = (float)lo[c];
                    qhi[c] = (float)hi[c];
                } else {
                    qlo[c] = nudge_down(__double2float_rd((double)lo[c] - (double)th));
                    qhi[c] = nudge_up(__double2float_ru((double)hi[c] + (double)th));
                }
            }
        }
        int sp = 0;
        int node = 0;
        const int limit = 4 * n + 64;
        for (int it = 0;; ++it) {
            if (it > limit) { atomicOr(&hdr->status, ST_MALFORMED_TREE); break; }
            const float4* np = reinterpret_cast<const float4*>(nd + node);
            float4 A = __ldg(np + 0), B = __ldg(np + 1), C = __ldg(np + 2);
            int4 D = __ldg(reinterpret_cast<const int4*>(np + 3));
            // child references inside this mesh: internal < n - 1, leaf position < n
            if (D.x >= n - 1 || D.y >= n - 1 || ~D.x >= n || ~D.y >= n) {
                atomicOr(&hdr->status, ST_MALFORMED_TREE);
                break;
            }
            bool ol = (qlo[0] <= A.w) && (qhi[0] >= A.x) && (qlo[1] <= B.x) && (qhi[1] >= A.y) && (qlo[2] <= B.y) &&
                      (qhi[2] >= A.z);
            bool orr = (qlo[0] <= C.y) && (qhi[0] >= B.z) && (qlo[1] <= C.z) && (qhi[1] >= B.w) && (qlo[2] <= C.w) &&
                       (qhi[2] >= C.x);
            if (!MASKED) {
                int rml = D.x < 0 ? ~D.x : D.z;
                int rmr = D.y < 0 ? ~D.y : D.w;
                if (p >= rml) ol = false;
                if (p >= rmr) orr = false;
            }
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                int ref = s ? D.y : D.x;
                bool hit = (s ? orr : ol) && ref < 0;
                if (hit) {
                    int cpos = ~ref;
                    int cid = s ? D.w : D.z;
                    if (MASKED && mask[po + cid] && !(qid < cid)) hit = false;
                    if (hit && !EXACT_F32) hit = overlap(q, leaves.box(m, vo, po, n, cpos), th);
                    if (hit) {
                        cbuf[nbuf++][tid] = make_int2(po + min(qid, cid), po + max(qid, cid));
                        if (nbuf == TRAV_BUF) {
                            cg::coalesced_group grp = cg::coalesced_threads();
                            int base = 0;
                            if (grp.thread_rank() == 0) base = atomicAdd(&hdr->cand_count, TRAV_BUF * (int)grp.size());
                            base = grp.shfl(base, 0) + TRAV_BUF * (int)grp.thread_rank();
                            flush_candidates(cbuf, tid, TRAV_BUF, base, cand, cand_cap, hdr);
                            nbuf = 0;
                        }
                    }
                }
            }
            bool tl = ol && D.x >= 0, tr = orr && D.y >= 0;
            if (!tl && !tr) {
                if (sp == 0) break;
                node = stack[--sp];
            } else {
                node = tl ? D.x : D.y;
                if (tl && tr) {
                    if (sp >= STACK_DEPTH) { atomicOr(&hdr->status, ST_STACK_OVERFLOW); break; }
                    stack[sp++] = D.y;
                }
            }
        }
    }
    if (nbuf > 0) flush_rest(cbuf, tid, nbuf, cand, cand_cap, hdr);
}

// ---------------------------------------------------------------------------------------
// Narrow phases.  Grid-stride over the candidate buffer; the count is read on the device.

// Output region of the mesh that owns data slot g: rows [poff[m] * per_tri, ... + F_m * per_tri)
struct OutRegion {
    int m;              // table index
    int po;             // first data slot
    long long cap;      // F_m * per_tri
};
__device__ __forceinline__ OutRegion out_region(const Forest& F, int M, long long g, int per_tri) {
    OutRegion r;
    r.m = forest_slot_mesh(F, M, g);
    r.po = __ldg(F.poff + r.m);
    r.cap = (long long)(__ldg(F.voff + r.m + 1) - __ldg(F.voff + r.m)) * per_tri;
    return r;
}

// per-mesh append of one row; returns the row index within the mesh region or -1 when full
__device__ __forceinline__ long long append_row(int* mesh_counters, const Forest& F, int m, long long cap,
                                                int* status) {
    cg::coalesced_group act = cg::coalesced_threads();
    cg::coalesced_group grp = cg::labeled_partition(act, m);
    int slot = 0;
    if (grp.thread_rank() == 0) slot = atomicAdd(mesh_counters + __ldg(F.sid + m), (int)grp.size());
    slot = grp.shfl(slot, 0) + grp.thread_rank();
    if ((long long)slot >= cap) {
        atomicOr(status, ST_OUT_OVERFLOW);
        return -1;
    }
    return slot;
}

// find_collisions: SAT + shared-vertex count (collisions_static.cu:123-159)
template <class T>
__global__ void __launch_bounds__(NARROW_THREADS)
k_static_narrow(const int2* __restrict__ cand, int cand_cap, WsHeader* hdr, const T* __restrict__ tri, Forest F,
                T th, long long* __restrict__ rows, int max_per_tri, int* __restrict__ mesh_counters) {
    chain_begin();
    const int M = forest_size(F);
    int n = min(hdr->cand_count, cand_cap);
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        int2 pr = cand[c];
        Tri<T> a = load_tri(tri, pr.x), b = load_tri(tri, pr.y);
        bool keep = sat(a, b, th) && !(count_shared(a, b) > 0);
        if (keep) {
            OutRegion R = out_region(F, M, pr.x, max_per_tri);
            long long r = append_row(mesh_counters, F, R.m, R.cap, &hdr->status);
            if (r >= 0) {
                long long o = (long long)R.po * max_per_tri + r;
                rows[o * 2 + 0] = pr.x - R.po;
                rows[o * 2 + 1] = pr.y - R.po;
            }
        }
    }
}

// find_triangle_edge_collisions (OP 0), _candidates (OP 1), _candidates2 (OP 2)
// (collisions_static.cu:588-942, icontour.cu:113-281): candidate pairs that intersect
// (separating axes, threshold 0) and share at most one vertex (none for OP 0), then the six
// edge sub-tests of each pair.  OP 0 / 1 append a row (i, j, cid, flag) per listed sub-test
// (OP 0 with the edge coefficient); OP 2 appends one row (i, j) per pair with its masks
// (bit cid set in x when the sub-test is listed, in y when it is a loop node).
// A lane's own six sub-tests one after the other ran with one or two lanes of a warp (one pair in
// 40 meets); they go to a lane each instead, and the pairs that share too many vertices, half of
// them on a mesh, end before the separating axes: 19.6 -> 11.3 us for 90,560 pairs of 10,952
// triangles (fp64), most of it now the latency of the separating axes.
enum TeOp { TE_COLLISIONS = 0, TE_CANDIDATES = 1, TE_CANDIDATES2 = 2 };

template <class T, int OP, int LIB>
__global__ void __launch_bounds__(NARROW_THREADS)
k_te_narrow(const int2* __restrict__ cand, int cand_cap, WsHeader* hdr, const T* __restrict__ tri, Forest F,
            long long* __restrict__ rows, T* __restrict__ coefs, int* __restrict__ masks, int max_per_tri,
            int* __restrict__ mesh_counters) {
    chain_begin();
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int M = forest_size(F);
    const int n = min(hdr->cand_count, cand_cap);
    const int step = gridDim.x * blockDim.x;
    const int group = lane / 6, cid = lane - 6 * group;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c - lane < n; c += step) {
        int2 pr = make_int2(0, 0);
        bool meets = false;
        if (c < n) {
            pr = cand[c];
            const Tri<T> a = load_tri(tri, pr.x), b = load_tri(tri, pr.y);
            meets = !(count_shared(a, b) > (OP == TE_COLLISIONS ? 0 : 1)) && sat(a, b, (T)0);
        }
        // five pairs at a time, a lane for each of their sub-tests
        for (unsigned pairs = __ballot_sync(FULL, meets); pairs;) {
            int own = -1;
            for (int g = 0; g < 5 && pairs; ++g, pairs &= pairs - 1)
                if (g == group) own = __ffs(pairs) - 1;
            const int i = __shfl_sync(FULL, pr.x, max(own, 0)), j = __shfl_sync(FULL, pr.y, max(own, 0));
            bool listed = false, node = false;
            int flag = -1;
            T coef = (T)-1;
            if (own >= 0) {
                Tri<T> face;
                V3<T> p0, p1;
                int e;
                te_edge(load_tri(tri, i), load_tri(tri, j), cid, face, p0, p1, e);
                if (OP == TE_COLLISIONS) {
                    listed = te_intersect<T, LIB>(face, p0, p1, cid, flag, coef);
                } else {
                    const int r = te_candidate(face, p0, p1, cid, e);
                    listed = r != 0;
                    node = (r & 2) != 0;
                    flag = node ? 0 : -1;
                }
            }
            if (OP == TE_CANDIDATES2) {
                const unsigned mx = __ballot_sync(FULL, listed), my = __ballot_sync(FULL, node);
                if (own >= 0 && cid == 0) {
                    const OutRegion R = out_region(F, M, i, max_per_tri);
                    const long long r = append_row(mesh_counters, F, R.m, R.cap, &hdr->status);
                    if (r >= 0) {
                        const long long o = (long long)R.po * max_per_tri + r;
                        rows[o * 2 + 0] = i - R.po;
                        rows[o * 2 + 1] = j - R.po;
                        masks[o * 2 + 0] = (int)(mx >> lane & 63u);
                        masks[o * 2 + 1] = (int)(my >> lane & 63u);
                    }
                }
            } else if (listed) {
                const OutRegion R = out_region(F, M, i, max_per_tri);
                const long long r = append_row(mesh_counters, F, R.m, R.cap, &hdr->status);
                if (r >= 0) {
                    const long long o = (long long)R.po * max_per_tri + r;
                    rows[o * 4 + 0] = i - R.po;
                    rows[o * 4 + 1] = j - R.po;
                    rows[o * 4 + 2] = cid;
                    rows[o * 4 + 3] = flag;
                    if (OP == TE_COLLISIONS) coefs[o] = coef;
                }
            }
        }
    }
}

// what becomes of a root that passes the filter: a row of find_collisions_continuous, or a
// contact whose impulses go to a sink
enum CcdMode { CCD_ROWS = 0, CCD_IMPULSES = 1 };
// where the continuous narrow phase takes its pairs and their sub-tests from: the candidate
// buffer with the masks that k_ccd_mask left in it (reference-format operations), or the
// engine's list of pairs with work (the collision step's shared sub-tests, k_ccd_stage_*, or
// the impulse loop's, k_ccd_mask)
enum CcdSource { SRC_PACKED = 0, SRC_STAGED = 1 };

// Receiver of the impulses of CCD_IMPULSES: per-corner sums and counters (F, 3, 3) / (F, 3)
// of the reference's compute_impulses.  Per-corner masses (F, 3) feed the contact.
template <class T> struct CornerSink {
    const T* masses;
    T* dv;
    T* dx;
    int* cnt;
    __device__ __forceinline__ void add(const MTet<T>& tet, long long gi, long long gj, int k, T root,
                                        const Contact<T>& ct, const Forest&, int, int*) const {
        apply_impulse(tet, gi, gj, k, root, ct, dv, dx, cnt);
    }
    // The contacts of a warp's lanes (of those with `valid`), all lanes taking part: the three
    // components of a point are added by neighbouring lanes, so that an instruction touches
    // some 16 sectors instead of 32.  What bounds k_ccd_contacts is those sectors in L2: 523 k
    // contacts (fp64) 82 -> 52 us, 34 k listed ones (fp32) 7.4 -> 5.4 us.
    static constexpr int MIN_BLOCKS = 1;    // k_ccd_contacts: 3 or 4 a SM (168, 128 registers) 55 us
    struct Points {
        T v[32 * 7];            // change of velocity and of position per lane, odd stride
        long long at[32];
    };
    __device__ __forceinline__ void add_all(bool valid, const MTet<T>& tet, long long gi, long long gj, int k, T root,
                                            const Contact<T>& ct, const Forest&, int, int*, Points& S) const {
        const int lane = threadIdx.x & 31;
        ImpulseScale<T> sc;
        if (valid) sc = impulse_scale(ct, root);
#pragma unroll
        for (int pt = 0; pt < 4; ++pt) {
            long long corner = -1;
            if (valid) {
                V3<T> imp, idx;
                impulse_point(tet, k, pt, ct, sc, imp, idx);
                corner = (tet_side(k, pt) ? gj : gi) * 3 + tet_corner(k, pt);
                T* v = S.v + 7 * lane;
                v[0] = imp.x; v[1] = imp.y; v[2] = imp.z;
                v[3] = idx.x; v[4] = idx.y; v[5] = idx.z;
                atomicAdd(cnt + corner, 1);
            }
            S.at[lane] = corner;
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const int l = (lane + 32 * r) / 3, d = lane + 32 * r - 3 * l;
                const long long at = S.at[l];
                if (at >= 0) {
                    atomicAdd(dv + at * 3 + d, S.v[7 * l + d]);
                    atomicAdd(dx + at * 3 + d, S.v[7 * l + 3 + d]);
                }
            }
            __syncwarp();
        }
    }
};

// Continuous narrow phase (collisions_continuous.cu:14-765, collisions_impulses.cu:24-1067),
// block-synchronous: blocks of CCD_BLOCK threads take CCD_BLOCK pairs at a time and queue
// their sub-tests, and each stage of the solve runs on a full block of its own queue's
// entries, so that every warp of the block runs the same stage's code at the same time:
//   (1) the cubic's coefficients; sub-tests that for certain have no root in [0, 1]
//       (cubic_misses) or none that passes the filter (roots_fail) end here, the others are queued
//       with their coefficients;
//   (2) the solver prefix, which classifies them, and the roots, ordered by solver branch; the
//       roots in [0, 1] are queued, edge-edge ones from the front of their array and
//       vertex-face ones from its back;
//   (3) the root filter, a warp at a time of one kind of root; the roots that pass leave a
//       record (or, for the reference's rows, a row).
// Sub-tests take different branches and have 0 to 3 roots: solved in arrival order they
// leave most lanes idle, and a kernel whose warps are in different stages needs all of its
// code in the instruction cache at once.  A stage that took only what the stage before it
// left of its batch would run with most of its threads idle between two barriers: on the
// 256 x 256 fold, three sub-tests in four have no root in [0, 1].
// Measured against one kernel that staged, solved and applied a batch from end to end (fp64):
// the fold's impulses 1,698 -> 109 (masks) + 752 + 82 us (contacts), ten served folds 931 ->
// 94 + 445 + 39 us an iteration, the cloth over the sphere 214 -> 21 + 161 us, 968 triangles
// 45 -> 5 + 15 + 6 us; the 64-mesh step, whose masks were apart already, 5,336 -> 4,950 us.
// roots_fail on top of that: the 64 meshes 4,913 -> 4,119 us, ten served folds 5,339 -> 4,813 us in
// all, 12 meshes 303 -> 249 us, the cloth over the sphere 159 -> 138 us, the fold the same (750 us:
// what it saves there it costs, most of it conversions to fp32 at 8 cycles a warp).
// What bounds it: instruction issue (52-57 % of the slots at 26-28 of 32 lanes; before roots_fail
// some 2,100 instructions per 32 sub-tests, a quarter of them in the FP64 pipe), with waits for fixed
// latencies 2.6, barriers 2.0 and memory 1.6-2.6 warps an issue.  Blocks of 128 threads: 5,219
// against 5,168 us on the 64 meshes, 801 against 759 us on the fold (before roots_fail).
static constexpr int CCD_BLOCK = 256;
// resident blocks per SM (80 registers a thread, 54 KB of shared memory a block); four of 64
// registers spill in roots_fail: 4,637 us on the 64 meshes, 793 us on the fold
constexpr int ccd_min_blocks(int bm) { return bm == 1 ? 3 : 2; }
static_assert(CCD_BLOCK % 32 == 0 && CCD_BLOCK <= 1024, "CCD_BLOCK");

constexpr size_t align16(size_t x) { return (x + 15) / 16 * 16; }

// dynamic shared memory of one block (byte offsets) for batches of NB sub-tests
template <class T, int NB> struct CcdLayout {
    static constexpr int ITEMS = NB + 3 * CCD_BLOCK;      // less than a batch, and an intake
    static constexpr int SURV = 2 * NB;                   // less than a batch, and a batch
    // less than a round of warps and two partial ones, and three roots of a batch
    static constexpr int ROOTS = 3 * NB + CCD_BLOCK + 32;
    static constexpr int OUT = CCD_BLOCK;
    static constexpr size_t coef = 0;                                                  // double [4][SURV]
    static constexpr size_t gh = coef + 4 * SURV * sizeof(double);                     // double [2][NB]
    static constexpr size_t out = gh + 2 * NB * sizeof(double);                        // int4 [OUT]
    static constexpr size_t root_val = out + OUT * sizeof(int4);                       // T [ROOTS]
    static constexpr size_t root_item = align16(root_val + ROOTS * sizeof(T));         // int2 [ROOTS]
    static constexpr size_t items = root_item + ROOTS * sizeof(int2);                  // int2 [ITEMS]
    static constexpr size_t surv = items + ITEMS * sizeof(int2);                       // int2 [SURV]
    static constexpr size_t clist = surv + SURV * sizeof(int2);                        // u16 [NB]
    static constexpr size_t pos = clist + NB * 2;                                      // u16 [NB]
    static constexpr size_t cls = pos + NB * 2;                                        // u8 [NB]
    static constexpr size_t ints = align16(cls + NB);                                  // int [64]
    static constexpr size_t bytes = ints + 64 * sizeof(int);
    static_assert(NB <= 65536, "batch indices are 16-bit");
};

// slots of the small int area: the intake's warp counts and total; the survivors queued since
// the kernel began; the solver classes' counts (two sets, used by alternate batches); the
// queued roots of each kind; the buffered records and where they go
enum CcdInts { CI_WARP = 0, CI_TOTAL = 32, CI_SURV = 33, CI_COUNT = 34, CI_EE = 42, CI_VF = 43, CI_OUT = 44, CI_BASE = 45 };

// a queued sub-test: triangle slots i and j, type k in the top bits of j (slots < 2^28),
// bit 28 of i set when the sub-test stands for all its repeats (see Weld)
constexpr int SLOT_MASK = 0x0fffffff;
__device__ __forceinline__ int2 pack_subtest(int i, int j, int k, int shared = 0) {
    return make_int2(i | (shared << 28), j | (k << 28));
}

// Repeated sub-tests (resident engine only).  On a mesh a vertex-face sub-test (v, face B)
// is the sub-test of every pair (A', B) whose triangle A' has a corner at v, and an
// edge-edge sub-test belongs to every pair of triangles carrying the two edges with their
// corners in the same order: the tetrahedra are bit for bit the same, and so are their
// roots, filter decisions and contacts.  The pairs that produce one of them are known from
// the corner classes alone:
//  * the corners of a mesh whose start positions are equal (==, the reference's
//    shared-vertex relation, figures.cu:527-544) form a class; a pair shares a vertex
//    exactly when its triangles have a class in common;
//  * every such pair is live (shares no vertex), is a candidate pair of the reference (a
//    vertex's swept sub-box lies in its triangle's leaf box, the merge of the triangle's
//    boxes at both ends of the step, when x0 + (x1 - x0) == x1 for its coordinates), and
//    has the sub-test's sub-box bit (the boxes of the same points);
//  * for vertex-face types 12..14 (vertex of the first triangle) they are the pairs
//    (A', B) with A' < B over the class's corners, for 9..11 the pairs (A, B') with
//    B' > A; for edge-edge types the pairs over each edge and its twin, the other
//    triangle edge whose corners are the same classes in the same order.
// The smallest of those (slot, slot, type) triples solves the sub-test and emits the rows
// or contacts of all of them; the others drop it.  A class is excluded (CLS_NODEDUP) when
// its corners are not bit-identical at both ends of the step, when x0 + (x1 - x0) != x1 for
// one of its coordinates, or when it has more than WELD_FANCAP corners; an edge with more
// than one twin is excluded too.  A sub-test touching an excluded class or edge is solved
// by each of its pairs, as without the classes.  Every pair finds the same members, so
// each repeat is solved exactly once.  Pairs with a rigid motion have no sub-test with a
// root (ccd_pair_subbox_mask), so it does not matter which of them is the smallest.
constexpr int CLS_MASK = (1 << 30) - 1;
constexpr int CLS_NODEDUP = 1 << 30;
constexpr int TWIN_NONE = -1, TWIN_MANY = -2;
constexpr int WELD_FANCAP = 16;
struct Weld {
    const int4* vid;       // per triangle slot: the class of each corner (its first entry in
                           // fan) | CLS_NODEDUP; in w the three class sizes (bits 5c..5c+4,
                           // sizes above 31 as 31) and whether each edge e has no twin, one
                           // or more (bits 15+2e..16+2e: 0, 1, 2); null: no classes
    const int4* fan;       // the classes' members, class by class in ascending corner id:
                           // (corner id 4 * slot + corner, the classes of its triangle)
    const int4* twin;      // per triangle slot and edge {01, 02, 12}: 4 * slot + edge of its
                           // twin, TWIN_NONE or TWIN_MANY
    const int4* third;     // per triangle slot and edge: the class of the twin's third corner
    const int4* live;      // the pairs with sub-tests to solve (hdr->live_count of them, from
                           // k_ccd_stage_*): slots i, j and the sub-tests it solves (bits
                           // 0..14) with those that stand for their repeats (bits 15..29)
    int4* expand;          // the roots that passed the filter, for k_ccd_expand or
                           // k_ccd_contacts (hdr->expand_count, at most expand_cap): slots
                           // i | shared << 28, j | type << 28, the root as a double (low, high
                           // words)
    int expand_cap;
};

__device__ __forceinline__ int int4_at(int4 v, int c) { return c == 0 ? v.x : (c == 1 ? v.y : v.z); }
__device__ __forceinline__ bool classes_meet(int4 a, int4 b) {
    const int a0 = a.x & CLS_MASK, a1 = a.y & CLS_MASK, a2 = a.z & CLS_MASK;
    const int b0 = b.x & CLS_MASK, b1 = b.y & CLS_MASK, b2 = b.z & CLS_MASK;
    return a0 == b0 || a0 == b1 || a0 == b2 || a1 == b0 || a1 == b1 || a1 == b2 || a2 == b0 || a2 == b1 ||
           a2 == b2;
}
__device__ __forceinline__ int class_size(int4 v, int c) { return (v.w >> (5 * c)) & 31; }
__device__ __forceinline__ int twin_kind(int4 v, int e) { return (v.w >> (15 + 2 * e)) & 3; }

// The edge-edge pairs of sub-test 3e + f of pair (A, B): over the edges' twins ta, tb
// (4 * slot + edge, or TWIN_NONE) whose third corners have classes ha, hb, the pairs
// (a < b) that share no vertex, the pair itself first.
template <class Fn>
__device__ __forceinline__ void weld_ee_members(int A, int B, int e, int f, int4 VA, int4 VB, int ta, int tb, int ha,
                                                int hb, Fn&& fn) {
    // edge {01, 02, 12}[e]: corners e > 1 ? 1 : 0 and e > 0 ? 2 : 1
    const int4 TA = make_int4(int4_at(VA, e > 1), int4_at(VA, e > 0 ? 2 : 1), ha, 0);
    const int4 TB = make_int4(int4_at(VB, f > 1), int4_at(VB, f > 0 ? 2 : 1), hb, 0);
    for (int i = 0; i < 2; ++i) {
        if (i == 1 && ta < 0) break;
        const int a = i ? ta >> 2 : A, sa = i ? ta & 3 : e;
        for (int j = 0; j < 2; ++j) {
            if (j == 1 && tb < 0) break;
            const int b = j ? tb >> 2 : B, sb = j ? tb & 3 : f;
            if (a >= b) continue;
            if ((i | j) && classes_meet(i ? TA : VA, j ? TB : VB)) continue;
            fn(a, b, 3 * sa + sb);
        }
    }
}

// Calls fn(a, b, type) for every pair that has sub-test k of pair (A, B) (A < B, live), the
// pair itself included, and returns true; returns false without a call when the sub-test
// is solved by each of its pairs.  VA, VB: W.vid[A], W.vid[B].
template <class Fn>
__device__ __forceinline__ bool weld_members(const Weld& W, int A, int B, int k, int4 VA, int4 VB, Fn&& fn) {
    if (k >= 9) {
        const bool vf = k >= 12;                 // vertex of A, face of B (else face of A)
        const int4 Vface = vf ? VB : VA;
        const int4 Vvert = vf ? VA : VB;
        const int c = vf ? k - 12 : k - 9;
        const int v = int4_at(Vvert, c);
        // (a class of one corner: the pair is the sub-test's only one)
        if (((v | Vface.x | Vface.y | Vface.z) & CLS_NODEDUP) || class_size(Vvert, c) < 2) return false;
        const int end = v + class_size(Vvert, c);
        for (int i = v; i < end; ++i) {
            const int4 en = __ldg(W.fan + i);
            const int t = en.x >> 2, cc = en.x & 3;
            if (vf ? t >= B : t <= A) continue;
            if (classes_meet(make_int4(en.y, en.z, en.w, 0), Vface)) continue;
            if (vf) fn(t, B, 12 + cc);
            else fn(A, t, 9 + cc);
        }
        return true;
    }
    const int e = k / 3, f = k - 3 * e;
    // (edges without a twin: the pair is the sub-test's only one)
    const int ka = twin_kind(VA, e), kb = twin_kind(VB, f);
    if (ka == 2 || kb == 2 || (ka | kb) == 0) return false;
    if ((int4_at(VA, e > 1) | int4_at(VA, e > 0 ? 2 : 1) | int4_at(VB, f > 1) | int4_at(VB, f > 0 ? 2 : 1)) &
        CLS_NODEDUP)
        return false;
    weld_ee_members(A, B, e, f, VA, VB, ka ? int4_at(__ldg(W.twin + A), e) : TWIN_NONE,
                    kb ? int4_at(__ldg(W.twin + B), f) : TWIN_NONE, ka ? int4_at(__ldg(W.third + A), e) : 0,
                    kb ? int4_at(__ldg(W.third + B), f) : 0, fn);
    return true;
}

// Whether pair (A, B) solves its shared vertex-face sub-test k, that is whether it is the smallest
// of the sub-test's pairs.  The members of a class are in ascending corner id, so the scan stops
// at the first pair that has the sub-test.
__device__ __forceinline__ bool weld_vf_solves(const Weld& W, int A, int B, int k, int4 VA, int4 VB) {
    const bool vf = k >= 12;                     // vertex of A, face of B (else face of A)
    const int4 Vface = vf ? VB : VA;
    const int4 Vvert = vf ? VA : VB;
    const int c = vf ? k - 12 : k - 9;
    const int v = int4_at(Vvert, c), end = v + class_size(Vvert, c), own = 4 * (vf ? A : B) + c;
    for (int i = v; i < end; ++i) {
        const int4 en = __ldg(W.fan + i);
        if (en.x == own) return true;            // (none before it)
        if (!vf && (en.x >> 2) <= A) continue;
        if (!classes_meet(make_int4(en.y, en.z, en.w, 0), Vface)) return false;
    }
    return true;    // (not reached: the pair itself has the sub-test)
}

// The pairs of sub-test k of pair (A, B) in (ma, mb, mk), at most WELD_FANCAP of them (a
// shared vertex-face sub-test has one per corner of its class, an edge-edge one at most
// four); the pair alone when the sub-test is not shared.  Returns their number.
__device__ __forceinline__ int weld_list(const Weld& W, int A, int B, int k, bool shared, int* ma, int* mb, int* mk) {
    int n = 0;
    if (shared)
        weld_members(W, A, B, k, __ldg(W.vid + A), __ldg(W.vid + B), [&](int a, int b, int kk) {
            if (n < WELD_FANCAP) {
                ma[n] = a;
                mb[n] = b;
                mk[n] = kk;
                ++n;
            }
        });
    if (n == 0) {
        ma[0] = A;
        mb[0] = B;
        mk[0] = k;
        n = 1;
    }
    return n;
}

__device__ __forceinline__ int warp_inclusive_scan(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// Row reservation for the lanes of mask, which call it together: each lane's nm rows in the
// region of its mesh m, with one atomic per mesh among them; returns the lane's first row
// (its prefix of the counts of the lanes in its mesh).  A whole warp in one mesh, the usual
// case, takes plain warp scans.
__device__ __forceinline__ int reserve_rows(int* mesh_counters, const Forest& F, int m, int nm, unsigned mask) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    __syncwarp(mask);
    if (mask == FULL && __all_sync(FULL, m == __shfl_sync(FULL, m, 0))) {
        const int incl = warp_inclusive_scan(nm, lane);
        int base = 0;
        if (lane == 31) base = atomicAdd(mesh_counters + __ldg(F.sid + m), incl);
        return __shfl_sync(FULL, base, 31) + incl - nm;
    }
    cg::coalesced_group g = cg::labeled_partition(cg::coalesced_threads(), m);
    const int before = cg::exclusive_scan(g, nm);
    const int all = cg::reduce(g, nm, cg::plus<int>());
    int base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(mesh_counters + __ldg(F.sid + m), all);
    return g.shfl(base, 0) + before;
}

// Staging of the resident engine's candidate pairs for k_ccd_narrow: the list Weld.live of
// the pairs with sub-tests to solve, in two kernels.
//  * k_ccd_stage_mask: pairs whose triangles share a vertex (a corner class in common, the
//    same relation as the reference's coordinate test) are dropped; the others queue per
//    warp in shared memory and are taken 32 at a time, for the sub-box mask with the exact
//    leaf-box test (the engine's candidates come from fp32 boxes rounded outward) and the
//    choice of the pair that solves each sub-test wherever the triangles' own records tell
//    it: every edge-edge sub-test (classes, twins and the twins' third corners) and the
//    vertex-face sub-tests that are not shared.  A pair left with shared vertex-face
//    sub-tests goes to the pending list, the others with work to the live list.
//    hdr->subtests counts the sub-tests of the masks.
//  * k_ccd_stage_pending: the pending pairs' vertex-face sub-tests, spread over the lanes
//    of a warp (a scan of the vertex's class each); then the pairs go to the live list.
//    (Each pair's lane lists its sub-tests; a search for the pair and the n-th bit by each
//    taking lane cost more than the scans: 765 -> 460 us on the 64-mesh step.)
// Records: (slot i, slot j, the sub-tests to solve in bits 0..14 with the shared ones in
// bits 15..29, pending vertex-face sub-tests).
static constexpr int STAGE_THREADS = 256;
static constexpr int STAGE_WARPS = STAGE_THREADS / 32;

// The edge-edge sub-tests among bits 0..8 of ee that pair (A, B) solves, from the records of A
// and B: those that are not shared, and the shared ones of which (A, B) is the smallest pair
// (weld_ee_members).  *shared: the shared ones among them.  All nine at once: a smaller pair is
// over the twin of A's edge (if that twin's triangle is before A) with B or with the twin of
// B's edge, or over A with the twin of B's edge, and whether such a pair shares a vertex depends
// on the twin's third corner only, not on the other edge.  One sub-test after the other took
// half of k_ccd_stage_mask (2,700 instructions per 32 pairs with 18 lanes active): 1,930 -> 978 us
// on the 64-mesh step, 118 -> 68 us on 12 meshes.
__device__ __forceinline__ unsigned weld_ee_choice(int A, int B, unsigned ee, int4 VA, int4 VB, int4 TWA, int4 TWB,
                                                   int4 THA, int4 THB, unsigned* shared) {
    // edges of A and B whose sub-tests may be shared, and those of them with a twin
    unsigned oka = 0, okb = 0, ta = 0, tb = 0;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const int c0 = e > 1, c1 = e > 0 ? 2 : 1;          // edge {01, 02, 12}[e]
        const int ka = twin_kind(VA, e), kb = twin_kind(VB, e);
        const bool fa = ka != 2 && !((int4_at(VA, c0) | int4_at(VA, c1)) & CLS_NODEDUP);
        const bool fb = kb != 2 && !((int4_at(VB, c0) | int4_at(VB, c1)) & CLS_NODEDUP);
        oka |= fa ? 1u << e : 0u;
        okb |= fb ? 1u << e : 0u;
        ta |= fa && ka == 1 ? 1u << e : 0u;
        tb |= fb && kb == 1 ? 1u << e : 0u;
    }
    // bit 3 e + f of edge e of A and edge f of B
    auto rows = [](unsigned x) { return (x & 1u ? 0x7u : 0u) | (x & 2u ? 0x38u : 0u) | (x & 4u ? 0x1c0u : 0u); };
    auto cols = [](unsigned x) { return x | (x << 3) | (x << 6); };
    const unsigned sh = ee & rows(oka) & cols(okb) & (rows(ta) | cols(tb));
    *shared = 0u;
    if (!sh) return ee;
    unsigned lost = 0;          // sub-tests that a smaller pair has
    bool own = false;           // a twin on the triangle itself (a degenerate triangle)
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const int c0 = e > 1, c1 = e > 0 ? 2 : 1;
        const int t = int4_at(TWA, e) >> 2;
        const bool has = ta >> e & 1u;
        own = own || (has && t == A);
        if (has && t < A && (sh & (7u << (3 * e)))) {
            const int4 TA = make_int4(int4_at(VA, c0), int4_at(VA, c1), int4_at(THA, e), 0);
            if (!classes_meet(TA, VB)) {
                lost |= 7u << (3 * e);
            } else {
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                    const int d0 = f > 1, d1 = f > 0 ? 2 : 1;
                    const int u = int4_at(TWB, f) >> 2;
                    if ((tb >> f & 1u) && t < u &&
                        !classes_meet(TA, make_int4(int4_at(VB, d0), int4_at(VB, d1), int4_at(THB, f), 0)))
                        lost |= 1u << (3 * e + f);
                }
            }
        }
        const int u = int4_at(TWB, e) >> 2;
        const bool hasb = tb >> e & 1u;
        own = own || (hasb && u == B);
        if (hasb && u < B && u > A && (sh & (0x49u << e)) &&
            !classes_meet(VA, make_int4(int4_at(VB, c0), int4_at(VB, c1), int4_at(THB, e), 0)))
            lost |= 0x49u << e;
    }
    if (own) {
        // pairs that differ in the sub-test's type only: each one by the full comparison
        lost = 0;
        for (unsigned x = sh; x; x &= x - 1) {
            const int k = __ffs(x) - 1, e = k / 3, f = k - 3 * e;
            weld_ee_members(A, B, e, f, VA, VB, ta >> e & 1u ? int4_at(TWA, e) : TWIN_NONE,
                            tb >> f & 1u ? int4_at(TWB, f) : TWIN_NONE, int4_at(THA, e), int4_at(THB, f),
                            [&](int a, int b, int kk) {
                                if (a < A || (a == A && (b < B || (b == B && kk < k)))) lost |= 1u << k;
                            });
        }
    }
    *shared = sh & ~lost;
    return ee & ~(sh & lost);
}

// the corners of V's triangle whose class has more than one corner, none excluded (bit c); the
// vertex-face sub-tests of such a corner are shared when the face's corners are not excluded
__device__ __forceinline__ unsigned weld_shared_corners(int4 V) {
    return (!(V.x & CLS_NODEDUP) && class_size(V, 0) >= 2 ? 1u : 0u) |
           (!(V.y & CLS_NODEDUP) && class_size(V, 1) >= 2 ? 2u : 0u) |
           (!(V.z & CLS_NODEDUP) && class_size(V, 2) >= 2 ? 4u : 0u);
}

// a record to the live list (work, no pending) or the pending list, warp-aggregated
__device__ __forceinline__ void stage_emit(WsHeader* hdr, int4* live, int4* pending, int2 pr, unsigned word,
                                           unsigned pend, bool valid) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const bool to_live = valid && pend == 0u && word != 0u, to_pend = valid && pend != 0u;
    const unsigned ml = __ballot_sync(FULL, to_live), mp = __ballot_sync(FULL, to_pend);
    int bl = 0, bp = 0;
    if (lane == 0 && ml) bl = atomicAdd(&hdr->live_count, __popc(ml));
    if (lane == 0 && mp) bp = atomicAdd(&hdr->pending_count, __popc(mp));
    bl = __shfl_sync(FULL, bl, 0) + __popc(ml & lt);
    bp = __shfl_sync(FULL, bp, 0) + __popc(mp & lt);
    // (at most one record per candidate in either list)
    if (to_live) live[bl] = make_int4(pr.x, pr.y, (int)word, 0);
    if (to_pend) pending[bp] = make_int4(pr.x, pr.y, (int)word, (int)pend);
}

template <class T>
__global__ void __launch_bounds__(STAGE_THREADS, 3)
k_ccd_stage_mask(const int2* __restrict__ cand, int cand_cap, WsHeader* hdr, const T* __restrict__ x0,
                 const T* __restrict__ x1, Weld W, int4* __restrict__ live, int4* __restrict__ pending) {
    chain_begin();
    __shared__ int2 q_pr[STAGE_WARPS][64];
    __shared__ int4 q_va[STAGE_WARPS][64], q_vb[STAGE_WARPS][64];
    const int n = min(*(volatile int*)&hdr->cand_count, cand_cap);
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int warps = gridDim.x * STAGE_WARPS;
    int masked = 0, qn = 0;             // qn: queued live pairs of this warp (warp-uniform)
    for (int base = (blockIdx.x * STAGE_WARPS + wq) * 32;; base += warps * 32) {
        const bool more = base < n;
        if (!more && qn == 0) break;
        if (more) {
            const int c = base + lane;
            int2 pr = make_int2(0, 0);
            int4 VA = make_int4(0, 0, 0, 0), VB = VA;
            bool lv = false;
            if (c < n) {
                pr = cand[c];
                VA = __ldg(W.vid + pr.x);
                VB = __ldg(W.vid + pr.y);
                lv = !classes_meet(VA, VB);
            }
            const unsigned m = __ballot_sync(FULL, lv);
            if (lv) {
                const int at = qn + __popc(m & lt);
                q_pr[wq][at] = pr;
                q_va[wq][at] = VA;
                q_vb[wq][at] = VB;
            }
            qn += __popc(m);
            __syncwarp();
        }
        while (qn >= 32 || (!more && qn > 0)) {
            const bool valid = lane < qn;
            int2 pr = make_int2(0, 0);
            unsigned word = 0u, pend = 0u;
            if (valid) {
                pr = q_pr[wq][lane];
                const int4 VA = q_va[wq][lane], VB = q_vb[wq][lane];
                const unsigned bits = ccd_pair_subbox_mask<T, true, true>(x0, x1, pr.x, pr.y);
                masked += __popc(bits);
                const unsigned ee = bits & 0x1ffu;
                int4 TWA = make_int4(0, 0, 0, 0), TWB = TWA, THA = TWA, THB = TWA;
                if (ee && ((VA.w | VB.w) >> 15)) {
                    TWA = __ldg(W.twin + pr.x);
                    TWB = __ldg(W.twin + pr.y);
                    THA = __ldg(W.third + pr.x);
                    THB = __ldg(W.third + pr.y);
                }
                unsigned shared;
                word = weld_ee_choice(pr.x, pr.y, ee, VA, VB, TWA, TWB, THA, THB, &shared);
                const bool fa = !((VA.x | VA.y | VA.z) & CLS_NODEDUP), fb = !((VB.x | VB.y | VB.z) & CLS_NODEDUP);
                pend = bits & ((fa ? weld_shared_corners(VB) << 9 : 0u) | (fb ? weld_shared_corners(VA) << 12 : 0u));
                word |= (bits & 0x7e00u & ~pend) | (shared << 15);
            }
            stage_emit(hdr, live, pending, pr, word, pend, valid);
            // the queue's second half moves to the front
            __syncwarp();
            if (lane + 32 < qn) {
                q_pr[wq][lane] = q_pr[wq][lane + 32];
                q_va[wq][lane] = q_va[wq][lane + 32];
                q_vb[wq][lane] = q_vb[wq][lane + 32];
            }
            qn = qn > 32 ? qn - 32 : 0;
            __syncwarp();
        }
    }
    masked = __reduce_add_sync(FULL, masked);
    if (lane == 0 && masked) atomicAdd(&hdr->subtests, masked);
}

static __global__ void __launch_bounds__(STAGE_THREADS, 8)
k_ccd_stage_pending(int cand_cap, WsHeader* hdr, Weld W, const int4* __restrict__ pending, int4* __restrict__ live) {
    chain_begin();
    // per warp: 32 pending pairs, their classes, the sub-tests they solve, and their pending
    // sub-tests (lane of the pair << 4 | type) one after the other; the lanes take those 32 at a
    // time
    __shared__ int2 s_pr[STAGE_THREADS];
    __shared__ int4 s_va[STAGE_THREADS], s_vb[STAGE_THREADS];
    __shared__ unsigned s_word[STAGE_THREADS];
    __shared__ unsigned short s_item[STAGE_WARPS][6 * 32];
    const int n = min(*(volatile int*)&hdr->pending_count, cand_cap);
    const int tid = threadIdx.x, lane = tid & 31, w0 = tid & ~31, wq = tid >> 5;
    const unsigned FULL = 0xffffffffu;
    const int warps = gridDim.x * STAGE_WARPS;
    for (int base = (blockIdx.x * STAGE_WARPS + wq) * 32; base < n; base += warps * 32) {
        const int c = base + lane;
        unsigned pend = 0u, word = 0u;
        int2 pr = make_int2(0, 0);
        if (c < n) {
            const int4 rec = pending[c];
            pr = make_int2(rec.x, rec.y);
            word = (unsigned)rec.z;
            pend = (unsigned)rec.w & 0x7e00u;        // (types 9 .. 14)
            s_va[tid] = __ldg(W.vid + pr.x);
            s_vb[tid] = __ldg(W.vid + pr.y);
        }
        s_pr[tid] = pr;
        s_word[tid] = word;
        const int incl = warp_inclusive_scan(__popc(pend), lane);
        int at = incl - __popc(pend);
        for (; pend; pend &= pend - 1) s_item[wq][at++] = (unsigned short)(lane << 4 | (__ffs(pend) - 1));
        const int total = __shfl_sync(FULL, incl, 31);
        __syncwarp();
        for (int r = lane; r < total; r += 32) {
            const int item = s_item[wq][r];
            const int p = w0 + (item >> 4), k = item & 15;
            if (weld_vf_solves(W, s_pr[p].x, s_pr[p].y, k, s_va[p], s_vb[p]))
                atomicOr(&s_word[p], (1u << k) | (1u << (15 + k)));
        }
        __syncwarp();
        word = s_word[tid];
        stage_emit(hdr, live, nullptr, pr, word, 0u, c < n);
        __syncwarp();
    }
}

// The sub-tests of every candidate pair of the operations without corner classes: pairs whose
// triangles share a vertex (equal coordinates) have none; the others queue per warp in shared
// memory and are taken 32 at a time for the swept sub-box tests, as in k_ccd_stage_mask (about
// half of the pairs are mesh neighbours, and gathering the rest keeps the warps full).
//  * MASK_PACK: the mask joins its pair in the candidate buffer: bits 0..7 above the first slot,
//    8..14 above the second (slots below 2^24), or in `masks` when that is given;
//  * MASK_LIST: the pairs with sub-tests go to the list `live` (the engine's impulse loop,
//    whose candidates come from fp32 boxes rounded outward: with the exact leaf-box test);
//  * MASK_ROWS: a row (i, j, type) per sub-test (find_mincol_cand).
enum MaskUse { MASK_PACK = 0, MASK_LIST = 1, MASK_ROWS = 2 };
constexpr int PACK_BITS = 24;
constexpr int PACK_MASK = (1 << PACK_BITS) - 1;

template <class T, int USE>
__global__ void __launch_bounds__(STAGE_THREADS, 3)
k_ccd_mask(int2* cand, int cand_cap, WsHeader* hdr, const T* __restrict__ x0, const T* __restrict__ x1,
           unsigned short* __restrict__ masks, int4* __restrict__ live, Forest F, long long* __restrict__ rows,
           int max_per_tri, int* __restrict__ mesh_counters) {
    chain_begin();
    __shared__ int2 q_pr[STAGE_WARPS][64];
    __shared__ int q_at[STAGE_WARPS][64];
    const int n = min(*(volatile int*)&hdr->cand_count, cand_cap);
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int warps = gridDim.x * STAGE_WARPS;
    int masked = 0, qn = 0;             // qn: queued pairs of this warp (warp-uniform)
    for (long long base = (blockIdx.x * STAGE_WARPS + wq) * 32LL;; base += warps * 32LL) {
        const bool more = base < n;
        if (!more && qn == 0) break;
        if (more) {
            const long long c = base + lane;
            int2 pr = make_int2(0, 0);
            bool lv = false;
            if (c < n) {
                pr = cand[c];
                lv = !ccd_pair_shares_vertex<T>(x0, pr.x, pr.y);
                if (USE == MASK_PACK && masks && !lv) masks[c] = 0;
            }
            const unsigned m = __ballot_sync(FULL, lv);
            if (lv) {
                const int at = qn + __popc(m & lt);
                q_pr[wq][at] = pr;
                q_at[wq][at] = (int)c;
            }
            qn += __popc(m);
            __syncwarp();
        }
        while (qn >= 32 || (!more && qn > 0)) {
            const bool valid = lane < qn;
            int2 pr = make_int2(0, 0);
            unsigned bits = 0u;
            if (valid) {
                pr = q_pr[wq][lane];
                bits = ccd_pair_subbox_mask<T, USE != MASK_ROWS, USE == MASK_LIST>(x0, x1, pr.x, pr.y);
                masked += __popc(bits);
                if (USE == MASK_PACK) {
                    const int at = q_at[wq][lane];
                    if (masks) masks[at] = (unsigned short)bits;
                    else if (bits)
                        cand[at] = make_int2(pr.x | (int)((bits & 0xffu) << PACK_BITS),
                                             pr.y | (int)((bits >> 8) << PACK_BITS));
                }
            }
            if (USE == MASK_LIST) {
                // (at most one record per candidate)
                const unsigned ml = __ballot_sync(FULL, bits != 0u);
                int b0 = 0;
                if (lane == 0 && ml) b0 = atomicAdd(&hdr->live_count, __popc(ml));
                b0 = __shfl_sync(FULL, b0, 0) + __popc(ml & lt);
                if (bits) live[b0] = make_int4(pr.x, pr.y, (int)bits, 0);
            }
            if (USE == MASK_ROWS) {
                while (bits) {
                    const int k = __ffs(bits) - 1;
                    bits &= bits - 1;
                    const OutRegion R = out_region(F, forest_size(F), pr.x, max_per_tri);
                    const long long r = append_row(mesh_counters, F, R.m, R.cap, &hdr->status);
                    if (r >= 0) {
                        const long long o = (long long)R.po * max_per_tri + r;
                        rows[o * 3 + 0] = pr.x - R.po;
                        rows[o * 3 + 1] = pr.y - R.po;
                        rows[o * 3 + 2] = k;
                    }
                }
            }
            // the queue's second half moves to the front
            __syncwarp();
            if (lane + 32 < qn) {
                q_pr[wq][lane] = q_pr[wq][lane + 32];
                q_at[wq][lane] = q_at[wq][lane + 32];
            }
            qn = qn > 32 ? qn - 32 : 0;
            __syncwarp();
        }
    }
    if (USE != MASK_ROWS) {
        masked = __reduce_add_sync(FULL, masked);
        if (lane == 0 && masked) atomicAdd(&hdr->subtests, masked);
    }
}

// What k_ccd_narrow and k_ccd_contacts work on.
template <class T> struct CcdArgs {
    const int2* cand;               // SRC_PACKED: the pairs with their masks
    const unsigned short* masks;    // ... null: packed into the pairs
    int cand_cap;
    WsHeader* hdr;
    const T* x0;
    const T* x1;
    Forest F;
    long long* rows;                // CCD_ROWS
    T* times;
    int max_per_tri;
    int* mesh_counters;
    int resident;                   // blocks of k_ccd_narrow that the chip holds at once
    Weld W;                         // live (SRC_STAGED), expand, and the classes when sub-tests are shared
};

// The continuous narrow phase is compiled in one translation unit only, ccc_narrow.cu, with
// nvcc's default multiply-add contraction as the reference is compiled (CUDA's pow, which the
// solver calls, computes slightly different results on rare arguments under -fmad=false);
// every operation of this library's own in it is contraction-proof (mulrn / addrn / subrn,
// fmaT).  The other units see only the launchers' declarations; ccc_narrow.cu instantiates
// the (type, mode, sink, math library) combinations the library launches.
template <class T, int MODE, class Sink, int LIB, int SRC, int BM = 1>
cudaError_t launch_ccd_narrow(int grid, cudaStream_t s, const CcdArgs<T>& A, const Sink& sink);
template <class T, int MODE, class Sink, int LIB, int SRC, int BM = 1> cudaError_t prepare_ccd_narrow();
// the contacts of the records that launch_ccd_narrow<CCD_IMPULSES> left
template <class T, class Sink, int LIB>
cudaError_t launch_ccd_contacts(int grid, cudaStream_t s, const CcdArgs<T>& A, const Sink& sink);

#ifdef CCC_NARROW_TU
// the contact of one root (i, j, type, time)
template <class T, class Sink, int LIB>
__device__ __forceinline__ Contact<T> contact_of_tet(const MTet<T>& tet, const Sink& sink, int i, int j, int k, T root) {
    T mq[4];
#pragma unroll
    for (int pt = 0; pt < 4; ++pt)
        mq[pt] = sink.masses[(long long)(tet_side(k, pt) ? j : i) * 3 + tet_corner(k, pt)];
    return contact<T, LIB>(tet, k, root, mq);
}

// ... and its impulses
template <class T, class Sink, int LIB>
__device__ __forceinline__ void contact_of_root(const CcdArgs<T>& A, const Sink& sink, int i, int j, int k, T root) {
    const MTet<T> tet = load_tet(A.x0, A.x1, i, j, k);
    const Contact<T> ct = contact_of_tet<T, Sink, LIB>(tet, sink, i, j, k, root);
    sink.add(tet, i, j, k, root, ct, A.F, forest_size(A.F), &A.hdr->status);
}

// The consequences of one record in place, for the records that do not fit their list (which
// has room for several a triangle): every row of the root, or its contact.
template <class T, int MODE, class Sink, int LIB>
__device__ __noinline__ void record_in_place(const CcdArgs<T>* A, const Sink* sink, int4 rec) {
    const int qx = rec.x & SLOT_MASK, qy = rec.y & SLOT_MASK, k = (rec.y >> 28) & 15;
    const T root = (T)__hiloint2double(rec.w, rec.z);
    if (MODE == CCD_ROWS) {
        const OutRegion R = out_region(A->F, forest_size(A->F), qx, A->max_per_tri);
        auto row = [&](int a, int b, int kk) {
            const long long r = append_row(A->mesh_counters, A->F, R.m, R.cap, &A->hdr->status);
            if (r >= 0) {
                const long long o = (long long)R.po * A->max_per_tri + r;
                A->rows[o * 3 + 0] = a - R.po;
                A->rows[o * 3 + 1] = b - R.po;
                A->rows[o * 3 + 2] = kk;
                A->times[o] = root;
            }
        };
        const bool shared = (rec.x >> 28) & 1;
        if (!(shared && weld_members(A->W, qx, qy, k, __ldg(A->W.vid + qx), __ldg(A->W.vid + qy), row))) row(qx, qy, k);
    } else {
        contact_of_root<T, Sink, LIB>(*A, *sink, qx, qy, k, root);
    }
}

template <class T, int MODE, class Sink, int LIB, int SRC, int BM>
__global__ void __launch_bounds__(CCD_BLOCK, ccd_min_blocks(BM))
k_ccd_narrow(const __grid_constant__ CcdArgs<T> A, const __grid_constant__ Sink sink) {
    chain_begin();
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int NB = BM * CCD_BLOCK;
    constexpr int NW = CCD_BLOCK / 32;
    using L = CcdLayout<T, NB>;
    double* coef = reinterpret_cast<double*>(smem + L::coef);
    double* gh = reinterpret_cast<double*>(smem + L::gh);
    int4* out = reinterpret_cast<int4*>(smem + L::out);
    T* root_val = reinterpret_cast<T*>(smem + L::root_val);
    int2* root_item = reinterpret_cast<int2*>(smem + L::root_item);
    int2* items = reinterpret_cast<int2*>(smem + L::items);
    int2* surv = reinterpret_cast<int2*>(smem + L::surv);
    unsigned short* clist = reinterpret_cast<unsigned short*>(smem + L::clist);
    unsigned short* cpos = reinterpret_cast<unsigned short*>(smem + L::pos);
    unsigned char* ccls = smem + L::cls;
    int* ints = reinterpret_cast<int*>(smem + L::ints);
    WsHeader* hdr = A.hdr;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned FULL = 0xffffffffu;
    const unsigned lt = (1u << lane) - 1u;
    const int n = min(*(volatile int*)(SRC == SRC_STAGED ? &hdr->live_count : &hdr->cand_count), A.cand_cap);
    // queue fills and positions (block-uniform)
    int ihead = 0, iq = 0;              // sub-tests: ring of ITEMS
    unsigned staken = 0;                // survivors: ring of SURV, taken so far (queued: ints[CI_SURV])
    int sq = 0;
    int nee = 0, nvf = 0;               // roots: edge-edge at [0, nee), vertex-face at [ROOTS - nvf, ROOTS)
    int par = 0;                        // the class counts' set
    int solved = 0, filtered = 0;       // totals of this block
    bool pend = false;                  // sub-tests of the current pairs that found no room yet
    int2 pr = make_int2(0, 0);
    unsigned bits = 0u, shared_bits = 0u;
    if (tid < 64) ints[tid] = 0;
    // pairs of an intake: a whole block's, or fewer when the blocks that run at once would not
    // all have work (a small call's blocks then end after one batch).  Spread over the whole grid
    // of two waves, three meshes' 13,401 pairs took the second wave as well: 23.0 -> 14.9 us.
    const int blocks = min((int)gridDim.x, A.resident);
    const int per = min(CCD_BLOCK, max(16, (int)((n + (long long)blocks - 1) / blocks)));
    // whether the sub-tests' work is worth roots_fail: a block with one short batch only waits for
    // it (968 triangles 14.3 us without, 16.5 us with it)
    const bool ahead = per == CCD_BLOCK;
    long long base = (long long)blockIdx.x * per;

    // a record of a passing root, past the block's buffer: to the list, or in place
    auto put = [&](int4 rec, int at) {
        if (at < A.W.expand_cap) A.W.expand[at] = rec;
        else record_in_place<T, MODE, Sink, LIB>(&A, &sink, rec);
    };
    // the buffered records (block-wide; between barriers)
    auto flush = [&]() {
        const int cnt = min(ints[CI_OUT], L::OUT);
        if (MODE == CCD_ROWS && SRC == SRC_PACKED) {
            // the rows themselves, one a record
            for (int i = tid; i < cnt; i += CCD_BLOCK) {
                const int4 rec = out[i];
                const int qx = rec.x & SLOT_MASK, qy = rec.y & SLOT_MASK;
                const OutRegion R = out_region(A.F, forest_size(A.F), qx, A.max_per_tri);
                const long long r = append_row(A.mesh_counters, A.F, R.m, R.cap, &hdr->status);
                if (r >= 0) {
                    const long long o = (long long)R.po * A.max_per_tri + r;
                    A.rows[o * 3 + 0] = qx - R.po;
                    A.rows[o * 3 + 1] = qy - R.po;
                    A.rows[o * 3 + 2] = (rec.y >> 28) & 15;
                    A.times[o] = (T)__hiloint2double(rec.w, rec.z);
                }
            }
        } else {
            if (tid == 0) ints[CI_BASE] = atomicAdd(&hdr->expand_count, cnt);
            __syncthreads();
            const int b0 = ints[CI_BASE];
            for (int i = tid; i < cnt; i += CCD_BLOCK) put(out[i], b0 + i);
        }
        __syncthreads();
        if (tid == 0) ints[CI_OUT] = 0;
    };

    __syncthreads();
    while (true) {
        // ---- sub-tests of the next pairs, until there is a batch of them
        while (iq < NB && (pend || base < n)) {
            if (!pend) {
                const long long c = base + tid;
                base += (long long)gridDim.x * per;
                bits = shared_bits = 0u;
                if (tid < per && c < n) {
                    if (SRC == SRC_STAGED) {
                        const int4 rec = A.W.live[c];
                        pr = make_int2(rec.x, rec.y);
                        bits = (unsigned)rec.z & 0x7fffu;
                        shared_bits = ((unsigned)rec.z >> 15) & 0x7fffu;
                    } else {
                        pr = A.cand[c];
                        if (A.masks) {
                            bits = A.masks[c];
                        } else {
                            bits = ((unsigned)pr.x >> PACK_BITS) | (((unsigned)pr.y >> PACK_BITS) << 8);
                            pr.x &= PACK_MASK;
                            pr.y &= PACK_MASK;
                        }
                    }
                }
            }
            // (block-wide exclusive scan of the counts)
            const int cnt = __popc(bits);
            const int incl = warp_inclusive_scan(cnt, lane);
            if (lane == 31) ints[CI_WARP + warp] = incl;
            __syncthreads();
            if (warp == 0) {
                const int v = lane < NW ? ints[CI_WARP + lane] : 0;
                const int sc = warp_inclusive_scan(v, lane);
                if (lane < NW) ints[CI_WARP + lane] = sc - v;
                if (lane == 31) ints[CI_TOTAL] = sc;
            }
            __syncthreads();
            const int room = L::ITEMS - iq, total = ints[CI_TOTAL];
            int at = ints[CI_WARP + warp] + incl - cnt;
            while (bits && at < room) {
                const int k = __ffs(bits) - 1;
                bits &= bits - 1;
                items[(ihead + iq + at) % L::ITEMS] = pack_subtest(pr.x, pr.y, k, (shared_bits >> k) & 1u);
                ++at;
            }
            pend = total > room;
            iq += min(total, room);
            __syncthreads();
        }
        const bool drained = !pend && base >= n;         // (block-uniform: base is)
        // ---- (1) coefficients
        if (iq > 0) {
            const int nb = min(NB, iq);
            for (int r0 = 0; r0 < nb; r0 += CCD_BLOCK) {
                const int ri = r0 + tid;
                bool go = false;
                int2 it = make_int2(0, 0);
                T cf[4] = {T(0), T(0), T(0), T(0)};
                if (ri < nb) {
                    it = items[(ihead + ri) % L::ITEMS];
                    const MTet<T> tet = load_tet(A.x0, A.x1, it.x & SLOT_MASK, it.y & SLOT_MASK, (it.y >> 28) & 15);
                    cubic_coeffs(tet, cf);
                    go = !(cf[0] == 0 && cf[1] == 0) &&          // (the linear case has no root that is kept)
                         !cubic_misses<T>((double)cf[0], (double)cf[1], (double)cf[2], (double)cf[3]) &&
                         !(ahead && roots_fail(tet, (it.y >> 28) & 15, cf));
                }
                const unsigned m = __ballot_sync(FULL, go);
                unsigned b0 = 0;
                if (lane == 0 && m) b0 = (unsigned)atomicAdd(&ints[CI_SURV], __popc(m));
                b0 = __shfl_sync(FULL, b0, 0) + __popc(m & lt);
                if (go) {
                    const unsigned slot = b0 % L::SURV;
                    surv[slot] = it;
                    coef[0 * L::SURV + slot] = (double)cf[0];
                    coef[1 * L::SURV + slot] = (double)cf[1];
                    coef[2 * L::SURV + slot] = (double)cf[2];
                    coef[3 * L::SURV + slot] = (double)cf[3];
                }
            }
            solved += nb;
            ihead = (ihead + nb) % L::ITEMS;
            iq -= nb;
            __syncthreads();
            sq = (int)((unsigned)ints[CI_SURV] - staken);
        }
        // ---- (2) solver prefix and roots
        if (sq >= NB || (drained && iq == 0 && sq > 0)) {
            const int nb = min(NB, sq);
            for (int r0 = 0; r0 < nb; r0 += CCD_BLOCK) {
                const int ri = r0 + tid;
                int cls = CUBIC_NONE;
                if (ri < nb) {
                    const unsigned slot = (staken + ri) % L::SURV;
                    double g, h;
                    cls = cubic_prefix<LIB>(coef[0 * L::SURV + slot], coef[1 * L::SURV + slot],
                                            coef[2 * L::SURV + slot], coef[3 * L::SURV + slot], g, h);
                    gh[ri] = g;
                    gh[NB + ri] = h;
                    ccls[ri] = (unsigned char)cls;
                }
                // its place in its class, one atomic a warp and class
#pragma unroll
                for (int c = CUBIC_QUAD; c <= CUBIC_ONE; ++c) {
                    const unsigned m = __ballot_sync(FULL, cls == c);
                    if (!m) continue;
                    int b0 = 0;
                    if (lane == 0) b0 = atomicAdd(&ints[CI_COUNT + 4 * par + c - 1], __popc(m));
                    b0 = __shfl_sync(FULL, b0, 0) + __popc(m & lt);
                    if (cls == c) cpos[ri] = (unsigned short)b0;
                }
            }
            __syncthreads();
            // ordered by class (every thread forms the class offsets itself)
            const int* counts = ints + CI_COUNT + 4 * par;
            const int o1 = counts[0];
            const int o2 = o1 + counts[1];
            const int o3 = o2 + counts[2];
            const int nsolve = o3 + counts[3];
            for (int ri = tid; ri < nb; ri += CCD_BLOCK) {
                const int cls = ccls[ri];
                if (cls != CUBIC_NONE) {
                    const int off = cls == 1 ? 0 : (cls == 2 ? o1 : (cls == 3 ? o2 : o3));
                    clist[off + cpos[ri]] = (unsigned short)ri;
                }
            }
            if (tid < 4) ints[CI_COUNT + 4 * (par ^ 1) + tid] = 0;
            __syncthreads();
            for (int j0 = 0; j0 < nsolve; j0 += CCD_BLOCK) {
                const int j = j0 + tid;
                T rr[3] = {(T)-1, (T)-1, (T)-1};
                int2 it = make_int2(0, 0);
                if (j < nsolve) {
                    const int ri = clist[j];
                    const unsigned slot = (staken + ri) % L::SURV;
                    it = surv[slot];
                    const int cc = (j >= o1) + (j >= o2) + (j >= o3);
                    class_roots<T, LIB>(cc + 1, coef[0 * L::SURV + slot], coef[1 * L::SURV + slot],
                                        coef[2 * L::SURV + slot], coef[3 * L::SURV + slot], gh[ri], gh[NB + ri], rr);
                }
                // (places of the three roots of every lane: one atomic a warp and kind)
                const bool ee = ((it.y >> 28) & 15) < 9;
                const unsigned mee = __ballot_sync(FULL, ee);
                unsigned keep[3];
#pragma unroll
                for (int s = 0; s < 3; ++s)
                    keep[s] = __ballot_sync(FULL, j < nsolve && (rr[s] >= 0 && rr[s] <= 1));
                int ae = 0, af = 0;
                const int ce = __popc(keep[0] & mee) + __popc(keep[1] & mee) + __popc(keep[2] & mee);
                const int ca = __popc(keep[0]) + __popc(keep[1]) + __popc(keep[2]);
                if (lane == 0 && ce) ae = atomicAdd(&ints[CI_EE], ce);
                if (lane == 0 && ca > ce) af = atomicAdd(&ints[CI_VF], ca - ce);
                ae = __shfl_sync(FULL, ae, 0);
                af = __shfl_sync(FULL, af, 0);
#pragma unroll
                for (int s = 0; s < 3; ++s) {
                    const unsigned mine = keep[s] & (ee ? mee : ~mee);
                    if ((keep[s] >> lane) & 1u) {
                        const int before = __popc(mine & lt);
                        const int at = ee ? ae + before : L::ROOTS - 1 - af - before;
                        root_item[at] = it;
                        root_val[at] = rr[s];
                    }
                    ae += __popc(keep[s] & mee);
                    af += __popc(keep[s] & ~mee);
                }
            }
            par ^= 1;
            staken += nb;
            sq -= nb;
            __syncthreads();
            nee = ints[CI_EE];
            nvf = ints[CI_VF];
        }
        // ---- (3) filter: whole rounds of full warps, or all that is left at the end
        const bool last = drained && iq == 0 && sq == 0;
        int we = nee >> 5, wv = nvf >> 5;
        if (last) {
            we = (nee + 31) >> 5;
            wv = (nvf + 31) >> 5;
        } else {
            const int w8 = (we + wv) / NW * NW;
            we = min(we, w8);
            wv = w8 - we;
        }
        if (we + wv > 0) {
            // (units are taken from the ends of the lists, so nothing moves)
            for (int u = warp; u < we + wv; u += NW) {
                const bool ee = u < we;
                const int at = ee ? nee - 1 - 32 * u - lane : L::ROOTS - nvf + 32 * (u - we) + lane;
                const bool valid = ee ? at >= 0 : at < L::ROOTS;
                bool pass = false;
                int4 rec = make_int4(0, 0, 0, 0);
                if (valid) {
                    const int2 it = root_item[at];
                    const T root = root_val[at];
                    const int k = (it.y >> 28) & 15;
                    const MTet<T> tet = load_tet(A.x0, A.x1, it.x & SLOT_MASK, it.y & SLOT_MASK, k);
                    pass = ccd_filter(tet, k, root);
                    const double tw = (double)root;
                    rec = make_int4(it.x, it.y, __double2loint(tw), __double2hiint(tw));
                }
                const unsigned pm = __ballot_sync(FULL, pass);
                int b0 = 0;
                if (lane == 0 && pm) b0 = atomicAdd(&ints[CI_OUT], __popc(pm));
                b0 = __shfl_sync(FULL, b0, 0) + __popc(pm & lt);
                if (pass) {
                    if (b0 < L::OUT) out[b0] = rec;
                    else if (MODE == CCD_ROWS && SRC == SRC_PACKED) record_in_place<T, MODE, Sink, LIB>(&A, &sink, rec);
                    else put(rec, atomicAdd(&hdr->expand_count, 1));
                }
            }
            filtered += last ? nee + nvf : 32 * (we + wv);
            nee = max(nee - 32 * we, 0);
            nvf = max(nvf - 32 * wv, 0);
            __syncthreads();
            if (tid == 0) {
                ints[CI_EE] = nee;
                ints[CI_VF] = nvf;
            }
            if (last || ints[CI_OUT] >= L::OUT / 2) flush();
        } else if (last && ints[CI_OUT] > 0) {
            flush();
        }
        if (last) break;
        __syncthreads();
    }
    if (tid == 0) {
        if (solved) atomicAdd(&hdr->solved, solved);
        if (filtered) atomicAdd(&hdr->roots, filtered);
    }
}

// Launch of k_ccd_narrow with its dynamic shared memory (the size is raised once per
// instantiation and device; prepare_ccd_narrow does it ahead of any stream capture).
// The flags are atomic because host threads may launch on different streams at once; two
// first calls may both set the attribute, which is harmless.
template <class T, int MODE, class Sink, int LIB, int SRC, int BM> cudaError_t prepare_ccd_narrow() {
    static std::atomic<bool> done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && done[dev].load(std::memory_order_acquire)) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_ccd_narrow<T, MODE, Sink, LIB, SRC, BM>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)CcdLayout<T, BM * CCD_BLOCK>::bytes);
    if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
    return e;
}

template <class T, int MODE, class Sink, int LIB, int SRC, int BM>
cudaError_t launch_ccd_narrow(int grid, cudaStream_t s, const CcdArgs<T>& A, const Sink& sink) {
    cudaError_t e = prepare_ccd_narrow<T, MODE, Sink, LIB, SRC, BM>();
    if (e != cudaSuccess) return e;
    return launch_chain(grid, CCD_BLOCK, CcdLayout<T, BM * CCD_BLOCK>::bytes, s,
                        k_ccd_narrow<T, MODE, Sink, LIB, SRC, BM>, A, sink);
}

// The contacts of the roots that passed the filter in k_ccd_narrow, one record a thread: the
// contact's registers and code stay out of the narrow kernel, and its lanes are full.  The sums
// are added by the warp together (Sink::add_all).
static constexpr int CONTACT_THREADS = 128;
template <class T, class Sink, int LIB>
__global__ void __launch_bounds__(CONTACT_THREADS, Sink::MIN_BLOCKS)
k_ccd_contacts(const __grid_constant__ CcdArgs<T> A, const __grid_constant__ Sink sink) {
    chain_begin();
    __shared__ typename Sink::Points S[CONTACT_THREADS / 32];
    const int lane = threadIdx.x & 31;
    const int n = min(*(volatile int*)&A.hdr->expand_count, A.W.expand_cap);
    for (int c = blockIdx.x * CONTACT_THREADS + threadIdx.x; c - lane < n; c += gridDim.x * CONTACT_THREADS) {
        int i = 0, j = 0, k = 0;
        T root = T(0);
        MTet<T> tet;
        Contact<T> ct;
        if (c < n) {
            const int4 rec = A.W.expand[c];
            i = rec.x & SLOT_MASK;
            j = rec.y & SLOT_MASK;
            k = (rec.y >> 28) & 15;
            root = (T)__hiloint2double(rec.w, rec.z);
            tet = load_tet(A.x0, A.x1, i, j, k);
            ct = contact_of_tet<T, Sink, LIB>(tet, sink, i, j, k, root);
        }
        sink.add_all(c < n, tet, i, j, k, root, ct, A.F, forest_size(A.F), &A.hdr->status, S[threadIdx.x >> 5]);
    }
}

template <class T, class Sink, int LIB>
cudaError_t launch_ccd_contacts(int grid, cudaStream_t s, const CcdArgs<T>& A, const Sink& sink) {
    return launch_chain(grid, CONTACT_THREADS, 0, s, k_ccd_contacts<T, Sink, LIB>, A, sink);
}
#endif  // CCC_NARROW_TU

// The rows of the roots that passed the filter in k_ccd_narrow (its records in Weld.expand),
// every pair's for a shared sub-test: one record a thread, the rows of a warp's lanes
// reserved with one atomic per mesh.
static constexpr int EXPAND_THREADS = 256;
template <class T>
__global__ void __launch_bounds__(EXPAND_THREADS)
k_ccd_expand(WsHeader* hdr, Weld W, Forest F, long long* __restrict__ rows, T* __restrict__ times, int max_per_tri,
             int* __restrict__ mesh_counters) {
    chain_begin();
    const unsigned FULL = 0xffffffffu;
    const int M = forest_size(F);
    const int n = min(*(volatile int*)&hdr->expand_count, W.expand_cap);
    const int lane = threadIdx.x & 31;
    const int nwarps = gridDim.x * (EXPAND_THREADS / 32);
    for (int base = ((blockIdx.x * EXPAND_THREADS + threadIdx.x) >> 5) * 32; base < n; base += nwarps * 32) {
        const int c = base + lane;
        int ma[WELD_FANCAP], mb[WELD_FANCAP], mk[WELD_FANCAP];
        int nm = 0, m = 0, po = 0;
        long long cap = 0;
        T tv = T(0);
        if (c < n) {
            const int4 rec = W.expand[c];
            const int qx = rec.x & SLOT_MASK, qy = rec.y & SLOT_MASK, k = (rec.y >> 28) & 15;
            tv = (T)__hiloint2double(rec.w, rec.z);
            const OutRegion R = out_region(F, M, qx, max_per_tri);
            m = R.m;
            po = R.po;
            cap = R.cap;
            nm = weld_list(W, qx, qy, k, (rec.x >> 28) & 1, ma, mb, mk);
        }
        const unsigned has = __ballot_sync(FULL, nm > 0);
        if (nm > 0) {
            const int first = reserve_rows(mesh_counters, F, m, nm, has);
            for (int i = 0; i < nm; ++i) {
                const long long r = (long long)first + i;
                if (r >= cap) {
                    atomicOr(&hdr->status, ST_OUT_OVERFLOW);
                    break;
                }
                const long long o = (long long)po * max_per_tri + r;
                rows[o * 3 + 0] = ma[i] - po;
                rows[o * 3 + 1] = mb[i] - po;
                rows[o * 3 + 2] = mk[i];
                times[o] = tv;
            }
        }
    }
}

// proximity (proximity_static.cu:11-508): the sub-box masks of 32 pairs a warp, then the
// distances of the sub-tests, queued in shared memory and taken 32 at a time, edge-edge and
// vertex-face ones apart.  A loop over each pair's own sub-tests ran with a few lanes of a
// warp at a time: 62 -> 19 us for 244 k pairs of 28,800 triangles (fp32).
static constexpr int PROX_WARPS = NARROW_THREADS / 32;
template <class T>
__global__ void __launch_bounds__(NARROW_THREADS)
k_prox_narrow(const int2* __restrict__ cand, int cand_cap, WsHeader* hdr, const T* __restrict__ tri, Forest F, T th,
              long long* __restrict__ rows, int max_per_tri, int* __restrict__ mesh_counters) {
    chain_begin();
    // less than 32 left over, and 32 pairs' sub-tests
    __shared__ int2 s_ee[PROX_WARPS][32 + 9 * 32], s_vf[PROX_WARPS][32 + 6 * 32];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
    const int M = forest_size(F);
    const int n = min(hdr->cand_count, cand_cap);
    const int warps = gridDim.x * PROX_WARPS;
    int ne = 0, nv = 0;                  // queued (warp-uniform)
    auto test = [&](const int2* q, int cnt) {
        bool hit = false;
        int2 it = make_int2(0, 0);
        int k = 0;
        if (lane < cnt) {
            it = q[lane];
            k = (it.y >> 28) & 15;
            it.y &= SLOT_MASK;
            V3<T> v[4];
            load_points(tri, it.x, it.y, k, v);
            const T d = prox_distance(v, k);
            hit = d <= th && d >= 0;
        }
        if (hit) {
            const OutRegion R = out_region(F, M, it.x, max_per_tri);
            const long long r = append_row(mesh_counters, F, R.m, R.cap, &hdr->status);
            if (r >= 0) {
                const long long o = (long long)R.po * max_per_tri + r;
                rows[o * 3 + 0] = it.x - R.po;
                rows[o * 3 + 1] = it.y - R.po;
                rows[o * 3 + 2] = k;
            }
        }
        __syncwarp();
    };
    for (long long base = (blockIdx.x * PROX_WARPS + wq) * 32LL; base < n; base += warps * 32LL) {
        const long long c = base + lane;
        uint32_t bits = 0;
        int2 pr = make_int2(0, 0);
        if (c < n) {
            pr = cand[c];
            const Tri<T> a = load_tri(tri, pr.x), b = load_tri(tri, pr.y);
            if (!share_vertex(a.v, b.v)) bits = prox_subbox_mask(a, b, th);
        }
        uint32_t e = bits & 0x1ffu, v = bits & ~0x1ffu;
        const int ie = warp_inclusive_scan(__popc(e), lane), iv = warp_inclusive_scan(__popc(v), lane);
        for (int at = ne + ie - __popc(e); e; e &= e - 1) s_ee[wq][at++] = pack_subtest(pr.x, pr.y, __ffs(e) - 1);
        for (int at = nv + iv - __popc(v); v; v &= v - 1) s_vf[wq][at++] = pack_subtest(pr.x, pr.y, __ffs(v) - 1);
        ne += __shfl_sync(FULL, ie, 31);
        nv += __shfl_sync(FULL, iv, 31);
        __syncwarp();
        for (; ne >= 32; ne -= 32) test(s_ee[wq] + ne - 32, 32);
        for (; nv >= 32; nv -= 32) test(s_vf[wq] + nv - 32, 32);
    }
    if (ne > 0) test(s_ee[wq], ne);
    if (nv > 0) test(s_vf[wq], nv);
}

// compute_impulses_from_collisions (collisions_impulses.cu:1738-1880) on caller rows.
// Rows with an index outside [0, F) or a type outside [0, 15) are skipped (the reference
// reads out of bounds on its -1 padding rows).
template <class T, int LIB>
__global__ void __launch_bounds__(NARROW_THREADS)
k_impulses_from_rows(const long long* __restrict__ rows, const T* __restrict__ roots, int B, long long N, int F,
                     const T* __restrict__ x0, const T* __restrict__ x1, const T* __restrict__ masses,
                     T* __restrict__ dv_out, T* __restrict__ dx_out, int* __restrict__ cnt_out) {
    chain_begin();
    using Sink = CornerSink<T>;
    __shared__ typename Sink::Points S[NARROW_THREADS / 32];
    const Sink sink{masses, dv_out, dx_out, cnt_out};
    const int lane = threadIdx.x & 31;
    const long long total = (long long)B * N;
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r - lane < total;
         r += (long long)gridDim.x * blockDim.x) {
        long long gi = 0, gj = 0;
        int k = 0;
        T root = T(0);
        MTet<T> tet;
        Contact<T> ct;
        bool valid = r < total;
        if (valid) {
            const long long b = r / N;
            const long long i = rows[r * 3 + 0], j = rows[r * 3 + 1], kk = rows[r * 3 + 2];
            valid = !(i < 0 || j < 0 || i >= F || j >= F || kk < 0 || kk >= 15);
            if (valid) {
                k = (int)kk;
                gi = b * F + i;
                gj = b * F + j;
                root = roots[r];
                tet = load_tet(x0, x1, gi, gj, k);
                T mq[4];
                for (int pt = 0; pt < 4; ++pt) mq[pt] = masses[(tet_side(k, pt) ? gj : gi) * 3 + tet_corner(k, pt)];
                ct = contact<T, LIB>(tet, k, root, mq);
            }
        }
        if (__any_sync(0xffffffffu, valid)) sink.add_all(valid, tet, gi, gj, k, root, ct, Forest{}, 0, nullptr, S[threadIdx.x >> 5]);
    }
}

// Test hooks of the solver's arithmetic (k_debug_math, k_debug_stage), compiled in
// ccc_narrow.cu with the continuous narrow phase, so that they compute what it computes.
cudaError_t launch_debug_math(int op, const double* in, double* out, int n, cudaStream_t s);
cudaError_t launch_debug_stage(int op, int lib, const double* in, int in_stride, double* out, int out_stride, int n,
                               cudaStream_t s);

}  // namespace ccc
