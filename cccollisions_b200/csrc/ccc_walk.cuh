// ccc_walk.cuh — four-wide tree nodes and the self-collision walk over them.
//
// Shared by the resident engine (nodes refit every step) and by the reference-format calls
// (nodes imported from the caller's tree tensors).
#pragma once

#include "ccc_kernels.cuh"

namespace ccc {

// Four-wide node over a binary tree: 2 to 4 slots, the node's children with (some of) the
// internal ones replaced by their own two children.  A slot holds a child box (fp32, rounded
// outward), a reference (>= 0: the QNode of an internal node; ~pos: the leaf at sorted
// position pos) and an aux word (the rightmost leaf position below an internal slot, the
// triangle id of a leaf slot).  Unused slots have the reference Q_EMPTY.  QNodes are indexed
// by their binary node.  One visit covers two binary levels, so a walk needs half as many
// dependent node fetches.
struct __align__(16) QNode {
    float4 lox, loy, loz, hix, hiy, hiz;
    int4 ref, aux;
};
static constexpr int Q_EMPTY = 0x7fffffff;

// The walk: every query leaf against the tree it is a leaf of, each unordered pair found once
// (a slot is skipped when its rightmost leaf position is not after the query's).
//
// A walk of one query is a chain of dependent node fetches, and with one query a thread the
// lanes of a warp end at different times (15 of 32 lanes active on the 64-mesh step) while a
// small mesh occupies a few warps for a hundred fetches in a row.  Here a warp takes up to 32
// consecutive queries and keeps their pending (query, node) visits on one stack in shared
// memory: every round, each lane pops one of the top 32 visits, tests the node's four slots
// and pushes the internal ones that the query's box meets, so that the lanes stay full and a
// round costs one fetch latency for 32 visits.  Slots are pushed one slot number at a time
// over all lanes, which leaves the visits of one node side by side (their fetches share
// lines).  Leaf hits queue up and are tested 32 at a time, the pairs that are kept go through a
// buffer of WALK_FLUSH pairs with one reservation on the shared counter.  Measured against
// one query a thread (fetch chains, a stack per thread): 5 small meshes of 7,468 triangles
// 96 -> 18 us, 12 meshes of 211 k 210 -> 90 us, 64 meshes of 2.69 M 1345 -> 895 us, the impulse
// loop's 149 k triangles 200 -> 85 us.  What bounds it now is instruction issue (55 % of the
// issue slots at 28 of 32 lanes on the 12 meshes; six blocks an SM instead of eight: 1128 us on
// the 64 meshes).
//
// The stack is popped in smaller bites when it fills up (at most one visit a round from
// WALK_RESERVE entries before its end), so it only overflows on a tree more than
// WALK_RESERVE / 3 four-wide levels deep below that point.
static constexpr int WALK_THREADS = 128;
static constexpr int WALK_WARPS = WALK_THREADS / 32;
static constexpr int WALK_STACK = 704;
static constexpr int WALK_RESERVE = 192;
static constexpr int WALK_FLUSH = 128;
static constexpr int WALK_LATE = 12;
static constexpr int WALK_TAIL = 8;
struct WalkWarp {
    unsigned stack[WALK_STACK];           // query of the group << shift | node
    uint2 leaf[32 + 128];                 // query << shift | leaf position, triangle id
    int2 out[WALK_FLUSH + 32];
    float lo[3][32], hi[3][32];           // the group's queries: boxes,
    int pos[32], id[32], base[32], n[32]; // leaf position, triangle, first slot and size of the mesh
};

// One query of the group, filled by the policy (the boxes conservative in fp32).
struct WalkQuery {
    float lo[3], hi[3];
    int pos, id, base, n;
};

// What the walk needs to know from its caller:
//   bool query(F, M, v, WalkQuery&)   the query of work item v, false when there is none
//   static ORDERED                    whether the order rule applies
//   bool keep(query, id, pos, cid...) whether the pair with the leaf at cpos (triangle cid) is
//                                     emitted; called on leaf hits
//   int rightmost(base, ref, aux)     rightmost leaf position below an internal slot
template <class Policy>
__device__ __forceinline__ void walk_forest(const Policy& pol, const QNode* __restrict__ qnodes, const Forest& F,
                                            int2* __restrict__ cand, int cand_cap, WsHeader* hdr, WalkWarp& S) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int M = forest_size(F);
    const int total = __ldg(F.voff + M);
    const int warps = gridDim.x * WALK_WARPS;
    // 27 bits of node and 32 queries, or 28 bits and 16
    const int shift = total <= (1 << 27) ? 27 : 28;
    const unsigned node_mask = (1u << shift) - 1u;
    // Groups of queries: the first `big` are as large as evenly spread work or the stack allows, the
    // last up to WALK_LATE queries a warp go out in groups of WALK_TAIL, all of them after the
    // warps' first ones to whichever warp is free.  Groups differ by how crowded their place
    // is, and with even ones dealt out beforehand a quarter of the walk's time was the slowest
    // warps' (64 meshes 888 -> 787 us, 12 meshes 90 -> 79 us, ten served folds 1,007 -> 952 us in
    // all).  Every group repeats the first visits, so small ones cost: all of them of 8 to 16
    // queries 115-119 us on the fold, against 113 us.  Calls with few queries a warp have one
    // group each (more of them would only walk later).
    const int most = total <= (1 << 27) ? 32 : 16;
    const int each = (total + warps - 1) / warps;
    const int late = each <= WALK_LATE ? 0 : min(total / 4, warps * WALK_LATE);
    const int per = min(most, max((total - late + warps - 1) / warps, 1));
    const int tail = min(per, WALK_TAIL);
    const int big = late ? (total - late) / per : (total + per - 1) / per;
    const int rest = max(total - big * per, 0);
    const int groups = big + (rest + tail - 1) / tail;
    int sp = 0, nl = 0, no = 0;           // stack, leaf queue and output fill (warp-uniform)

    auto flush_out = [&](int cnt) {
        int b0 = 0;
        if (lane == 0) b0 = atomicAdd(&hdr->cand_count, cnt);
        b0 = __shfl_sync(FULL, b0, 0);
        for (int i = lane; i < cnt; i += 32) {
            const long long slot = (long long)b0 + i;
            if (b0 >= 0 && slot < cand_cap) cand[slot] = S.out[i];
            else atomicOr(&hdr->status, ST_CAND_OVERFLOW);
        }
        __syncwarp();
    };
    auto test_leaves = [&](int cnt) {
        bool keep = false;
        int2 pr = make_int2(0, 0);
        if (lane < cnt) {
            const uint2 e = S.leaf[nl - cnt + lane];
            const int q = (int)(e.x >> shift), cpos = (int)(e.x & node_mask), cid = (int)e.y;
            const int base = S.base[q], id = S.id[q];
            keep = pol.keep(base, S.n[q], S.pos[q], id, cpos, cid);
            pr = make_int2(base + min(id, cid), base + max(id, cid));
        }
        nl -= cnt;
        const unsigned mk = __ballot_sync(FULL, keep);
        if (keep) S.out[no + __popc(mk & lt)] = pr;
        no += __popc(mk);
        __syncwarp();
        if (no >= WALK_FLUSH) {
            flush_out(WALK_FLUSH);
            no -= WALK_FLUSH;
            if (lane < no) S.out[lane] = S.out[WALK_FLUSH + lane];
            __syncwarp();
        }
    };

    auto next_group = [&]() {
        if (groups <= warps) return groups;
        int g = 0;
        if (lane == 0) g = atomicAdd(&hdr->walk_next, 1);
        return warps + __shfl_sync(FULL, g, 0);
    };
    for (int g = blockIdx.x * WALK_WARPS + (threadIdx.x >> 5); g < groups; g = next_group()) {
        const int v = min(g, big) * per + max(g - big, 0) * tail + lane;
        WalkQuery Q;
        const bool act = lane < (g < big ? per : tail) && v < total && pol.query(F, M, v, hdr, Q);
        const unsigned am = __ballot_sync(FULL, act);
        if (!am) continue;
        if (act) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                S.lo[c][lane] = Q.lo[c];
                S.hi[c][lane] = Q.hi[c];
            }
            S.pos[lane] = Q.pos;
            S.id[lane] = Q.id;
            S.base[lane] = Q.base;
            S.n[lane] = Q.n;
            S.stack[__popc(am & lt)] = (unsigned)lane << shift;       // the root
        }
        sp = __popc(am);
        // A query visits each node of its tree at most once, and a round that takes all the pending
        // visits leaves only deeper ones, so that there are no more of those rounds than nodes: counted
        // as 32 visits each, they bound a walk that goes in circles to some 2 n rounds, however few of
        // the group's queries do.
        long long left = 64 + (sp + 32LL) * __reduce_max_sync(FULL, act ? (unsigned)Q.n : 0u);
        __syncwarp();
        while (sp > 0) {
            if (left < 0 || sp > WALK_STACK - 3) {
                if (lane == 0) atomicOr(&hdr->status, left < 0 ? ST_MALFORMED_TREE : ST_STACK_OVERFLOW);
                sp = 0;
                break;
            }
            const int k = min(min(sp, 32), max(1, (WALK_STACK - WALK_RESERVE - sp) / 3));
            left -= k == sp ? 32 : k;
            const bool has = lane < k;
            const unsigned e = has ? S.stack[sp - k + lane] : 0u;
            sp -= k;
            const int q = (int)(e >> shift), node = (int)(e & node_mask);
            const int base = S.base[q], n = S.n[q], p = S.pos[q];
            int4 R = make_int4(Q_EMPTY, Q_EMPTY, Q_EMPTY, Q_EMPTY), A = R;
            float4 LX, LY, LZ, HX, HY, HZ;
            LX = LY = LZ = HX = HY = HZ = make_float4(0.f, 0.f, 0.f, 0.f);
            if (has) {
                const float4* f = reinterpret_cast<const float4*>(qnodes + (base + node));
                LX = __ldg(f + 0); LY = __ldg(f + 1); LZ = __ldg(f + 2);
                HX = __ldg(f + 3); HY = __ldg(f + 4); HZ = __ldg(f + 5);
                R = __ldg(reinterpret_cast<const int4*>(f + 6));
                A = __ldg(reinterpret_cast<const int4*>(f + 7));
            }
            const float lo0 = S.lo[0][q], lo1 = S.lo[1][q], lo2 = S.lo[2][q];
            const float hi0 = S.hi[0][q], hi1 = S.hi[1][q], hi2 = S.hi[2][q];
            __syncwarp();          // the popped entries are read
            const float lx[4] = {LX.x, LX.y, LX.z, LX.w}, ly[4] = {LY.x, LY.y, LY.z, LY.w};
            const float lz[4] = {LZ.x, LZ.y, LZ.z, LZ.w}, hx[4] = {HX.x, HX.y, HX.z, HX.w};
            const float hy[4] = {HY.x, HY.y, HY.z, HY.w}, hz[4] = {HZ.x, HZ.y, HZ.z, HZ.w};
            const int rr[4] = {R.x, R.y, R.z, R.w}, aa[4] = {A.x, A.y, A.z, A.w};
            const unsigned qbits = e & ~node_mask;
            bool bad = false;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int ref = rr[s];
                bool hit = ref != Q_EMPTY && lo0 <= hx[s] && hi0 >= lx[s] && lo1 <= hy[s] && hi1 >= ly[s] &&
                           lo2 <= hz[s] && hi2 >= lz[s];
                // child references inside the mesh: internal < n - 1, leaf position < n
                if (hit && (ref >= n - 1 || (ref < 0 && ~ref >= n))) {
                    bad = true;
                    hit = false;
                }
                if (Policy::ORDERED && hit) hit = p < (ref < 0 ? ~ref : pol.rightmost(base, ref, aa[s]));
                const unsigned mi = __ballot_sync(FULL, hit && ref >= 0), ml = __ballot_sync(FULL, hit && ref < 0);
                if (mi) {
                    if (hit && ref >= 0) S.stack[sp + __popc(mi & lt)] = qbits | (unsigned)ref;
                    sp += __popc(mi);
                }
                if (ml) {
                    if (hit && ref < 0)
                        S.leaf[nl + __popc(ml & lt)] = make_uint2(qbits | (unsigned)~ref, (unsigned)aa[s]);
                    nl += __popc(ml);
                }
            }
            if (bad) atomicOr(&hdr->status, ST_MALFORMED_TREE);
            __syncwarp();
            while (nl >= 32) test_leaves(32);
        }
        if (nl > 0) test_leaves(nl);
    }
    if (no > 0) flush_out(no);
}

}  // namespace ccc
