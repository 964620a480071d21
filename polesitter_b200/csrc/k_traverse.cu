// The interaction pass of the FMM tick: MAC + M2L + L2L, and for leaves also
// P2P + L2P, producing the final forces.
//
// Reference (PS_MULTITHREADING build): every node at depth 2, and every leaf
// above it, is paired with the root (ps_impl_dispatch_fmm, polesitter.h:
// 1772-1801, :1883-1885), and each pair (t, s) is walked by the dual
// recursion of ps_impl_fmm_interaction_pass (:1050-1146):
//   separated (MAC)        -> M2L: t.local += field of s's monopole+dipole
//   both leaves            -> P2P (the P2P pass :1258-1494 walks the same
//                             pairs with the same MAC)
//   t leaf                 -> (t, each child of s)
//   s leaf                 -> (each child of t, s)
//   otherwise              -> (each child of t) x (each child of s)
// then L2L adds every parent's field to its children (:1238-1251), L2P sets
// F = m * field at the leaves (:1224-1233) and P2P adds the direct sums
// f_t += m_t * sum_{j in s} m_j d / (|d|^2 + 0.1)^{3/2} (:1279-1449).
//
// B200 formulation (target-major, no interaction lists in HBM).  The pairs
// an internal target t hands to its children are its "near list" NS(t) =
// the sources it was not separated from, so all children of an internal
// node p (a "group") start from the same candidates
//   cand(p) = {root}                                         if depth(p) <= 1
//   cand(p) = U_{s in NS(p)} (s leaf ? {s} : children(s))    otherwise.
// One warp owns a group (with the closure's order-1 accumulators, half a
// group: children 0-3 or 4-7, so that the 4 x 9 accumulators leave room for
// 4 blocks per SM).  Candidates are tested 32 at a time, one per lane;
// each carries the set of the group's children it must be tested against,
// and the lane loads the candidate once and runs the MAC (and M2L, into
// per-child register accumulators) for each of those children.  What is
// not separated is dealt with once per chunk:
//
//  * MODE_INTERNAL, levels k = 2..10, targets = the internal children of the
//    depth-(k-1) nodes: near candidates form NS(u) in HBM for level k+1;
//    L(u) = M2L(u) + L(p) is stored.  One launch runs a range of levels: the
//    work queue is in level order, and a group waits (bounded) until its
//    parent's list and field are marked final by the warp that made them,
//    which took an earlier item, so some warp can always go on.
//  * MODE_LEAF, one launch after all levels, targets = the leaf children of
//    every node: a near leaf candidate is a P2P source, staged in shared
//    memory with the set of children it serves (spilled to HBM chunks past
//    128); a near internal candidate is the "t leaf" recursion -- it goes
//    onto a DFS stack in shared memory with the set of children that still
//    need it opened, so sibling leaves share every descent.  The warp then
//    finishes each leaf: L(u) = M2L(u) + L(p) and, per particle,
//    F = m * (L(u) + its P2P sum) -- written once, no atomics.  Running all
//    levels' leaves in one launch lets the long descents of shallow leaves
//    overlap with everything else.
//
// The MAC replays the reference's rounded float sequence exactly
// (mac_separated), so the interaction set is identical, ties included.
// Bound: FP32 pipe (M2L ~35 flop + 1 MUFU per pair; P2P ~20 flop + 1 MUFU
// per particle pair) and the latency of the candidate loads.
#include <type_traits>

#include "psg_common.cuh"
#include "psg_kernels.h"

namespace psg {

constexpr int kTravWarps = 4;
constexpr int kTravThreads = kTravWarps * 32;
constexpr int kCandBuf = 256;             // children of 32 opened entries
constexpr int kStackCap = 384;            // DFS stack (node, child mask)
constexpr int kStackSlack = 72;           // 9 levels x 7: growth of a single-entry descent
constexpr int kP2PCap = 128;              // staged P2P sources of a group
constexpr uint32_t kSegChunks = 32;       // chunks of source list per dense work record

enum { MODE_INTERNAL = 0, MODE_LEAF = 1 };

struct SmemInternal {
    float4 cgeo[8];  // the targets: centre + half width
    float4 cgp[4][2];  // ... pair-packed for the MAC (cgp_put)
    uint8_t tq[8];     // ... and which of the group's children each is
    uint32_t cand_node[kCandBuf];
    uint32_t ns_cnt[8];
    uint32_t dbg_m2l[8];
    unsigned long long ns_next, ns_end;
    uint8_t cand_mask[kCandBuf];
};

struct SmemLeaf {
    float4 cgeo[8];
    float4 cgp[4][2];
    uint8_t tq[8];
    float4 chain_geo[8];    // chain groups: the ancestors a_{K+1} .. p under test
    float4 sL[8];           // the children's local fields
    float4 sG0[8];          // closure order 1: the children's field gradients
    float2 sG1[8];
    uint2 cpart[8];         // the children's particle ranges
    // staged P2P sources: leaves (p2p_node), or, where neighbours are merged and
    // in stream_p2p, their first particle and count (p2p_range)
    uint2 p2p_range[kP2PCap];
    uint32_t p2p_node[kP2PCap];
    uint32_t cand_node[kCandBuf];
    uint32_t stk_node[kStackCap];
    uint32_t chunk_next, chunk_end;
    // DENSE: the group's source list so far -- chunks in the open segment,
    // segments recorded, the first and the latest recorded segment's slots
    uint32_t seg_chunks, seg_cnt, seg_first, seg_prev;
    uint32_t dbg_m2l[8];
    uint32_t dbg_p2p[8];
    uint8_t cand_mask[kCandBuf];
    uint8_t stk_mask[kStackCap];
    uint8_t p2p_mask[kP2PCap];
    uint8_t cand_lvl[kCandBuf];  // 0: tested against the children in the mask;
    uint8_t stk_lvl[kStackCap];  // c > 0: against chain target c (chain groups)
};

template <int MODE>
struct SmemOf { using T = SmemInternal; };
template <>
struct SmemOf<MODE_LEAF> { using T = SmemLeaf; };

__device__ __forceinline__ void m2l_field(float dx, float dy, float dz, float d2, float4 mp,
                                          float& fx, float& fy, float& fz) {
    // polesitter.h:1065-1092 with rsqrt: 1/r^3 and 1/r^5 of the softened distance
    const float soft = d2 + 0.1f;
    const float inv = rsqrt_soft(soft);
    const float inv2 = inv * inv;
    const float ir3 = inv2 * inv;
    const float ir5 = ir3 * inv2;
    const float mdr = fmaf(mp.y, dx, fmaf(mp.z, dy, mp.w * dz));
    const float a = fmaf(mp.x, ir3, -3.0f * mdr * ir5);
    fx = fmaf(dx, a, mp.y * ir3);
    fy = fmaf(dy, a, mp.z * ir3);
    fz = fmaf(dz, a, mp.w * ir3);
}

// m2l_field plus what the closure's order-1 local expansion needs: the
// gradient of the monopole field at the target centre is
// g3 * d d^T - gi * I with g3 = 3 m0 / r^5, gi = m0 / r^3 (softened r).
__device__ __forceinline__ void m2l_field_grad(float dx, float dy, float dz, float d2, float4 mp,
                                               float& fx, float& fy, float& fz, float& g3,
                                               float& gi) {
    const float soft = d2 + 0.1f;
    const float inv = rsqrt_soft(soft);
    const float inv2 = inv * inv;
    const float ir3 = inv2 * inv;
    const float ir5 = ir3 * inv2;
    const float mdr = fmaf(mp.y, dx, fmaf(mp.z, dy, mp.w * dz));
    const float a = fmaf(mp.x, ir3, -3.0f * mdr * ir5);
    fx = fmaf(dx, a, mp.y * ir3);
    fy = fmaf(dy, a, mp.z * ir3);
    fz = fmaf(dz, a, mp.w * ir3);
    g3 = 3.0f * mp.x * ir5;
    gi = mp.x * ir3;
}

// G v for the symmetric gradient stored as (xx, yy, zz, xy) + (xz, yz)
__device__ __forceinline__ float3 grad_apply(float4 g0, float2 g1, float vx, float vy, float vz) {
    return make_float3(fmaf(g0.x, vx, fmaf(g0.w, vy, g1.x * vz)),
                       fmaf(g0.w, vx, fmaf(g0.y, vy, g1.y * vz)),
                       fmaf(g1.x, vx, fmaf(g1.y, vy, g0.z * vz)));
}

// Children 2k and 2k + 1 of the group, pair-packed for the paired FP32
// instructions: cgp[k][0] = (x, x', y, y'), cgp[k][1] = (z, z', w, w');
// zeros past the nc children, so that every lane computes with finite
// values (a masked term is x * 0, which a NaN would survive).
// Warp-collective.
__device__ __forceinline__ void cgp_put(float4 (*cgp)[2], const float4* cgeo, uint32_t nc) {
    const uint32_t lane = lane_id();
    __syncwarp();
    if (lane < 4) {
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 a = 2 * lane < nc ? cgeo[2 * lane] : z;
        const float4 b = 2 * lane + 1 < nc ? cgeo[2 * lane + 1] : z;
        cgp[lane][0] = make_float4(a.x, b.x, a.y, b.y);
        cgp[lane][1] = make_float4(a.z, b.z, a.w, b.w);
    }
    __syncwarp();
}

// the run of consecutive children that starts at the lowest bit of m (its
// particles are contiguous): child mask, first particle, particles; taken off m
__device__ __forceinline__ uint32_t next_run(const SmemLeaf& sm, uint32_t& m, uint32_t& first,
                                             uint32_t& count) {
    const uint32_t q0 = __ffs(m) - 1;
    uint32_t q1 = q0;
    first = sm.cpart[q0].x;
    count = sm.cpart[q0].y;
    while (q1 + 1 < 8 && ((m >> (q1 + 1)) & 1u)) count += sm.cpart[++q1].y;
    m &= ~((2u << q1) - 1u);
    return ((2u << q1) - 1u) & ~((1u << q0) - 1u);
}

// k_dense_p2p work records for the leaf children in mask of the group whose
// children start at node fc, over the source chain phead: each run of
// consecutive children is cut into records of up to kDenseTargets particles.
// A long source list is recorded in segments of kSegChunks chunks (last: the
// warp's last segment), so that the records of a shallow leaf, whose list
// reaches most of the tree, are shared out over many warps; the segments'
// sums meet in slots (DenseStore).  One warp per whole list took 7.7 of a
// 131K closure tick's 9.9 ms, as segments 0.8 ms; 32 chunks (at most 1,024
// sources) keep a record to tens of microseconds while most lists of a 1M tick
// stay whole (16 chunks: 3 % faster at 131K, 2 % slower at 1M).  part: the list is
// one of several warps' (a split group, whose last warp links the lists and fills
// in the items).
// Record: {fc, phead, first particle, count | run's child mask << 8}, slot or
// kNone.
__device__ __noinline__ void record_dense(SmemLeaf& sm, const DenseStore& ds, uint32_t mask,
                                          uint32_t fc, uint32_t phead, bool last, bool part,
                                          Status* status) {
    const uint32_t lane = lane_id();
    const uint32_t segs = sm.seg_cnt;
    const bool split = !last || part || segs != 0;
    uint32_t nall = 0, first, count;
    for (uint32_t m = mask; m;) {
        next_run(sm, m, first, count);
        nall += (count + kDenseTargets - 1) / kDenseTargets;
    }
    uint32_t r0 = 0, s0 = kNone;
    if (lane == 0) {
        r0 = atomicAdd(&status->run.dense_count, nall);
        if (split) s0 = atomicAdd(&status->run.dense_slots, nall);
    }
    r0 = __shfl_sync(0xFFFFFFFFu, r0, 0);
    s0 = __shfl_sync(0xFFFFFFFFu, s0, 0);
    const uint32_t prev_slot = segs ? sm.seg_prev : kNone;
    uint32_t ord = 0;
    for (uint32_t m = mask; m;) {
        const uint32_t run = next_run(sm, m, first, count);
        const uint32_t nrec = (count + kDenseTargets - 1) / kDenseTargets;
        for (uint32_t k = lane; k < nrec; k += 32) {
            const uint32_t r = r0 + ord + k, sl = s0 + ord + k, c0 = k * kDenseTargets;
            if (r < ds.rec_cap) {
                ds.rec[r] = make_uint4(fc, phead, first + c0,
                                       min(kDenseTargets, count - c0) | (run << 8));
                ds.rec_slot[r] = split ? sl : kNone;
            }
            if (split && sl < ds.slot_cap) {
                ds.prev[sl] = prev_slot == kNone ? kNone : prev_slot + ord + k;
                if (last && !part) ds.item[first + c0] = make_uint4(sl, segs + 1, 0u, 0u);
            }
        }
        ord += nrec;
    }
    if (lane == 0 && (r0 + nall > ds.rec_cap || (split && s0 + nall > ds.slot_cap)))
        set_err(status, PSG_ERR_DENSE_OVERFLOW);
    __syncwarp();
    if (lane == 0) {
        if (segs == 0) sm.seg_first = s0;
        sm.seg_prev = s0;
        sm.seg_cnt = segs + 1;
        sm.seg_chunks = 0;
    }
    __syncwarp();
}

// The last warp of a split group: the warps' source lists (SplitStore::list,
// in warp order) become one list per target chunk -- each list's first slot
// is linked to the list before it -- and the chunk's item holds its end.
__device__ __noinline__ void link_split(SmemLeaf& sm, const TravArgs& A, uint32_t mask,
                                        uint32_t fc, uint32_t sidx) {
    const uint32_t lane = lane_id();
    const DenseStore& ds = A.dense;
    // lane w: warp w's list (first slot, last segment's slot, segments)
    uint4 l = make_uint4(kNone, kNone, 0u, 0u);
    if (lane < (uint32_t)kSplitParts) l = __ldcg(&A.split.list[(size_t)sidx * kSplitParts + lane]);
    const uint32_t lists = __ballot_sync(0xFFFFFFFFu, l.z != 0u);
    if (lists == 0) {  // no source at all: records that only add the field
        if (lane == 0) sm.seg_chunks = sm.seg_cnt = 0;
        __syncwarp();
        record_dense(sm, ds, mask, fc, kNone, true, false, A.status);
        return;
    }
    const uint32_t nseg = __reduce_add_sync(0xFFFFFFFFu, l.z);
    uint32_t ord = 0, first, count;
    for (uint32_t m = mask; m;) {
        next_run(sm, m, first, count);
        const uint32_t nrec = (count + kDenseTargets - 1) / kDenseTargets;
        for (uint32_t k0 = 0; k0 < nrec; k0 += 32) {
            const uint32_t k = k0 + lane;
            uint32_t end = kNone;
            for (uint32_t w = lists; w; w &= w - 1) {
                const uint32_t fs = __shfl_sync(0xFFFFFFFFu, l.x, __ffs(w) - 1),
                               ls = __shfl_sync(0xFFFFFFFFu, l.y, __ffs(w) - 1);
                if (k < nrec && fs + ord + k < ds.slot_cap) ds.prev[fs + ord + k] = end;
                end = ls + ord + k;
            }
            if (k < nrec && end < ds.slot_cap)
                ds.item[first + k * kDenseTargets] = make_uint4(end, nseg, 0u, 0u);
        }
        ord += nrec;
    }
    __syncwarp();
}

// a listed P2P source's particles: first, count
__device__ __forceinline__ uint2 source_range(const TreeView& tv, uint2 r) {
    if (r.y != kNone) return r;
    const uint4 si = tv.info[r.x];
    return make_uint2(si.x, si.y);
}

// Spill the group's staged P2P sources [0, fill) to HBM chunks of
// kP2PChunk (particle range, child mask) entries, chained to the group's earlier
// chunks.  Warp-collective; chunk ids come from a per-warp pool.  Returns the
// new chain head.  record: the list is for k_dense_p2p, so after kSegChunks
// chunks a segment is recorded and the chain starts over.
__device__ __noinline__ uint32_t spill_p2p(SmemLeaf& sm, uint32_t fill, uint32_t head,
                                           const TravArgs& A, uint32_t tgt_mask, uint32_t fc,
                                           bool record, bool merged) {
    const uint32_t lane = lane_id();
    const P2PStore& st = A.p2p;
    Status* status = A.status;
    if (record && sm.seg_chunks >= kSegChunks) {
        record_dense(sm, A.dense, tgt_mask, fc, head, false, false, status);
        head = kNone;
    }
    for (uint32_t e0 = 0; e0 < fill; e0 += kP2PChunk) {
        if (sm.chunk_next >= sm.chunk_end) {
            uint32_t c = 0;
            if (lane == 0) c = atomicAdd(&status->run.p2p_chunks, kChunkPool);
            c = __shfl_sync(0xFFFFFFFFu, c, 0);
            __syncwarp();
            if (lane == 0) {
                sm.chunk_next = c;
                sm.chunk_end = c + kChunkPool;
            }
            __syncwarp();
        }
        const uint32_t c = sm.chunk_next;
        const uint32_t cnt = min((uint32_t)kP2PChunk, fill - e0);
        if (c < st.cap_chunks) {
            if (lane < cnt) {
                st.src[(size_t)c * kP2PChunk + lane] =
                    merged ? sm.p2p_range[e0 + lane] : make_uint2(sm.p2p_node[e0 + lane], kNone);
                st.mask[(size_t)c * kP2PChunk + lane] = sm.p2p_mask[e0 + lane];
            }
            if (lane == 0) {
                st.next[c] = head;
                st.cnt[c] = cnt;
            }
            head = c;
        } else if (lane == 0) {
            set_err(status, PSG_ERR_P2P_OVERFLOW);
        }
        __syncwarp();
        if (lane == 0) sm.chunk_next = c + 1;
        __syncwarp();
    }
    __syncwarp();
    if (lane == 0) sm.seg_chunks += (fill + kP2PChunk - 1) / kP2PChunk;
    __syncwarp();
    return head;
}

// Direct sum of the particles [r.x, r.x + r.y) on target particle t
// (polesitter.h:1424-1444 with rsqrt), optionally Kahan-compensated.
__device__ __forceinline__ void p2p_range(const float4* __restrict__ xyzm, uint2 r, float4 t,
                                          bool kahan, float& ax, float& ay, float& az, float& cx,
                                          float& cy, float& cz) {
    for (uint32_t j = 0; j < r.y; ++j) {
        const float4 p = xyzm[r.x + j];
        const float dx = p.x - t.x, dy = p.y - t.y, dz = p.z - t.z;
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) + 0.1f;
        const float inv = rsqrt_soft(r2);
        const float f = p.w * (inv * inv * inv);
        if (kahan) {
            const float yx = __fsub_rn(__fmul_rn(dx, f), cx);
            const float yy = __fsub_rn(__fmul_rn(dy, f), cy);
            const float yz = __fsub_rn(__fmul_rn(dz, f), cz);
            const float tx = __fadd_rn(ax, yx);
            const float ty = __fadd_rn(ay, yy);
            const float tz = __fadd_rn(az, yz);
            cx = __fsub_rn(__fsub_rn(tx, ax), yx);
            cy = __fsub_rn(__fsub_rn(ty, ay), yy);
            cz = __fsub_rn(__fsub_rn(tz, az), yz);
            ax = tx;
            ay = ty;
            az = tz;
        } else {
            ax = fmaf(dx, f, ax);
            ay = fmaf(dy, f, ay);
            az = fmaf(dz, f, az);
        }
    }
}

// The P2P sums of the staged sources [0, pfill), and of the chain phead of
// spilled ones, for every target particle of the work item's leaf children
// (tgt_mask).  The children's particles are enumerated flat (children in mask
// order), 32 at a time; T lanes own targets (T the smallest power of two >=
// their count) and the 32 / T slices of lanes split the source leaves; the
// slices' sums are added in a fixed order.  fin: also L2P, F = m (L + all P2P
// sums), with order 1's shift to the particle.
// STREAM: the sums are taken when the stage is full instead of spilling it to
// HBM, so that no store grows with the size of a source list; they are kept in
// the force arrays between flushes (accum: add to what an earlier flush of
// this item left there; fin: the item's last flush).
template <bool DEBUG, bool GRAD>
__device__ __noinline__ void stream_p2p(SmemLeaf& sm, const TravArgs& o, uint32_t tgt_mask,
                                        uint32_t fc, uint32_t pfill, uint32_t phead, bool accum,
                                        bool fin, unsigned long long& inter) {
    const uint32_t lane = lane_id();
    for (uint32_t e = lane; e < pfill; e += 32)
        sm.p2p_range[e] = source_range(o.tv, make_uint2(sm.p2p_node[e], kNone));
    __syncwarp();
    uint32_t total = 0;
    for (uint32_t m = tgt_mask; m; m &= m - 1) total += sm.cpart[__ffs(m) - 1].y;
    for (uint32_t r0 = 0; r0 < total; r0 += 32) {
        const uint32_t cnt = min(32u, total - r0);
        uint32_t T = 1;
        while (T < cnt) T <<= 1;
        const uint32_t S = 32u / T, tl = lane & (T - 1u), slice = lane / T;
        const bool active = tl < cnt;
        const uint32_t f = r0 + (active ? tl : 0u);
        uint32_t q = 0, i = 0, acc = 0;
        for (uint32_t m = tgt_mask; m; m &= m - 1) {
            const uint32_t qq = __ffs(m) - 1;
            const uint2 cp = sm.cpart[qq];
            if (f >= acc && f < acc + cp.y) {
                q = qq;
                i = cp.x + (f - acc);
            }
            acc += cp.y;
        }
        const float4 t = o.xyzm[i];
        float bx = 0.f, by = 0.f, bz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
        uint32_t used = 0;
        for (uint32_t e = slice; e < pfill; e += S) {
            if ((sm.p2p_mask[e] >> q) & 1u) {
                const uint2 r = sm.p2p_range[e];
                p2p_range(o.xyzm, r, t, o.kahan, bx, by, bz, cx, cy, cz);
                used += r.y;
            }
        }
        for (uint32_t c = phead; c != kNone; c = o.p2p.next[c]) {
            const uint32_t n = o.p2p.cnt[c];
            for (uint32_t e = slice; e < n; e += S) {
                if ((o.p2p.mask[(size_t)c * kP2PChunk + e] >> q) & 1u) {
                    const uint2 r = source_range(o.tv, o.p2p.src[(size_t)c * kP2PChunk + e]);
                    p2p_range(o.xyzm, r, t, o.kahan, bx, by, bz, cx, cy, cz);
                    used += r.y;
                }
            }
        }
        bx -= cx;
        by -= cy;
        bz -= cz;
        for (uint32_t d = T; d < 32u; d <<= 1) {
            bx += __shfl_xor_sync(0xFFFFFFFFu, bx, d);
            by += __shfl_xor_sync(0xFFFFFFFFu, by, d);
            bz += __shfl_xor_sync(0xFFFFFFFFu, bz, d);
        }
        if (DEBUG) inter += active ? used : 0u;
        if (active && slice == 0) {
            if (accum) {
                bx += o.fx[i];
                by += o.fy[i];
                bz += o.fz[i];
            }
            if (!fin) {
                o.fx[i] = bx;
                o.fy[i] = by;
                o.fz[i] = bz;
            } else {
                const float4 L = sm.sL[q];
                float lx = L.y, ly = L.z, lz = L.w;
                if constexpr (GRAD) {
                    const float4 cu = sm.cgeo[q];
                    const float3 sh = grad_apply(sm.sG0[q], sm.sG1[q], t.x - cu.x, t.y - cu.y,
                                                 t.z - cu.z);
                    lx += sh.x;
                    ly += sh.y;
                    lz += sh.z;
                    if (o.leaf_of) o.leaf_of[i] = fc + sm.tq[q];
                }
                const double mm = (double)t.w;
                o.fx[i] = (float)(mm * ((double)lx + (double)bx));
                o.fy[i] = (float)(mm * ((double)ly + (double)by));
                o.fz[i] = (float)(mm * ((double)lz + (double)bz));
            }
        }
    }
    __syncwarp();
}

// L2P + P2P of a group's leaf children once its candidates are done: with
// DENSE, every group is handed to k_dense_p2p (which adds L and the P2P sum);
// otherwise, and where the P2P is streamed, F = m (L + P2P sum) here.
template <bool DEBUG, bool GRAD, bool DENSE>
__device__ __forceinline__ void leaf_epilogue(SmemLeaf& sm, const TravArgs& o, uint32_t tgt_mask,
                                           uint32_t fc, uint32_t pfill, uint32_t phead,
                                           bool merged, bool stream, bool flushed,
                                           unsigned long long inter) {
    const uint32_t lane = lane_id();
    Status* status = o.status;
    if (!DENSE || stream) {
        stream_p2p<DEBUG, GRAD>(sm, o, tgt_mask, fc, pfill, phead, flushed, true, inter);
        if (DEBUG) {
            inter = warp_sum(inter);
            if (lane == 0) atomicAdd(&status->stat[PSG_STAT_P2P_INTER], inter);
        }
    } else {
        // the group's whole source list to HBM chunks, then k_dense_p2p work
        // records of up to kDenseTargets target particles
        if (pfill) phead = spill_p2p(sm, pfill, phead, o, tgt_mask, fc, true, merged);
        record_dense(sm, o.dense, tgt_mask, fc, phead, true, false, status);
    }
    if (DEBUG && lane == 0) {
        for (uint32_t m = tgt_mask; m; m &= m - 1) {
            const uint32_t q = __ffs(m) - 1;
            o.tv.dbg_p2p[fc + sm.tq[q]] = sm.dbg_p2p[q];
            atomicAdd(&status->stat[PSG_STAT_P2P_PAIRS], (unsigned long long)sm.dbg_p2p[q]);
        }
    }
    __syncwarp();
}

// Wait until a node's near list and field are final (ready set by the warp that
// makes them, in this launch); false after kReadyPolls polls (a poll takes 0.26 us
// alone and up to 0.65 us on a full GPU: 0.27 to 0.7 s) or once another wait has
// given up.  The longest waits are for groups whose candidates are most of a
// level's nodes: 9,100 polls measured (256K cube at theta 48; 5,700 for 1M clumpy
// there, 114 for 1M Plummer at theta 2).  A group that gives up leaves its
// children's lists and offsets as an earlier run left them, or never written: every
// later kernel of the run returns at once (PSG_ERR_VOID).  Warp-collective.
constexpr int kReadyPolls = 1 << 20;

__device__ __noinline__ bool wait_ready(const uint32_t* flag, int polls, Status* status) {
    uint32_t ok = 0;
    if (lane_id() == 0) {
        for (int i = 0; i < polls; ++i) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(ok) : "l"(flag) : "memory");
            if (ok) break;
            if ((i & 255) == 255 && (*(volatile uint32_t*)&status->err & PSG_ERR_READY_SPIN)) break;
            __nanosleep(64);
        }
        if (!ok) set_err(status, PSG_ERR_READY_SPIN);
    }
    ok = __shfl_sync(0xFFFFFFFFu, ok, 0);
    __syncwarp();  // (orders the other lanes' reads after lane 0's acquire)
    return ok != 0u;
}

// DENSE (leaf pass only): the variant for trees whose fullest leaf holds at
// least kDenseSwitch particles or whose leaf capacity is kDenseCap or more,
// which hands every leaf's P2P to k_dense_p2p.  Below kDenseCap the host does not
// know the fullest leaf: the sparse and the dense variant are both launched, and
// each returns at once unless the tree is its kind.
// XL (leaf pass only): the variant that also serves chain groups and
// streamed P2P, launched only when the near lists stop short of the deepest
// level or the P2P is streamed, so the other variants keep their registers.
// Blocks per SM, measured: the plain sparse leaf variant (the reference's tree
// and far field) 7 (72 registers; 5, 6 and 8 took a 1M tick's leaf pass from
// 1.43 to 1.62, 1.48 and 1.70 ms), the order-1 leaf variants 4 (128; 3 and 5 took
// a 1M closure tick's from 4.35 to 4.70 and 5.14 ms), the internal levels 5, with
// order 1 4 (3, 4, 5 blocks: 0.49, 0.50, 0.45 ms of a 1M plain tick, 0.24, 0.26,
// 0.30 of a 131K closure tick).
// SPLIT (leaf pass only): the groups of the depths < shallow, whose leaves'
// walks reach a large part of the tree, kSplitParts warps each (every warp
// takes every kSplitParts-th candidate and what lies below it), on trees of
// either kind; their P2P always goes to k_dense_p2p.  A launch of its own
// beside the rest, so that the other variants keep their registers.
// MERGE (leaf pass only): the dense variant for leaf capacities of kDenseCap and
// more (SPLIT_MERGE: of the split groups), which lists neighbouring source
// leaves as one range, so that k_dense_p2p walks fewer entries (5.51 against 6.17 ms of
// P2P in a 1M closure tick, 5.36 against 6.10 in a 250K one at theta 10, for
// 0.18 and 0.08 ms of leaf pass).  One-particle leaves are listed singly:
// merging cost a 100K tick at theta 8 and leaf capacity 1 0.45 ms of leaf pass.
// The dense variants run 4 blocks per SM (128 registers; 3 blocks: 3.48 against
// 2.88 ms of leaf pass in that tick, 6: 3.42).
enum { VAR_PLAIN = 0, VAR_XL = 1, VAR_SPLIT = 2, VAR_MERGE = 3, VAR_SPLIT_MERGE = 4 };

template <int MODE, bool DEBUG, bool GRAD, bool DENSE, int VAR>
__global__ void __launch_bounds__(
    kTravThreads,
    (DEBUG || VAR == VAR_XL) ? 1
    : MODE == MODE_INTERNAL  ? (GRAD ? 4 : 5)
                             : (GRAD ? 4 : (DENSE ? 4 : 7)))
    k_trav(const __grid_constant__ TravArgs A) {
    constexpr bool XL = VAR == VAR_XL, SPLIT = VAR == VAR_SPLIT || VAR == VAR_SPLIT_MERGE;
    constexpr bool MERGE = VAR == VAR_MERGE || VAR == VAR_SPLIT_MERGE;
    constexpr bool COMPACT = MODE == MODE_INTERNAL || !DENSE;
    using Smem = typename SmemOf<MODE>::T;
    __shared__ Smem smem[kTravWarps];
    const uint32_t lane = lane_id();
    const uint32_t lt_mask = lanemask_lt();
    Smem& sm = smem[threadIdx.x >> 5];
    const TreeView& tv = A.tv;
    Status* status = A.status;
    if (status->err & PSG_ERR_VOID) return;
    // a run whose near lists ran out is void (the host grows them and runs
    // again): the internal levels below the one that failed did not run, so
    // their lists must not be read
    if (MODE == MODE_LEAF && (status->err & PSG_ERR_NS_OVERFLOW)) return;
    // the variant for this tree (batched systems: each group takes its
    // system's variant, so a system sums exactly as it does alone)
    if (MODE == MODE_LEAF && !SPLIT && !MERGE && !tv.part_sys &&
        ((status->max_leaf >= kDenseSwitch || A.leaf_cap >= kDenseCap) != DENSE))
        return;
    // a shallower level's near lists did not fit: this level's are void
    if (MODE == MODE_INTERNAL && A.level == A.level_end &&
        (status->run.ns_fail & ((1u << A.level) - 1u)))
        return;
    const float theta2 = __fmul_rn(A.theta, A.theta);

    // the closure's order-1 accumulators take a group's children 4 at a time:
    // a work item is (group, half)
    constexpr uint32_t SL = GRAD ? 4u : 8u;
    constexpr uint32_t NH = 8u / SL;
    // work items: MODE_INTERNAL = the (halves of the) internal nodes at depth
    // k-1; MODE_LEAF = those at depths shallow..9, level after level (SPLIT: at
    // depths 0..shallow-1, each kSplitParts times)
    uint32_t cum[kMaxDepth + 1];
    uint32_t total = 0;
    uint32_t* work;
    if (MODE == MODE_INTERNAL) {
#pragma unroll
        for (int d = 0; d < kMaxDepth; ++d) {
            cum[d] = total;
            if (d + 1 >= A.level && d < A.level_end) total += status->group_count[d] * NH;
        }
        cum[kMaxDepth] = total;
        work = &status->run.work[A.level];
    } else {
#pragma unroll
        for (int d = 0; d < kMaxDepth; ++d) {
            cum[d] = total;
            if ((d < A.shallow) == SPLIT)
                total += status->group_count[d] * NH * (SPLIT ? kSplitParts : 1u);
        }
        cum[kMaxDepth] = total;
        // batched systems run both variants over all groups, each with its
        // own counter (work[1] is no internal level's); one system: work[0]
        work = SPLIT   ? (MERGE ? &status->run.split_work : &status->run.heavy_work)
               : MERGE ? &status->run.work[kLevels]
                       : &status->run.work[(tv.part_sys && DENSE) ? 1 : 0];
    }
    if (lane == 0) {
        if constexpr (MODE == MODE_INTERNAL) {
            sm.ns_next = 0;
            sm.ns_end = 0;
        } else {
            sm.chunk_next = 0;
            sm.chunk_end = 0;
        }
    }
    __syncwarp();
    // items taken per atomic: one, since whole work queues are a few items per
    // warp (4 at a time cost the internal levels of a 65K tick 70 of 104 us; as a
    // loop without the inner one the merging leaf variant spills more, for 0.5 % of
    // a 131K closure tick)
    constexpr uint32_t batch = 1u;
    const uint32_t items = total;

    for (;;) {
        uint32_t g0 = 0;
        if (lane == 0) {
            g0 = atomicAdd(work, batch);
            // once k_heavy_leaf, beside it, has run out of frontier the run is void
            // (first tick of 1M clumpy at theta 48: 28.4 s when it was taken to its
            // end and then done again, 13.8 so)
            if (XL && (*(volatile uint32_t*)&status->err & PSG_ERR_HEAVY_OVERFLOW)) g0 = items;
        }
        g0 = __shfl_sync(0xFFFFFFFFu, g0, 0);
        if (g0 >= items) break;
#pragma unroll 1
        for (uint32_t gi = g0; gi < g0 + batch && gi < items; ++gi) {
            uint32_t pid, dp, base;
            // SPLIT: this is warp `part` of the group's `parts`
            uint32_t parts = 1, part = 0;
            {
                dp = 0;
                uint32_t off = 0;
#pragma unroll
                for (int d = 1; d < kMaxDepth; ++d) {
                    if (gi >= cum[d] && cum[d + 1] > cum[d]) {
                        dp = d;
                        off = cum[d];
                    }
                }
                uint32_t k = gi - off;
                if constexpr (SPLIT) {
                    parts = kSplitParts;
                    part = k % kSplitParts;
                    k /= kSplitParts;
                }
                pid = tv.groups[tv.lvl_base[dp] + k / NH];
                base = (k % NH) * SL;
            }
            const long long t_group = DEBUG ? clock64() : 0;
            const uint32_t plink = tv.link[pid];
            const uint32_t nc = plink >> 28;
            const uint32_t fc = plink & kLinkMask;
            // batched systems: the group's own system, theta and root; its
            // shallow leaves belong to the split groups or k_heavy_leaf
            uint32_t gsys = 0;
            float th2 = theta2;
            if (tv.part_sys) {
                gsys = tv.part_sys[tv.info[pid].x];
                th2 = tv.sys_theta2[gsys];
                const bool many = tv.sys_cap[gsys] >= kDenseCap;
                if (SPLIT && ((int)dp >= tv.sys_shallow[gsys] || many != MERGE)) continue;
                if (MODE == MODE_LEAF && !SPLIT) {
                    const bool dense = many || tv.sys_maxleaf[gsys] >= kDenseSwitch;
                    if ((int)dp < tv.sys_shallow[gsys] ||
                        (MERGE ? !many : (DENSE && !XL) ? !dense || many : dense != DENSE))
                        continue;
                }
            }
            uint32_t cl = 0;
            float4 cg = make_float4(0.f, 0.f, 0.f, 0.f);
            if (lane < nc) {
                cg = tv.geo[fc + lane];
                cl = tv.link[fc + lane];
            }
            const uint32_t leaf_mask =
                __ballot_sync(0xFFFFFFFFu, lane < nc && (cl >> 28) == 0) & 0xFFu;
            uint32_t tgt_mask = MODE == MODE_INTERNAL ? (((1u << nc) - 1u) & ~leaf_mask)
                                                      : leaf_mask;
            // The targets are numbered without gaps, so that the pairs (and
            // order 1's halves) run full; where k_dense_p2p takes the P2P they
            // keep their child numbers, which its source masks refer to.
            uint32_t slot = lane;
            bool tgt = lane < nc;
            if constexpr (COMPACT) {
                slot = __popc(tgt_mask & lt_mask);
                tgt = (tgt_mask >> lane) & 1u;
                tgt_mask = (1u << __popc(tgt_mask)) - 1u;
            }
            const uint32_t nt = COMPACT ? __popc(tgt_mask) : nc;
            tgt_mask &= ((1u << SL) - 1u) << base;
            if (tgt_mask == 0) continue;
            if (tgt) {
                sm.cgeo[slot] = cg;
                sm.tq[slot] = (uint8_t)lane;
            }
            cgp_put(sm.cgp, sm.cgeo, nt);
            if constexpr (MODE == MODE_LEAF) {
                if ((tgt_mask >> lane) & 1u) {
                    const uint4 ci = tv.info[fc + sm.tq[lane]];
                    sm.cpart[lane] = make_uint2(ci.x, ci.y);
                }
            }
            const float thw = sm.cgeo[base].w;  // (siblings are equally wide)
            if (lane < 8) {
                if (DEBUG) sm.dbg_m2l[lane] = 0;
                if constexpr (MODE == MODE_INTERNAL) {
                    sm.ns_cnt[lane] = 0;
                } else {
                    if (DEBUG) sm.dbg_p2p[lane] = 0;
                    if (lane == 0) sm.seg_chunks = sm.seg_cnt = 0;
                }
            }
            // a parent made in this launch: wait until it is final
            if (MODE == MODE_INTERNAL && (int)dp >= A.level && dp >= 2u) {
                const int polls = A.ready_spin > 0 ? A.ready_spin : kReadyPolls;
                if (!wait_ready(&tv.ready[pid], polls, status)) continue;
            }
            // chain group (leaf pass, parent deeper than the near lists
            // reach, K = ns_levels): start from the near list of p's ancestor
            // a at depth K and test its candidates down p's ancestor chain
            // a_{K+1} .. a_dp = p, as the reference's pair recursion does
            // (polesitter.h:1097-1145); what p is not separated from is
            // opened for the leaf children.  No near list below depth K is
            // stored, so nothing grows with theta.
            uint32_t nchain = 0, bnode = pid;
            if constexpr (MODE == MODE_LEAF) {
                if (XL && (int)dp > A.ns_levels) {
                    nchain = dp - (uint32_t)A.ns_levels;
                    uint32_t a = pid;
                    if (lane == 0) {
                        for (uint32_t c = nchain; c > 0; --c) {
                            sm.chain_geo[c - 1] = tv.geo[a];
                            a = tv.parent[a];
                        }
                    }
                    bnode = __shfl_sync(0xFFFFFFFFu, a, 0);
                    __syncwarp();
                    if (GRAD) {
                        // order 1 needs every ancestor's own gradient: chain
                        // groups serve the reference's order 0 only
                        if (lane == 0) set_err(status, PSG_ERR_CHAIN_ORDER);
                        continue;
                    }
                }
            }
            const float4 Lp = tv.lt[bnode];
            bool root_only = dp <= 1;
            const uint32_t* nsl = nullptr;
            uint32_t nsn = 0, nfirst = 0;
            if (!root_only) {
                nsl = A.ns + tv.ns_off[bnode];
                nsn = tv.ns_cnt[bnode];
            }
            if constexpr (SPLIT) {
                if (root_only) {
                    // the candidates of a group below the root are the root
                    // alone: its warps start from the root's grandchildren,
                    // unless a target is separated from the root or one of
                    // its children (a tiny theta, or centres that rounding
                    // has pulled together): then the first warp takes it whole
                    const uint32_t rl = tv.link[gsys];
                    const uint32_t rc = rl >> 28;
                    bool far = false;
                    if (lane <= rc) {
                        const float4 sg = tv.geo[lane < rc ? (rl & kLinkMask) + lane : gsys];
                        for (uint32_t m = tgt_mask; m; m &= m - 1) {
                            const float4 c = sm.cgeo[__ffs(m) - 1];
                            float dx, dy, dz, d2;
                            far |= mac_separated(c.x, c.y, c.z, c.w, sg.x, sg.y, sg.z, sg.w, th2,
                                                 dx, dy, dz, d2);
                        }
                    }
                    if (__any_sync(0xFFFFFFFFu, far)) {
                        if (part) continue;
                        parts = 1;
                    } else {
                        root_only = false;
                        nfirst = rl & kLinkMask;
                        nsn = rc;
                    }
                }
            }
            // MODE_INTERNAL: reserve |cand| near-list entries per target child
            uint32_t cand_total = 1;
            unsigned long long ns_base = 0;
            bool ns_ok = true;
            if constexpr (MODE == MODE_INTERNAL) {
                if (!root_only) {
                    uint32_t c = 0;
                    for (uint32_t e = lane; e < nsn; e += 32) {
                        const uint32_t nch = nsl[e] >> 28;
                        c += nch ? nch : 1u;
                    }
                    cand_total = warp_sum(c);
                }
                const unsigned long long need =
                    (unsigned long long)__popc(tgt_mask) * cand_total;
                __syncwarp();
                if (need && sm.ns_next + need > sm.ns_end) {
                    const unsigned long long take = need > A.ns_pool ? need : A.ns_pool;
                    unsigned long long b = 0;
                    if (lane == 0) b = atomicAdd(&status->run.ns_used, take);
                    b = __shfl_sync(0xFFFFFFFFu, b, 0);
                    __syncwarp();
                    if (lane == 0) {
                        sm.ns_next = b;
                        sm.ns_end = b + take;
                    }
                    __syncwarp();
                }
                ns_base = sm.ns_next;
                ns_ok = ns_base + need <= A.ns_cap;
                if (!ns_ok && lane == 0) {
                    set_err(status, PSG_ERR_NS_OVERFLOW);
                    atomicOr(&status->run.ns_fail, 1u << (dp + 1));
                }
                __syncwarp();
                if (lane == 0) sm.ns_next = ns_base + need;
            }
            __syncwarp();

            // per pair of children (2k, 2k + 1): field and, for order 1, its
            // gradient, one child in each half of a float2
            float2 acc[SL / 2][3];
#pragma unroll
            for (int k = 0; k < (int)SL / 2; ++k)
                acc[k][0] = acc[k][1] = acc[k][2] = make_float2(0.f, 0.f);
            float2 gacc[GRAD ? SL / 2 : 1][6];
            if constexpr (GRAD) {
#pragma unroll
                for (int k = 0; k < (int)SL / 2; ++k)
#pragma unroll
                    for (int c = 0; c < 6; ++c) gacc[k][c] = make_float2(0.f, 0.f);
            }
            uint32_t ssize = 0, e0 = 0;
            uint32_t pfill = 0, phead = kNone;  // MODE_LEAF: staged / spilled P2P sources
            bool root_pending = root_only;
            float cacc0 = 0.f, cacc1 = 0.f, cacc2 = 0.f;  // chain groups: ancestors' M2L
            bool flushed = false;                         // STREAM: a flush has run
            unsigned long long sinter = 0;                // ... its pairs (debug)
            uint32_t crun = 0;                            // split: candidates passed

            for (;;) {
                // ---- next batch of candidates into cand[0, tot) ----
                uint32_t tot;
                if (root_pending) {
                    if (lane == 0) {
                        sm.cand_node[0] = gsys;  // the (system's) root
                        sm.cand_mask[0] = (uint8_t)tgt_mask;
                        if constexpr (MODE == MODE_LEAF && XL) sm.cand_lvl[0] = 0;
                    }
                    tot = 1;
                    root_pending = false;
                } else if (e0 < nsn &&
                           (MODE == MODE_INTERNAL ||
                            ssize <= (uint32_t)(kStackCap - kStackSlack - kCandBuf))) {
                    // a split group's warp keeps every parts-th candidate, and
                    // reads on until it has a warp's worth of them
                    tot = 0;
                    do {
                        const uint32_t e = e0 + lane;
                        // an entry is an internal source's link or a leaf's id
                        uint32_t s0 = 0, c = 0, link = 0;
                        if (e < nsn) {
                            if (SPLIT && !nsl) {
                                s0 = nfirst + e;
                                link = tv.link[s0];
                            } else {
                                s0 = link = nsl[e];
                            }
                            const uint32_t nch = link >> 28;
                            c = nch ? nch : 1u;
                        }
                        const uint32_t inc = warp_incl_scan(c);
                        const uint32_t all = __shfl_sync(0xFFFFFFFFu, inc, 31);
                        const uint32_t ex = inc - c;
                        const bool lf = (link >> 28) == 0;
                        if (SPLIT && parts > 1u) {
                            const uint32_t off = (part - crun) % kSplitParts;
                            for (uint32_t i = 0; i < c; ++i) {
                                const uint32_t k = ex + i - off;
                                if (k % kSplitParts == 0) {
                                    sm.cand_node[tot + k / kSplitParts] =
                                        lf ? s0 : (link & kLinkMask) + i;
                                    sm.cand_mask[tot + k / kSplitParts] = (uint8_t)tgt_mask;
                                }
                            }
                            if (all > off) tot += (all - off + kSplitParts - 1) / kSplitParts;
                            crun += all;
                        } else {
                            tot = all;
                            // a chain group's candidates are first tested against its
                            // ancestor a_{K+1} alone (level 1, no children)
                            const uint8_t cmk = (uint8_t)((XL && nchain) ? 0u : tgt_mask);
                            for (uint32_t i = 0; i < c; ++i) {
                                sm.cand_node[ex + i] = lf ? s0 : (link & kLinkMask) + i;
                                sm.cand_mask[ex + i] = cmk;
                                if constexpr (MODE == MODE_LEAF && XL)
                                    sm.cand_lvl[ex + i] = nchain ? 1 : 0;
                            }
                        }
                        e0 += 32;
                    } while (SPLIT && parts > 1u && tot < 32u && e0 < nsn);
                } else if (MODE == MODE_LEAF && ssize > 0) {
                    // pop entries (bounded so the stack cannot overflow) and
                    // open them: an internal node's candidates are its
                    // children, a leaf's (pushed by a chain test) itself
                    const int room = ((int)kStackCap - kStackSlack - (int)ssize) / 7;
                    const uint32_t kp = (uint32_t)min(32, min((int)ssize, max(1, room)));
                    uint32_t node = 0, mask = 0, lvl = 0;
                    if constexpr (MODE == MODE_LEAF) {
                        if (lane < kp) {
                            node = sm.stk_node[ssize - kp + lane];
                            mask = sm.stk_mask[ssize - kp + lane];
                            if constexpr (XL) lvl = sm.stk_lvl[ssize - kp + lane];
                        }
                    }
                    __syncwarp();
                    ssize -= kp;
                    const uint32_t link = node;  // (a leaf's id in chain groups)
                    const uint32_t nch = link >> 28;
                    const uint32_t c = lane < kp ? (XL && nch == 0 ? 1u : nch) : 0u;
                    const uint32_t inc = warp_incl_scan(c);
                    tot = __shfl_sync(0xFFFFFFFFu, inc, 31);
                    const uint32_t ex = inc - c;
                    for (uint32_t i = 0; i < c; ++i) {
                        sm.cand_node[ex + i] = nch ? (link & kLinkMask) + i : node;
                        sm.cand_mask[ex + i] = (uint8_t)mask;
                        if constexpr (MODE == MODE_LEAF && XL) sm.cand_lvl[ex + i] = (uint8_t)lvl;
                    }
                } else {
                    break;
                }
                __syncwarp();

                // ---- test the candidates, one per lane; the next chunk's node
                // records are loaded while the current one is processed ----
                uint32_t n_s = 0, n_mask = 0, n_link = 0, n_lvl = 0;
                float4 n_g = make_float4(0.f, 0.f, 0.f, 0.f), n_mp = n_g;
                if (lane < tot) {
                    n_s = sm.cand_node[lane];
                    n_mask = sm.cand_mask[lane];
                    if constexpr (MODE == MODE_LEAF && XL) n_lvl = sm.cand_lvl[lane];
                    n_g = tv.geo[n_s];
                    n_mp = tv.mp[n_s];
                    n_link = tv.link[n_s];
                }
#pragma unroll 1
                for (uint32_t j0 = 0; j0 < tot; j0 += 32) {
                    const uint32_t s = n_s, smask = n_mask, slink = n_link, slvl = n_lvl;
                    const float4 sg = n_g, smp = n_mp;
                    {
                        const uint32_t jn = j0 + 32 + lane;
                        n_mask = 0;
                        n_lvl = 0;
                        if (jn < tot) {
                            n_s = sm.cand_node[jn];
                            n_mask = sm.cand_mask[jn];
                            if constexpr (MODE == MODE_LEAF && XL) n_lvl = sm.cand_lvl[jn];
                            n_g = tv.geo[n_s];
                            n_mp = tv.mp[n_s];
                            n_link = tv.link[n_s];
                        }
                    }
                    const uint32_t chunk_mask = __reduce_or_sync(0xFFFFFFFFu, smask);
                    uint32_t sep = 0;  // targets the candidate is separated from
                    const float hs = __fadd_rn(thw, sg.w);
                    const float mac = __fmul_rn(th2, __fmul_rn(hs, hs));
                    // children two at a time: the MAC per child (mac_separated,
                    // scalar, so its decisions are the reference's), then the
                    // M2L of m2l_field(_grad) for both children in paired FP32
                    // instructions, each half rounding as the scalar form does
#pragma unroll
                    for (uint32_t k = 0; k < SL / 2; ++k) {
                        const uint32_t q = base + 2 * k;  // children q and q + 1
                        if (!((chunk_mask >> q) & 3u)) continue;
                        const float4 ga = sm.cgp[q >> 1][0], gb = sm.cgp[q >> 1][1];
                        float dx0, dy0, dz0, d20, dx1, dy1, dz1, d21;
                        const bool m0 = mac_far(ga.x, ga.z, gb.x, sg, mac, dx0, dy0, dz0, d20);
                        const bool m1 = mac_far(ga.y, ga.w, gb.y, sg, mac, dx1, dy1, dz1, d21);
                        sep |= (m0 ? 1u << q : 0u) | (m1 ? 2u << q : 0u);
                        const float2 dx = make_float2(dx0, dx1), dy = make_float2(dy0, dy1),
                                     dz = make_float2(dz0, dz1), d2 = make_float2(d20, d21);
                        const bool s0 = m0 && ((smask >> q) & 1u),
                                   s1 = m1 && ((smask >> (q + 1)) & 1u);
                        // branch-free: every lane evaluates; a pair that is not
                        // separated has its 1/r zeroed and adds zeros
                        const float2 soft = __fadd2_rn(d2, make_float2(0.1f, 0.1f));
                        const float2 inv = make_float2(s0 ? rsqrt_soft(soft.x) : 0.f,
                                                       s1 ? rsqrt_soft(soft.y) : 0.f);
                        const float2 inv2 = __fmul2_rn(inv, inv);
                        const float2 ir3 = __fmul2_rn(inv2, inv);
                        const float2 ir5 = __fmul2_rn(ir3, inv2);
                        const float2 mx = make_float2(smp.x, smp.x),
                                     my = make_float2(smp.y, smp.y),
                                     mz = make_float2(smp.z, smp.z),
                                     mw = make_float2(smp.w, smp.w);
                        const float2 mdr =
                            __ffma2_rn(my, dx, __ffma2_rn(mz, dy, __fmul2_rn(mw, dz)));
                        const float2 a = __ffma2_rn(
                            mx, ir3, __fmul2_rn(__fmul2_rn(make_float2(-3.f, -3.f), mdr), ir5));
                        acc[k][0] = __ffma2_rn(dx, a, __ffma2_rn(my, ir3, acc[k][0]));
                        acc[k][1] = __ffma2_rn(dy, a, __ffma2_rn(mz, ir3, acc[k][1]));
                        acc[k][2] = __ffma2_rn(dz, a, __ffma2_rn(mw, ir3, acc[k][2]));
                        if constexpr (GRAD) {
                            // g3 d d^T - gi I, g3 = 3 m0 / r^5, gi = m0 / r^3
                            const float2 g3 =
                                __fmul2_rn(__fmul2_rn(make_float2(3.f, 3.f), mx), ir5);
                            const float2 ngi = __fmul2_rn(make_float2(-mx.x, -mx.y), ir3);
                            const float2 gx = __fmul2_rn(g3, dx), gy = __fmul2_rn(g3, dy);
                            gacc[k][0] = __fadd2_rn(gacc[k][0], __ffma2_rn(gx, dx, ngi));
                            gacc[k][1] = __fadd2_rn(gacc[k][1], __ffma2_rn(gy, dy, ngi));
                            gacc[k][2] = __fadd2_rn(gacc[k][2],
                                                    __ffma2_rn(__fmul2_rn(g3, dz), dz, ngi));
                            gacc[k][3] = __ffma2_rn(gx, dy, gacc[k][3]);
                            gacc[k][4] = __ffma2_rn(gx, dz, gacc[k][4]);
                            gacc[k][5] = __ffma2_rn(gy, dz, gacc[k][5]);
                        }
                        if (DEBUG) {
                            const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, s0);
                            const uint32_t b1 = __ballot_sync(0xFFFFFFFFu, s1);
                            if (lane == 0) {
                                sm.dbg_m2l[q] += __popc(b0);
                                sm.dbg_m2l[q + 1] += __popc(b1);
                            }
                        }
                    }
                    const uint32_t near_bits = smask & ~sep;
                    if constexpr (MODE == MODE_INTERNAL) {
                        // near candidates of internal children: their near lists
                        const uint32_t near_any = __reduce_or_sync(0xFFFFFFFFu, near_bits);
#pragma unroll 1
                        for (uint32_t m = near_any; m; m &= m - 1) {
                            const uint32_t q = __ffs(m) - 1;
                            const bool nr = (near_bits >> q) & 1u;
                            const uint32_t nm = __ballot_sync(0xFFFFFFFFu, nr);
                            const uint32_t have = sm.ns_cnt[q];
                            if (ns_ok && nr) {
                                const uint32_t sub = q - base;
                                A.ns[ns_base + (unsigned long long)sub * cand_total + have +
                                     __popc(nm & lt_mask)] = (slink >> 28) ? slink : s;
                            }
                            __syncwarp();
                            if (lane == 0) sm.ns_cnt[q] = have + __popc(nm);
                            __syncwarp();
                        }
                    } else {
                        const bool sleaf = (slink >> 28) == 0;
                        // chain candidates: the MAC against their ancestor
                        // target; separated -> M2L into the chain's field,
                        // else opened for the next ancestor (past p: for the
                        // leaf children, with the whole target mask)
                        bool cpush = false;
                        uint32_t cmask = 0, clvl = 0;
                        if (XL && nchain && __any_sync(0xFFFFFFFFu, slvl != 0)) {
                            if (slvl) {
                                const float4 cg = sm.chain_geo[slvl - 1];
                                float dx, dy, dz, d2;
                                if (mac_separated(cg.x, cg.y, cg.z, cg.w, sg.x, sg.y, sg.z, sg.w,
                                                  th2, dx, dy, dz, d2)) {
                                    float fx, fy, fz;
                                    m2l_field(dx, dy, dz, d2, smp, fx, fy, fz);
                                    cacc0 += fx;
                                    cacc1 += fy;
                                    cacc2 += fz;
                                } else {
                                    cpush = true;
                                    cmask = slvl == nchain ? tgt_mask : 0u;
                                    clvl = slvl == nchain ? 0u : slvl + 1;
                                }
                            }
                        }
                        // near leaf candidate: a P2P source of these children
                        const uint32_t pbits = sleaf ? near_bits : 0u;
                        const uint32_t pb = __ballot_sync(0xFFFFFFFFu, pbits != 0);
                        if (pb) {
                            // neighbouring leaves that follow one another in
                            // memory and serve the same children (siblings, as
                            // a rule) make one source range, which ends with the
                            // last source before the next one's
                            uint32_t hb = pb;
                            uint2 r = make_uint2(0u, 0u);
                            if (MERGE) {
                                uint32_t end = 0;
                                if (pbits) {
                                    const uint4 si = tv.info[s];
                                    r.x = si.x;
                                    end = si.x + si.y;
                                }
                                const uint32_t below = pb & lt_mask;
                                const int prev = below ? 31 - __clz(below) : (int)lane;
                                const uint32_t pe = __shfl_sync(0xFFFFFFFFu, end, prev),
                                               pm = __shfl_sync(0xFFFFFFFFu, pbits, prev);
                                hb = __ballot_sync(0xFFFFFFFFu,
                                                   pbits && !(below && pm == pbits && pe == r.x));
                                const uint32_t after = hb & ~(lt_mask | (1u << lane));
                                const uint32_t upto =
                                    after ? pb & ((after & (0u - after)) - 1u) : pb;
                                r.y = __shfl_sync(0xFFFFFFFFu, end, 31 - __clz(upto)) - r.x;
                            }
                            if (pfill + __popc(hb) > (uint32_t)kP2PCap) {
                                if (XL && A.stream) {
                                    stream_p2p<DEBUG, GRAD>(sm, A, tgt_mask, fc, pfill, kNone,
                                                            flushed, false, sinter);
                                    flushed = true;
                                } else {
                                    phead = spill_p2p(sm, pfill, phead, A, tgt_mask, fc, DENSE,
                                                      MERGE);
                                }
                                pfill = 0;
                            }
                            if (MERGE ? ((hb >> lane) & 1u) : pbits) {
                                const uint32_t pos = pfill + __popc(hb & lt_mask);
                                if (MERGE)
                                    sm.p2p_range[pos] = r;
                                else
                                    sm.p2p_node[pos] = s;
                                sm.p2p_mask[pos] = (uint8_t)pbits;
                            }
                            pfill += __popc(hb);
                            if (DEBUG) {
                                const uint32_t pany = __reduce_or_sync(0xFFFFFFFFu, pbits);
                                for (uint32_t m = pany; m; m &= m - 1) {
                                    const uint32_t q = __ffs(m) - 1;
                                    const uint32_t c =
                                        __popc(__ballot_sync(0xFFFFFFFFu, (pbits >> q) & 1u));
                                    if (lane == 0) sm.dbg_p2p[q] += c;
                                }
                            }
                        }
                        // near internal candidate: open it later for these children
                        const uint32_t qbits = sleaf ? 0u : near_bits;
                        const bool push = qbits != 0 || cpush;
                        const uint32_t qb = __ballot_sync(0xFFFFFFFFu, push);
                        if (qb) {
                            const uint32_t pos = ssize + __popc(qb & lt_mask);
                            if (push && pos < (uint32_t)kStackCap) {
                                sm.stk_node[pos] = (XL && sleaf) ? s : slink;
                                sm.stk_mask[pos] = (uint8_t)(cpush ? cmask : qbits);
                                if constexpr (XL) sm.stk_lvl[pos] = (uint8_t)(cpush ? clvl : 0u);
                            }
                            ssize += __popc(qb);
                            if (ssize > (uint32_t)kStackCap) {
                                if (lane == 0) set_err(status, PSG_ERR_STACK);
                                ssize = kStackCap;
                            }
                        }
                    }
                    __syncwarp();
                }
                if (MODE == MODE_LEAF && DEBUG && lane == 0) atomicMax(&status->max_stack, ssize);
            }

            // ---- L2L: L(u) = M2L(u) + L(parent)  (polesitter.h:1248-1250) ----
            // closure order 1 shifts the parent's field to the child's centre:
            // L(u) = M2L(u) + L(p) + G(p) (c_u - c_p), G(u) = M2L_G(u) + G(p).
            // A chain group's parent field is L(a) + the chain's M2L.
            float4 Lb = Lp;
            if (XL && nchain) {
                Lb.y = __fadd_rn(Lb.y, warp_sum(cacc0));
                Lb.z = __fadd_rn(Lb.z, warp_sum(cacc1));
                Lb.w = __fadd_rn(Lb.w, warp_sum(cacc2));
            }
            // a split group: this warp's sums and source list are put down, and
            // the warp that comes last adds them all up in warp order
            const float* psum = nullptr;
            if constexpr (SPLIT) {
                if (parts > 1u) {
                    const uint32_t sidx = gi / kSplitParts;
                    float* own = A.split.sums + (size_t)gi * kSplitSums;
#pragma unroll
                    for (uint32_t k = 0; k < SL; ++k) {
                        if (!((tgt_mask >> (base + k)) & 1u)) continue;
#pragma unroll
                        for (uint32_t c = 0; c < (GRAD ? 9u : 3u); ++c) {
                            const float2 v2 = c < 3u ? acc[k >> 1][c]
                                                     : gacc[GRAD ? (k >> 1) : 0][c < 3u ? 0 : c - 3u];
                            const float v = warp_sum((k & 1) ? v2.y : v2.x);
                            if (lane == 0) __stcg(own + k * (GRAD ? 9u : 3u) + c, v);
                        }
                        if (DEBUG && lane == 0) {
                            const uint32_t q = base + k;
                            atomicAdd(&tv.dbg_m2l[fc + q], sm.dbg_m2l[q]);
                            atomicAdd(&tv.dbg_p2p[fc + q], sm.dbg_p2p[q]);
                            atomicAdd(&status->stat[PSG_STAT_M2L],
                                      (unsigned long long)sm.dbg_m2l[q]);
                            atomicAdd(&status->stat[PSG_STAT_P2P_PAIRS],
                                      (unsigned long long)sm.dbg_p2p[q]);
                        }
                    }
                    if (pfill) phead = spill_p2p(sm, pfill, phead, A, tgt_mask, fc, true, MERGE);
                    if (phead != kNone)
                        record_dense(sm, A.dense, tgt_mask, fc, phead, true, true, status);
                    uint32_t done = 0;
                    if (lane == 0) {
                        __stcg(&A.split.list[gi],
                               make_uint4(sm.seg_first, sm.seg_prev, sm.seg_cnt, 0u));
                        __threadfence();
                        done = atomicAdd(&A.split.count[sidx], 1u);
                    }
                    done = __shfl_sync(0xFFFFFFFFu, done, 0);
                    if (done + 1u != parts) continue;
                    __threadfence();
                    link_split(sm, A, tgt_mask, fc, sidx);
                    psum = A.split.sums + (size_t)sidx * kSplitParts * kSplitSums +
                           lane * kSplitSums;
                }
            }
            // the sum of a lane's value over the warp, or of the split group's
            // warps' sums
            auto total_of = [&](float v, uint32_t k, uint32_t c) {
                if (SPLIT && psum)
                    v = lane < (uint32_t)kSplitParts ? __ldcg(psum + k * (GRAD ? 9u : 3u) + c)
                                                     : 0.f;
                return warp_sum(v);
            };
            float4 Gp0 = make_float4(0.f, 0.f, 0.f, 0.f), cp = Gp0;
            float2 Gp1 = make_float2(0.f, 0.f);
            if constexpr (GRAD) {
                cp = tv.geo[pid];
                if (dp >= 2) {
                    Gp0 = tv.lg0[pid];
                    Gp1 = tv.lg1[pid];
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < SL; ++k) {
                const uint32_t q = base + k;
                if (!((tgt_mask >> q) & 1u)) continue;
                const float2* ak = acc[k >> 1];
                const float ax = total_of((k & 1) ? ak[0].y : ak[0].x, k, 0);
                const float ay = total_of((k & 1) ? ak[1].y : ak[1].x, k, 1);
                const float az = total_of((k & 1) ? ak[2].y : ak[2].x, k, 2);
                float4 L = make_float4(0.f, __fadd_rn(ax, Lb.y), __fadd_rn(ay, Lb.z),
                                       __fadd_rn(az, Lb.w));
                float4 G0 = Gp0;
                float2 G1 = Gp1;
                if constexpr (GRAD) {
                    const float4 cu = sm.cgeo[q];
                    const float3 sh = grad_apply(Gp0, Gp1, cu.x - cp.x, cu.y - cp.y, cu.z - cp.z);
                    L.y += sh.x;
                    L.z += sh.y;
                    L.w += sh.z;
                    const float2* gk = gacc[k >> 1];
                    G0.x += total_of((k & 1) ? gk[0].y : gk[0].x, k, 3);
                    G0.y += total_of((k & 1) ? gk[1].y : gk[1].x, k, 4);
                    G0.z += total_of((k & 1) ? gk[2].y : gk[2].x, k, 5);
                    G0.w += total_of((k & 1) ? gk[3].y : gk[3].x, k, 6);
                    G1.x += total_of((k & 1) ? gk[4].y : gk[4].x, k, 7);
                    G1.y += total_of((k & 1) ? gk[5].y : gk[5].x, k, 8);
                }
                if (lane == 0) {
                    const uint32_t u = fc + sm.tq[q];
                    tv.lt[u] = L;
                    if constexpr (GRAD) {
                        tv.lg0[u] = G0;
                        tv.lg1[u] = G1;
                    }
                    if constexpr (MODE == MODE_LEAF) {
                        sm.sL[q] = L;
                        if constexpr (GRAD) {
                            sm.sG0[q] = G0;
                            sm.sG1[q] = G1;
                        }
                    } else {
                        const uint32_t sub = q - base;
                        tv.ns_off[u] = (uint32_t)(ns_base + (unsigned long long)sub * cand_total);
                        tv.ns_cnt[u] = ns_ok ? sm.ns_cnt[q] : 0u;
                    }
                    if (DEBUG && !(SPLIT && parts > 1u)) {
                        tv.dbg_m2l[u] = sm.dbg_m2l[q];
                        atomicAdd(&status->stat[PSG_STAT_M2L], (unsigned long long)sm.dbg_m2l[q]);
                    }
                }
            }
            __syncwarp();
            if constexpr (MODE == MODE_INTERNAL) {
                // lists and fields of this group's children are final
                if (A.ready_spin > 0 && (int)dp + 1 == A.level) publish_late();
                if ((tgt_mask >> lane) & 1u) {
                    __threadfence();
                    __stcg(&tv.ready[fc + sm.tq[lane]], 1u);
                }
            }

            if constexpr (MODE == MODE_LEAF) {
                if (SPLIT && parts > 1u) continue;  // (its P2P and L2P: k_dense_p2p)
                leaf_epilogue<DEBUG, GRAD, DENSE>(sm, A, tgt_mask, fc, pfill, phead,
                                                  MERGE,
                                                  XL && A.stream != 0, flushed, sinter);
                if (DEBUG && lane == 0) {
                    const unsigned long long cyc = (unsigned long long)(clock64() - t_group);
                    atomicMax(&status->stat[PSG_STAT_SLOWEST_GROUP],
                              (min(cyc, (1ull << 36) - 1) << 28) | pid);
                }
            }
        }
    }
}

// L2P + P2P of the full leaves recorded by the leaf pass.  A warp takes one
// record at a time from a shared counter: up to 16 target particles of a run
// of leaves, and the chain of source leaves (or a segment of it) that their
// group found.  The lanes own sources: the source leaves' particles are laid
// end to end over the lanes, and each lane sums its particle into its own
// accumulators of every target, two targets at a time in the paired FP32
// instructions (__fadd2_rn, __ffma2_rn, __fmul2_rn; one issued instruction
// does a step of two pairs).  At the record's end the lanes' sums are added.
// So targets are padded to the pair only, sources not at all, a source's
// load and lookup serve all targets, and no source passes through shared
// memory.  A source that serves only some leaves of the record (its child
// mask) has its mass zeroed for the other targets; such sources are set aside
// and summed 32 or more at a time, so that every other step skips the masks
// (one mixed stream, masked wherever a lane needed it: 6.48 against 6.17 ms in
// the 1M tick below).
//
// Bound: the FP32 pipe.  A step on a pair of targets is 12 paired FP32
// instructions of two cycles and 2 MUFU; alone in a loop that takes 32 cycles
// per scheduler (2.3e12 particle pairs/s on 148 SMs).  16 targets a record
// and 4 blocks per SM (128 registers) is the best of 8-24 targets and 2-6
// blocks measured: the accumulators' registers trade against the warps that
// hide the chain's latency.  Measured at 1M clumpy, theta 6.25, leaf capacity
// 16 (8.2 G pairs): closure tick 14.2 -> 13.0 ms against lanes that owned
// targets, with sources staged in shared-memory tiles and a second walk per
// leaf for partly wanted sources; with the masked sources apart and merged
// source leaves this kernel takes 5.5 ms of it (1.5e12 pairs/s).
//
// Sums are taken in chain order, the lanes and the segments added in a fixed
// order, so the result does not depend on scheduling.

// a spilled chunk as one lane sees it: the chunk's entry count and link,
// and the lane's entry (its source and child mask; slots past the count hold
// stale values and are not used)
struct ChunkHead {
    uint32_t cnt, next, mask;
    uint2 src;
};

__device__ __forceinline__ ChunkHead load_chunk(const P2PStore& st, uint32_t c, uint32_t lane) {
    ChunkHead h{0u, kNone, 0u, make_uint2(0u, 0u)};
    if (c != kNone) {
        h.cnt = st.cnt[c];
        h.next = st.next[c];
        h.src = st.src[(size_t)c * kP2PChunk + lane];
        h.mask = st.mask[(size_t)c * kP2PChunk + lane];
    }
    return h;
}

// Two of a record's targets (negated, one in each half of a float2) and this
// lane's sums for them.
template <bool KAHAN>
struct DensePair {
    float2 sx, sy, sz;
};
template <>
struct DensePair<true> {
    float2 sx, sy, sz, cx, cy, cz;
};

struct DenseSmem {
    uint2 ent[32];
    uint2 part[64];   // partly wanted entries: first particle, particles
    uint16_t ptm[64]; // ... and the targets that want them
    float4 txy[kDenseTargets / 2];  // a pair's targets, negated: x, x', y, y'
    float2 tz[kDenseTargets / 2];
};

__device__ __forceinline__ void kahan_add(float2& s, float2& c, float2 v) {
    const float2 y = __fadd2_rn(v, make_float2(-c.x, -c.y));
    const float2 t = __fadd2_rn(s, y);
    const float2 d = __fadd2_rn(t, make_float2(-s.x, -s.y));
    c = __fadd2_rn(d, make_float2(-y.x, -y.y));
    s = t;
}

// source particle p on target pair k, where the set tm holds the targets that
// want it (polesitter.h:1424-1444 with rsqrt)
template <bool KAHAN, bool MASKED>
__device__ __forceinline__ void dense_pair(DensePair<KAHAN>& a, const DenseSmem& sm, float4 p,
                                           uint32_t tm, int k) {
    const float4 txy = sm.txy[k];
    const float2 tz = sm.tz[k];
    float2 pw = make_float2(p.w, p.w);
    if constexpr (MASKED) {
        if (!(tm & (1u << (2 * k)))) pw.x = 0.f;
        if (!(tm & (2u << (2 * k)))) pw.y = 0.f;
    }
    const float2 dx = __fadd2_rn(make_float2(p.x, p.x), make_float2(txy.x, txy.y));
    const float2 dy = __fadd2_rn(make_float2(p.y, p.y), make_float2(txy.z, txy.w));
    const float2 dz = __fadd2_rn(make_float2(p.z, p.z), tz);
    float2 r = __ffma2_rn(dz, dz, make_float2(0.1f, 0.1f));
    r = __ffma2_rn(dy, dy, r);
    r = __ffma2_rn(dx, dx, r);
    const float2 i = make_float2(rsqrt_soft(r.x), rsqrt_soft(r.y));
    const float2 f = __fmul2_rn(pw, __fmul2_rn(__fmul2_rn(i, i), i));
    if constexpr (KAHAN) {
        kahan_add(a.sx, a.cx, __fmul2_rn(dx, f));
        kahan_add(a.sy, a.cy, __fmul2_rn(dy, f));
        kahan_add(a.sz, a.cz, __fmul2_rn(dz, f));
    } else {
        a.sx = __ffma2_rn(dx, f, a.sx);
        a.sy = __ffma2_rn(dy, f, a.sy);
        a.sz = __ffma2_rn(dz, f, a.sz);
    }
}

constexpr int kDensePairs = (int)kDenseTargets / 2;
constexpr int kDenseBlock = 2;
constexpr uint32_t kDenseMany = 64;  // records a warp from which they are loaded ahead

// one step: a lane's source p on the record's np target pairs, kDenseBlock
// pairs at a time (their chains of dependent instructions overlap; 1 or 4 at a
// time: 6.87 and 6.48 against 6.17 ms in the 1M tick below).  MASKED: tm
// are the targets that want p, want those that any lane's source is wanted by.
template <bool KAHAN, bool MASKED>
__device__ __forceinline__ void dense_step(DensePair<KAHAN> (&a)[kDensePairs],
                                           const DenseSmem& sm, float4 p, uint32_t tm,
                                           uint32_t want, uint32_t np) {
#pragma unroll
    for (int k = 0; k < kDensePairs; k += kDenseBlock) {
        constexpr uint32_t block = (1u << (2 * kDenseBlock)) - 1u;
        if (MASKED ? ((want >> (2 * k)) & block) != 0u : (k == 0 || np > (uint32_t)k)) {
#pragma unroll
            for (int j = 0; j < kDenseBlock; ++j)
                dense_pair<KAHAN, MASKED>(a[k + j], sm, p, tm, k + j);
        }
    }
}

// Entries of source leaves held one per lane (en particles, 0: none), laid end
// to end from position start; ent holds each one's first particle less its
// start (and its targets), compacted past empty entries.
struct DenseRun {
    uint32_t en, start, before, b;
    // the entry (in ent) of this lane's position b + lane: the last to start at
    // or before it; warp-collective, for successive b
    __device__ __forceinline__ uint32_t entry(uint32_t le_mask) {
        const uint32_t d = start - b;
        const uint32_t bits =
            __reduce_or_sync(0xFFFFFFFFu, (en != 0u && d < 32u) ? 1u << d : 0u);
        const uint32_t e = before + __popc(bits & le_mask);
        before += __popc(bits);
        return e ? e - 1u : 0u;
    }
};

// one record
template <bool KAHAN>
__device__ __forceinline__ void dense_record(const TravArgs& A, DenseSmem& sm, uint4 rec,
                                             uint32_t slot, unsigned long long& inter) {
    const TreeView& tv = A.tv;
    const float4* __restrict__ xyzm = A.xyzm;
    const uint32_t lane = lane_id(), le_mask = lanemask_lt() | (1u << lane);
    const uint32_t fc = rec.x, run = rec.w >> 8, cnt = rec.w & 0xFFu, first = rec.z;
    const uint32_t np = (cnt + 1u) >> 1;
    // lane k < cnt: target k, its leaf (the child of the run that holds it)
    const uint32_t ti = first + min(lane, cnt - 1u);
    uint32_t q = __ffs(run) - 1;
    for (uint32_t m = run & (run - 1u); m; m &= m - 1) {
        const uint32_t qq = __ffs(m) - 1;
        if (tv.info[fc + qq].x <= ti) q = qq;
    }
    const float4 t = xyzm[ti];
    // the record's leaves, and per leaf (in lane q) the set of its targets
    const uint32_t leaves = __reduce_or_sync(0xFFFFFFFFu, 1u << q);
    uint32_t tset = 0;
    for (uint32_t m = leaves; m; m &= m - 1) {
        const uint32_t qq = __ffs(m) - 1;
        const uint32_t b = __ballot_sync(0xFFFFFFFFu, lane < cnt && q == qq);
        if (lane == qq) tset = b;
    }
    DensePair<KAHAN> a[kDensePairs];
#pragma unroll
    for (int k = 0; k < kDensePairs; ++k) {
        a[k].sx = a[k].sy = a[k].sz = make_float2(0.f, 0.f);
        if constexpr (KAHAN) a[k].cx = a[k].cy = a[k].cz = make_float2(0.f, 0.f);
    }
    __syncwarp();
    if (lane < kDenseTargets) {  // (slots past cnt: the last target again, not used)
        float* xy = reinterpret_cast<float*>(&sm.txy[lane >> 1]);
        xy[lane & 1u] = -t.x;
        xy[2 + (lane & 1u)] = -t.y;
        reinterpret_cast<float*>(&sm.tz[lane >> 1])[lane & 1u] = -t.z;
    }
    __syncwarp();
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    // chunks one ahead: the next chunk's source ranges and the header after
    // it are in flight while a chunk is summed
    auto src_range = [&](const ChunkHead& hh) -> uint2 {
        if (lane < hh.cnt && (hh.mask & leaves) != 0u) return source_range(tv, hh.src);
        return make_uint2(0u, 0u);
    };
    ChunkHead h = load_chunk(A.p2p, rec.y, lane);
    uint2 hr = src_range(h);
    ChunkHead hn = load_chunk(A.p2p, h.next, lane);
    uint32_t c = rec.y;
    // wholly wanted sources: positions left over from a chunk (fewer than 32)
    // are carried into the next, and the particle loaded in one step is summed
    // in the next one
    uint32_t carry = 0, carry_idx = 0, npart = 0;
    float4 p = none;
    for (bool more = true; more;) {
        uint32_t em = 0, en_all = 0, es = 0;
        more = c != kNone;
        if (more) {
            em = lane < h.cnt ? (h.mask & leaves) : 0u;
            es = hr.x;
            en_all = hr.y;
            c = h.next;
            h = hn;
            hr = src_range(h);
            hn = load_chunk(A.p2p, h.next, lane);
        }
        DenseRun w;
        w.en = em == leaves ? en_all : 0u;
        w.before = w.b = 0;
        const uint32_t incl = warp_incl_scan(w.en);
        const uint32_t total = carry + __shfl_sync(0xFFFFFFFFu, incl, 31);
        w.start = carry + incl - w.en;
        const uint32_t full = __ballot_sync(0xFFFFFFFFu, w.en != 0u);
        // partly wanted entries: collected, and summed when 32 are in
        const bool partial = em != 0u && em != leaves;
        const uint32_t pb = __ballot_sync(0xFFFFFFFFu, partial);
        __syncwarp();
        if (w.en) sm.ent[__popc(full & lanemask_lt())].x = es - w.start;
        if (pb) {
            uint32_t tm = 0;
            for (uint32_t m = leaves; m; m &= m - 1) {
                const uint32_t qq = __ffs(m) - 1;
                const uint32_t v = __shfl_sync(0xFFFFFFFFu, tset, qq);
                tm |= ((em >> qq) & 1u) ? v : 0u;
            }
            if (partial) {
                const uint32_t pos = npart + __popc(pb & lanemask_lt());
                sm.part[pos] = make_uint2(es, en_all);
                sm.ptm[pos] = (uint16_t)tm;
            }
            npart += __popc(pb);
            if (A.debug) inter += partial ? (unsigned long long)en_all * __popc(tm) : 0ull;
        }
        __syncwarp();
        if (A.debug) inter += (unsigned long long)w.en * cnt;
        // at the chain's end: the remainder, and the step that sums it
        const uint32_t steps = more ? total >> 5 : ((total + 31u) >> 5) + 1u;
#pragma unroll 1
        for (uint32_t st = 0; st < steps; ++st, w.b += 32) {
            const uint32_t f = w.b + lane;
            const uint32_t at = sm.ent[w.entry(le_mask)].x + f;
            const float4 pn = f < total ? xyzm[f < carry ? carry_idx : at] : none;
            dense_step<KAHAN, false>(a, sm, p, 0u, 0u, np);
            p = pn;
        }
        if (more && w.b < total) {
            const uint32_t f = w.b + lane;
            const uint32_t at = sm.ent[w.entry(le_mask)].x + f;
            if (f >= carry) carry_idx = at;  // (lanes past the remainder are not used)
        }
        carry = more ? total - w.b : 0u;
        while (npart >= 32u || (!more && npart)) {
            const uint32_t take = min(npart, 32u);
            __syncwarp();
            const uint2 e0 = lane < take ? sm.part[lane] : make_uint2(0u, 0u);
            const uint32_t t0 = sm.ptm[lane];
            const uint2 e1 = sm.part[32 + lane];
            const uint16_t t1 = sm.ptm[32 + lane];
            __syncwarp();
            sm.part[lane] = e1;
            sm.ptm[lane] = t1;
            npart -= take;
            DenseRun v;
            v.en = e0.y;
            v.before = v.b = 0;
            const uint32_t pincl = warp_incl_scan(v.en);
            const uint32_t ptot = __shfl_sync(0xFFFFFFFFu, pincl, 31);
            v.start = pincl - v.en;
            const uint32_t pfull = __ballot_sync(0xFFFFFFFFu, v.en != 0u);
            if (v.en) sm.ent[__popc(pfull & lanemask_lt())] = make_uint2(e0.x - v.start, t0);
            __syncwarp();
            float4 pp = none;
            uint32_t tm = 0;
#pragma unroll 1
            for (; v.b < ptot + 32u; v.b += 32) {
                const uint32_t f = v.b + lane;
                const uint2 at = sm.ent[v.entry(le_mask)];
                const bool in = f < ptot;
                const float4 pn = in ? xyzm[at.x + f] : none;
                const uint32_t want = __reduce_or_sync(0xFFFFFFFFu, tm);
                dense_step<KAHAN, true>(a, sm, pp, tm, want, np);
                pp = pn;
                tm = in ? at.y : 0u;
            }
        }
    }
    // the lanes' sums; lane k keeps target k's
    double bx = 0.0, by = 0.0, bz = 0.0;
#pragma unroll
    for (int k = 0; k < kDensePairs; ++k) {
        if (k > 0 && np <= (uint32_t)k) continue;
        using Sum = typename std::conditional<KAHAN, double, float>::type;
        Sum v[6] = {a[k].sx.x, a[k].sx.y, a[k].sy.x, a[k].sy.y, a[k].sz.x, a[k].sz.y};
        if constexpr (KAHAN) {
            v[0] -= a[k].cx.x;
            v[1] -= a[k].cx.y;
            v[2] -= a[k].cy.x;
            v[3] -= a[k].cy.y;
            v[4] -= a[k].cz.x;
            v[5] -= a[k].cz.y;
        }
#pragma unroll
        for (int j = 0; j < 6; ++j) v[j] = warp_sum(v[j]);
        if ((lane >> 1) == (uint32_t)k) {
            bx = (lane & 1u) ? v[1] : v[0];
            by = (lane & 1u) ? v[3] : v[2];
            bz = (lane & 1u) ? v[5] : v[4];
        }
    }
    // a segment of a longer list: its sums go to its slot, and the segment
    // that comes last adds them all, from the list's end
    if (slot != kNone) {
        const DenseStore& ds = A.dense;
        double* own = ds.sums + (size_t)slot * kDenseTargets * 3;
        if (lane < cnt) {
            __stcg(own + 3 * lane, bx);
            __stcg(own + 3 * lane + 1, by);
            __stcg(own + 3 * lane + 2, bz);
        }
        __threadfence();
        __syncwarp();
        uint4* item = ds.item + first;
        uint32_t done = 0;
        if (lane == 0) done = atomicAdd(&item->z, 1u);
        done = __shfl_sync(0xFFFFFFFFu, done, 0);
        if (done + 1u != item->y) return;
        __threadfence();
        bx = by = bz = 0.0;
        for (uint32_t sl = item->x; sl != kNone; sl = ds.prev[sl]) {
            if (lane < cnt) {
                const double* v = ds.sums + (size_t)sl * kDenseTargets * 3 + 3 * lane;
                bx += __ldcg(v);
                by += __ldcg(v + 1);
                bz += __ldcg(v + 2);
            }
        }
    }
    if (lane < cnt) {
        const uint32_t u = fc + q;
        const float4 L = tv.lt[u];
        float lx = L.y, ly = L.z, lz = L.w;
        if (A.order >= 1) {
            const float4 cu = tv.geo[u];
            const float3 sh = grad_apply(tv.lg0[u], tv.lg1[u], t.x - cu.x, t.y - cu.y,
                                         t.z - cu.z);
            lx += sh.x;
            ly += sh.y;
            lz += sh.z;
            if (A.leaf_of) A.leaf_of[ti] = u;
        }
        const double mm = (double)t.w;
        A.fx[ti] = (float)(mm * ((double)lx + bx));
        A.fy[ti] = (float)(mm * ((double)ly + by));
        A.fz[ti] = (float)(mm * ((double)lz + bz));
    }
}

template <bool KAHAN>
__global__ void __launch_bounds__(kDenseThreads, KAHAN ? 2 : kDenseBlocksPerSm)
    k_dense_p2p(const __grid_constant__ TravArgs A) {
    __shared__ DenseSmem smem[kDenseWarpsPerBlock];
    DenseSmem& sm = smem[threadIdx.x >> 5];
    Status* status = A.status;
    if (status->err & (PSG_ERR_VOID | PSG_ERR_DENSE_OVERFLOW)) return;
    const uint32_t lane = lane_id();
    const uint32_t total = min(status->run.dense_count, A.dense.rec_cap);
    unsigned long long inter = 0;
    // Many records a warp are short ones, bound by the chain of loads: they are
    // taken two ahead and loaded one ahead (lanes 0-3: the record, lane 4: its
    // slot), while the one before is summed (4M particles, leaf capacity 1, two
    // ticks: 13.05 -> 12.78 ms).  Fewer are taken one by one, since long ones
    // held back leave other warps idle (a 131K closure tick: 0.81 against 0.96
    // ms).
    auto take = [&]() {
        return lane == 0 ? atomicAdd(&status->run.dense_work, 1u) : 0u;
    };
    auto load = [&](uint32_t r) -> uint32_t {
        if (r >= total || lane > 4u) return 0u;
        return lane < 4u ? reinterpret_cast<const uint32_t*>(&A.dense.rec[r])[lane]
                         : A.dense.rec_slot[r];
    };
    const bool many = total >= kDenseMany * gridDim.x * kDenseWarpsPerBlock;
    uint32_t r = __shfl_sync(0xFFFFFFFFu, take(), 0);
    uint32_t word = load(r), ahead = many ? take() : 0u;
    while (r < total) {
        const uint4 rec = make_uint4(__shfl_sync(0xFFFFFFFFu, word, 0),
                                     __shfl_sync(0xFFFFFFFFu, word, 1),
                                     __shfl_sync(0xFFFFFFFFu, word, 2),
                                     __shfl_sync(0xFFFFFFFFu, word, 3));
        const uint32_t slot = __shfl_sync(0xFFFFFFFFu, word, 4);
        if (many) {
            r = __shfl_sync(0xFFFFFFFFu, ahead, 0);
            word = load(r);
            ahead = take();
        }
        dense_record<KAHAN>(A, sm, rec, slot, inter);
        __syncwarp();
        if (!many) {
            r = __shfl_sync(0xFFFFFFFFu, take(), 0);
            word = load(r);
        }
    }
    if (A.debug) {
        inter = warp_sum(inter);
        if (lane == 0 && inter) {
            atomicAdd(&status->stat[PSG_STAT_P2P_INTER], inter);
            atomicAdd(&status->stat[PSG_STAT_DENSE_INTER], inter);
        }
    }
}

// L2L + L2P + P2P of the shallow leaves (depth <= heavy_depth; the leaf
// pass starts below them), one block each.  A shallow leaf is a large cell,
// so its walk -- the reference's (t leaf, s) recursion over the whole
// candidate set -- reaches a large part of the tree; the block runs it
// level-synchronously: the frontier of candidates at one level is tested by
// all threads (separated: M2L, leaf: P2P, else: its children go to the next
// frontier, placed by a block scan).
// Frontier order and the final reduction are fixed, so the result does not
// depend on scheduling.  A one-particle leaf sums its P2P during the walk; a
// leaf holding more (leaf capacity > 1) lists its P2P sources in frontier
// order and sums them per particle afterwards.
constexpr int kHeavyThreads = 512;
constexpr int kHeavyWarps = kHeavyThreads / 32;
constexpr int kHeavyTargets = 8;  // particles of a multi-particle leaf summed together

// exclusive block scan of v; returns the block total
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t& excl, uint32_t* s_w) {
    const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
    const uint32_t inc = warp_incl_scan(v);
    if (lane == 31) s_w[w] = inc;
    __syncthreads();
    uint32_t base = 0, total = 0;
    for (int k = 0; k < kHeavyWarps; ++k) {
        const uint32_t x = s_w[k];
        if (k < (int)w) base += x;
        total += x;
    }
    __syncthreads();
    excl = base + inc - v;
    return total;
}

template <bool DEBUG, bool GRAD>
__global__ void __launch_bounds__(kHeavyThreads, 2) k_heavy_leaf(const __grid_constant__ TravArgs A) {
    __shared__ uint32_t s_w[kHeavyWarps];
    __shared__ uint32_t s_rec;
    __shared__ float s_red[kHeavyWarps][12];
    __shared__ float4 s_g[2];  // multi-particle leaf: field gradient (xx yy zz xy), local field
    __shared__ float2 s_g1;
    __shared__ unsigned long long s_cnt[kHeavyWarps][3];
    __shared__ float s_redt[kHeavyWarps][3 * kHeavyTargets];
    Status* status = A.status;
    // (a run whose near lists ran out is void: see k_trav)
    if (status->err & (PSG_ERR_VOID | PSG_ERR_HEAVY_OVERFLOW | PSG_ERR_NS_OVERFLOW)) return;
    const TreeView& tv = A.tv;
    // work items: the leaf children of the nodes at depths 0 .. heavy_depth-1
    uint32_t cum[kMaxDepth + 1];
    uint32_t total = 0;
    for (int d = 0; d < A.heavy_depth && d < kMaxDepth; ++d) {
        cum[d] = total;
        total += status->lvl_count[d];
    }
    if (total == 0) return;
    const uint32_t tid = threadIdx.x, lane = lane_id(), w = tid >> 5;
    const float theta2 = __fmul_rn(A.theta, A.theta);
    uint32_t* fa = A.heavy_frontier + (size_t)blockIdx.x * 3 * A.heavy_fcap;
    uint32_t* fb = fa + A.heavy_fcap;
    uint32_t* const fp = fa + 2 * (size_t)A.heavy_fcap;  // P2P sources of a multi-particle leaf
    uint32_t leaves = 0, pid = 0, dp = 0, fc = 0;  // current group's leaf children
    uint32_t gsys = 0;                              // ... its system (batched systems)
    float th2 = theta2;
    for (;;) {
        if (leaves == 0) {
            // next group with leaf children
            if (tid == 0) s_rec = atomicAdd(&status->run.heavy_work, 1u);
            __syncthreads();
            const uint32_t g = s_rec;
            __syncthreads();
            if (g >= total) break;
            dp = 0;
            for (int d = 1; d < A.heavy_depth && d < kMaxDepth; ++d)
                if (g >= cum[d]) dp = d;
            pid = tv.lvl_base[dp] + (g - cum[dp]);
            if (tv.part_sys) {
                // batched systems: only the groups shallow for their own system
                gsys = tv.part_sys[tv.info[pid].x];
                if ((int)dp >= tv.sys_shallow[gsys]) continue;
                th2 = tv.sys_theta2[gsys];
            }
            const uint32_t plink = tv.link[pid];
            fc = plink & kLinkMask;
            for (uint32_t q = 0; q < (plink >> 28); ++q)
                if ((tv.link[fc + q] >> 28) == 0) leaves |= 1u << q;
            if (leaves == 0) continue;
        }
        const uint32_t u = fc + __ffs(leaves) - 1;
        leaves &= leaves - 1;
        const float4 ug = tv.geo[u];
        const uint4 ui = tv.info[u];
        const float4 t = A.xyzm[ui.x];
        const bool multi = ui.y > 1u;  // the same for the whole block
        uint32_t np2p = 0;
        // initial candidates: cand(p)
        uint32_t F = 0;
        if (dp <= 1) {
            if (tid == 0) fa[0] = gsys;  // the (system's) root
            F = 1;
        } else {
            const uint32_t* nsl = A.ns + tv.ns_off[pid];
            const uint32_t nsn = tv.ns_cnt[pid];
            for (uint32_t e0 = 0; e0 < nsn; e0 += kHeavyThreads) {
                const uint32_t e = e0 + tid;
                uint32_t s0 = 0, link = 0, c = 0;
                if (e < nsn) {
                    s0 = link = nsl[e];  // an internal source's link or a leaf's id
                    c = (link >> 28) ? (link >> 28) : 1u;
                }
                uint32_t ex;
                const uint32_t tot = block_scan(c, ex, s_w);
                if (F + tot > A.heavy_fcap) {
                    if (tid == 0) set_err(status, PSG_ERR_HEAVY_OVERFLOW);
                    return;
                }
                for (uint32_t i = 0; i < c; ++i)
                    fa[F + ex + i] = (link >> 28) ? (link & kLinkMask) + i : s0;
                F += tot;
            }
        }
        __syncthreads();
        float ax = 0.f, ay = 0.f, az = 0.f;
        float g[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float bx = 0.f, by = 0.f, bz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
        unsigned long long n_m2l = 0, n_p2p = 0, n_inter = 0;
        // one candidate: MAC, then M2L, a P2P source or its children
        auto visit = [&](uint32_t sn, float4 sg, uint32_t& c, uint32_t& link, uint32_t& pf) {
            float dx, dy, dz, d2;
            if (mac_separated(ug.x, ug.y, ug.z, ug.w, sg.x, sg.y, sg.z, sg.w, th2, dx, dy, dz,
                              d2)) {
                const float4 mp = tv.mp[sn];
                float fx, fy, fz;
                if constexpr (GRAD) {
                    float g3, gi;
                    m2l_field_grad(dx, dy, dz, d2, mp, fx, fy, fz, g3, gi);
                    g[0] += fmaf(g3 * dx, dx, -gi);
                    g[1] += fmaf(g3 * dy, dy, -gi);
                    g[2] += fmaf(g3 * dz, dz, -gi);
                    g[3] += g3 * dx * dy;
                    g[4] += g3 * dx * dz;
                    g[5] += g3 * dy * dz;
                } else {
                    m2l_field(dx, dy, dz, d2, mp, fx, fy, fz);
                }
                ax += fx;
                ay += fy;
                az += fz;
                ++n_m2l;
            } else {
                link = tv.link[sn];
                c = link >> 28;
                if (c == 0) {  // leaf x leaf: P2P
                    const uint4 si = tv.info[sn];
                    if (multi) {
                        pf = 1;
                    } else {
                        p2p_range(A.xyzm, make_uint2(si.x, si.y), t, A.kahan, bx, by, bz, cx, cy,
                                  cz);
                    }
                    ++n_p2p;
                    n_inter += (unsigned long long)si.y * ui.y;
                }
            }
        };
        while (F > 0) {
            uint32_t Fn = 0;
            // two candidates per thread and step (candidates i and i + 512 of
            // the step's 1024), their loads in flight together; one block
            // scan places both threads' children and P2P sources
            for (uint32_t i0 = 0; i0 < F; i0 += 2 * kHeavyThreads) {
                const uint32_t ia = i0 + tid, ib = ia + kHeavyThreads;
                const uint32_t sa = ia < F ? fa[ia] : kNone, sb = ib < F ? fa[ib] : kNone;
                const float4 ga = sa != kNone ? tv.geo[sa] : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 gb = sb != kNone ? tv.geo[sb] : make_float4(0.f, 0.f, 0.f, 0.f);
                uint32_t ca = 0, la = 0, pa = 0, cb = 0, lb = 0, pb = 0;
                if (sa != kNone) visit(sa, ga, ca, la, pa);
                if (sb != kNone) visit(sb, gb, cb, lb, pb);
                // children counts in bits 0..15 (at most 8 x 1024 a step), P2P
                // sources above
                uint32_t ex;
                const uint32_t tot = block_scan((ca + cb) | ((pa + pb) << 16), ex, s_w);
                const uint32_t ctot = tot & 0xFFFFu, ptot = tot >> 16;
                const uint32_t cex = ex & 0xFFFFu, pex = ex >> 16;
                if (Fn + ctot > A.heavy_fcap || np2p + ptot > A.heavy_fcap) {
                    if (tid == 0) set_err(status, PSG_ERR_HEAVY_OVERFLOW);
                    return;
                }
                if (pa) fp[np2p + pex] = sa;
                if (pb) fp[np2p + pex + pa] = sb;
                np2p += ptot;
                for (uint32_t k = 0; k < ca; ++k) fb[Fn + cex + k] = (la & kLinkMask) + k;
                for (uint32_t k = 0; k < cb; ++k) fb[Fn + cex + ca + k] = (lb & kLinkMask) + k;
                Fn += ctot;
            }
            __syncthreads();
            uint32_t* tmp = fa;
            fa = fb;
            fb = tmp;
            F = Fn;
        }
        // fixed-order block reduction
        float v[12] = {ax, ay, az, g[0], g[1], g[2], g[3], g[4], g[5], bx - cx, by - cy, bz - cz};
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            const float x = warp_sum(v[k]);
            if (lane == 0) s_red[w][k] = x;
        }
        if (DEBUG) {
            const unsigned long long c0 = warp_sum(n_m2l), c1 = warp_sum(n_p2p),
                                     c2 = warp_sum(n_inter);
            if (lane == 0) {
                s_cnt[w][0] = c0;
                s_cnt[w][1] = c1;
                s_cnt[w][2] = c2;
            }
        }
        __syncthreads();
        if (tid == 0) {
            float sum[12];
            for (int k = 0; k < 12; ++k) {
                sum[k] = 0.f;
                for (int q = 0; q < kHeavyWarps; ++q) sum[k] += s_red[q][k];
            }
            // L2L from the parent, then L2P at the particle
            const float4 Lp = tv.lt[pid];
            float4 L = make_float4(0.f, __fadd_rn(sum[0], Lp.y), __fadd_rn(sum[1], Lp.z),
                                   __fadd_rn(sum[2], Lp.w));
            float lx = L.y, ly = L.z, lz = L.w;
            if constexpr (GRAD) {
                float4 G0 = make_float4(sum[3], sum[4], sum[5], sum[6]);
                float2 G1 = make_float2(sum[7], sum[8]);
                if (dp >= 2) {
                    const float4 cp = tv.geo[pid];
                    const float4 Gp0 = tv.lg0[pid];
                    const float2 Gp1 = tv.lg1[pid];
                    const float3 sh = grad_apply(Gp0, Gp1, ug.x - cp.x, ug.y - cp.y, ug.z - cp.z);
                    L.y += sh.x;
                    L.z += sh.y;
                    L.w += sh.z;
                    G0.x += Gp0.x;
                    G0.y += Gp0.y;
                    G0.z += Gp0.z;
                    G0.w += Gp0.w;
                    G1.x += Gp1.x;
                    G1.y += Gp1.y;
                }
                tv.lg0[u] = G0;
                tv.lg1[u] = G1;
                s_g[0] = G0;
                s_g1 = G1;
                const float3 at = grad_apply(G0, G1, t.x - ug.x, t.y - ug.y, t.z - ug.z);
                lx = L.y + at.x;
                ly = L.z + at.y;
                lz = L.w + at.z;
                if (A.leaf_of && !multi) A.leaf_of[ui.x] = u;
            }
            tv.lt[u] = L;
            s_g[1] = L;
            if (!multi) {
                const double mm = (double)t.w;
                A.fx[ui.x] = (float)(mm * ((double)lx + (double)sum[9]));
                A.fy[ui.x] = (float)(mm * ((double)ly + (double)sum[10]));
                A.fz[ui.x] = (float)(mm * ((double)lz + (double)sum[11]));
            }
            if (DEBUG) {
                unsigned long long c0 = 0, c1 = 0, c2 = 0;
                for (int q = 0; q < kHeavyWarps; ++q) {
                    c0 += s_cnt[q][0];
                    c1 += s_cnt[q][1];
                    c2 += s_cnt[q][2];
                }
                tv.dbg_m2l[u] = (uint32_t)c0;
                tv.dbg_p2p[u] = (uint32_t)c1;
                atomicAdd(&status->stat[PSG_STAT_M2L], c0);
                atomicAdd(&status->stat[PSG_STAT_P2P_PAIRS], c1);
                atomicAdd(&status->stat[PSG_STAT_P2P_INTER], c2);
            }
        }
        __syncthreads();
        if (multi) {
            // P2P + L2P of the leaf's particles over the listed sources,
            // kHeavyTargets particles a pass: each source particle is loaded
            // once a pass and summed into every target's accumulators;
            // fixed-order sums over warps, then over the block
            const float4 L = s_g[1];
            for (uint32_t k0 = 0; k0 < ui.y; k0 += kHeavyTargets) {
                const uint32_t nk = min((uint32_t)kHeavyTargets, ui.y - k0);
                float4 tk[kHeavyTargets];
                float acc[kHeavyTargets][3];
#pragma unroll
                for (int k = 0; k < kHeavyTargets; ++k) {
                    tk[k] = A.xyzm[ui.x + k0 + min((uint32_t)k, nk - 1)];
                    acc[k][0] = acc[k][1] = acc[k][2] = 0.f;
                }
                if (A.kahan) {
                    // compensated sums: one target at a time (a rare mode)
                    for (uint32_t k = 0; k < nk; ++k) {
                        float px = 0.f, py = 0.f, pz = 0.f, qx = 0.f, qy = 0.f, qz = 0.f;
                        const float4 t1 = A.xyzm[ui.x + k0 + k];
                        for (uint32_t e = tid; e < np2p; e += kHeavyThreads) {
                            const uint4 si = tv.info[fp[e]];
                            p2p_range(A.xyzm, make_uint2(si.x, si.y), t1, true, px, py, pz, qx,
                                      qy, qz);
                        }
#pragma unroll
                        for (int kk = 0; kk < kHeavyTargets; ++kk)
                            if ((uint32_t)kk == k) {
                                acc[kk][0] = px - qx;
                                acc[kk][1] = py - qy;
                                acc[kk][2] = pz - qz;
                            }
                    }
                } else {
                    // the listed source leaves, 32 a warp at a time, their
                    // particles laid end to end (a warp prefix sum) and dealt
                    // one per lane, so that no lane idles on a short leaf;
                    // the targets two at a time in paired FP32 instructions
                    constexpr int KP = kHeavyTargets / 2;
                    float2 ntx[KP], nty[KP], ntz[KP], sx[KP], sy[KP], sz[KP];
#pragma unroll
                    for (int k = 0; k < KP; ++k) {
                        ntx[k] = make_float2(-tk[2 * k].x, -tk[2 * k + 1].x);
                        nty[k] = make_float2(-tk[2 * k].y, -tk[2 * k + 1].y);
                        ntz[k] = make_float2(-tk[2 * k].z, -tk[2 * k + 1].z);
                        sx[k] = sy[k] = sz[k] = make_float2(0.f, 0.f);
                    }
                    const float2 eps = make_float2(0.1f, 0.1f);
                    for (uint32_t e0 = w * 32u; e0 < np2p; e0 += kHeavyThreads) {
                        uint32_t es = 0, en = 0;
                        if (e0 + lane < np2p) {
                            const uint4 si = tv.info[fp[e0 + lane]];
                            es = si.x;
                            en = si.y;
                        }
                        const uint32_t incl = warp_incl_scan(en);
                        const uint32_t ptot = __shfl_sync(0xFFFFFFFFu, incl, 31);
                        const uint32_t excl = incl - en;
                        for (uint32_t b = 0; b < ptot; b += 32) {
                            // lane's particle: the entry whose prefix holds b + lane
                            const uint32_t f = b + lane;
                            uint32_t ee = 0;
#pragma unroll
                            for (uint32_t step = 16; step > 0; step >>= 1) {
                                const uint32_t v = __shfl_sync(0xFFFFFFFFu, incl, ee + step - 1);
                                if (v <= f) ee += step;
                            }
                            const uint32_t s0 = __shfl_sync(0xFFFFFFFFu, es, ee);
                            const uint32_t x0 = __shfl_sync(0xFFFFFFFFu, excl, ee);
                            if (f < ptot) {
                                const float4 p = A.xyzm[s0 + (f - x0)];
                                const float2 px = make_float2(p.x, p.x), py = make_float2(p.y, p.y),
                                             pz = make_float2(p.z, p.z), pw = make_float2(p.w, p.w);
#pragma unroll
                                for (int k = 0; k < KP; ++k) {
                                    const float2 dx = __fadd2_rn(px, ntx[k]);
                                    const float2 dy = __fadd2_rn(py, nty[k]);
                                    const float2 dz = __fadd2_rn(pz, ntz[k]);
                                    float2 r = __ffma2_rn(dz, dz, eps);
                                    r = __ffma2_rn(dy, dy, r);
                                    r = __ffma2_rn(dx, dx, r);
                                    const float2 i = make_float2(rsqrt_soft(r.x), rsqrt_soft(r.y));
                                    const float2 fw =
                                        __fmul2_rn(pw, __fmul2_rn(__fmul2_rn(i, i), i));
                                    sx[k] = __ffma2_rn(dx, fw, sx[k]);
                                    sy[k] = __ffma2_rn(dy, fw, sy[k]);
                                    sz[k] = __ffma2_rn(dz, fw, sz[k]);
                                }
                            }
                        }
                    }
#pragma unroll
                    for (int k = 0; k < KP; ++k) {
                        acc[2 * k][0] = sx[k].x;
                        acc[2 * k + 1][0] = sx[k].y;
                        acc[2 * k][1] = sy[k].x;
                        acc[2 * k + 1][1] = sy[k].y;
                        acc[2 * k][2] = sz[k].x;
                        acc[2 * k + 1][2] = sz[k].y;
                    }
                }
#pragma unroll
                for (int k = 0; k < kHeavyTargets; ++k) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const float x = warp_sum(acc[k][c]);
                        if (lane == 0) s_redt[w][3 * k + c] = x;
                    }
                }
                __syncthreads();
                if (tid < nk) {
                    float sx = 0.f, sy = 0.f, sz = 0.f;
                    for (int q = 0; q < kHeavyWarps; ++q) {
                        sx += s_redt[q][3 * tid];
                        sy += s_redt[q][3 * tid + 1];
                        sz += s_redt[q][3 * tid + 2];
                    }
                    const uint32_t i = ui.x + k0 + tid;
                    const float4 t1 = A.xyzm[i];
                    float lx = L.y, ly = L.z, lz = L.w;
                    if constexpr (GRAD) {
                        const float3 at =
                            grad_apply(s_g[0], s_g1, t1.x - ug.x, t1.y - ug.y, t1.z - ug.z);
                        lx += at.x;
                        ly += at.y;
                        lz += at.z;
                        if (A.leaf_of) A.leaf_of[i] = u;
                    }
                    const double mm = (double)t1.w;
                    A.fx[i] = (float)(mm * ((double)lx + (double)sx));
                    A.fy[i] = (float)(mm * ((double)ly + (double)sy));
                    A.fz[i] = (float)(mm * ((double)lz + (double)sz));
                }
                __syncthreads();
            }
        }
    }
}

void launch_heavy_leaf(const TravArgs& A, int grid, cudaStream_t st) {
    if (A.order >= 1) {
        if (A.debug) k_heavy_leaf<true, true><<<grid, kHeavyThreads, 0, st>>>(A);
        else k_heavy_leaf<false, true><<<grid, kHeavyThreads, 0, st>>>(A);
    } else {
        if (A.debug) k_heavy_leaf<true, false><<<grid, kHeavyThreads, 0, st>>>(A);
        else k_heavy_leaf<false, false><<<grid, kHeavyThreads, 0, st>>>(A);
    }
}

void launch_dense_p2p(const TravArgs& A, int grid, cudaStream_t st) {
    if (A.kahan) k_dense_p2p<true><<<grid, kDenseThreads, 0, st>>>(A);
    else k_dense_p2p<false><<<grid, kDenseThreads, 0, st>>>(A);
}

template <int MODE, bool DENSE, int VAR>
static void launch_mode(const TravArgs& A, int grid, cudaStream_t st) {
    if (A.order >= 1) {
        if (A.debug) k_trav<MODE, true, true, DENSE, VAR><<<grid, kTravThreads, 0, st>>>(A);
        else k_trav<MODE, false, true, DENSE, VAR><<<grid, kTravThreads, 0, st>>>(A);
    } else {
        if (A.debug) k_trav<MODE, true, false, DENSE, VAR><<<grid, kTravThreads, 0, st>>>(A);
        else k_trav<MODE, false, false, DENSE, VAR><<<grid, kTravThreads, 0, st>>>(A);
    }
}

static bool leaf_xl(const TravArgs& A) { return A.ns_levels < kMaxDepth || A.stream; }

void launch_traverse_internal(const TravArgs& args, int level, int level_end, int grid,
                              cudaStream_t st) {
    TravArgs A = args;
    A.level = level;
    A.level_end = level_end;
    launch_mode<MODE_INTERNAL, false, VAR_PLAIN>(A, grid, st);
}

// which: 1 the variants for leaf capacities below kDenseCap (sparse and dense:
// each returns at once unless the tree is its kind), 2 the one for the others
void launch_traverse_leaves(const TravArgs& args, const int grid[2], int which, cudaStream_t st) {
    if (leaf_xl(args)) {
        if (which & 1) launch_mode<MODE_LEAF, false, VAR_XL>(args, grid[0], st);
        launch_mode<MODE_LEAF, true, VAR_XL>(args, grid[1], st);
    } else {
        if (which & 1) launch_mode<MODE_LEAF, false, VAR_PLAIN>(args, grid[0], st);
        if (which & 1) launch_mode<MODE_LEAF, true, VAR_PLAIN>(args, grid[1], st);
        if (which & 2) launch_mode<MODE_LEAF, true, VAR_MERGE>(args, grid[1], st);
    }
}

void launch_traverse_split(const TravArgs& args, int grid, int which, cudaStream_t st) {
    if (which & 1) launch_mode<MODE_LEAF, true, VAR_SPLIT>(args, grid, st);
    if (which & 2) launch_mode<MODE_LEAF, true, VAR_SPLIT_MERGE>(args, grid, st);
}

int traverse_threads() { return kTravThreads; }
const void* traverse_kernel_ptr(int order, int dense, int xl) {
    if (xl) {
        if (order) {
            return dense ? (const void*)k_trav<MODE_LEAF, false, true, true, VAR_XL>
                         : (const void*)k_trav<MODE_LEAF, false, true, false, VAR_XL>;
        }
        return dense ? (const void*)k_trav<MODE_LEAF, false, false, true, VAR_XL>
                     : (const void*)k_trav<MODE_LEAF, false, false, false, VAR_XL>;
    }
    if (order) {
        return dense ? (const void*)k_trav<MODE_LEAF, false, true, true, VAR_PLAIN>
                     : (const void*)k_trav<MODE_LEAF, false, true, false, VAR_PLAIN>;
    }
    return dense ? (const void*)k_trav<MODE_LEAF, false, false, true, VAR_PLAIN>
                 : (const void*)k_trav<MODE_LEAF, false, false, false, VAR_PLAIN>;
}
const void* traverse_internal_kernel_ptr(int order) {
    return order ? (const void*)k_trav<MODE_INTERNAL, false, true, false, VAR_PLAIN>
                 : (const void*)k_trav<MODE_INTERNAL, false, false, false, VAR_PLAIN>;
}

}  // namespace psg
