// Octree build from the sorted Morton codes, and the upward pass (P2M/M2M).
//
// Reference: ps_impl_build_tree (polesitter.h:906-967) recursively splits a
// node [s, e) at depth d < 10 holding >= 2 particles into one child per
// non-empty octant of digit (code >> (27 - 3d)) & 7; a node is a leaf when
// d == 10 or it holds <= 1 particle (:911-916).  Equivalently, with
// cpl(i) = the number of leading octal digits codes[i-1] and codes[i] share,
// a depth-d node starts at position i iff
//     (i == 0 or cpl(i) < d)                        -- a depth-d run starts
// and (cpl(i) >= d-1 or cpl(i+1) >= d-1)            -- its parent run has >= 2
// so the whole tree comes from one pass of flags and a 10-wide prefix scan,
// with no recursion.  Levels are stored contiguously in Morton order.
//
// Leaf capacity B > 1 (an extension: nodes holding <= B particles are
// leaves): "its parent run has >= 2" becomes "> B".  The depth-k runs
// around i shrink as k grows, and the depth-k run holding i has > B
// particles iff some window [j, j+B] containing i lies inside it, so a
// depth-d node starts at i iff a depth-d run starts there and
//     d - 1 <= W(i) = max over j in [i-B, i] of cpl2(codes[j], codes[j+B])
// (cpl2 = common octal prefix length).  With B = 1 this is the rule above.
// The root is split whenever it holds >= 2 particles, so every particle has
// a leaf below the root (W(i) >= 0).
//
// Child centres follow the reference's float chain exactly (:935-939):
// hw_child = hw * 0.5 and c_child = c_parent +/- hw_child, replayed from the
// root for each node.
#include "psg_common.cuh"
#include "psg_kernels.h"

namespace psg {

constexpr int kTreeThreads = 256;
constexpr int kTreePer = 4;
constexpr int kTreeTile = kTreeThreads * kTreePer;  // 1024 positions

// bytes of the build's scratch: counts per tile and depth, flags per position
size_t tree_scratch_bytes(size_t n) {
    const size_t tiles = (n + kTreeTile - 1) / kTreeTile;
    return tiles * (kMaxDepth * sizeof(uint32_t) + kTreeTile * sizeof(unsigned short));
}

__device__ __forceinline__ int cpl2(uint32_t a, uint32_t b) {
    // common octal prefix length of two codes (0 .. 10)
    const uint32_t x = (a ^ b) & 0x3FFFFFFFu;
    if (x == 0u) return kMaxDepth;
    return (__clz(x) - 2) / 3;
}

__device__ __forceinline__ int cpl_at(const uint32_t* __restrict__ c, size_t i, size_t lo,
                                      size_t hi) {
    // common octal prefix length of codes[i-1], codes[i]; -1 outside (lo, hi)
    if (i <= lo || i >= hi) return -1;
    return cpl2(c[i - 1], c[i]);
}

// 10 one-bit flags (bit d-1 <=> a depth-d node starts at i); w = W(i), the
// deepest level whose run around i holds more than the leaf capacity
__device__ __forceinline__ uint32_t node_flags(int cpl_i, int w, bool first) {
    uint32_t f = 0;
#pragma unroll
    for (int d = 1; d <= kMaxDepth; ++d) {
        bool start = first || cpl_i < d;
        if (start && w >= d - 1) f |= 1u << (d - 1);
    }
    return f;
}

// counters of depths 1..5 in lo, 6..10 in hi, 12 bits each
__device__ __forceinline__ void add_flags(unsigned long long& lo, unsigned long long& hi,
                                          uint32_t f) {
#pragma unroll
    for (int d = 0; d < 5; ++d) {
        lo += (unsigned long long)((f >> d) & 1u) << (12 * d);
        hi += (unsigned long long)((f >> (d + 5)) & 1u) << (12 * d);
    }
}

__device__ __forceinline__ uint32_t get_cnt(unsigned long long lo, unsigned long long hi,
                                            int d /*1..10*/) {
    return d <= 5 ? (uint32_t)((lo >> (12 * (d - 1))) & 0xFFFull)
                  : (uint32_t)((hi >> (12 * (d - 6))) & 0xFFFull);
}

// the flags of the positions p0 .. p0 + kTreePer - 1 of the system whose
// particles are [lo, hi)
__device__ __forceinline__ void thread_flags(const uint32_t* __restrict__ codes, size_t lo,
                                             size_t hi, size_t p0, uint32_t cap,
                                             uint32_t (&f)[kTreePer]) {
    int cprev = cpl_at(codes, p0, lo, hi);
    if (cap <= 1u) {
        // W(i) = max(cpl(i), cpl(i+1))
#pragma unroll
        for (int q = 0; q < kTreePer; ++q) {
            size_t i = p0 + q;
            int cnext = cpl_at(codes, i + 1, lo, hi);
            f[q] = (i < hi) ? node_flags(cprev, max(cprev, cnext), i == lo) : 0u;
            cprev = cnext;
        }
        return;
    }
    // W over the windows [j, j + cap] with j in [p0 - cap, p0 + kTreePer - 1],
    // lo <= j and j + cap < hi; at least 0 (the root is split) once it holds 2
    int w[kTreePer];
#pragma unroll
    for (int q = 0; q < kTreePer; ++q) w[q] = hi - lo >= 2 ? 0 : -1;
    const long long jlo = max((long long)lo, (long long)p0 - (long long)cap);
    const long long jhi = min((long long)p0 + kTreePer - 1, (long long)hi - 1 - (long long)cap);
#pragma unroll 4
    for (long long j = jlo; j <= jhi; ++j) {
        const int c = cpl2(codes[j], codes[j + cap]);
#pragma unroll
        for (int q = 0; q < kTreePer; ++q) {
            const long long i = (long long)p0 + q;
            if (j <= i && j + (long long)cap >= i) w[q] = max(w[q], c);
        }
    }
#pragma unroll
    for (int q = 0; q < kTreePer; ++q) {
        size_t i = p0 + q;
        f[q] = (i < hi) ? node_flags(cprev, w[q], i == lo) : 0u;
        cprev = cpl_at(codes, i + 1, lo, hi);
    }
}

// Many systems in one array: the same rules inside each system's range,
// with its own leaf capacity; a system's first position starts its root (a
// depth-0 node, node k of level 0) and no run crosses a system boundary.
__device__ __forceinline__ void thread_flags_forest(const uint32_t* __restrict__ codes, size_t n,
                                                    size_t p0, const TreeView& tv,
                                                    uint32_t (&f)[kTreePer]) {
    if (p0 + kTreePer <= n) {
        const uint32_t k = tv.part_sys[p0];
        if (tv.part_sys[p0 + kTreePer - 1] == k) {
            thread_flags(codes, tv.sys_off[k], tv.sys_off[k + 1], p0, tv.sys_cap[k], f);
            return;
        }
    }
#pragma unroll 1
    for (int q = 0; q < kTreePer; ++q) {
        const size_t i = p0 + q;
        f[q] = 0u;
        if (i >= n) continue;
        const uint32_t k = tv.part_sys[i];
        uint32_t g[kTreePer];
        thread_flags(codes, tv.sys_off[k], tv.sys_off[k + 1], i, tv.sys_cap[k], g);
        f[q] = g[0];
    }
}

// The flags of every position, and per tile the nodes that start in it at
// each depth.
__global__ void __launch_bounds__(kTreeThreads) k_tree_count(const uint32_t* __restrict__ codes,
                                                            size_t n, uint32_t cap,
                                                            uint32_t* __restrict__ tile_cnt,
                                                            ushort4* __restrict__ flags,
                                                            const TreeView tv) {
    const size_t p0 = (size_t)blockIdx.x * kTreeTile + (size_t)threadIdx.x * kTreePer;
    uint32_t f[kTreePer];
    if (tv.part_sys) thread_flags_forest(codes, n, p0, tv, f);
    else thread_flags(codes, 0, n, p0, cap, f);
    flags[p0 / kTreePer] = make_ushort4((unsigned short)f[0], (unsigned short)f[1],
                                        (unsigned short)f[2], (unsigned short)f[3]);
    unsigned long long lo = 0, hi = 0;
#pragma unroll
    for (int q = 0; q < kTreePer; ++q) add_flags(lo, hi, f[q]);
    lo = warp_sum(lo);
    hi = warp_sum(hi);
    __shared__ unsigned long long s[2][kTreeThreads / 32];
    if (lane_id() == 0) {
        s[0][threadIdx.x >> 5] = lo;
        s[1][threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x < kMaxDepth) {
        const int d = threadIdx.x + 1;
        uint32_t c = 0;
        for (int w = 0; w < kTreeThreads / 32; ++w) c += get_cnt(s[0][w], s[1][w], d);
        tile_cnt[(size_t)blockIdx.x * kMaxDepth + threadIdx.x] = c;
    }
}

// a level's node count, held to its capacity
__device__ __forceinline__ uint32_t level_count(const TreeView& tv, Status* status, int d,
                                                uint32_t total) {
    if (total > tv.lvl_cap[d]) {
        set_err(status, PSG_ERR_NODES);
        total = tv.lvl_cap[d];
    }
    return total;
}

// Exclusive scan of the tile counts, one block of 1024 threads per depth (one
// block for all depths took 12 us at 1M, where this takes 4).
__global__ void __launch_bounds__(1024) k_tree_scan(uint32_t* __restrict__ tile_cnt, int tiles,
                                                    TreeView tv, Status* status) {
    __shared__ uint32_t wsum[32];
    const int d = blockIdx.x + 1;
    const uint32_t w = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (int b0 = 0; b0 < tiles; b0 += 1024) {
        const int b = b0 + threadIdx.x;
        const uint32_t v = b < tiles ? tile_cnt[(size_t)b * kMaxDepth + d - 1] : 0u;
        const uint32_t inc = warp_incl_scan(v);
        if (lane_id() == 31) wsum[w] = inc;
        __syncthreads();
        const uint32_t ws = wsum[lane_id()];
        const uint32_t wi = warp_incl_scan(ws);
        const uint32_t add = carry + __shfl_sync(0xFFFFFFFFu, wi - ws, w);
        if (b < tiles) tile_cnt[(size_t)b * kMaxDepth + d - 1] = inc - v + add;
        carry += __shfl_sync(0xFFFFFFFFu, wi, 31);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        status->lvl_count[d] = level_count(tv, status, d, carry);
        if (d == 1) {
            status->lvl_count[0] = tv.part_sys ? tv.nsys : 1u;
            status->lvl_count[kLevels] = 0;
        }
    }
}

// end of the run of codes sharing code[i]'s first d octal digits, at least
// up to position `from` (gallop, then binary search)
__device__ __forceinline__ size_t run_end(const uint32_t* __restrict__ c, size_t n, size_t i,
                                          size_t from, int d) {
    const int sh = 30 - 3 * d;
    const uint32_t key = (c[i] & 0x3FFFFFFFu) >> sh;
    size_t lo = from, step = 1;  // invariant: prefix(c[lo]) == key
    while (lo + step < n && ((c[lo + step] & 0x3FFFFFFFu) >> sh) == key) {
        lo += step;
        step <<= 1;
    }
    size_t hi = (lo + step < n) ? lo + step : n;  // prefix(c[hi]) != key or hi == n
    while (hi - lo > 1) {
        size_t mid = lo + ((hi - lo) >> 1);
        if (((c[mid] & 0x3FFFFFFFu) >> sh) == key) lo = mid; else hi = mid;
    }
    return hi;
}

// Nodes.  A depth-d node that starts at i ends where the next node of depth <= d
// starts (or its system ends), which the block looks up in its tile's flags; only
// a node that runs past the tile searches the codes.  Up to kSelfScanTiles tiles
// every block adds up the tile counts before it itself (no k_tree_scan).
// Measured (whole build; flags computed twice, a scan of all depths in one block
// and a search of the codes per node / now): 1K 48 / 34 us, 33K 56 / 44 us, 1M
// 144 / 130 us, 4M 379 / 317 us.
constexpr int kSelfScanTiles = 64;

__global__ void __launch_bounds__(kTreeThreads) k_tree_emit(const uint32_t* __restrict__ codes,
                                                           size_t n, int tiles,
                                                           const uint32_t* __restrict__ tile_off,
                                                           const ushort4* __restrict__ flags,
                                                           TreeView tv, Status* status,
                                                           float cx, float cy, float cz,
                                                           float hw,
                                                           const float* __restrict__ bbox) {
    if (bbox) {
        // root from a device-side bounding box (min, max, range), as the
        // caller's loop derives it: c = min + range / 2, hw = range / 2
        // (README.md:76-78)
        hw = __fdiv_rn(bbox[2], 2.0f);
        cx = cy = cz = __fadd_rn(bbox[0], hw);
    }
    const size_t p0 = (size_t)blockIdx.x * kTreeTile + (size_t)threadIdx.x * kTreePer;
    uint32_t f[kTreePer];
    const bool forest = tv.part_sys != nullptr;
    {
        const ushort4 v = flags[p0 / kTreePer];
        f[0] = v.x;
        f[1] = v.y;
        f[2] = v.z;
        f[3] = v.w;
    }
    unsigned long long lo = 0, hi = 0;
#pragma unroll
    for (int q = 0; q < kTreePer; ++q) add_flags(lo, hi, f[q]);
    // the shallowest depth that starts at each position (11: none), and its
    // minimum over a thread's and a warp's positions
    __shared__ uint8_t s_md[kTreeTile], s_tmd[kTreeThreads], s_wmd[kTreeThreads / 32];
    {
        uint32_t m = kMaxDepth + 1;
#pragma unroll
        for (int q = 0; q < kTreePer; ++q) {
            const uint32_t md = f[q] ? __ffs(f[q]) : kMaxDepth + 1;
            s_md[threadIdx.x * kTreePer + q] = (uint8_t)md;
            m = min(m, md);
        }
        s_tmd[threadIdx.x] = (uint8_t)m;
        m = __reduce_min_sync(0xFFFFFFFFu, m);
        if (lane_id() == 0) s_wmd[threadIdx.x >> 5] = (uint8_t)m;
    }
    // block exclusive scan of the packed counters
    unsigned long long ilo = lo, ihi = hi;
    const uint32_t l = lane_id(), w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long a = __shfl_up_sync(0xFFFFFFFFu, ilo, o);
        unsigned long long b = __shfl_up_sync(0xFFFFFFFFu, ihi, o);
        if (l >= (uint32_t)o) {
            ilo += a;
            ihi += b;
        }
    }
    __shared__ unsigned long long s[2][kTreeThreads / 32];
    __shared__ uint32_t s_off[kMaxDepth + 1], s_lvl[kMaxDepth + 1];
    const bool self = tiles <= kSelfScanTiles;
    if (threadIdx.x <= kMaxDepth) s_off[threadIdx.x] = s_lvl[threadIdx.x] = 0;
    if (l == 31) {
        s[0][w] = ilo;
        s[1][w] = ihi;
    }
    __syncthreads();
    if (self) {
        constexpr int kParts = kTreeThreads / kMaxDepth;  // 25 threads per depth
        const int d = threadIdx.x % kMaxDepth, part = threadIdx.x / kMaxDepth;
        uint32_t before = 0, all = 0;
        if (part < kParts) {
            for (int b = part; b < tiles; b += kParts) {
                const uint32_t v = tile_off[(size_t)b * kMaxDepth + d];
                all += v;
                if (b < (int)blockIdx.x) before += v;
            }
            if (before) atomicAdd(&s_off[d + 1], before);
            if (all) atomicAdd(&s_lvl[d + 1], all);
        }
        __syncthreads();
        if (threadIdx.x < kMaxDepth) {
            const int dd = threadIdx.x + 1;
            const uint32_t c = min(s_lvl[dd], tv.lvl_cap[dd]);
            if (blockIdx.x == 0) status->lvl_count[dd] = level_count(tv, status, dd, s_lvl[dd]);
            s_lvl[dd] = c;
        }
        if (blockIdx.x == 0 && threadIdx.x == kMaxDepth) {
            status->lvl_count[0] = forest ? tv.nsys : 1u;
            status->lvl_count[kLevels] = 0;
        }
    } else if (threadIdx.x < kMaxDepth) {
        s_off[threadIdx.x + 1] = tile_off[(size_t)blockIdx.x * kMaxDepth + threadIdx.x];
        s_lvl[threadIdx.x + 1] = status->lvl_count[threadIdx.x + 1];
    }
    __syncthreads();
    // the tile position after li at which a node of depth <= d starts
    // (kTreeTile: none), position by position to the thread's end, thread by
    // thread to the warp's, and down again
    auto next_start = [&](int li, int d) -> int {
        int j = li + 1;
        for (; j & (kTreePer - 1); ++j)
            if (s_md[j] <= d) return j;
        int t = j / kTreePer;
        for (; t < kTreeThreads && (t & 31) && s_tmd[t] > d; ++t) {
        }
        if (t < kTreeThreads && !(t & 31)) {
            int w2 = t >> 5;
            while (w2 < kTreeThreads / 32 && s_wmd[w2] > d) ++w2;
            if (w2 == kTreeThreads / 32) return kTreeTile;
            for (t = w2 * 32; s_tmd[t] > d; ++t) {
            }
        }
        if (t >= kTreeThreads) return kTreeTile;
        for (j = t * kTreePer; s_md[j] > d; ++j) {
        }
        return j;
    };
    unsigned long long elo = ilo - lo, ehi = ihi - hi;
    for (uint32_t j = 0; j < w; ++j) {
        elo += s[0][j];
        ehi += s[1][j];
    }
    uint32_t rank[kMaxDepth + 2];
#pragma unroll
    for (int d = 1; d <= kMaxDepth; ++d)
        rank[d] = tv.lvl_base[d] + s_off[d] + get_cnt(elo, ehi, d);
    rank[kMaxDepth + 1] = 0;

    if (p0 == 0 && !forest) {  // root
        tv.geo[0] = make_float4(cx, cy, cz, hw);
        tv.info[0] = make_uint4(0u, (uint32_t)n, tv.lvl_base[1], pack_flags(0, 0, 0));
        tv.parent[0] = kNone;
        tv.cbase[0] = tv.lvl_base[1];
        tv.arrive[0] = 0;
        tv.lt[0] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < kTreePer; ++q) {
        const size_t i = p0 + q;
        const uint32_t fq = f[q];
        uint32_t sys = 0;
        if (forest && i < n) {
            // this position's system: its root box (README.md:76-78) and, at
            // its first position, its root node
            sys = tv.part_sys[i];
            const float* bb = tv.sys_bbox + 4 * sys;
            hw = __fdiv_rn(bb[2], 2.0f);
            cx = cy = cz = __fadd_rn(bb[0], hw);
            const uint32_t lo_s = tv.sys_off[sys];
            if (i == lo_s) {
                tv.geo[sys] = make_float4(cx, cy, cz, hw);
                tv.info[sys] = make_uint4(lo_s, tv.sys_off[sys + 1] - lo_s, rank[1],
                                          pack_flags(0, 0, 0));
                tv.parent[sys] = kNone;
                tv.cbase[sys] = rank[1];
                tv.arrive[sys] = 0;
                tv.lt[sys] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        if (fq) {
            const uint32_t code = codes[i];
            const size_t run_n = forest ? tv.sys_off[sys + 1] : n;
            // centre and half width down the code's digits: the reference's
            // chain of rounded adds from the root centre
            float4 g = make_float4(cx, cy, cz, hw);
#pragma unroll 1
            for (int d = 1; d <= kMaxDepth; ++d) {
                const uint32_t dig = (code >> (30 - 3 * d)) & 7u;
                g.w = __fmul_rn(g.w, 0.5f);
                g.x = __fadd_rn(g.x, (dig & 1u) ? g.w : -g.w);
                g.y = __fadd_rn(g.y, (dig & 2u) ? g.w : -g.w);
                g.z = __fadd_rn(g.z, (dig & 4u) ? g.w : -g.w);
                if (!((fq >> (d - 1)) & 1u)) continue;
                const uint32_t id = rank[d];
                if (id - tv.lvl_base[d] >= s_lvl[d]) continue;  // capacity guard
                const int ne = next_start((int)threadIdx.x * kTreePer + q, d);
                const size_t tile_end = (size_t)blockIdx.x * kTreeTile + (size_t)ne;
                size_t end = tile_end < run_n ? tile_end : run_n;
                if (ne == kTreeTile && tile_end < run_n)
                    end = run_end(codes, run_n, i, tile_end - 1, d);
                const uint32_t cnt = (uint32_t)(end - i);
                uint32_t par = forest ? sys : 0u;
                if (d > 1) par = rank[d - 1] + ((fq >> (d - 2)) & 1u) - 1u;
                const uint32_t cb = d < kMaxDepth ? rank[d + 1] : 0u;
                tv.geo[id] = g;
                tv.info[id] = make_uint4((uint32_t)i, cnt, cb,
                                         pack_flags(0, d, dig));
                tv.parent[id] = par;
                tv.cbase[id] = cb;
                tv.arrive[id] = 0;
            }
        }
#pragma unroll
        for (int d = 1; d <= kMaxDepth; ++d) rank[d] += (fq >> (d - 1)) & 1u;
    }
}

// child count = next node's first-child rank - this node's (same level); also
// the particle count of the fullest leaf, and the list of each level's
// internal nodes (the traversal's groups: without the leaves, 3 of 4 nodes,
// its work queues hold no empty items), in Morton order but for the order in
// which warps append
__global__ void __launch_bounds__(256) k_tree_link(TreeView tv, Status* status) {
    const uint32_t total = tv.lvl_base[kLevels];
    const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
    int d = 0;
    while (d < kMaxDepth && id >= tv.lvl_base[d + 1]) ++d;
    const uint32_t r = id - tv.lvl_base[d];
    const uint32_t cnt_d = status->lvl_count[d];
    const bool node = id < total && r < cnt_d;
    if (!__any_sync(0xFFFFFFFFu, node)) return;
    uint32_t nch = 0, max_leaf = 0;
    if (node) {
        if (d < kMaxDepth) {
            const uint32_t next = (r + 1 < cnt_d) ? tv.cbase[id + 1]
                                                  : tv.lvl_base[d + 1] + status->lvl_count[d + 1];
            nch = next - tv.cbase[id];
            if (nch > 8u) {  // codes not sorted by their 30-bit prefix
                set_err(status, PSG_ERR_NODES);
                nch = 0;
            }
        }
        uint4 inf = tv.info[id];
        inf.w = (inf.w & ~0xFu) | (nch & 0xFu);
        tv.info[id] = inf;
        tv.link[id] = nch ? ((inf.z & kLinkMask) | (nch << 28)) : 0u;
        tv.lt[id] = make_float4(0.f, 0.f, 0.f, 0.f);
        tv.ready[id] = 0;
        if (nch == 0) max_leaf = inf.y;
        // batched systems: each system picks its own leaf-pass variant
        if (nch == 0 && tv.part_sys && inf.y >= kDenseSwitch)
            atomicMax(&tv.sys_maxleaf[tv.part_sys[inf.x]], inf.y);
    }
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, nch ? (uint32_t)d : kNone);
    if (nch) {
        const int leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if ((int)lane_id() == leader) base = atomicAdd(&status->group_count[d], __popc(peers));
        base = __shfl_sync(peers, base, leader);
        tv.groups[tv.lvl_base[d] + base + __popc(peers & lanemask_lt())] = id;
    }
    max_leaf = __reduce_max_sync(0xFFFFFFFFu, max_leaf);
    if (lane_id() == 0 && max_leaf) atomicMax(&status->max_leaf, max_leaf);
}

// Upward pass: P2M (a leaf's particles) and M2M (a node's children).
// Operation order matches polesitter.h:978-1045 exactly (sequential sums over
// the leaf's particles; children in octant order), every op rounded to nearest,
// whichever thread does it.
// Bound: latency -- the sequential sum of the fullest leaf (its loads run
// kP2mBatch ahead of the adds) and the way from the leaves to the root.
constexpr int kP2mBatch = 8;

__device__ __forceinline__ float4 p2m(const float4* __restrict__ xyzm, uint4 inf, float4 c) {
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [&](const float4& p) {
        o.x = __fadd_rn(o.x, p.w);
        o.y = __fadd_rn(o.y, __fmul_rn(p.w, __fsub_rn(p.x, c.x)));
        o.z = __fadd_rn(o.z, __fmul_rn(p.w, __fsub_rn(p.y, c.y)));
        o.w = __fadd_rn(o.w, __fmul_rn(p.w, __fsub_rn(p.z, c.z)));
    };
    uint32_t k = 0;
    for (; k + kP2mBatch <= inf.y; k += kP2mBatch) {
        float4 p[kP2mBatch];
#pragma unroll
        for (int j = 0; j < kP2mBatch; ++j) p[j] = xyzm[inf.x + k + j];
#pragma unroll
        for (int j = 0; j < kP2mBatch; ++j) add(p[j]);
    }
    for (; k < inf.y; ++k) add(xyzm[inf.x + k]);
    return o;
}

__device__ __forceinline__ float4 m2m(const TreeView& tv, uint32_t link, float4 c) {
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t fc = link & kLinkMask, nch = link >> 28;
    for (uint32_t j = 0; j < nch; ++j) {
        const float4 cm = __ldcg(&tv.mp[fc + j]);
        const float4 cg = tv.geo[fc + j];
        o.x = __fadd_rn(o.x, cm.x);
        o.y = __fadd_rn(o.y, __fadd_rn(cm.y, __fmul_rn(cm.x, __fsub_rn(cg.x, c.x))));
        o.z = __fadd_rn(o.z, __fadd_rn(cm.z, __fmul_rn(cm.x, __fsub_rn(cg.y, c.y))));
        o.w = __fadd_rn(o.w, __fadd_rn(cm.w, __fmul_rn(cm.x, __fsub_rn(cg.z, c.z))));
    }
    return o;
}

// the nodes of one level (their children are done)
__global__ void __launch_bounds__(256) k_upward_level(TreeView tv, const Status* status,
                                                      const float4* __restrict__ xyzm, int d) {
    if (status->err & (PSG_ERR_NODES | PSG_ERR_SORT_SPIN)) return;
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= status->lvl_count[d]) return;
    const uint32_t id = tv.lvl_base[d] + r;
    const float4 c = tv.geo[id];
    const uint32_t link = tv.link[id];
    tv.mp[id] = (link >> 28) == 0 ? p2m(xyzm, tv.info[id], c) : m2m(tv, link, c);
}

// the levels bottom .. 0 in one launch: a thread takes a node of the bottom
// level (any deeper ones are done) or a leaf above it and climbs; of a node's
// children the last to arrive (per-node counters, zeroed by k_tree_emit) adds
// their multipoles and climbs on
__global__ void __launch_bounds__(256) k_upward_climb(TreeView tv, const Status* status,
                                                      const float4* __restrict__ xyzm,
                                                      int bottom) {
    if (status->err & (PSG_ERR_NODES | PSG_ERR_SORT_SPIN)) return;
    const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= tv.lvl_base[bottom + 1]) return;
    int d = 0;
    while (d < bottom && id >= tv.lvl_base[d + 1]) ++d;
    if (id - tv.lvl_base[d] >= status->lvl_count[d]) return;
    uint32_t link = tv.link[id];
    if ((link >> 28) != 0 && d < bottom) return;
    const float4 c0 = tv.geo[id];
    __stcg(&tv.mp[id], (link >> 28) == 0 ? p2m(xyzm, tv.info[id], c0) : m2m(tv, link, c0));
    for (uint32_t cur = tv.parent[id]; cur != kNone; cur = tv.parent[cur]) {
        link = tv.link[cur];
        __threadfence();
        if (atomicAdd(&tv.arrive[cur], 1u) + 1u != (link >> 28)) return;
        __threadfence();
        __stcg(&tv.mp[cur], m2m(tv, link, tv.geo[cur]));
    }
}

void launch_tree(const uint32_t* codes, size_t n, uint32_t* tile_buf, TreeView tv,
                 Status* status, float cx, float cy, float cz, float hw, int grid,
                 cudaStream_t st, const float* bbox, uint32_t leaf_cap) {
    const int tiles = (int)((n + kTreeTile - 1) / kTreeTile);
    ushort4* const flags = (ushort4*)(tile_buf + (size_t)tiles * kMaxDepth);
    k_tree_count<<<tiles, kTreeThreads, 0, st>>>(codes, n, leaf_cap, tile_buf, flags, tv);
    if (tiles > kSelfScanTiles)
        k_tree_scan<<<kMaxDepth, 1024, 0, st>>>(tile_buf, tiles, tv, status);
    k_tree_emit<<<tiles, kTreeThreads, 0, st>>>(codes, n, tiles, tile_buf, flags, tv, status, cx,
                                                cy, cz, hw, bbox);
    k_tree_link<<<grid, 256, 0, st>>>(tv, status);
}

constexpr size_t kClimbParticles = 262144;

void launch_upward(TreeView tv, const Status* status, const float4* xyzm, size_t n,
                   cudaStream_t st) {
    // One climbing launch for a small system, where launches cost more than the
    // climb; the three deepest (and widest) levels of a large one in launches of
    // their own, since a fence and an atomic per leaf cost more than those.
    // Measured (one launch / the 3 deepest levels apart): 33K Plummer 39 / 50 us,
    // 262K 53 / 50, 1M 113 / 65, 4M 309 / 142; 262K clumpy at leaf capacity 16
    // 51 / 69.  One launch per level: 65K 64 us, 1M 80 us.
    const int bottom = n < kClimbParticles ? kMaxDepth : kMaxDepth - 3;
    for (int d = kMaxDepth; d > bottom; --d)
        k_upward_level<<<(tv.lvl_cap[d] + 255) / 256, 256, 0, st>>>(tv, status, xyzm, d);
    k_upward_climb<<<(tv.lvl_base[bottom + 1] + 255) / 256, 256, 0, st>>>(tv, status, xyzm,
                                                                         bottom);
}

}  // namespace psg
