// Device runtime behind the C ABI: per-context device memory, the tick's
// launch sequence, host-pointer mirrors, status checks with capacity regrow,
// the learned closure's per-tick steps and training driver, the device tick
// loop, and the batched ensemble's CUDA graphs.
//
// Ownership follows the reference (polesitter.h:1699-1767): the caller owns
// every particle array and the ps_config_t buffer, and the host-side state
// lives inside that buffer.  The device scratch (sorted particles, tree,
// near lists) is cudaMalloc'ed in ps_init from max_particles and freed in
// ps_destroy; it replaces the reference's arena + radix temporaries.
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <cmath>
#include <mutex>
#include <new>
#include <vector>

#include "psg_closure.cuh"
#include "psg_common.cuh"
#include "psg_kernels.h"

namespace psg {

static thread_local char g_err[256];

static void note(const char* what, cudaError_t e) {
    std::snprintf(g_err, sizeof(g_err), "%s: %s", what, cudaGetErrorString(e));
}

#define PSG_CHECK(call)                        \
    do {                                       \
        cudaError_t _e = (call);               \
        if (_e != cudaSuccess) {               \
            ::psg::note(#call, _e);            \
            return PSG_EDEVICE;                \
        }                                      \
    } while (0)

#define PSG_ALLOC(ptr, bytes)                                        \
    do {                                                             \
        cudaError_t _e = cudaMalloc((void**)&(ptr), (bytes) ? (bytes) : 16); \
        if (_e != cudaSuccess) {                                     \
            ::psg::note("cudaMalloc " #ptr, _e);                     \
            return PSG_EALLOC;                                       \
        }                                                            \
    } while (0)

constexpr uint32_t kMagic = 0x50534732u;  // "PSG2"
constexpr int kPhases = 9;  // timing events
enum Phase { PH_SORT = 0, PH_GATHER, PH_TREE, PH_UP, PH_TRAV, PH_END, PH_BEGIN, PH_CLOSURE,
             PH_DENSE };

// device mirrors of host arrays: one block of 9 rows of cap elements, in the
// order x y z m id codes fx fy fz; stage: pinned rows that a small call's
// pageable arrays pass through
struct Mirror {
    float *x, *y, *z, *m, *fx, *fy, *fz;
    uint32_t *id, *codes;
    size_t cap;
    uint32_t* stage;
    size_t stage_cap;
};

// the learned closure's device buffers (allocated when it is first enabled)
struct ClosureState {
    int mode;            // 0 off (the reference), 1 order-1 local, 2 order-1 + MLP
    int judge;           // run the sampled FP64 judge in mode 1 too
    int judge_bps;       // blocks per SM of the judge's FP64 direct sum (1..8)
    int judge_samples;   // particles of the judge's sample (64..kJudgeSamples)
    float4* lg0;         // per node: field gradient xx yy zz xy
    float2* lg1;         //           xz yz
    uint32_t* leaf_of;   // per sorted particle: its leaf
    float4* dF;          // per sorted particle: the MLP's correction
    float* params;       // FP32 parameter vector (kMlpParams)
    MlpPacked* packed;   // BF16 device copy
    int have_weights;
    uint32_t* judge_tg;  // judge sample (sorted indices)
    double* judge_f64;   // FP64 direct forces of the sample
    double* judge_part;  // ... their partial sums per source split
    size_t judge_part_n;
    JudgeOut* d_judge;
    JudgeOut* h_judge;
    uint32_t tick;       // ticks run in closure mode (varies the judge sample)
    JudgeOut last;       // judge result of the last tick (samples 0: none)
    int valid;           // the last completed tick ran the order-1 traversal
    cudaStream_t side;   // the judge's direct sum, beside the tree and traversal
    cudaEvent_t ev_sorted, ev_judge;
};

struct State {
    uint32_t magic;
    int device;
    int sms;
    int trav_grid[2][2][2];  // leaf-pass grid [closure order 0 / 1][sparse / dense variant]
                             // [plain / chain + stream variant]
    int trav_int_grid[2];
    size_t max_particles;
    float theta;
    int morton_variant;
    int debug;
    int timing;
    cudaStream_t stream;
    float4* xyzm;
    uint32_t* ids;
    SortBuffers sort;
    uint32_t* tree_tiles;
    TreeView tv;
    uint32_t* ns;
    unsigned long long ns_cap;
    P2PStore p2p;
    DenseStore dense;      // full-leaf P2P work records
    SplitStore split;      // sums of the groups that several warps share
    int forest_caps;       // many systems: leaf capacities below kDenseCap (1), others (2)
    int forest_split;      // many systems: the deepest of their split depths
    const int32_t* sys_heavy;  // ... and each one's shallow-leaf and split depth
    const int32_t* sys_split;
    uint32_t* heavy_frontier;
    uint32_t heavy_fcap;
    int heavy_slots;       // blocks of k_heavy_leaf
    bool heavy_off;        // its frontiers overflowed and could not be grown
    cudaStream_t aux;      // split groups or k_heavy_leaf, beside the leaf pass
    cudaEvent_t ev_levels, ev_heavy;
    // host-array calls: the sorted arrays (final after the gather) go back to
    // pinned host buffers on their own stream while the traversal runs
    struct EarlyCopy {
        void* h;
        const void* dv;
    } early[6];
    int n_early = 0;
    size_t early_bytes = 0;
    bool early_issued = false;
    cudaStream_t copy_out = nullptr;
    cudaEvent_t ev_written = nullptr;
    int heavy_depth;       // option; < 0: derived from theta
    int forest_heavy;      // many systems: the deepest of their shallow-leaf depths
    int ns_levels;         // near lists are stored for node depths <= this (kMaxDepth: all);
                           // lowered when they do not fit, deeper groups walk their chains
    bool level_by_level;   // one launch per internal level: the lists once did not fit
    int stream_p2p;        // P2P summed in the leaf pass as found (no spill store)
    int force_ns_levels;   // option: store near lists for depths <= this at most
    int force_stream;      // option: always stream the P2P
    int sort_spin_limit;   // look-back polls before the sort gives up (option; 0: default)
    int ready_spin_limit;  // ... and a traversal group's polls for its parent
    uint32_t leaf_cap;     // option: nodes holding more particles are split (1: the reference)
    double grid_scale;     // traversal grids x this (ensemble autotuner); 0: 1
    int kahan;
    Status* d_status;
    Status* h_status;
    Mirror mir;
    cudaEvent_t ev[kPhases];
    float ms[kPhases];
    unsigned long long stats[24];
    uint32_t last_nodes;
    uint32_t lvl_count[kLevels];  // node counts of the last completed tick
    void* work;            // workspace of one call at a time (struct Work)
    size_t work_bytes;
    // device tick loop scratch (allocated by its first call)
    int tk_grid;
    float2* tk_partial;
    float* tk_bbox;
    float* tk_v[3];
    float* tk_vmir[3];
    ClosureState cl;
    int order;  // traversal's local expansion order: 0 (reference) or 1
    size_t last_n;  // particles of the last completed tick
    bool trav_fresh;  // no traversal has run on the current tree yet
    size_t trav_n;  // particles of the tick whose traversal is being enqueued
    int attempts;   // traversal runs of the last tick (> 1: a capacity regrow)
};

// the near-list levels and the P2P mode start over when what they depend
// on (theta, leaf capacity, expansion order, store sizes) changes
static void reset_near_levels(State* s) {
    s->level_by_level = false;
    s->heavy_off = false;
    s->ns_levels = kMaxDepth;
    s->stream_p2p = 0;
}

static int grid_for(const State* s, size_t n, int per_block_items) {
    size_t want = (n + per_block_items - 1) / per_block_items;
    size_t cap = (size_t)s->sms * 8;
    if (want < 1) want = 1;
    return (int)(want < cap ? want : cap);
}

// near-list entries a warp reserves at once: a warp of a small system takes few
// groups, and pools for all warps would dwarf its lists
static uint32_t ns_pool(size_t n) { return n < 262144 ? kNsPool / 8 : kNsPool; }

static int alloc_ns(State* s, unsigned long long cap) {
    if (s->ns) cudaFree(s->ns);
    s->ns = nullptr;
    s->ns_cap = 0;
    PSG_ALLOC(s->ns, cap * sizeof(uint32_t));
    s->ns_cap = cap;
    return PSG_OK;
}

// one allocation for several arrays, the first of which is its address: a
// cudaMalloc or cudaFree of more than some 100 KB takes 50-200 us whatever its size
// (ps_init with the arrays that keep their size allocated one by one / together:
// 1K particles 1.5 / 1.2 ms, 64K 3.9 / 1.6, 4M 6.7 / 1.9; ps_destroy of 64K
// 4.0 / 1.7 ms)
struct Carve {
    size_t total = 0;
    size_t add(size_t bytes, size_t align = 256) {
        total = (total + align - 1) & ~(align - 1);
        const size_t at = total;
        total += (bytes + 255) & ~(size_t)255;
        return at;
    }
};
template <typename T>
static T* carved(void* base, size_t at) {
    return reinterpret_cast<T*>(static_cast<char*>(base) + at);
}

// The device workspace of a call that brings data of its own (direct sums; the
// closure's features, network, gradient and training), one call at a time.  It
// stays with the context, so that repeated calls allocate nothing: with an
// allocation per array a call paid 0.64 ms more whenever its small arrays needed
// a page that the driver had just taken back (8192 samples trained 0.99 / 0.33 ms,
// the network on 5000 0.78 / 0.14 ms).  Past kWorkKeep it is given back at the
// call's end.
constexpr size_t kWorkKeep = (size_t)64 << 20;

struct Work {
    State* s;
    Carve c;
    explicit Work(State* state) : s(state) {}
    ~Work() {
        if (s->work_bytes <= kWorkKeep) return;
        cudaFree(s->work);
        s->work = nullptr;
        s->work_bytes = 0;
    }
    // (after every add)
    int alloc() {
        if (s->work_bytes >= c.total) return PSG_OK;
        if (s->work) cudaFree(s->work);
        s->work = nullptr;
        s->work_bytes = 0;
        PSG_ALLOC(s->work, c.total);
        s->work_bytes = c.total;
        return PSG_OK;
    }
    template <typename T>
    T* at(size_t off) const { return carved<T>(s->work, off); }
};

static int alloc_p2p(State* s, uint32_t chunks) {
    P2PStore& p = s->p2p;
    if (p.src) cudaFree(p.src);
    p = P2PStore{};
    Carve c;
    c.add((size_t)chunks * kP2PChunk * sizeof(uint2));
    const size_t next = c.add((size_t)chunks * 4), cnt = c.add((size_t)chunks * 4),
                 mask = c.add((size_t)chunks * kP2PChunk);
    PSG_ALLOC(p.src, c.total);
    p.next = carved<uint32_t>(p.src, next);
    p.cnt = carved<uint32_t>(p.src, cnt);
    p.mask = carved<uint8_t>(p.src, mask);
    p.cap_chunks = chunks;
    return PSG_OK;
}

static int alloc_dense(State* s, uint32_t recs, uint32_t slots) {
    DenseStore& d = s->dense;
    if (d.rec) cudaFree(d.rec);
    uint4* const item = d.item;  // (sized by the particles, not by the records)
    d = DenseStore{};
    d.item = item;
    Carve c;
    c.add((size_t)recs * sizeof(uint4));
    const size_t rec_slot = c.add((size_t)recs * 4), prev = c.add((size_t)slots * 4),
                 sums = c.add((size_t)slots * kDenseTargets * 3 * sizeof(double));
    PSG_ALLOC(d.rec, c.total);
    d.rec_slot = carved<uint32_t>(d.rec, rec_slot);
    d.prev = carved<uint32_t>(d.rec, prev);
    d.sums = carved<double>(d.rec, sums);
    d.rec_cap = recs;
    d.slot_cap = slots;
    return PSG_OK;
}

static int alloc_split(SplitStore& p, uint32_t groups) {
    if (p.sums) cudaFree(p.sums);
    p = SplitStore{};
    Carve c;
    c.add((size_t)groups * kSplitParts * kSplitSums * sizeof(float));
    const size_t list = c.add((size_t)groups * kSplitParts * sizeof(uint4)),
                 count = c.add((size_t)groups * 4);
    PSG_ALLOC(p.sums, c.total);
    p.list = carved<uint4>(p.sums, list);
    p.count = carved<uint32_t>(p.sums, count);
    p.cap = groups;
    return PSG_OK;
}

// sums and lists of the groups split over several warps: the groups (two
// halves each) of the depths above `depth`; false when the device cannot hold
// them (many systems: 2.5 KB a group half, 3 MB a system at depth 4): the leaf
// pass then takes every group in one warp
static bool ensure_split(State* s, int depth) {
    uint32_t groups = 0;
    for (int d = 0; d < depth; ++d) groups += 2 * s->tv.lvl_cap[d];
    if (s->split.cap >= groups || alloc_split(s->split, groups) == PSG_OK) return true;
    cudaGetLastError();
    return false;
}

// blocks of k_dense_p2p for n particles: the blocks that fit on the SMs,
// fewer for a small system (whose records, if any, are few), so an ensemble
// of small systems does not launch thousands of idle blocks each
static size_t dense_grid(const State* s, size_t n) {
    return std::min<size_t>((size_t)s->sms * kDenseBlocksPerSm, std::max<size_t>(4, n / 64));
}

// frontier buffers of k_heavy_leaf: 2 x cap candidates per block
static int alloc_heavy(State* s, uint32_t cap) {
    if (s->heavy_frontier) cudaFree(s->heavy_frontier);
    s->heavy_frontier = nullptr;
    s->heavy_fcap = 0;
    // per block: two frontiers and the P2P source list of a multi-particle leaf
    PSG_ALLOC(s->heavy_frontier, (size_t)s->heavy_slots * 3 * cap * 4);
    s->heavy_fcap = cap;
    return PSG_OK;
}

// ... allocated when that kernel first has work (most contexts never run it; 192
// bytes a particle).  A frontier holds at most one level's nodes plus the parent's
// near list.  On a full device they take the place of the P2P stores where the P2P
// is streamed.  False when the device cannot hold them: the leaf pass then takes
// the shallow leaves too.
static bool ensure_heavy(State* s) {
    if (s->heavy_frontier) return true;
    if (s->heavy_off) return false;
    const uint32_t cap = (uint32_t)(s->max_particles / 4 + 4096);
    if (alloc_heavy(s, cap) == PSG_OK) return true;
    cudaGetLastError();
    if (s->stream_p2p && alloc_p2p(s, 64) == PSG_OK && alloc_dense(s, 64, 64) == PSG_OK &&
        alloc_heavy(s, cap) == PSG_OK)
        return true;
    cudaGetLastError();
    return false;
}

static void free_mirror(Mirror& mi) {
    if (mi.x) cudaFree(mi.x);
    if (mi.stage) cudaFreeHost(mi.stage);
    std::memset(&mi, 0, sizeof(mi));
}

static int ensure_mirror(Mirror& mi, size_t n) {
    if (mi.cap >= n && mi.x) return PSG_OK;
    free_mirror(mi);
    const size_t cap = n ? n : 4;
    float* base = nullptr;
    const cudaError_t e = cudaMalloc((void**)&base, 9 * cap * 4);
    if (e != cudaSuccess) {
        note("cudaMalloc mirror", e);
        return PSG_EALLOC;
    }
    mi.x = base;
    mi.y = base + cap;
    mi.z = base + 2 * cap;
    mi.m = base + 3 * cap;
    mi.id = (uint32_t*)(base + 4 * cap);
    mi.codes = (uint32_t*)(base + 5 * cap);
    mi.fx = base + 6 * cap;
    mi.fy = base + 7 * cap;
    mi.fz = base + 8 * cap;
    mi.cap = cap;
    return PSG_OK;
}

// Up to this many particles, pageable arrays go through pinned rows in one copy
// each way: with a pageable copy per array (19 a tick, the ones back each
// waiting for the GPU) a 1K tick took 390 us, so it takes 245.  Above it the
// copies themselves are the cost, and the driver's staging does them.
constexpr size_t kStageMax = 32768;

static int ensure_stage(Mirror& mi, size_t n) {
    if (mi.stage_cap >= n) return PSG_OK;
    if (mi.stage) cudaFreeHost(mi.stage);
    mi.stage = nullptr;
    mi.stage_cap = 0;
    const cudaError_t e = cudaMallocHost((void**)&mi.stage, 9 * n * 4);
    if (e != cudaSuccess) {
        note("cudaMallocHost stage", e);
        return PSG_EALLOC;
    }
    mi.stage_cap = n;
    return PSG_OK;
}

// where p lives: device (or managed) memory, pinned or pageable host memory
enum Place { PAGEABLE = 0, PINNED, DEVICE };

static Place place_of(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return PAGEABLE;
    }
    if (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) return DEVICE;
    return a.type == cudaMemoryTypeHost ? PINNED : PAGEABLE;
}

// true when the GPU can dereference p (device or managed memory)
static bool on_device(const void* p) { return place_of(p) == DEVICE; }

static void free_state(State* s) {
    void* ps[] = {s->xyzm, s->ns, s->p2p.src, s->dense.rec, s->work, s->split.sums,
                  s->heavy_frontier, s->tk_partial, s->tk_bbox, s->tk_v[0], s->tk_v[1], s->tk_v[2],
                  s->tk_vmir[0], s->tk_vmir[1], s->tk_vmir[2], s->cl.lg0, s->cl.lg1,
                  s->cl.leaf_of, s->cl.dF, s->cl.params, s->cl.packed, s->cl.judge_tg,
                  s->cl.judge_f64, s->cl.judge_part, s->cl.d_judge};
    for (void* p : ps)
        if (p) cudaFree(p);
    if (s->h_status) cudaFreeHost(s->h_status);
    if (s->cl.h_judge) cudaFreeHost(s->cl.h_judge);
    if (s->cl.side) cudaStreamSynchronize(s->cl.side);
    if (s->cl.ev_sorted) cudaEventDestroy(s->cl.ev_sorted);
    if (s->cl.ev_judge) cudaEventDestroy(s->cl.ev_judge);
    if (s->cl.side) cudaStreamDestroy(s->cl.side);
    free_mirror(s->mir);
    for (int i = 0; i < kPhases; ++i)
        if (s->ev[i]) cudaEventDestroy(s->ev[i]);
    if (s->aux) {
        cudaStreamSynchronize(s->aux);
        cudaStreamDestroy(s->aux);
    }
    if (s->ev_levels) cudaEventDestroy(s->ev_levels);
    if (s->ev_heavy) cudaEventDestroy(s->ev_heavy);
    if (s->copy_out) {
        cudaStreamSynchronize(s->copy_out);
        cudaStreamDestroy(s->copy_out);
    }
    if (s->ev_written) cudaEventDestroy(s->ev_written);
    if (s->stream) cudaStreamDestroy(s->stream);
    s->magic = 0;
}

// lvl_caps (optional): node capacity of each level, for a tree pass over
// many systems; sort_passes: radix passes the look-back flags must serve
static int init_state(State* s, size_t maxp, float theta, const uint32_t* lvl_caps = nullptr,
                      int sort_passes = 4) {
    std::memset(s, 0, sizeof(State));
    PSG_CHECK(cudaGetDevice(&s->device));
    PSG_CHECK(cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, s->device));
    PSG_CHECK(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
    for (int i = 0; i < kPhases; ++i) PSG_CHECK(cudaEventCreate(&s->ev[i]));
    s->max_particles = maxp;
    s->theta = theta;
    s->morton_variant = PSG_MORTON_AVX2;
    const size_t n = maxp ? maxp : 1;
    // level capacities: min(8^d, n) nodes at depth d
    uint32_t base = 0;
    for (int d = 0; d <= kMaxDepth; ++d) {
        unsigned long long cap8 = 1ull << (3 * d);
        uint32_t cap = (uint32_t)(cap8 < n ? cap8 : n);
        if (d == 0) cap = 1;
        if (lvl_caps) cap = lvl_caps[d];
        s->tv.lvl_base[d] = base;
        s->tv.lvl_cap[d] = cap;
        base += cap;
    }
    s->tv.lvl_base[kLevels] = base;
    s->tv.lvl_cap[kLevels] = 0;
    const size_t nodes = base, stiles = (n + sort_tile_size() - 1) / sort_tile_size();
    {
        // everything that keeps its size, in one allocation (xyzm is its address)
        TreeView& t = s->tv;
        const struct { void* p; size_t bytes; } part[] = {
            {&s->xyzm, n * sizeof(float4)}, {&s->ids, n * 4},
            {&s->sort.key_a, n * 4}, {&s->sort.key_b, n * 4},
            {&s->sort.val_a, n * 4}, {&s->sort.val_b, n * 4},
            {&s->sort.hist, ((size_t)sort_passes * stiles + 4) * 256 * 4},
            {&s->tree_tiles, tree_scratch_bytes(n)},
            {&t.geo, nodes * 16}, {&t.mp, nodes * 16}, {&t.lt, nodes * 16},
            {&t.info, nodes * 16}, {&t.parent, nodes * 4}, {&t.arrive, nodes * 4},
            {&t.cbase, nodes * 4}, {&t.ns_off, nodes * 4}, {&t.ns_cnt, nodes * 4},
            {&t.dbg_m2l, nodes * 4}, {&t.dbg_p2p, nodes * 4}, {&t.link, nodes * 4},
            {&t.ready, nodes * 4}, {&t.groups, nodes * 4},
            {&s->dense.item, n * sizeof(uint4)}, {&s->d_status, sizeof(Status)}};
        // (large ones start at 2 MB, as an allocation of their own would: end to end
        // a 1M tick took 2.29 instead of 2.28 ms)
        auto align = [](size_t bytes) -> size_t { return bytes < (1u << 20) ? 256 : 2u << 20; };
        Carve c, at;
        for (const auto& q : part) c.add(q.bytes, align(q.bytes));
        char* fixed = nullptr;
        PSG_ALLOC(fixed, c.total);
        for (const auto& q : part) {
            void* const p = fixed + at.add(q.bytes, align(q.bytes));
            std::memcpy(q.p, &p, sizeof(p));
        }
        s->sort.lookback = s->sort.hist + 4 * 256;
    }
    PSG_CHECK(cudaMallocHost((void**)&s->h_status, sizeof(Status)));
    std::memset(s->h_status, 0, sizeof(Status));
    // first sizes of the stores that the warps take pools from: what the lists
    // need as a rule, and a pool for every warp that can hold one (without, the
    // first tick of a system of up to some 100K particles was run twice: 1.33
    // against 0.49 ms at 65K, 4.0 against 0.64 at 8K with leaves of 16)
    const unsigned long long warps = std::min<unsigned long long>(n / 4 + 1, s->sms * 20ull);
    int r = alloc_ns(s, (unsigned long long)(n < 1024 ? 1024 : n) * 48ull + warps * ns_pool(n));
    if (r != PSG_OK) return r;
    r = alloc_p2p(s, (uint32_t)((n < 4096 ? 4096 : n / 4) + warps * kChunkPool));
    if (r != PSG_OK) return r;
    r = alloc_dense(s, (uint32_t)(n / 2 + 1024), (uint32_t)(n / 8 + 8192));
    if (r != PSG_OK) return r;
    s->heavy_slots = 64;
    s->heavy_depth = -1;
    s->ns_levels = kMaxDepth;
    s->force_ns_levels = kMaxDepth;
    s->leaf_cap = 1;
    PSG_CHECK(cudaStreamCreateWithFlags(&s->aux, cudaStreamNonBlocking));
    PSG_CHECK(cudaEventCreateWithFlags(&s->ev_levels, cudaEventDisableTiming));
    PSG_CHECK(cudaEventCreateWithFlags(&s->ev_heavy, cudaEventDisableTiming));
    for (int o = 0; o < 2; ++o) {
        int bps = 0;
        for (int dn = 0; dn < 2; ++dn) {
            for (int xl = 0; xl < 2; ++xl) {
                PSG_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                    &bps, traverse_kernel_ptr(o, dn, xl), traverse_threads(), 0));
                s->trav_grid[o][dn][xl] = s->sms * (bps > 0 ? bps : 1);
            }
        }
        PSG_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &bps, traverse_internal_kernel_ptr(o), traverse_threads(), 0));
        s->trav_int_grid[o] = s->sms * (bps > 0 ? bps : 1);
    }
    s->magic = kMagic;
    return PSG_OK;
}

static int closure_alloc(State* s) {
    ClosureState& c = s->cl;
    if (c.lg0) return PSG_OK;
    const size_t nodes = s->tv.lvl_base[kLevels];
    const size_t n = s->max_particles ? s->max_particles : 1;
    PSG_ALLOC(c.lg0, nodes * sizeof(float4));
    PSG_ALLOC(c.lg1, nodes * sizeof(float2));
    PSG_ALLOC(c.leaf_of, n * 4);
    PSG_ALLOC(c.dF, n * sizeof(float4));
    PSG_ALLOC(c.params, kMlpParams * sizeof(float));
    PSG_ALLOC(c.packed, sizeof(MlpPacked));
    PSG_ALLOC(c.judge_tg, kJudgeSamples * 4);
    PSG_ALLOC(c.judge_f64, kJudgeSamples * 3 * sizeof(double));
    c.judge_part_n = direct_f64_part_doubles(n, kJudgeSamples, s->sms * 8);
    if (c.judge_bps == 0) c.judge_bps = 4;
    if (c.judge_samples == 0) c.judge_samples = kJudgeDefault;
    PSG_ALLOC(c.judge_part, c.judge_part_n * sizeof(double));
    PSG_ALLOC(c.d_judge, sizeof(JudgeOut));
    PSG_CHECK(cudaMallocHost((void**)&c.h_judge, sizeof(JudgeOut)));
    std::memset(c.h_judge, 0, sizeof(JudgeOut));
    PSG_CHECK(cudaStreamCreateWithFlags(&c.side, cudaStreamNonBlocking));
    PSG_CHECK(cudaEventCreateWithFlags(&c.ev_sorted, cudaEventDisableTiming));
    PSG_CHECK(cudaEventCreateWithFlags(&c.ev_judge, cudaEventDisableTiming));
    return PSG_OK;
}

// A leaf at depth d (half width H / 2^d of the root's H) stays unseparated
// from the sources within about theta H / 2^(d-1), a large part of the tree
// once 2^d <= 4 theta.  The leaf pass shares such groups out over kSplitParts
// warps each (split_depth_of).  The leaf pass that walks ancestor chains or
// streams its P2P takes each group in one warp; beside it such leaves are
// walked block-parallel by k_heavy_leaf (also on demand:
// PS_B200_OPT_HEAVY_DEPTH), but not below kHeavyMinParticles, where a walk
// over the whole tree is still short and shallow leaves are most leaves.
constexpr size_t kHeavyMinParticles = 131072;

static int heavy_depth_of(float theta, size_t n) {
    if (n < kHeavyMinParticles) return 0;
    int d = 0;
    while (d < 5 && (float)(2 << d) <= 4.0f * theta) ++d;
    return d < 2 ? 2 : d;
}

// Depth above which the leaf pass splits groups over kSplitParts warps: 3 from
// theta 3 and 4 from theta 4 on, where a shallow leaf's walk is long, none below
// theta 3, and only above the depth at which n particles spread evenly would have
// their leaves (8^d * cap < n), since groups that are the rule need no help.
// Measured (leaf pass and
// full-leaf P2P, one warp per group / split): 32K clumpy at theta 8 7.0 / 2.8
// ms, 131K clumpy at theta 6.25 and leaf capacity 16 1.87 / 1.42 ms; theta 3
// 32K clumpy 0.41 / 0.42 ms; without the second limit 32K cube at theta 10 and
// leaf capacity 16 0.61 / 0.61 ms but 0.11 ms more a tick, 1K cube at theta 8
// 0.21 / 0.41 ms.
constexpr int kSplitBlocksPerSm = 4;

static int split_depth_of(float theta, size_t n, uint32_t cap) {
    if (theta < 3.0f) return 0;
    int d = theta < 4.0f ? 3 : 4;
    while (d > 0 && ((unsigned long long)cap << (3 * d)) >= n) --d;
    return d;
}

static int heavy_depth_for(const State* s) {
    if (s->tv.part_sys) return s->forest_heavy;  // many systems: the deepest of theirs
    if (s->heavy_depth >= 0) return s->heavy_depth > 5 ? 5 : s->heavy_depth;
    return heavy_depth_of(s->theta, s->trav_n);
}

// Depth of the deepest nodes whose near lists this traversal stores.  The
// shallow-leaf walk reads the lists of depths < heavy_depth, so they always
// exist; the order-1 expansion needs every level's (its chain groups would
// need each ancestor's own gradient).
static int near_levels(const State* s) {
    if (s->order >= 1) return kMaxDepth;
    int k = std::min(s->ns_levels, s->force_ns_levels);
    return std::max(k, std::max(2, heavy_depth_for(s) - 1));
}

static void record(State* s, int ph) {
    if (s->timing) cudaEventRecord(s->ev[ph], s->stream);
}

// one traversal run (internal levels, leaf pass, shallow leaves, full
// leaves) enqueued on s->stream; no host synchronisation
static int enqueue_traversal(State* s, const float4* xyzm, float* fx, float* fy, float* fz) {
    if (!s->trav_fresh) {  // (a new tree comes with its counters and flags zeroed)
        Status* const ds = s->d_status;
        PSG_CHECK(cudaMemsetAsync(&ds->run, 0, sizeof(ds->run), s->stream));
        PSG_CHECK(cudaMemsetAsync(s->tv.ready, 0, (size_t)s->tv.lvl_base[kLevels] * 4,
                                  s->stream));
    }
    s->trav_fresh = false;
    TravArgs A;
    A.tv = s->tv;
    A.ns = s->ns;
    A.ns_cap = s->ns_cap;
    A.ns_pool = ns_pool(s->max_particles);
    A.status = s->d_status;
    A.theta = s->theta;
    A.level = 0;
    A.ready_spin = s->ready_spin_limit;
    A.debug = s->debug;
    A.kahan = s->kahan;
    A.xyzm = xyzm;
    A.fx = fx;
    A.fy = fy;
    A.fz = fz;
    const int o = s->order >= 1 ? 1 : 0;
    A.order = o;
    A.leaf_of = o ? s->cl.leaf_of : nullptr;
    A.tv.lg0 = o ? s->cl.lg0 : nullptr;
    A.tv.lg1 = o ? s->cl.lg1 : nullptr;
    const bool xl = near_levels(s) < kMaxDepth || s->stream_p2p || s->force_stream;
    // the shallow groups: split over several warps, or (XL, or on demand)
    // k_heavy_leaf's
    const bool forest = s->tv.part_sys != nullptr;
    const bool heavy = xl || s->heavy_depth >= 0;
    int depth = heavy    ? heavy_depth_for(s)
                : forest ? s->forest_split
                         : split_depth_of(s->theta, s->trav_n, s->leaf_cap);
    if (!heavy && !ensure_split(s, depth)) depth = 0;
    if (heavy && depth && !ensure_heavy(s)) {
        if (forest) return PSG_EALLOC;  // (its groups read their systems' depths)
        depth = 0;
    }
    if (forest) A.tv.sys_shallow = heavy ? s->sys_heavy : s->sys_split;
    A.shallow = forest ? 0 : depth;
    // (not reset by the kernel: a void run may stop half way)
    if (!heavy && depth)
        PSG_CHECK(cudaMemsetAsync(s->split.count, 0, (size_t)s->split.cap * 4, s->stream));
    A.p2p = s->p2p;
    A.dense = s->dense;
    A.split = s->split;
    A.heavy_depth = depth;
    A.heavy_frontier = s->heavy_frontier;
    A.heavy_fcap = s->heavy_fcap;
    A.ns_levels = near_levels(s);
    A.leaf_cap = s->leaf_cap;
    A.stream = (s->stream_p2p || s->force_stream) ? 1 : 0;
    const double gs = s->grid_scale > 0.0 ? s->grid_scale : 1.0;
    auto scaled = [&](int g) {
        const int v = (int)(g * gs);
        return v < 1 ? 1 : v;
    };
    // leaf capacities below kDenseCap (1), others (2), systems of both kinds (3)
    const int caps = forest ? s->forest_caps : s->leaf_cap >= kDenseCap ? 2 : 1;
    // The shallow groups on the aux stream.  They read the near lists and
    // fields of the nodes above `depth`, final once the internal level of
    // depth - 1 is done, so they start there and run beside the deeper levels
    // and the leaf pass (which starts at the groups of that depth).
    bool started = depth == 0;
    auto start_shallow = [&]() -> int {
        PSG_CHECK(cudaEventRecord(s->ev_levels, s->stream));
        PSG_CHECK(cudaStreamWaitEvent(s->aux, s->ev_levels, 0));
        if (heavy) {
            launch_heavy_leaf(A, scaled(s->heavy_slots), s->aux);
        } else {
            TravArgs S = A;
            S.shallow = depth;
            launch_traverse_split(S, scaled(s->sms * kSplitBlocksPerSm), caps, s->aux);
        }
        PSG_CHECK(cudaEventRecord(s->ev_heavy, s->aux));
        started = true;
        return PSG_OK;
    };
    if (!started && depth - 1 < 2) {
        const int r = start_shallow();
        if (r != PSG_OK) return r;
    }
    // the internal levels in one launch, two when the shallow groups start
    // between them; one launch per level while the lists are short of memory
    // (the first level that does not fit is then the same in every run)
    for (int k = 2; k <= A.ns_levels;) {
        int end = A.ns_levels;
        if (s->level_by_level) end = k;
        if (!started) end = std::min(end, std::max(k, depth - 1));
        launch_traverse_internal(A, k, end, scaled(s->trav_int_grid[o]), s->stream);
        if (!started && end >= depth - 1) {
            const int r = start_shallow();
            if (r != PSG_OK) return r;
        }
        k = end + 1;
    }
    record(s, PH_TRAV);
    if (!started) {
        const int r = start_shallow();
        if (r != PSG_OK) return r;
    }
    const int lg[2] = {scaled(s->trav_grid[o][0][xl]), scaled(s->trav_grid[o][1][xl])};
    launch_traverse_leaves(A, lg, caps, s->stream);
    record(s, PH_DENSE);
    // (the split groups' records too; k_heavy_leaf leaves none)
    if (depth && !heavy) PSG_CHECK(cudaStreamWaitEvent(s->stream, s->ev_heavy, 0));
    launch_dense_p2p(A, scaled((int)dense_grid(s, s->trav_n)), s->stream);
    if (depth && heavy) PSG_CHECK(cudaStreamWaitEvent(s->stream, s->ev_heavy, 0));
    record(s, PH_END);
    return PSG_OK;
}

// bytes a growing store may take: what the device has free plus what the
// store holds now (freed before the new one is allocated), less 1/16 of the
// device for everything else
static unsigned long long store_budget(unsigned long long held) {
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
        cudaGetLastError();
        return held;
    }
    const unsigned long long avail = (unsigned long long)fr + held, margin = tot / 16;
    return avail > margin ? avail - margin : 0ull;
}

// a store of another size, or the old one back when the device refuses
static bool try_alloc_ns(State* s, unsigned long long cap) {
    const unsigned long long old = s->ns_cap;
    if (alloc_ns(s, cap) == PSG_OK) return true;
    cudaGetLastError();
    alloc_ns(s, old);
    return false;
}

static bool try_alloc_p2p(State* s, uint32_t chunks) {
    const uint32_t old = s->p2p.cap_chunks;
    if (alloc_p2p(s, chunks) == PSG_OK) return true;
    cudaGetLastError();
    alloc_p2p(s, old);
    return false;
}

static bool try_alloc_dense(State* s, uint32_t recs, uint32_t slots) {
    const uint32_t old_recs = s->dense.rec_cap, old_slots = s->dense.slot_cap;
    if (alloc_dense(s, recs, slots) == PSG_OK) return true;
    cudaGetLastError();
    alloc_dense(s, old_recs, old_slots);
    return false;
}

// After a traversal run read back its status, makes room for every store
// that ran out, for the rerun and later ticks:
//  * near lists: grown to twice what the run reserved while the device has
//    the memory and 32-bit offsets reach; past that (order 0), they stop at
//    the level before the first that did not fit, the groups below walk
//    their ancestor chains, and the P2P is streamed, so no store grows with
//    theta any more;
//  * P2P chunks: grown likewise, else the P2P is streamed;
//  * full-leaf records: grown (a segment of a source list takes a slot of 384
//    bytes per record, so they too grow with theta), else the P2P is streamed;
//  * shallow-leaf frontiers: grown, else (one system) the leaf pass takes the
//    shallow leaves.
// PSG_EOOM when nothing can give.
static int regrow(State* s, uint32_t err) {
    if (err & PSG_ERR_NS_OVERFLOW) {
        const unsigned long long used = s->h_status->run.ns_used;
        const uint32_t fail = s->h_status->run.ns_fail;
        const int kf = fail ? __builtin_ctz(fail) : kMaxDepth;
        const unsigned long long limit =
            std::min(0xFFFFFFF0ull, store_budget(s->ns_cap * 4) / 4);
        const unsigned long long want = 2 * used + (1ull << 20);
        const int floor_k = std::max(2, heavy_depth_for(s) - 1);
        bool done = false;
        if (want <= limit) {
            done = try_alloc_ns(s, want);
        } else if (s->ns_cap < limit && used + (1ull << 20) <= limit) {
            // what the run reserved fits, twice that does not: the largest
            // store, and the levels below show whether it is enough
            done = try_alloc_ns(s, limit);
        }
        if (!done && s->order == 0 && !s->level_by_level) {
            // which level is the first that does not fit: run level by level
            s->level_by_level = true;
            done = true;
        }
        if (!done && s->order == 0 && kf - 1 >= floor_k) {
            s->ns_levels = kf - 1;
            s->stream_p2p = 1;
            done = true;
        }
        if (!done && s->order >= 1 && limit > s->ns_cap) done = try_alloc_ns(s, limit);
        if (!done) {
            std::snprintf(g_err, sizeof(g_err),
                          "near lists need %llu entries at level %d; the device holds %llu",
                          want, kf, limit);
            return PSG_EOOM;
        }
    }
    if (err & PSG_ERR_HEAVY_OVERFLOW) {
        unsigned long long cap = 2ull * s->heavy_fcap;
        const unsigned long long most = 2ull * s->max_particles + 1024;
        int r = alloc_heavy(s, (uint32_t)(cap < most ? cap : most));
        if (r != PSG_OK && s->tv.part_sys) return r;
        if (r != PSG_OK) {
            cudaGetLastError();
            s->heavy_off = true;
        }
    }
    if (err & PSG_ERR_P2P_OVERFLOW) {
        // the chunk counter is 32-bit: below the capacity it has wrapped
        const unsigned long long used = s->h_status->run.p2p_chunks;
        const unsigned long long need = used < s->p2p.cap_chunks ? ~0ull : 2 * used + 1024;
        const unsigned long long per = kP2PChunk * 9 + 8;
        const unsigned long long limit =
            std::min(0x7FFFFFFFull, store_budget(s->p2p.cap_chunks * per) / per);
        if (!(need <= limit && try_alloc_p2p(s, (uint32_t)need))) s->stream_p2p = 1;
    }
    if ((err & PSG_ERR_DENSE_OVERFLOW) && !s->stream_p2p) {
        auto room = [](uint32_t used, uint32_t cap) {
            if (used <= cap) return cap;
            const unsigned long long need = (unsigned long long)used + used / 4 + 1024;
            return (uint32_t)std::min<unsigned long long>(need, 0x7FFFFFFFull);
        };
        const uint32_t recs = room(s->h_status->run.dense_count, s->dense.rec_cap),
                       slots = room(s->h_status->run.dense_slots, s->dense.slot_cap);
        // (both below their capacity: a 32-bit counter has wrapped)
        const bool wrapped = recs == s->dense.rec_cap && slots == s->dense.slot_cap;
        if (wrapped || !try_alloc_dense(s, recs, slots)) s->stream_p2p = 1;
    }
    return PSG_OK;
}

// traversal of all levels + P2P/L2P; regrows the near-list regions or the
// P2P chunk store and reruns when a capacity flag comes back
static int run_traversal(State* s, const float4* xyzm, float* fx, float* fy, float* fz,
                         uint32_t* err_out) {
    for (int attempt = 0; attempt < 8; ++attempt) {
        s->attempts = attempt + 1;
        int r0 = enqueue_traversal(s, xyzm, fx, fy, fz);
        if (r0 != PSG_OK) return r0;
        PSG_CHECK(cudaGetLastError());
        PSG_CHECK(cudaMemcpyAsync(s->h_status, s->d_status, sizeof(Status),
                                  cudaMemcpyDeviceToHost, s->stream));
        PSG_CHECK(cudaStreamSynchronize(s->stream));
        const uint32_t err = s->h_status->err;
        if (!(err & (PSG_ERR_NS_OVERFLOW | PSG_ERR_P2P_OVERFLOW | PSG_ERR_DENSE_OVERFLOW |
                     PSG_ERR_HEAVY_OVERFLOW))) {
            *err_out = err;
            return PSG_OK;
        }
        int rg = regrow(s, err);
        if (rg != PSG_OK) return rg;
        PSG_CHECK(cudaMemsetAsync(&s->d_status->err, 0, 4, s->stream));
        PSG_CHECK(cudaMemsetAsync(&s->d_status->stat[0], 0, sizeof(s->d_status->stat), s->stream));
        if (s->debug) {
            const size_t bytes = (size_t)s->tv.lvl_base[kLevels] * 4;
            PSG_CHECK(cudaMemsetAsync(s->tv.dbg_m2l, 0, bytes, s->stream));
            PSG_CHECK(cudaMemsetAsync(s->tv.dbg_p2p, 0, bytes, s->stream));
        }
        if (s->timing) cudaEventRecord(s->ev[PH_UP], s->stream);
    }
    std::snprintf(g_err, sizeof(g_err), "traversal stores still too small after 8 runs");
    return PSG_EOOM;
}

// the caller's arrays as the GPU sees them: in place when it can reach them,
// else device mirrors in the context
struct DevArrays {
    float *x, *y, *z, *m, *fx, *fy, *fz;
    uint32_t *id, *codes;
    bool dev[9];      // (rows as in Mirror) no copy back is due
    bool pinned[9];
    bool any_host;
    bool staged;      // all through the mirror's pinned rows
};

static int map_arrays(State* s, const psg_arrays_t* a, DevArrays& d, bool upload_codes) {
    const size_t n = a->n;
    d.x = a->x; d.y = a->y; d.z = a->z; d.m = a->mass;
    d.fx = a->fx; d.fy = a->fy; d.fz = a->fz; d.id = a->id; d.codes = a->codes;
    void* const ps[9] = {d.x, d.y, d.z, d.m, d.id, d.codes, d.fx, d.fy, d.fz};
    d.any_host = false;
    d.staged = n <= kStageMax;
    for (int i = 0; i < 9; ++i) {
        const Place p = place_of(ps[i]);
        d.dev[i] = p == DEVICE;
        d.pinned[i] = p == PINNED;
        d.any_host |= p != DEVICE;
        d.staged &= p == PAGEABLE;
    }
    if (!d.any_host) return PSG_OK;
    Mirror& mi = s->mir;
    int r = ensure_mirror(mi, s->max_particles);
    if (r == PSG_OK && d.staged) r = ensure_stage(mi, std::min(s->max_particles, kStageMax));
    if (r != PSG_OK) return r;
    void* const rows[9] = {mi.x, mi.y, mi.z, mi.m, mi.id, mi.codes, mi.fx, mi.fy, mi.fz};
    const int in = upload_codes ? 6 : 5;
    if (d.staged) {
        for (int i = 0; i < in; ++i) std::memcpy(mi.stage + (size_t)i * n, ps[i], n * 4);
        PSG_CHECK(cudaMemcpy2DAsync(mi.x, mi.cap * 4, mi.stage, n * 4, n * 4, in,
                                    cudaMemcpyHostToDevice, s->stream));
    } else {
        for (int i = 0; i < in; ++i)
            if (!d.dev[i])
                PSG_CHECK(cudaMemcpyAsync(rows[i], ps[i], n * 4, cudaMemcpyHostToDevice,
                                          s->stream));
    }
    if (!d.dev[0]) d.x = mi.x;
    if (!d.dev[1]) d.y = mi.y;
    if (!d.dev[2]) d.z = mi.z;
    if (!d.dev[3]) d.m = mi.m;
    if (!d.dev[4]) d.id = mi.id;
    if (!d.dev[5]) d.codes = mi.codes;
    if (!d.dev[6]) d.fx = mi.fx;
    if (!d.dev[7]) d.fy = mi.fy;
    if (!d.dev[8]) d.fz = mi.fz;
    return PSG_OK;
}

// the results back into the caller's host arrays, final when this returns
static int unmap_arrays(State* s, const psg_arrays_t* a, const DevArrays& d) {
    const size_t n = a->n;
    Mirror& mi = s->mir;
    void* const hs[9] = {a->x, a->y, a->z, a->mass, a->id, a->codes, a->fx, a->fy, a->fz};
    if (d.staged && d.any_host) {
        PSG_CHECK(cudaMemcpy2DAsync(mi.stage, n * 4, mi.x, mi.cap * 4, n * 4, 9,
                                    cudaMemcpyDeviceToHost, s->stream));
        PSG_CHECK(cudaStreamSynchronize(s->stream));
        for (int i = 0; i < 9; ++i) std::memcpy(hs[i], mi.stage + (size_t)i * n, n * 4);
        return PSG_OK;
    }
    const void* const ds[9] = {d.x, d.y, d.z, d.m, d.id, d.codes, d.fx, d.fy, d.fz};
    for (int i = 0; d.any_host && i < 9; ++i)
        if (!d.dev[i])
            PSG_CHECK(cudaMemcpyAsync(hs[i], ds[i], n * 4, cudaMemcpyDeviceToHost, s->stream));
    PSG_CHECK(cudaStreamSynchronize(s->stream));
    return PSG_OK;
}

// ps_calc_forces on device-resident arrays: sort -> gather -> tree -> upward
// -> traversal (polesitter.h:1840-1909).  The root is (cx, cy, cz, hw), or,
// when bbox is set, derived on the device from this tick's bounding box.
static int tick_core(State* s, const DevArrays& d, size_t n, float cx, float cy, float cz,
                     float hw, const float* bbox) {
    cudaStream_t st = s->stream;
    record(s, PH_BEGIN);
    PSG_CHECK(cudaMemsetAsync(s->d_status, 0, sizeof(Status), st));
    const int g = grid_for(s, n, 1024);
    if (sort_small_fits(n) && s->sort_spin_limit == 0) {
        launch_sort_small(d.codes, n, d.x, d.y, d.z, d.m, d.id, s->xyzm, s->ids, st);
        record(s, PH_SORT);
    } else {
        launch_sort(s->sort, d.codes, n, g, s->d_status, st, s->sort_spin_limit);
        record(s, PH_SORT);
        launch_gather(s->sort.perm, d.x, d.y, d.z, d.m, d.id, n, s->xyzm, s->ids, g, st);
        launch_writeback(s->xyzm, s->ids, n, d.x, d.y, d.z, d.m, d.id, g, st);
    }
    if (s->n_early && !s->early_issued) {
        PSG_CHECK(cudaEventRecord(s->ev_written, st));
        PSG_CHECK(cudaStreamWaitEvent(s->copy_out, s->ev_written, 0));
        for (int k = 0; k < s->n_early; ++k)
            PSG_CHECK(cudaMemcpyAsync(s->early[k].h, s->early[k].dv, s->early_bytes,
                                      cudaMemcpyDeviceToHost, s->copy_out));
        s->early_issued = true;
    }
    record(s, PH_GATHER);
    // closure judge: its FP64 direct sum needs only the sorted particles, so
    // it runs on a side stream under the tree build and traversal, on a
    // quarter of the GPU's block slots
    ClosureState& cj = s->cl;
    const bool judge = s->order >= 1 && n > 1 && ((cj.mode == 2 && cj.have_weights) || cj.judge);
    const int smp = n < (size_t)cj.judge_samples ? (int)n : cj.judge_samples;
    if (judge) {
        PSG_CHECK(cudaEventRecord(cj.ev_sorted, st));
        PSG_CHECK(cudaStreamWaitEvent(cj.side, cj.ev_sorted, 0));
        launch_judge_direct(s->xyzm, n, cj.judge_tg, smp, cj.judge_f64, cj.tick,
                            s->sms * cj.judge_bps,
                            cj.side, cj.judge_part, cj.judge_part_n);
        PSG_CHECK(cudaEventRecord(cj.ev_judge, cj.side));
    }
    const int gt = (int)((s->tv.lvl_base[kLevels] + 255) / 256);
    if (s->debug) {
        PSG_CHECK(cudaMemsetAsync(s->tv.dbg_m2l, 0, (size_t)s->tv.lvl_base[kLevels] * 4, st));
        PSG_CHECK(cudaMemsetAsync(s->tv.dbg_p2p, 0, (size_t)s->tv.lvl_base[kLevels] * 4, st));
    }
    launch_tree(d.codes, n, s->tree_tiles, s->tv, s->d_status, cx, cy, cz, hw, gt, st, bbox,
                s->leaf_cap);
    record(s, PH_TREE);
    launch_upward(s->tv, s->d_status, s->xyzm, n, st);
    s->trav_fresh = true;
    record(s, PH_UP);
    PSG_CHECK(cudaGetLastError());
    uint32_t err = 0;
    if (n == 1) {
        // a single particle: the root is a leaf and its only P2P term is
        // the zero self-interaction (polesitter.h:1279-1449)
        PSG_CHECK(cudaMemsetAsync(d.fx, 0, 4, st));
        PSG_CHECK(cudaMemsetAsync(d.fy, 0, 4, st));
        PSG_CHECK(cudaMemsetAsync(d.fz, 0, 4, st));
        record(s, PH_TRAV);
        record(s, PH_DENSE);
        record(s, PH_END);
        PSG_CHECK(cudaMemcpyAsync(s->h_status, s->d_status, sizeof(Status),
                                  cudaMemcpyDeviceToHost, st));
        PSG_CHECK(cudaStreamSynchronize(st));
        err = s->h_status->err;
    } else {
        s->trav_n = n;
        int r = run_traversal(s, s->xyzm, d.fx, d.fy, d.fz, &err);
        if (r != PSG_OK) {
            if (judge) cudaStreamSynchronize(cj.side);  // leave no judge work running
            return r;
        }
    }
    if (err & PSG_ERR_FATAL) {
        if (judge) cudaStreamSynchronize(cj.side);
        const bool nodes = (err & PSG_ERR_FATAL) == PSG_ERR_NODES;
        std::snprintf(g_err, sizeof(g_err), nodes ? "morton codes not sorted/30-bit (0x%x)"
                                                  : "device status error 0x%x", err);
        return nodes ? PSG_EINVAL : PSG_EDEVICE;
    }
    s->cl.last.samples = 0;
    s->cl.valid = s->order >= 1 && n > 1;
    if (judge) {
        // learned closure: MLP correction, the judge's decision, fallback
        ClosureState& c = s->cl;
        const bool mlp = c.mode == 2 && c.have_weights;
        {
            TreeView tv = s->tv;
            tv.lg0 = c.lg0;
            tv.lg1 = c.lg1;
            if (mlp) {
                launch_closure_mlp(tv, c.leaf_of, s->xyzm, n, c.packed, c.dF, s->sms,
                                   &s->d_status->err, st);
            } else {
                PSG_CHECK(cudaMemsetAsync(c.dF, 0, n * sizeof(float4), st));
            }
            PSG_CHECK(cudaStreamWaitEvent(st, c.ev_judge, 0));
            launch_judge_decide(c.judge_tg, smp, c.judge_f64, d.fx, d.fy, d.fz, c.dF,
                                mlp ? 1 : 0, c.d_judge, st);
            if (mlp) launch_closure_apply(d.fx, d.fy, d.fz, c.dF, n, c.d_judge, s->sms, st);
            PSG_CHECK(cudaGetLastError());
            PSG_CHECK(cudaMemcpyAsync(c.h_judge, c.d_judge, sizeof(JudgeOut),
                                      cudaMemcpyDeviceToHost, st));
            if (mlp)
                PSG_CHECK(cudaMemcpyAsync(&s->h_status->err, &s->d_status->err, 4,
                                          cudaMemcpyDeviceToHost, st));
            PSG_CHECK(cudaStreamSynchronize(st));
            if (mlp && (s->h_status->err & PSG_ERR_TC_TIMEOUT)) {
                std::snprintf(g_err, sizeof(g_err),
                              "closure network: a tensor-core MMA did not complete");
                return PSG_EDEVICE;
            }
            c.last = *c.h_judge;
            ++c.tick;
        }
    }
    record(s, PH_CLOSURE);
    uint32_t nodes = 0;
    for (int k = 0; k <= kMaxDepth; ++k) {
        s->lvl_count[k] = s->h_status->lvl_count[k];
        nodes += s->lvl_count[k];
    }
    s->last_nodes = nodes;
    s->last_n = n;
    for (int i = 0; i < 8; ++i) s->stats[i] = s->h_status->stat[i];
    s->stats[8] = nodes;
    s->stats[9] = s->h_status->max_stack;
    for (int i = 8; i < 16; ++i) s->stats[i + 8] = s->h_status->stat[i];
    s->stats[10] = s->h_status->run.p2p_chunks;
    s->stats[11] = (unsigned long long)s->attempts;
    s->stats[12] = s->h_status->max_leaf;
    s->stats[13] = s->h_status->run.dense_count;
    s->stats[14] = (unsigned long long)near_levels(s);
    s->stats[15] = (s->stream_p2p || s->force_stream) ? 1ull : 0ull;
    if (s->timing) {
        cudaEventSynchronize(s->ev[PH_CLOSURE]);
        const int order[7] = {PH_BEGIN, PH_SORT, PH_GATHER, PH_TREE, PH_UP, PH_TRAV, PH_DENSE};
        for (int i = 0; i + 1 < 7; ++i)
            cudaEventElapsedTime(&s->ms[i], s->ev[order[i]], s->ev[order[i + 1]]);
        cudaEventElapsedTime(&s->ms[6], s->ev[PH_BEGIN], s->ev[PH_CLOSURE]);
        cudaEventElapsedTime(&s->ms[7], s->ev[PH_END], s->ev[PH_CLOSURE]);
        cudaEventElapsedTime(&s->ms[8], s->ev[PH_DENSE], s->ev[PH_END]);
    }
    return PSG_OK;
}

static int calc(State* s, const psg_arrays_t* a, float cx, float cy, float cz, float hw) {
    const size_t n = a->n;
    if (n > s->max_particles) return PSG_EINVAL;
    if (n == 0) return PSG_OK;
    PSG_CHECK(cudaSetDevice(s->device));
    DevArrays d;
    int r = map_arrays(s, a, d, true);
    if (r != PSG_OK) return r;
    // sorted positions, masses, ids and codes into pinned host arrays go back
    // while the traversal runs (a pageable copy would block this thread, so
    // those wait for the end); the forces go back at the end
    s->n_early = 0;
    s->early_issued = false;
    s->early_bytes = n * 4;
    if (d.any_host) {
        void* const hs[6] = {a->x, a->y, a->z, a->mass, a->id, a->codes};
        const void* const ds[6] = {d.x, d.y, d.z, d.m, d.id, d.codes};
        for (int k = 0; k < 6; ++k) {
            if (d.dev[k] || !d.pinned[k]) continue;
            s->early[s->n_early++] = State::EarlyCopy{hs[k], ds[k]};
            d.dev[k] = true;  // (unmap_arrays skips it)
        }
        if (s->n_early && !s->copy_out) {
            PSG_CHECK(cudaStreamCreateWithFlags(&s->copy_out, cudaStreamNonBlocking));
            PSG_CHECK(cudaEventCreateWithFlags(&s->ev_written, cudaEventDisableTiming));
        }
    }
    r = tick_core(s, d, n, cx, cy, cz, hw, nullptr);
    if (r == PSG_OK) r = unmap_arrays(s, a, d);
    if (s->early_issued) {
        // the early copies are done too when the call returns
        const cudaError_t e = cudaStreamSynchronize(s->copy_out);
        if (e != cudaSuccess && r == PSG_OK) {
            note("cudaStreamSynchronize copy_out", e);
            r = PSG_EDEVICE;
        }
    }
    s->n_early = 0;
    s->early_issued = false;
    return r;
}

// `ticks` iterations of the caller's loop (README.md:65-111) without leaving
// the device: ids reset, prepare, calc with the root derived on the device,
// velocities permuted through ids, semi-implicit Euler.  Host arrays are
// copied in once and out once.
static int run_ticks(State* s, const psg_arrays_t* a, float* vx, float* vy, float* vz, float dt,
                     uint32_t ticks, int variant) {
    const size_t n = a->n;
    if (n > s->max_particles) return PSG_EINVAL;
    if (n == 0 || ticks == 0) return PSG_OK;
    PSG_CHECK(cudaSetDevice(s->device));
    cudaStream_t st = s->stream;
    if (!s->tk_bbox) {
        s->tk_grid = s->sms * 4;
        PSG_ALLOC(s->tk_partial, s->tk_grid * sizeof(float2));
        PSG_ALLOC(s->tk_bbox, 4 * sizeof(float));
        for (int c = 0; c < 3; ++c) PSG_ALLOC(s->tk_v[c], s->max_particles * 4);
        for (int c = 0; c < 3; ++c) PSG_ALLOC(s->tk_vmir[c], s->max_particles * 4);
    }
    DevArrays d;
    int r = map_arrays(s, a, d, false);
    if (r != PSG_OK) return r;
    float* vh[3] = {vx, vy, vz};
    float* vin[3];
    float* vout[3];
    for (int c = 0; c < 3; ++c) {
        if (on_device(vh[c])) {
            vin[c] = vh[c];
        } else {
            vin[c] = s->tk_vmir[c];
            PSG_CHECK(cudaMemcpyAsync(vin[c], vh[c], n * 4, cudaMemcpyHostToDevice, st));
        }
        vout[c] = s->tk_v[c];
    }
    float* const vdst[3] = {vin[0], vin[1], vin[2]};
    const int g = grid_for(s, n, 1024);
    int gp = (int)((n + 1023) / 1024);
    if (gp > s->tk_grid) gp = s->tk_grid;
    for (uint32_t t = 0; t < ticks; ++t) {
        launch_tick_reset_ids(d.id, n, g, st);
        launch_prepare(d.x, d.y, d.z, n, s->tk_partial, gp, d.codes, s->tk_bbox, variant, st);
        r = tick_core(s, d, n, 0.f, 0.f, 0.f, 0.f, s->tk_bbox);
        if (r != PSG_OK) return r;
        TickState ts;
        ts.id = d.id;
        ts.vx_in = vin[0]; ts.vy_in = vin[1]; ts.vz_in = vin[2];
        ts.vx_out = vout[0]; ts.vy_out = vout[1]; ts.vz_out = vout[2];
        ts.x = d.x; ts.y = d.y; ts.z = d.z; ts.m = d.m;
        ts.fx = d.fx; ts.fy = d.fy; ts.fz = d.fz;
        launch_tick_euler(ts, n, dt, g, st);
        PSG_CHECK(cudaGetLastError());
        for (int c = 0; c < 3; ++c) {
            float* tmp = vin[c];
            vin[c] = vout[c];
            vout[c] = tmp;
        }
    }
    for (int c = 0; c < 3; ++c) {
        if (vin[c] != vdst[c])
            PSG_CHECK(cudaMemcpyAsync(vdst[c], vin[c], n * 4, cudaMemcpyDeviceToDevice, st));
        if (vdst[c] != vh[c])
            PSG_CHECK(cudaMemcpyAsync(vh[c], vdst[c], n * 4, cudaMemcpyDeviceToHost, st));
    }
    return unmap_arrays(s, a, d);  // (and all before it)
}

// ---- process-wide workspace of ps_prepare_particles (it takes no context) ----
struct PrepWs {
    std::mutex mu;
    int device = -1;
    cudaStream_t stream = nullptr;
    float2* partial = nullptr;
    float* bbox = nullptr;
    float* h_bbox = nullptr;
    int grid = 0;
    Mirror mir{};
};
static PrepWs g_prep;

static int prepare(const psg_arrays_t* a, float* out_min, float* out_max, float* out_range,
                   int variant) {
    std::lock_guard<std::mutex> lock(g_prep.mu);
    int dev = 0;
    PSG_CHECK(cudaGetDevice(&dev));
    if (g_prep.device != dev) {
        if (g_prep.stream) {
            cudaSetDevice(g_prep.device);
            cudaStreamDestroy(g_prep.stream);
            cudaFree(g_prep.partial);
            cudaFree(g_prep.bbox);
            cudaFreeHost(g_prep.h_bbox);
            free_mirror(g_prep.mir);
            cudaSetDevice(dev);
        }
        int sms = 0;
        PSG_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        PSG_CHECK(cudaStreamCreateWithFlags(&g_prep.stream, cudaStreamNonBlocking));
        g_prep.grid = sms * 4;
        PSG_ALLOC(g_prep.partial, g_prep.grid * sizeof(float2));
        PSG_ALLOC(g_prep.bbox, 4 * sizeof(float));
        PSG_CHECK(cudaMallocHost((void**)&g_prep.h_bbox, 4 * sizeof(float)));
        g_prep.device = dev;
    }
    const size_t n = a->n;
    cudaStream_t st = g_prep.stream;
    const float* x = a->x; const float* y = a->y; const float* z = a->z;
    uint32_t* codes = a->codes;
    Mirror& mi = g_prep.mir;
    const void* const hs[3] = {x, y, z};
    const Place at[4] = {place_of(x), place_of(y), place_of(z), place_of(codes)};
    const bool dc = at[3] == DEVICE;
    // (pageable arrays of a small call: as in map_arrays)
    const bool staged = n <= kStageMax && at[0] == PAGEABLE && at[1] == PAGEABLE &&
                        at[2] == PAGEABLE && at[3] == PAGEABLE;
    if (!(at[0] == DEVICE && at[1] == DEVICE && at[2] == DEVICE && dc)) {
        int r = ensure_mirror(mi, n);
        if (r == PSG_OK && staged) r = ensure_stage(mi, n);
        if (r != PSG_OK) return r;
        float* const rows[3] = {mi.x, mi.y, mi.z};
        if (staged) {
            for (int i = 0; i < 3; ++i) std::memcpy(mi.stage + (size_t)i * n, hs[i], n * 4);
            PSG_CHECK(cudaMemcpy2DAsync(mi.x, mi.cap * 4, mi.stage, n * 4, n * 4, 3,
                                        cudaMemcpyHostToDevice, st));
        } else {
            for (int i = 0; i < 3; ++i)
                if (at[i] != DEVICE)
                    PSG_CHECK(cudaMemcpyAsync(rows[i], hs[i], n * 4, cudaMemcpyHostToDevice, st));
        }
        if (at[0] != DEVICE) x = mi.x;
        if (at[1] != DEVICE) y = mi.y;
        if (at[2] != DEVICE) z = mi.z;
        if (!dc) codes = mi.codes;
    }
    int grid = (int)((n + 1023) / 1024);
    if (grid > g_prep.grid) grid = g_prep.grid;
    if (grid < 1) grid = 1;
    launch_prepare(x, y, z, n, g_prep.partial, grid, codes, g_prep.bbox, variant, st);
    PSG_CHECK(cudaGetLastError());
    if (!dc)
        PSG_CHECK(cudaMemcpyAsync(staged ? mi.stage : a->codes, codes, n * 4,
                                  cudaMemcpyDeviceToHost, st));
    PSG_CHECK(cudaMemcpyAsync(g_prep.h_bbox, g_prep.bbox, 4 * sizeof(float), cudaMemcpyDeviceToHost, st));
    PSG_CHECK(cudaStreamSynchronize(st));
    if (staged) std::memcpy(a->codes, mi.stage, n * 4);
    if (out_min) *out_min = g_prep.h_bbox[0];
    if (out_max) *out_max = g_prep.h_bbox[1];
    if (out_range) *out_range = g_prep.h_bbox[2];
    return PSG_OK;
}

// ---- batched ensemble: many independent systems in one tree pass ----------
//
// All systems share one set of device buffers: their particles are the
// caller's concatenated arrays (system k at [off_k, off_k + N_k)), and every
// phase of the tick is one launch over all of them -- the segmented bounding
// box and Morton codes, the radix sort (four code passes, then stable passes
// on the system index, so each system ends sorted within its range), the
// tree build (a system's first position starts its root, node k of level 0;
// no run crosses a system boundary), the upward pass, and the persistent
// traversal kernels, whose work queues run over the groups of every system
// with each group's own theta, root, leaf-pass variant, split depth and
// shallow-leaf depth.  Per system the arithmetic is exactly that of its own
// tick, so the results equal each system's ps_b200_run_ticks bit for bit.
// One tick is two CUDA graphs captured once and replayed (forces; velocity
// permutation + Euler); between them the host reads the one status block and
// regrows a store that ran out (then that traversal is rerun and the graphs
// are captured again).

constexpr uint32_t kEnsMagic = 0x50534745u;  // "PSGE"
constexpr uint32_t kForestBlock = 1024;      // particles per prepare block

struct Ensemble {
    uint32_t magic = 0;
    int device = 0;
    size_t nsys = 0, total = 0;
    std::vector<size_t> count, offset;
    std::vector<float> theta;       // per system
    std::vector<uint32_t> cap;      // leaf capacity per system
    State* fs = nullptr;            // the device state of all systems together
    // per-system tables (device)
    uint32_t* part_sys = nullptr;   // system of each particle position
    uint32_t* sys_off = nullptr;    // [nsys + 1]
    uint32_t* sys_cap = nullptr;
    float* sys_theta2 = nullptr;
    int32_t* sys_heavy = nullptr;
    int32_t* sys_split = nullptr;
    float* sys_bbox = nullptr;      // [nsys][4]
    uint32_t* sys_maxleaf = nullptr;
    uint32_t* sys_sort_hist = nullptr;  // digit counts of the system sort passes
    int sys_passes = 1;
    uint4* blk = nullptr;           // prepare blocks: (system, first, end)
    uint32_t* sys_blk = nullptr;    // [nsys + 1]
    float2* partial = nullptr;
    int nblk = 0;
    float* vtmp = nullptr;          // 3 x total velocity scratch
    cudaGraphExec_t g_force = nullptr, g_step = nullptr;
    bool dirty = true;
    DevArrays cap_arr{};            // arrays the graphs were captured with
    float* cap_v[3] = {nullptr, nullptr, nullptr};
    float cap_dt = 0.f;
    double grid_scale = 1.0;
    int variant = PSG_MORTON_AVX2;
    std::vector<uint32_t> leaf_ladder{1u, 16u, 32u, 64u};  // leaf capacities the autotuner tries
    int order = 0;                     // local expansion: 0 the reference's, 1 order-1
    std::vector<int> order_ladder{0, 1};  // expansion orders the autotuner tries
};

static DevArrays slice(const DevArrays& a, size_t off) {
    DevArrays d = a;
    d.x += off; d.y += off; d.z += off; d.m += off;
    d.fx += off; d.fy += off; d.fz += off; d.id += off; d.codes += off;
    return d;
}

static int ensure_tick_scratch(State* s) {
    if (s->tk_bbox) return PSG_OK;
    s->tk_grid = s->sms * 4;
    PSG_ALLOC(s->tk_partial, s->tk_grid * sizeof(float2));
    PSG_ALLOC(s->tk_bbox, 4 * sizeof(float));
    for (int c = 0; c < 3; ++c) PSG_ALLOC(s->tk_v[c], s->max_particles * 4);
    for (int c = 0; c < 3; ++c) PSG_ALLOC(s->tk_vmir[c], s->max_particles * 4);
    return PSG_OK;
}

// the local expansion of a state's traversal: 0 the reference's order 0,
// 1 the order-1 expansion (closure mode 1: its field gradients per node)
static int set_order(State* s, int order) {
    if (order >= 1) {
        const int r = closure_alloc(s);
        if (r != PSG_OK) return r;
    }
    s->cl.mode = order >= 1 ? 1 : 0;
    s->order = order >= 1 ? 1 : 0;
    reset_near_levels(s);
    return PSG_OK;
}

// theta, theta^2 (rounded as the MAC rounds it), shallow-leaf depth and leaf
// capacity of every system to the device tables
static int upload_systems(Ensemble* e) {
    std::vector<float> th2(e->nsys);
    std::vector<int32_t> hv(e->nsys), sp(e->nsys);
    int hmax = 0, smax = 0;
    int caps = 0;
    for (size_t k = 0; k < e->nsys; ++k) {
        const float t = e->theta[k];
        th2[k] = t * t;
        hv[k] = heavy_depth_of(t, e->count[k]);
        hmax = std::max(hmax, (int)hv[k]);
        caps |= e->cap[k] >= kDenseCap ? 2 : 1;
        sp[k] = split_depth_of(t, e->count[k], e->cap[k]);
        smax = std::max(smax, (int)sp[k]);
    }
    const SplitStore before = e->fs->split;  // (allocated here: not while capturing)
    if (!ensure_split(e->fs, smax)) {
        std::fill(sp.begin(), sp.end(), 0);
        smax = 0;
    }
    if (before.sums != e->fs->split.sums || before.cap != e->fs->split.cap) e->dirty = true;
    PSG_CHECK(cudaMemcpy(e->sys_theta2, th2.data(), e->nsys * 4, cudaMemcpyHostToDevice));
    PSG_CHECK(cudaMemcpy(e->sys_heavy, hv.data(), e->nsys * 4, cudaMemcpyHostToDevice));
    PSG_CHECK(cudaMemcpy(e->sys_split, sp.data(), e->nsys * 4, cudaMemcpyHostToDevice));
    PSG_CHECK(cudaMemcpy(e->sys_cap, e->cap.data(), e->nsys * 4, cudaMemcpyHostToDevice));
    if (hmax != e->fs->forest_heavy) e->dirty = true;  // a launch parameter changes
    e->fs->forest_heavy = hmax;
    if (smax != e->fs->forest_split || caps != e->fs->forest_caps) e->dirty = true;
    e->fs->forest_caps = caps;
    e->fs->forest_split = smax;
    // the stores' near-list depth and P2P mode start over with the settings
    // (both are launch parameters of the captured graphs)
    if (e->fs->ns_levels != kMaxDepth || e->fs->stream_p2p || e->fs->level_by_level)
        e->dirty = true;
    reset_near_levels(e->fs);
    return PSG_OK;
}

static void drop_graphs(Ensemble* e) {
    if (e->g_force) cudaGraphExecDestroy(e->g_force);
    if (e->g_step) cudaGraphExecDestroy(e->g_step);
    e->g_force = e->g_step = nullptr;
    e->dirty = true;
}

// one tick's forces of all systems, enqueued on the forest stream without
// any host synchronisation (capturable)
static int enqueue_forest_forces(Ensemble* e, const DevArrays& d) {
    State* s = e->fs;
    cudaStream_t st = s->stream;
    const size_t n = e->total;
    const int g = grid_for(s, n, 1024);
    launch_forest_reset_ids(d.id, n, e->part_sys, e->sys_off, g, st);
    launch_prepare_forest(d.x, d.y, d.z, e->blk, e->nblk, e->sys_blk, e->sys_off, e->partial,
                          d.codes, e->sys_bbox, e->variant, st);
    PSG_CHECK(cudaMemsetAsync(s->d_status, 0, sizeof(Status), st));
    PSG_CHECK(cudaMemsetAsync(e->sys_maxleaf, 0, e->nsys * 4, st));
    launch_sort_forest(s->sort, d.codes, n, g, s->d_status, st, e->part_sys, e->sys_passes,
                       e->sys_sort_hist);
    launch_gather(s->sort.perm, d.x, d.y, d.z, d.m, d.id, n, s->xyzm, s->ids, g, st);
    launch_writeback(s->xyzm, s->ids, n, d.x, d.y, d.z, d.m, d.id, g, st);
    const int gt = (int)((s->tv.lvl_base[kLevels] + 255) / 256);
    launch_tree(d.codes, n, s->tree_tiles, s->tv, s->d_status, 0.f, 0.f, 0.f, 0.f, gt, st,
                nullptr, 1);
    launch_upward(s->tv, s->d_status, s->xyzm, n, st);
    s->trav_fresh = true;
    s->trav_n = n;
    int r = enqueue_traversal(s, s->xyzm, d.fx, d.fy, d.fz);
    if (r != PSG_OK) return r;
    launch_forest_single_forces(e->sys_off, (uint32_t)e->nsys, d.fx, d.fy, d.fz, st);
    PSG_CHECK(cudaMemcpyAsync(s->h_status, s->d_status, sizeof(Status), cudaMemcpyDeviceToHost,
                              st));
    return PSG_OK;
}

// every system's velocity permutation through its ids + semi-implicit Euler
static int enqueue_forest_step(Ensemble* e, const DevArrays& d, float* const v[3], float dt) {
    State* s = e->fs;
    cudaStream_t st = s->stream;
    const size_t n = e->total;
    TickState ts;
    ts.id = d.id;
    ts.vx_in = v[0]; ts.vy_in = v[1]; ts.vz_in = v[2];
    ts.vx_out = e->vtmp; ts.vy_out = e->vtmp + n; ts.vz_out = e->vtmp + 2 * n;
    ts.x = d.x; ts.y = d.y; ts.z = d.z; ts.m = d.m;
    ts.fx = d.fx; ts.fy = d.fy; ts.fz = d.fz;
    launch_forest_euler(ts, n, dt, e->part_sys, e->sys_off, grid_for(s, n, 1024), st);
    for (int c = 0; c < 3; ++c)
        PSG_CHECK(cudaMemcpyAsync(v[c], e->vtmp + c * n, n * 4, cudaMemcpyDeviceToDevice, st));
    return PSG_OK;
}

static int capture(Ensemble* e, bool forces, const DevArrays& a, float* const v[3], float dt,
                   cudaGraphExec_t* out) {
    cudaStream_t st = e->fs->stream;
    PSG_CHECK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    int r = forces ? enqueue_forest_forces(e, a) : enqueue_forest_step(e, a, v, dt);
    cudaGraph_t graph = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(st, &graph);
    if (r == PSG_OK && ce != cudaSuccess) {
        note("cudaStreamEndCapture", ce);
        r = PSG_EDEVICE;
    }
    if (r == PSG_OK) {
        const cudaError_t ie = cudaGraphInstantiate(out, graph, 0ull);
        if (ie != cudaSuccess) {
            note("cudaGraphInstantiate", ie);
            r = PSG_EDEVICE;
        }
    }
    if (graph) cudaGraphDestroy(graph);
    return r;
}

static int ensure_graphs(Ensemble* e, const DevArrays& a, float* const v[3], float dt) {
    const bool same = !e->dirty && std::memcmp(&e->cap_arr, &a, sizeof(DevArrays)) == 0 &&
                      e->cap_v[0] == v[0] && e->cap_v[1] == v[1] && e->cap_v[2] == v[2] &&
                      e->cap_dt == dt;
    if (same) return PSG_OK;
    drop_graphs(e);
    e->fs->grid_scale = e->grid_scale;
    int r = capture(e, true, a, v, dt, &e->g_force);
    if (r == PSG_OK) r = capture(e, false, a, v, dt, &e->g_step);
    if (r != PSG_OK) {
        drop_graphs(e);
        return r;
    }
    e->cap_arr = a;
    for (int c = 0; c < 3; ++c) e->cap_v[c] = v[c];
    e->cap_dt = dt;
    e->dirty = false;
    return PSG_OK;
}

// after a forces replay: fatal status -> error; capacity bits -> regrow and
// rerun the traversal, and capture again before the next tick
static int check_forest(Ensemble* e, const DevArrays& a) {
    State* s = e->fs;
    const uint32_t err = s->h_status->err;
    if (err & PSG_ERR_FATAL) {
        std::snprintf(g_err, sizeof(g_err), "ensemble: device status 0x%x", err);
        return (err & PSG_ERR_NODES) ? PSG_EINVAL : PSG_EDEVICE;
    }
    if (err & (PSG_ERR_NS_OVERFLOW | PSG_ERR_P2P_OVERFLOW | PSG_ERR_DENSE_OVERFLOW |
               PSG_ERR_HEAVY_OVERFLOW)) {
        e->dirty = true;  // (the captured graphs hold the stores' old addresses)
        int r = regrow(s, err);
        if (r != PSG_OK) return r;
        PSG_CHECK(cudaMemsetAsync(&s->d_status->err, 0, 4, s->stream));
        uint32_t err2 = 0;
        r = run_traversal(s, s->xyzm, a.fx, a.fy, a.fz, &err2);
        if (r != PSG_OK) return r;
        if (err2 & PSG_ERR_FATAL) {
            std::snprintf(g_err, sizeof(g_err), "ensemble: device status 0x%x", err2);
            return PSG_EDEVICE;
        }
    }
    return PSG_OK;
}

static int ens_map(Ensemble* e, const psg_arrays_t* a, DevArrays& d) {
    if (a->n != e->total) {
        std::snprintf(g_err, sizeof(g_err), "ensemble: %zu particles given, %zu expected", a->n,
                      e->total);
        return PSG_EINVAL;
    }
    d.x = a->x; d.y = a->y; d.z = a->z; d.m = a->mass;
    d.fx = a->fx; d.fy = a->fy; d.fz = a->fz; d.id = a->id; d.codes = a->codes;
    void* ps[9] = {d.x, d.y, d.z, d.m, d.fx, d.fy, d.fz, d.id, d.codes};
    for (void* p : ps) {
        if (!on_device(p)) {
            std::snprintf(g_err, sizeof(g_err), "ensemble arrays must be device memory");
            return PSG_EINVAL;
        }
    }
    d.any_host = false;
    return PSG_OK;
}

static void free_ensemble(Ensemble* e) {
    if (e->fs && e->fs->stream) cudaStreamSynchronize(e->fs->stream);
    drop_graphs(e);
    if (e->fs) {
        if (e->fs->magic == kMagic) free_state(e->fs);
        delete e->fs;
        e->fs = nullptr;
    }
    void* ps[] = {e->part_sys, e->sys_off, e->sys_cap, e->sys_theta2, e->sys_heavy,
                  e->sys_split, e->sys_bbox, e->sys_maxleaf, e->sys_sort_hist, e->blk, e->sys_blk,
                  e->partial, e->vtmp};
    for (void* p : ps)
        if (p) cudaFree(p);
    e->magic = 0;
}

static int ens_create(Ensemble* e, const size_t* counts, size_t nsys, const float* theta) {
    PSG_CHECK(cudaGetDevice(&e->device));
    e->nsys = nsys;
    e->count.assign(counts, counts + nsys);
    e->offset.resize(nsys);
    size_t off = 0;
    for (size_t k = 0; k < nsys; ++k) {
        e->offset[k] = off;
        off += counts[k];
    }
    e->total = off;
    if (off >= 0xFFFFFFF0ull || nsys > 65536) {
        std::snprintf(g_err, sizeof(g_err), "ensemble: at most 65,536 systems and 2^32 particles");
        return PSG_EINVAL;
    }
    e->theta.resize(nsys);
    for (size_t k = 0; k < nsys; ++k) e->theta[k] = theta && theta[k] > 0.f ? theta[k] : 2.0f;
    e->cap.assign(nsys, 1u);
    // level capacities: the sum over systems of min(8^d, N_k); level 0 holds
    // the roots
    uint32_t caps[kLevels];
    for (int d = 0; d <= kMaxDepth; ++d) {
        unsigned long long c = 0;
        for (size_t k = 0; k < nsys; ++k)
            c += d == 0 ? 1ull : std::min<unsigned long long>(1ull << (3 * d), counts[k]);
        if (c >= 0xFFFFFFF0ull) return PSG_EINVAL;
        caps[d] = (uint32_t)c;
    }
    e->sys_passes = nsys > 256 ? 2 : 1;
    e->fs = new (std::nothrow) State;
    if (!e->fs) return PSG_EALLOC;
    int r = init_state(e->fs, e->total, 2.0f, caps, 4 + e->sys_passes);
    if (r != PSG_OK) return r;
    r = ensure_tick_scratch(e->fs);
    if (r != PSG_OK) return r;
    // the shallow-leaf walk serves the shallow groups of every system: more
    // blocks, each frontier sized for the largest system
    {
        size_t maxn = 1;
        for (size_t k = 0; k < nsys; ++k) maxn = std::max(maxn, counts[k]);
        e->fs->heavy_slots = e->fs->sms * 2;
        r = alloc_heavy(e->fs, (uint32_t)(maxn / 4 + 4096));
        if (r != PSG_OK) return r;
    }
    // per-system tables
    std::vector<uint32_t> psys(e->total), soff(nsys + 1), sblk(nsys + 1);
    std::vector<uint4> blk;
    for (size_t k = 0; k < nsys; ++k) {
        soff[k] = (uint32_t)e->offset[k];
        sblk[k] = (uint32_t)blk.size();
        for (size_t i = 0; i < counts[k]; ++i) psys[e->offset[k] + i] = (uint32_t)k;
        for (size_t b = 0; b < counts[k]; b += kForestBlock)
            blk.push_back(make_uint4((uint32_t)k, (uint32_t)(e->offset[k] + b),
                                     (uint32_t)(e->offset[k] + std::min<size_t>(b + kForestBlock,
                                                                               counts[k])),
                                     0u));
    }
    soff[nsys] = (uint32_t)e->total;
    sblk[nsys] = (uint32_t)blk.size();
    e->nblk = (int)blk.size();
    // digit counts of the system passes, from the system sizes
    std::vector<uint32_t> so(256 * e->sys_passes, 0u);
    for (int q = 0; q < e->sys_passes; ++q)
        for (size_t k = 0; k < nsys; ++k)
            so[256 * q + ((k >> (8 * q)) & 0xFFu)] += (uint32_t)counts[k];
    PSG_ALLOC(e->part_sys, e->total * 4);
    PSG_ALLOC(e->sys_off, (nsys + 1) * 4);
    PSG_ALLOC(e->sys_cap, nsys * 4);
    PSG_ALLOC(e->sys_theta2, nsys * 4);
    PSG_ALLOC(e->sys_heavy, nsys * 4);
    PSG_ALLOC(e->sys_split, nsys * 4);
    PSG_ALLOC(e->sys_bbox, nsys * 16);
    PSG_ALLOC(e->sys_maxleaf, nsys * 4);
    PSG_ALLOC(e->sys_sort_hist, so.size() * 4);
    PSG_ALLOC(e->blk, blk.size() * sizeof(uint4));
    PSG_ALLOC(e->sys_blk, (nsys + 1) * 4);
    PSG_ALLOC(e->partial, blk.size() * sizeof(float2));
    PSG_ALLOC(e->vtmp, 3 * e->total * sizeof(float));
    PSG_CHECK(cudaMemcpy(e->part_sys, psys.data(), e->total * 4, cudaMemcpyHostToDevice));
    PSG_CHECK(cudaMemcpy(e->sys_off, soff.data(), (nsys + 1) * 4, cudaMemcpyHostToDevice));
    PSG_CHECK(cudaMemcpy(e->sys_sort_hist, so.data(), so.size() * 4, cudaMemcpyHostToDevice));
    PSG_CHECK(cudaMemcpy(e->blk, blk.data(), blk.size() * sizeof(uint4), cudaMemcpyHostToDevice));
    PSG_CHECK(cudaMemcpy(e->sys_blk, sblk.data(), (nsys + 1) * 4, cudaMemcpyHostToDevice));
    TreeView& tv = e->fs->tv;
    tv.part_sys = e->part_sys;
    tv.sys_off = e->sys_off;
    tv.sys_cap = e->sys_cap;
    tv.sys_bbox = e->sys_bbox;
    tv.sys_theta2 = e->sys_theta2;
    e->fs->sys_heavy = e->sys_heavy;
    e->fs->sys_split = e->sys_split;
    tv.sys_maxleaf = e->sys_maxleaf;
    tv.nsys = (uint32_t)nsys;
    r = upload_systems(e);
    if (r != PSG_OK) return r;
    e->magic = kEnsMagic;
    return PSG_OK;
}

static int ens_run(Ensemble* e, const psg_arrays_t* a, float* const v[3], float dt,
                   uint32_t ticks) {
    DevArrays d{};
    int r = ens_map(e, a, d);
    if (r != PSG_OK) return r;
    for (int c = 0; c < 3; ++c) {
        if (!on_device(v[c])) {
            std::snprintf(g_err, sizeof(g_err), "ensemble velocities must be device memory");
            return PSG_EINVAL;
        }
    }
    PSG_CHECK(cudaSetDevice(e->device));
    cudaStream_t st = e->fs->stream;
    for (uint32_t t = 0; t < ticks; ++t) {
        r = ensure_graphs(e, d, v, dt);
        if (r != PSG_OK) return r;
        PSG_CHECK(cudaGraphLaunch(e->g_force, st));
        PSG_CHECK(cudaStreamSynchronize(st));
        r = check_forest(e, d);
        if (r != PSG_OK) return r;
        PSG_CHECK(cudaGraphLaunch(e->g_step, st));
    }
    PSG_CHECK(cudaStreamSynchronize(st));
    return PSG_OK;
}

// Autotuner.  Per size class (the systems with the same floor(log2 N)) and
// per leaf capacity of its ladder: the smallest theta of {1, 1.5, 2, 3, 4, 6,
// 8} whose median relative force error against an FP64 direct sum on up to
// 1024 particles of the class's first system is at most `target` (a tick of
// that system alone).  Then, class by class from the one holding the most
// particles: the leaf capacity (with its theta) whose whole-ensemble forces
// replay is fastest, among those that met the target.  Last, the traversal
// grids' scale among {1, 1/2, 1/4} by the same replay time.  Works on copies;
// the caller's arrays are left as they are.
static int ens_autotune(Ensemble* e, const psg_arrays_t* a, float target, float* theta_out,
                        double* scale_out) {
    DevArrays d{};
    int r = ens_map(e, a, d);
    if (r != PSG_OK) return r;
    PSG_CHECK(cudaSetDevice(e->device));
    cudaStream_t st = e->fs->stream;
    const size_t T = e->total;
    float* buf = nullptr;  // scratch copy: x y z m fx fy fz (7 T floats), id, codes
    PSG_ALLOC(buf, (size_t)9 * T * 4 + 16);
    DevArrays c{};
    c.x = buf; c.y = buf + T; c.z = buf + 2 * T; c.m = buf + 3 * T;
    c.fx = buf + 4 * T; c.fy = buf + 5 * T; c.fz = buf + 6 * T;
    c.id = (uint32_t*)(buf + 7 * T); c.codes = (uint32_t*)(buf + 8 * T);
    c.any_host = false;
    auto restore = [&]() -> int {
        PSG_CHECK(cudaMemcpyAsync(c.x, d.x, T * 4, cudaMemcpyDeviceToDevice, st));
        PSG_CHECK(cudaMemcpyAsync(c.y, d.y, T * 4, cudaMemcpyDeviceToDevice, st));
        PSG_CHECK(cudaMemcpyAsync(c.z, d.z, T * 4, cudaMemcpyDeviceToDevice, st));
        PSG_CHECK(cudaMemcpyAsync(c.m, d.m, T * 4, cudaMemcpyDeviceToDevice, st));
        PSG_CHECK(cudaStreamSynchronize(st));
        return PSG_OK;
    };
    static const float ladder[] = {1.0f, 1.5f, 2.0f, 3.0f, 4.0f, 6.0f, 8.0f};
    const int nl = (int)(sizeof(ladder) / sizeof(ladder[0]));
    std::vector<int> cls(e->nsys);
    for (size_t k = 0; k < e->nsys; ++k)
        cls[k] = (int)std::floor(std::log2((double)e->count[k] + 1));
    std::vector<int> classes;  // distinct classes, by the particles they hold (most first)
    std::vector<size_t> rep;   // the first system of each class
    {
        std::vector<std::pair<unsigned long long, int>> held;
        for (size_t k = 0; k < e->nsys; ++k) {
            auto it = std::find(classes.begin(), classes.end(), cls[k]);
            if (it == classes.end()) {
                classes.push_back(cls[k]);
                rep.push_back(k);
                held.push_back({0ull, (int)classes.size() - 1});
                it = classes.end() - 1;
            }
            held[it - classes.begin()].first += e->count[k];
        }
        std::sort(held.begin(), held.end(), [](auto& x, auto& y) { return x.first > y.first; });
        std::vector<int> c2;
        std::vector<size_t> r2;
        for (auto& h : held) {
            c2.push_back(classes[h.second]);
            r2.push_back(rep[h.second]);
        }
        classes = c2;
        rep = r2;
    }
    const size_t ncls = classes.size(), nlc = e->leaf_ladder.size();
    const size_t nor = e->order_ladder.size();
    std::vector<std::vector<std::vector<float>>> thx(
        nor, std::vector<std::vector<float>>(nlc, std::vector<float>(ncls, ladder[nl - 1])));
    std::vector<std::vector<std::vector<bool>>> metx(
        nor, std::vector<std::vector<bool>>(nlc, std::vector<bool>(ncls, false)));
    const size_t kSample = 1024;
    uint32_t* d_tg = nullptr;
    double* d_f64 = nullptr;
    PSG_ALLOC(d_tg, kSample * 4);
    PSG_ALLOC(d_f64, kSample * 3 * sizeof(double));
    size_t maxn = 1;
    for (size_t k = 0; k < e->nsys; ++k) maxn = std::max(maxn, e->count[k]);
    const int dsms = e->fs->sms * 8;
    const size_t part_n = direct_f64_part_doubles(maxn, kSample, dsms);
    double* d_part = nullptr;
    PSG_ALLOC(d_part, part_n * sizeof(double));
    std::vector<uint32_t> tg(kSample);
    std::vector<double> f64(kSample * 3);
    // theta per (leaf capacity, class): ticks of the class's first system alone
    for (size_t ci = 0; ci < ncls && r == PSG_OK; ++ci) {
        const size_t k = rep[ci], n = e->count[k];
        State* s = new (std::nothrow) State;
        if (!s) { r = PSG_EALLOC; break; }
        r = init_state(s, n, 2.0f);
        if (r == PSG_OK) r = ensure_tick_scratch(s);
        const DevArrays ck = slice(c, e->offset[k]);
        for (size_t oi = 0; oi < nor && r == PSG_OK; ++oi)
        for (size_t li = 0; li < nlc && r == PSG_OK; ++li) {
            if ((r = set_order(s, e->order_ladder[oi])) != PSG_OK) break;
            auto& th = thx[oi];
            auto& met = metx[oi];
            s->leaf_cap = e->leaf_ladder[li];
            for (int ti = 0; ti < nl && r == PSG_OK; ++ti) {
                s->theta = ladder[ti];
                reset_near_levels(s);
                if ((r = restore()) != PSG_OK) break;
                launch_tick_reset_ids(ck.id, n, grid_for(s, n, 1024), s->stream);
                int gp = (int)((n + 1023) / 1024);
                if (gp > s->tk_grid) gp = s->tk_grid;
                launch_prepare(ck.x, ck.y, ck.z, n, s->tk_partial, gp, ck.codes, s->tk_bbox,
                               e->variant, s->stream);
                if ((r = tick_core(s, ck, n, 0.f, 0.f, 0.f, 0.f, s->tk_bbox)) != PSG_OK) break;
                const size_t ns = n < kSample ? n : kSample;
                for (size_t i = 0; i < ns; ++i) tg[i] = (uint32_t)(i * n / ns);
                PSG_CHECK(cudaMemcpyAsync(d_tg, tg.data(), ns * 4, cudaMemcpyHostToDevice,
                                          s->stream));
                launch_direct_f64(s->xyzm, n, d_tg, ns, d_f64, dsms, s->stream, d_part, part_n);
                PSG_CHECK(cudaMemcpyAsync(f64.data(), d_f64, ns * 3 * sizeof(double),
                                          cudaMemcpyDeviceToHost, s->stream));
                std::vector<float> hf[3] = {std::vector<float>(n), std::vector<float>(n),
                                            std::vector<float>(n)};
                PSG_CHECK(cudaMemcpyAsync(hf[0].data(), ck.fx, n * 4, cudaMemcpyDeviceToHost,
                                          s->stream));
                PSG_CHECK(cudaMemcpyAsync(hf[1].data(), ck.fy, n * 4, cudaMemcpyDeviceToHost,
                                          s->stream));
                PSG_CHECK(cudaMemcpyAsync(hf[2].data(), ck.fz, n * 4, cudaMemcpyDeviceToHost,
                                          s->stream));
                PSG_CHECK(cudaStreamSynchronize(s->stream));
                std::vector<double> rel(ns);
                for (size_t i = 0; i < ns; ++i) {
                    const double gx = f64[3 * i], gy = f64[3 * i + 1], gz = f64[3 * i + 2];
                    const double ex = hf[0][tg[i]] - gx, ey = hf[1][tg[i]] - gy,
                                 ez = hf[2][tg[i]] - gz;
                    const double nr = std::sqrt(gx * gx + gy * gy + gz * gz);
                    rel[i] = nr > 0 ? std::sqrt(ex * ex + ey * ey + ez * ez) / nr : 0.0;
                }
                std::nth_element(rel.begin(), rel.begin() + ns / 2, rel.end());
                if (rel[ns / 2] <= (double)target) {
                    th[li][ci] = ladder[ti];
                    met[li][ci] = true;
                    break;
                }
            }
        }
        if (s->magic == kMagic) free_state(s);
        delete s;
    }
    cudaFree(d_tg);
    cudaFree(d_f64);
    cudaFree(d_part);
    // one forces replay of the copies with the current settings: its time
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    PSG_CHECK(cudaEventCreate(&t0));
    PSG_CHECK(cudaEventCreate(&t1));
    float* vdummy[3] = {c.fx, c.fy, c.fz};
    auto replay = [&](float* ms) -> int {
        int rr = PSG_OK;
        for (int rep2 = 0; rep2 < 2 && rr == PSG_OK; ++rep2) {  // the first grows stores
            if ((rr = restore()) != PSG_OK) break;
            if ((rr = ensure_graphs(e, c, vdummy, 0.f)) != PSG_OK) break;
            PSG_CHECK(cudaEventRecord(t0, st));
            PSG_CHECK(cudaGraphLaunch(e->g_force, st));
            PSG_CHECK(cudaEventRecord(t1, st));
            PSG_CHECK(cudaStreamSynchronize(st));
            if ((rr = check_forest(e, c)) != PSG_OK) break;
            cudaEventElapsedTime(ms, t0, t1);
        }
        return rr;
    };
    // per expansion order: the class-by-class descent below, then the order
    // whose final replay is fastest
    size_t oi = 0;
    auto set_class = [&](size_t ci, size_t li) {
        for (size_t k = 0; k < e->nsys; ++k) {
            if (cls[k] != classes[ci]) continue;
            e->cap[k] = e->leaf_ladder[li];
            e->theta[k] = thx[oi][li][ci];
        }
    };
    std::vector<std::vector<size_t>> picks(nor, std::vector<size_t>(ncls, 0));
    std::vector<double> order_ms(nor, 1e300);
    for (oi = 0; oi < nor && r == PSG_OK; ++oi) {
        const auto& met = metx[oi];
        auto& pick = picks[oi];
        e->order = e->order_ladder[oi];
        if ((r = set_order(e->fs, e->order)) != PSG_OK) break;
        e->dirty = true;
        // start from each class's first leaf capacity that met the target
        for (size_t ci = 0; ci < ncls; ++ci)
            for (size_t li = 0; li < nlc; ++li)
                if (met[li][ci]) {
                    pick[ci] = li;
                    break;
                }
        for (size_t ci = 0; ci < ncls; ++ci) set_class(ci, pick[ci]);
        if ((r = upload_systems(e)) != PSG_OK) break;
        // then class by class the fastest whole replay
        double best = 1e300;
        for (size_t ci = 0; ci < ncls && r == PSG_OK; ++ci) {
            best = 1e300;
            size_t best_li = pick[ci];
            for (size_t li = 0; li < nlc && r == PSG_OK; ++li) {
                if (nlc > 1 && !met[li][ci] && met[pick[ci]][ci]) continue;
                if (nlc == 1 && li != pick[ci]) continue;
                set_class(ci, li);
                if ((r = upload_systems(e)) != PSG_OK) break;
                e->dirty = true;
                float ms = 0.f;
                if ((r = replay(&ms)) != PSG_OK) break;
                if (ms < best) {
                    best = ms;
                    best_li = li;
                }
            }
            pick[ci] = best_li;
            set_class(ci, best_li);
            if (r == PSG_OK) r = upload_systems(e);
        }
        order_ms[oi] = best;
    }
    if (r == PSG_OK) {
        oi = (size_t)(std::min_element(order_ms.begin(), order_ms.end()) - order_ms.begin());
        e->order = e->order_ladder[oi];
        r = set_order(e->fs, e->order);
        for (size_t ci = 0; ci < ncls; ++ci) set_class(ci, picks[oi][ci]);
        if (r == PSG_OK) r = upload_systems(e);
        e->dirty = true;
    }
    // launch shape: the traversal grids' scale
    if (r == PSG_OK) {
        static const double scales[] = {1.0, 0.5, 0.25};
        double best = 1e300, best_scale = 1.0;
        for (double sc : scales) {
            e->grid_scale = sc;
            e->dirty = true;
            float ms = 0.f;
            if ((r = replay(&ms)) != PSG_OK) break;
            if (ms < best) {
                best = ms;
                best_scale = sc;
            }
        }
        e->grid_scale = best_scale;
        drop_graphs(e);
        if (scale_out) *scale_out = best_scale;
        if (theta_out)
            for (size_t k = 0; k < e->nsys; ++k) theta_out[k] = e->theta[k];
    }
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    cudaFree(buf);
    return r;
}

}  // namespace psg

using psg::State;


extern "C" {

size_t psg_state_bytes(void) { return (sizeof(State) + 63) & ~(size_t)63; }

int psg_init(void* mem, size_t max_particles, float theta) {
    State* s = static_cast<State*>(mem);
    int r = psg::init_state(s, max_particles, theta);
    if (r != PSG_OK) psg::free_state(s);
    return r;
}

int psg_destroy(void* mem) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic) return PSG_EINVAL;
    cudaSetDevice(s->device);
    cudaStreamSynchronize(s->stream);
    psg::free_state(s);
    return PSG_OK;
}

int psg_prepare(const psg_arrays_t* a, float* out_min, float* out_max, float* out_range,
                int variant) {
    return psg::prepare(a, out_min, out_max, out_range, variant);
}

int psg_calc(void* mem, const psg_arrays_t* a, float cx, float cy, float cz, float hw) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic) return PSG_EINVAL;
    return psg::calc(s, a, cx, cy, cz, hw);
}

int psg_run_ticks(void* mem, const psg_arrays_t* a, float* vx, float* vy, float* vz, float dt,
                  uint32_t ticks, int variant) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic) return PSG_EINVAL;
    return psg::run_ticks(s, a, vx, vy, vz, dt, ticks, variant);
}

int psg_set_option(void* mem, int key, double value) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic) return PSG_EINVAL;
    switch (key) {
        case PSG_OPT_DEBUG: s->debug = value != 0.0; return PSG_OK;
        case PSG_OPT_THETA:
            s->theta = value > 0.0 ? (float)value : 1.0f;
            psg::reset_near_levels(s);
            return PSG_OK;
        case PSG_OPT_MORTON_VARIANT:
            if (value < 0 || value > 2) return PSG_EINVAL;
            s->morton_variant = (int)value;
            return PSG_OK;
        case PSG_OPT_TIMING: s->timing = value != 0.0; return PSG_OK;
        case PSG_OPT_KAHAN: s->kahan = value != 0.0; return PSG_OK;
        case PSG_OPT_CLOSURE: {
            const int mode = (int)value;
            if (mode < 0 || mode > 2 || (double)mode != value) return PSG_EINVAL;
            if (mode >= 1) {
                PSG_CHECK(cudaSetDevice(s->device));
                const int r = psg::closure_alloc(s);
                if (r != PSG_OK) return r;
            }
            s->cl.mode = mode;
            s->order = mode >= 1 ? 1 : 0;
            psg::reset_near_levels(s);
            return PSG_OK;
        }
        case PSG_OPT_JUDGE: s->cl.judge = value != 0.0; return PSG_OK;
        case PSG_OPT_JUDGE_BLOCKS:
            if (value < 1 || value > 8 || (double)(int)value != value) return PSG_EINVAL;
            s->cl.judge_bps = (int)value;
            return PSG_OK;
        case PSG_OPT_JUDGE_SAMPLES:
            if (value < 64 || value > psg::kJudgeSamples || (double)(int)value != value)
                return PSG_EINVAL;
            s->cl.judge_samples = (int)value;
            return PSG_OK;
        case PSG_OPT_HEAVY_DEPTH:
            if (value > 5) return PSG_EINVAL;
            s->heavy_depth = value < 0 ? -1 : (int)value;
            return PSG_OK;
        case PSG_OPT_LEAF_CAP:
            if (value < 1 || value > PSG_MAX_LEAF_CAP || (double)(int)value != value)
                return PSG_EINVAL;
            s->leaf_cap = (uint32_t)value;
            psg::reset_near_levels(s);
            return PSG_OK;
        case PSG_OPT_NEAR_LEVELS:
            if (value < 2 || value > psg::kMaxDepth || (double)(int)value != value)
                return PSG_EINVAL;
            s->force_ns_levels = (int)value;
            return PSG_OK;
        case PSG_OPT_STREAM: s->force_stream = value != 0.0; return PSG_OK;
        case PSG_OPT_SHRINK_STORES: {
            if (value != 1.0) return PSG_EINVAL;
            PSG_CHECK(cudaSetDevice(s->device));
            PSG_CHECK(cudaStreamSynchronize(s->stream));
            int r = psg::alloc_ns(s, 1024);
            if (r == PSG_OK) r = psg::alloc_p2p(s, 64);
            if (r == PSG_OK) r = psg::alloc_dense(s, 64, 64);
            psg::reset_near_levels(s);
            return r;
        }
        case PSG_OPT_SORT_SPIN:
            if (value < 0 || value > (1 << 22) || (double)(int)value != value) return PSG_EINVAL;
            s->sort_spin_limit = (int)value;
            return PSG_OK;
        case PSG_OPT_READY_SPIN:
            if (value < 0 || value > (1 << 22) || (double)(int)value != value) return PSG_EINVAL;
            s->ready_spin_limit = (int)value;
            return PSG_OK;
        default: return PSG_EINVAL;
    }
}

int psg_get_stats(void* mem, uint64_t* out, size_t n_out) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic || !out) return PSG_EINVAL;
    for (size_t i = 0; i < n_out && i < 24; ++i) out[i] = s->stats[i];
    return PSG_OK;
}

int psg_last_timing(void* mem, float* out_ms, size_t n_out) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic || !out_ms) return PSG_EINVAL;
    for (size_t i = 0; i < n_out && i < (size_t)psg::kPhases; ++i) out_ms[i] = s->ms[i];
    return PSG_OK;
}

size_t psg_tree_nodes(void* mem) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic) return 0;
    return s->last_nodes;
}

// canonical table (level-major, Morton order per level) copied to the host
int psg_tree_dump(void* mem, size_t cap, int32_t* depth, uint32_t* start, uint32_t* count,
                  uint32_t* nchild, int32_t* octant, uint32_t* first_child, uint32_t* parent,
                  float* geo, float* mp, float* lt, uint32_t* m2l_cnt, uint32_t* p2p_cnt) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic) return PSG_EINVAL;
    if (cap < s->last_nodes || s->last_nodes == 0) return cap < s->last_nodes ? PSG_EOOM : PSG_OK;
    PSG_CHECK(cudaSetDevice(s->device));
    // global (capacity-strided) ids -> compact level-major ids
    uint32_t cstart[psg::kLevels + 1];
    cstart[0] = 0;
    for (int d = 0; d <= psg::kMaxDepth; ++d) cstart[d + 1] = cstart[d] + s->lvl_count[d];
    auto compact = [&](uint32_t g, int d) -> uint32_t {
        return g - s->tv.lvl_base[d] + cstart[d];
    };
    size_t k = 0;
    for (int d = 0; d <= psg::kMaxDepth; ++d) {
        const uint32_t cnt = s->lvl_count[d];
        const uint32_t b = s->tv.lvl_base[d];
        if (!cnt) continue;
        uint4* inf = new uint4[cnt];
        PSG_CHECK(cudaMemcpy(inf, s->tv.info + b, cnt * 16, cudaMemcpyDeviceToHost));
        PSG_CHECK(cudaMemcpy(geo + 4 * k, s->tv.geo + b, cnt * 16, cudaMemcpyDeviceToHost));
        PSG_CHECK(cudaMemcpy(mp + 4 * k, s->tv.mp + b, cnt * 16, cudaMemcpyDeviceToHost));
        PSG_CHECK(cudaMemcpy(lt + 4 * k, s->tv.lt + b, cnt * 16, cudaMemcpyDeviceToHost));
        PSG_CHECK(cudaMemcpy(parent + k, s->tv.parent + b, cnt * 4, cudaMemcpyDeviceToHost));
        PSG_CHECK(cudaMemcpy(m2l_cnt + k, s->tv.dbg_m2l + b, cnt * 4, cudaMemcpyDeviceToHost));
        PSG_CHECK(cudaMemcpy(p2p_cnt + k, s->tv.dbg_p2p + b, cnt * 4, cudaMemcpyDeviceToHost));
        for (uint32_t i = 0; i < cnt; ++i) {
            depth[k + i] = d;
            start[k + i] = inf[i].x;
            count[k + i] = inf[i].y;
            nchild[k + i] = psg::flags_nchild(inf[i].w);
            octant[k + i] = d ? (int32_t)psg::flags_octant(inf[i].w) : -1;
            first_child[k + i] = nchild[k + i] ? compact(inf[i].z, d + 1) : 0u;
            parent[k + i] = d ? compact(parent[k + i], d - 1) : 0xFFFFFFFFu;
        }
        delete[] inf;
        k += cnt;
    }
    return PSG_OK;
}

// FP64 direct-sum forces (tests/accuracy.c:42-72) for n_t sampled targets;
// x/y/z/mass, targets and out may each be host or device memory.
int psg_direct_f64(void* mem, const psg_arrays_t* a, const uint32_t* targets, size_t n_t,
                   double* out) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic || !a || !targets || !out) return PSG_EINVAL;
    const size_t n = a->n;
    if (n == 0 || n > s->max_particles) return PSG_EINVAL;
    PSG_CHECK(cudaSetDevice(s->device));
    cudaStream_t st = s->stream;
    // host arrays come in through the context's mirrors
    const float* src[4] = {a->x, a->y, a->z, a->mass};
    for (int c = 0; c < 4; ++c) {
        if (psg::on_device(src[c])) continue;
        const int r = psg::ensure_mirror(s->mir, s->max_particles);
        if (r != PSG_OK) return r;
        float* const rows[4] = {s->mir.x, s->mir.y, s->mir.z, s->mir.m};
        PSG_CHECK(cudaMemcpyAsync(rows[c], src[c], n * 4, cudaMemcpyHostToDevice, st));
        src[c] = rows[c];
    }
    const bool ht = !psg::on_device(targets), ho = !psg::on_device(out);
    const size_t part_n = psg::direct_f64_part_doubles(n, n_t, s->sms * 8);
    psg::Work ws(s);
    const size_t o_part = ws.c.add(part_n * sizeof(double)),
                 o_out = ws.c.add(n_t * 3 * sizeof(double)), o_tg = ws.c.add(n_t * 4);
    const int rw = ws.alloc();
    if (rw != PSG_OK) return rw;
    double* const part = ws.at<double>(o_part);
    double* const dout = ho ? ws.at<double>(o_out) : out;
    const uint32_t* dt = targets;
    if (ht) {
        uint32_t* const d = ws.at<uint32_t>(o_tg);
        PSG_CHECK(cudaMemcpyAsync(d, targets, n_t * 4, cudaMemcpyHostToDevice, st));
        dt = d;
    }
    psg::launch_direct_pack(src[0], src[1], src[2], src[3], n, s->xyzm, st);
    psg::launch_direct_f64(s->xyzm, n, dt, n_t, dout, s->sms * 8, st, part, part_n);
    PSG_CHECK(cudaGetLastError());
    if (ho) PSG_CHECK(cudaMemcpyAsync(out, dout, n_t * 3 * sizeof(double), cudaMemcpyDeviceToHost, st));
    PSG_CHECK(cudaStreamSynchronize(st));
    return PSG_OK;
}

// ---- batched ensemble ------------------------------------------------------------

int psg_ensemble_create(void** out, const size_t* counts, size_t n_systems, const float* theta) {
    if (!out || !counts || n_systems == 0) return PSG_EINVAL;
    for (size_t k = 0; k < n_systems; ++k)
        if (counts[k] == 0 || counts[k] > 60000000u) return PSG_EINVAL;
    psg::Ensemble* e = new (std::nothrow) psg::Ensemble;
    if (!e) return PSG_EALLOC;
    int r = psg::ens_create(e, counts, n_systems, theta);
    if (r != PSG_OK) {
        psg::free_ensemble(e);
        delete e;
        return r;
    }
    *out = e;
    return PSG_OK;
}

int psg_ensemble_destroy(void* h) {
    psg::Ensemble* e = static_cast<psg::Ensemble*>(h);
    if (!e || e->magic != psg::kEnsMagic) return PSG_EINVAL;
    cudaSetDevice(e->device);
    psg::free_ensemble(e);
    delete e;
    return PSG_OK;
}

int psg_ensemble_run(void* h, const psg_arrays_t* a, float* vx, float* vy, float* vz, float dt,
                     uint32_t ticks) {
    psg::Ensemble* e = static_cast<psg::Ensemble*>(h);
    if (!e || e->magic != psg::kEnsMagic || !a || !vx || !vy || !vz) return PSG_EINVAL;
    float* const v[3] = {vx, vy, vz};
    return psg::ens_run(e, a, v, dt, ticks);
}

int psg_ensemble_autotune(void* h, const psg_arrays_t* a, float target, float* theta_out,
                          double* grid_scale_out) {
    psg::Ensemble* e = static_cast<psg::Ensemble*>(h);
    if (!e || e->magic != psg::kEnsMagic || !a || !(target > 0.f)) return PSG_EINVAL;
    return psg::ens_autotune(e, a, target, theta_out, grid_scale_out);
}

int psg_ensemble_systems(void* h, float* theta_out, size_t n) {
    psg::Ensemble* e = static_cast<psg::Ensemble*>(h);
    if (!e || e->magic != psg::kEnsMagic || !theta_out || n != e->nsys) return PSG_EINVAL;
    for (size_t k = 0; k < n; ++k) theta_out[k] = e->theta[k];
    return PSG_OK;
}

int psg_ensemble_leaf_caps(void* h, uint32_t* cap_out, size_t n) {
    psg::Ensemble* e = static_cast<psg::Ensemble*>(h);
    if (!e || e->magic != psg::kEnsMagic || !cap_out || n != e->nsys) return PSG_EINVAL;
    for (size_t k = 0; k < n; ++k) cap_out[k] = e->cap[k];
    return PSG_OK;
}

int psg_ensemble_set_leaf_caps(void* h, const uint32_t* caps, size_t n, int ladder) {
    psg::Ensemble* e = static_cast<psg::Ensemble*>(h);
    if (!e || e->magic != psg::kEnsMagic || !caps || n == 0) return PSG_EINVAL;
    for (size_t k = 0; k < n; ++k)
        if (caps[k] < 1u || caps[k] > (uint32_t)PSG_MAX_LEAF_CAP) return PSG_EINVAL;
    if (ladder) {
        e->leaf_ladder.assign(caps, caps + n);
        return PSG_OK;
    }
    if (n != e->nsys) return PSG_EINVAL;
    PSG_CHECK(cudaSetDevice(e->device));
    for (size_t k = 0; k < n; ++k) e->cap[k] = caps[k];
    e->dirty = true;
    return psg::upload_systems(e);
}

int psg_ensemble_set_order(void* h, int order) {
    psg::Ensemble* e = static_cast<psg::Ensemble*>(h);
    if (!e || e->magic != psg::kEnsMagic || order > 1) return PSG_EINVAL;
    PSG_CHECK(cudaSetDevice(e->device));
    if (order < 0) {
        e->order_ladder = {0, 1};
        return PSG_OK;
    }
    e->order_ladder = {order};
    e->order = order;
    e->dirty = true;
    const int r = psg::set_order(e->fs, order);
    return r == PSG_OK ? psg::upload_systems(e) : r;
}

int psg_ensemble_order(void* h, int* out) {
    psg::Ensemble* e = static_cast<psg::Ensemble*>(h);
    if (!e || e->magic != psg::kEnsMagic || !out) return PSG_EINVAL;
    *out = e->order;
    return PSG_OK;
}

// (no recapture: captured graphs keep the limit they have, reruns take the new one)
int psg_ensemble_set_option(void* h, int key, double value) {
    psg::Ensemble* e = static_cast<psg::Ensemble*>(h);
    if (!e || e->magic != psg::kEnsMagic || key != PSG_OPT_READY_SPIN) return PSG_EINVAL;
    return psg_set_option(e->fs, key, value);
}

// ---- learned closure ----------------------------------------------------------

int psg_closure_set_weights(void* mem, const float* params, size_t n_params) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic || !params) return PSG_EINVAL;
    if (n_params != (size_t)psg::kMlpParams) {
        std::snprintf(psg::g_err, sizeof(psg::g_err), "closure weights: %zu parameters, want %d",
                      n_params, psg::kMlpParams);
        return PSG_EINVAL;
    }
    PSG_CHECK(cudaSetDevice(s->device));
    int r = psg::closure_alloc(s);
    if (r != PSG_OK) return r;
    PSG_CHECK(cudaMemcpyAsync(s->cl.params, params, n_params * 4, cudaMemcpyHostToDevice,
                              s->stream));
    psg::launch_mlp_pack(s->cl.params, s->cl.packed, s->stream);
    PSG_CHECK(cudaGetLastError());
    PSG_CHECK(cudaStreamSynchronize(s->stream));
    s->cl.have_weights = 1;
    return PSG_OK;
}

int psg_closure_last(void* mem, double* median_base, double* median_mlp, int* used,
                     int* samples) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic) return PSG_EINVAL;
    if (median_base) *median_base = s->cl.last.median_base;
    if (median_mlp) *median_mlp = s->cl.last.median_mlp;
    if (used) *used = s->cl.last.use_mlp;
    if (samples) *samples = s->cl.last.samples;
    return PSG_OK;
}

// features of sorted particles idx[0, k) after a closure tick (host arrays)
int psg_closure_features(void* mem, const uint32_t* idx, size_t k, float* x_out,
                         float* scale_out) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic || !idx || !x_out || !scale_out) return PSG_EINVAL;
    if (!s->cl.valid) {
        std::snprintf(psg::g_err, sizeof(psg::g_err), "closure features need a closure tick");
        return PSG_EINVAL;
    }
    if (k == 0) return PSG_OK;
    PSG_CHECK(cudaSetDevice(s->device));
    cudaStream_t st = s->stream;
    psg::Work ws(s);
    const size_t o_idx = ws.c.add(k * 4), o_x = ws.c.add(k * 17 * 4);
    const int rw = ws.alloc();
    if (rw != PSG_OK) return rw;
    uint32_t* const d_idx = ws.at<uint32_t>(o_idx);
    float* const d_x = ws.at<float>(o_x);
    PSG_CHECK(cudaMemcpyAsync(d_idx, idx, k * 4, cudaMemcpyHostToDevice, st));
    psg::TreeView tv = s->tv;
    tv.lg0 = s->cl.lg0;
    tv.lg1 = s->cl.lg1;
    psg::launch_closure_features(tv, s->cl.leaf_of, s->xyzm, s->last_n, d_idx, k, d_x,
                                 d_x + k * 16, st);
    PSG_CHECK(cudaGetLastError());
    PSG_CHECK(cudaMemcpyAsync(x_out, d_x, k * 16 * 4, cudaMemcpyDeviceToHost, st));
    PSG_CHECK(cudaMemcpyAsync(scale_out, d_x + k * 16, k * 4, cudaMemcpyDeviceToHost, st));
    PSG_CHECK(cudaStreamSynchronize(st));
    return PSG_OK;
}

// Train the closure MLP with Adam on (x, t) pairs (host arrays, n x 16 and
// n x 3), the learning rate decaying from lr along a cosine to 5 % of it.  params (kMlpParams) holds the initial values and receives the
// trained ones; loss_out (epochs) receives each epoch's mean squared error.
int psg_closure_train(void* mem, const float* x, const float* t, size_t n, float* params,
                      uint32_t epochs, uint32_t batch, float lr, uint64_t seed, float* loss_out) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic || !x || !t || !params || n == 0 || batch == 0)
        return PSG_EINVAL;
    PSG_CHECK(cudaSetDevice(s->device));
    cudaStream_t st = s->stream;
    PSG_CHECK(psg::prepare_mlp_grad_kernel());
    const int P = psg::kMlpParams;
    psg::Work ws(s);
    const size_t o_x = ws.c.add(n * 16 * 4), o_t = ws.c.add(n * 3 * 4), o_perm = ws.c.add(n * 4),
                 o_p = ws.c.add(P * 4), o_m = ws.c.add(P * 4), o_v = ws.c.add(P * 4),
                 o_g = ws.c.add(P * 4), o_loss = ws.c.add((size_t)(epochs ? epochs : 1) * 4),
                 o_w = ws.c.add(sizeof(psg::MlpPacked));
    const int rw = ws.alloc();
    if (rw != PSG_OK) return rw;
    float *const d_x = ws.at<float>(o_x), *const d_t = ws.at<float>(o_t),
          *const d_p = ws.at<float>(o_p), *const d_m = ws.at<float>(o_m),
          *const d_v = ws.at<float>(o_v), *const d_g = ws.at<float>(o_g),
          *const d_loss = ws.at<float>(o_loss);
    uint32_t* const d_perm = ws.at<uint32_t>(o_perm);
    psg::MlpPacked* const d_w = ws.at<psg::MlpPacked>(o_w);
    PSG_CHECK(cudaMemcpyAsync(d_x, x, n * 16 * 4, cudaMemcpyHostToDevice, st));
    PSG_CHECK(cudaMemcpyAsync(d_t, t, n * 3 * 4, cudaMemcpyHostToDevice, st));
    PSG_CHECK(cudaMemcpyAsync(d_p, params, P * 4, cudaMemcpyHostToDevice, st));
    PSG_CHECK(cudaMemsetAsync(d_m, 0, P * 4, st));
    PSG_CHECK(cudaMemsetAsync(d_v, 0, P * 4, st));
    PSG_CHECK(cudaMemsetAsync(d_g, 0, P * 4, st));
    psg::launch_mlp_pack(d_p, d_w, st);
    PSG_CHECK(cudaMemsetAsync(d_loss, 0, (epochs ? epochs : 1) * 4, st));
    uint32_t* perm = nullptr;
    PSG_CHECK(cudaMallocHost((void**)&perm, n * 4));
    uint64_t rng = seed ^ 0x9E3779B97F4A7C15ull;
    auto next = [&rng]() {  // splitmix64
        uint64_t z = (rng += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    };
    const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    uint64_t step = 0;
    int r = PSG_OK;
    for (uint32_t ep = 0; ep < epochs && r == PSG_OK; ++ep) {
        PSG_CHECK(cudaStreamSynchronize(st));  // perm is reused
        for (size_t i = 0; i < n; ++i) perm[i] = (uint32_t)i;
        for (size_t i = n - 1; i > 0; --i) {
            const size_t j = (size_t)(next() % (i + 1));
            const uint32_t tmp = perm[i];
            perm[i] = perm[j];
            perm[j] = tmp;
        }
        PSG_CHECK(cudaMemcpyAsync(d_perm, perm, n * 4, cudaMemcpyHostToDevice, st));
        // cosine decay of the learning rate over the epochs, to 5 % of lr
        const float lr_ep =
            lr * (0.05f + 0.95f * 0.5f * (1.0f + cosf(3.14159265f * (float)ep / (float)epochs)));
        for (size_t b0 = 0; b0 < n; b0 += batch) {
            const size_t cnt = n - b0 < batch ? n - b0 : batch;
            psg::launch_mlp_grad(d_x, d_t, d_perm, b0, cnt, d_w, 1.0f / (3.0f * (float)cnt), d_g,
                                 d_loss + ep, st);
            ++step;
            const float bc1 = 1.0f - powf(beta1, (float)step);
            const float bc2 = 1.0f - powf(beta2, (float)step);
            psg::launch_mlp_adam(d_p, d_m, d_v, d_g, d_w, P, lr_ep, beta1, beta2, eps, bc1, bc2,
                                 st);
        }
        if (cudaGetLastError() != cudaSuccess) r = PSG_EDEVICE;
    }
    if (r == PSG_OK) {
        PSG_CHECK(cudaMemcpyAsync(params, d_p, P * 4, cudaMemcpyDeviceToHost, st));
        if (loss_out && epochs)
            PSG_CHECK(cudaMemcpyAsync(loss_out, d_loss, epochs * 4, cudaMemcpyDeviceToHost, st));
        PSG_CHECK(cudaStreamSynchronize(st));
        if (loss_out)
            for (uint32_t ep = 0; ep < epochs; ++ep) loss_out[ep] /= (float)(3 * n);
    }
    cudaFreeHost(perm);
    if (r != PSG_OK) std::snprintf(psg::g_err, sizeof(psg::g_err), "closure training failed");
    return r;
}

// loss (mean squared error) and its gradient w.r.t. params for one batch of
// n samples (host arrays): the training step's own kernels, no update
int psg_closure_grad(void* mem, const float* x, const float* t, size_t n, const float* params,
                     float* grad_out, float* loss_out) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic || !x || !t || !params || !grad_out || n == 0)
        return PSG_EINVAL;
    PSG_CHECK(cudaSetDevice(s->device));
    cudaStream_t st = s->stream;
    PSG_CHECK(psg::prepare_mlp_grad_kernel());
    const int P = psg::kMlpParams;
    psg::Work ws(s);
    const size_t o_x = ws.c.add(n * 16 * 4), o_t = ws.c.add(n * 3 * 4), o_p = ws.c.add(P * 4),
                 o_g = ws.c.add(P * 4), o_loss = ws.c.add(4),
                 o_w = ws.c.add(sizeof(psg::MlpPacked));
    const int rw = ws.alloc();
    if (rw != PSG_OK) return rw;
    float *const d_x = ws.at<float>(o_x), *const d_t = ws.at<float>(o_t),
          *const d_p = ws.at<float>(o_p), *const d_g = ws.at<float>(o_g),
          *const d_loss = ws.at<float>(o_loss);
    psg::MlpPacked* const d_w = ws.at<psg::MlpPacked>(o_w);
    PSG_CHECK(cudaMemcpyAsync(d_x, x, n * 16 * 4, cudaMemcpyHostToDevice, st));
    PSG_CHECK(cudaMemcpyAsync(d_t, t, n * 3 * 4, cudaMemcpyHostToDevice, st));
    PSG_CHECK(cudaMemcpyAsync(d_p, params, P * 4, cudaMemcpyHostToDevice, st));
    PSG_CHECK(cudaMemsetAsync(d_g, 0, P * 4, st));
    PSG_CHECK(cudaMemsetAsync(d_loss, 0, 4, st));
    psg::launch_mlp_pack(d_p, d_w, st);
    psg::launch_mlp_grad(d_x, d_t, nullptr, 0, n, d_w, 1.0f / (3.0f * (float)n), d_g, d_loss, st);
    PSG_CHECK(cudaGetLastError());
    PSG_CHECK(cudaMemcpyAsync(grad_out, d_g, P * 4, cudaMemcpyDeviceToHost, st));
    float loss = 0.f;
    PSG_CHECK(cudaMemcpyAsync(&loss, d_loss, 4, cudaMemcpyDeviceToHost, st));
    PSG_CHECK(cudaStreamSynchronize(st));
    if (loss_out) *loss_out = loss / (float)(3 * n);
    return PSG_OK;
}

// MLP outputs (n x 8, before scaling) for inputs x (n x 16), host arrays:
// the inference kernel's network on the tensor cores
int psg_closure_forward(void* mem, const float* x, size_t n, const float* params, float* y_out) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic || !x || !params || !y_out || n == 0) return PSG_EINVAL;
    PSG_CHECK(cudaSetDevice(s->device));
    cudaStream_t st = s->stream;
    psg::Work ws(s);
    const size_t o_x = ws.c.add(n * 16 * 4), o_p = ws.c.add(psg::kMlpParams * 4),
                 o_y = ws.c.add(n * 8 * 4), o_w = ws.c.add(sizeof(psg::MlpPacked));
    const int rw = ws.alloc();
    if (rw != PSG_OK) return rw;
    float *const d_x = ws.at<float>(o_x), *const d_p = ws.at<float>(o_p),
          *const d_y = ws.at<float>(o_y);
    psg::MlpPacked* const d_w = ws.at<psg::MlpPacked>(o_w);
    PSG_CHECK(cudaMemcpyAsync(d_x, x, n * 16 * 4, cudaMemcpyHostToDevice, st));
    PSG_CHECK(cudaMemcpyAsync(d_p, params, psg::kMlpParams * 4, cudaMemcpyHostToDevice, st));
    psg::launch_mlp_pack(d_p, d_w, st);
    PSG_CHECK(cudaMemsetAsync(&s->d_status->err, 0, 4, st));
    psg::launch_mlp_forward(d_x, n, d_w, d_y, s->sms, &s->d_status->err, st);
    PSG_CHECK(cudaGetLastError());
    PSG_CHECK(cudaMemcpyAsync(y_out, d_y, n * 8 * 4, cudaMemcpyDeviceToHost, st));
    PSG_CHECK(cudaMemcpyAsync(&s->h_status->err, &s->d_status->err, 4, cudaMemcpyDeviceToHost,
                              st));
    PSG_CHECK(cudaStreamSynchronize(st));
    if (s->h_status->err & PSG_ERR_TC_TIMEOUT) {
        std::snprintf(psg::g_err, sizeof(psg::g_err),
                      "closure network: a tensor-core MMA did not complete");
        return PSG_EDEVICE;
    }
    return PSG_OK;
}

// the last closure tick's per-particle correction (sorted order, n x 3)
int psg_closure_correction(void* mem, float* out, size_t n) {
    State* s = static_cast<State*>(mem);
    if (!s || s->magic != psg::kMagic || !out || !s->cl.dF) return PSG_EINVAL;
    if (n != s->last_n || !s->cl.valid) return PSG_EINVAL;
    PSG_CHECK(cudaSetDevice(s->device));
    PSG_CHECK(cudaMemcpy2DAsync(out, 12, s->cl.dF, 16, 12, n, cudaMemcpyDeviceToHost, s->stream));
    PSG_CHECK(cudaStreamSynchronize(s->stream));
    return PSG_OK;
}

const char* psg_last_error(void) { return psg::g_err; }

void psg_set_error(const char* msg) { std::snprintf(psg::g_err, sizeof(psg::g_err), "%s", msg); }

}  // extern "C"
