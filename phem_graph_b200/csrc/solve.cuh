// solve.cuh -- the device code that the one-graph solve (msf.cu) and the grid
// batch (batch_grid.cu) share: the grid barrier, the offers, the survivor
// lists and the passes over them.
#pragma once

#include "internal.h"

namespace phem {

struct SolveArgs {
    const void *e0;
    uint64_t m;
    uint32_t n;
    uint32_t *parent;
    unsigned long long *best;      // two arrays of best_stride words: minimum key offered, by round parity
    uint64_t best_stride;
    uint32_t *samples;             // the threshold select's sample: weights, then one endpoint each
    uint32_t nsamp;                // 0: no select
    uint32_t *bitmap;              // MSF membership, one bit per edge id
    uint32_t *chunk_off;           // offset of each chunk of edge ids' MSF edges within a CTA's range of chunks
    uint32_t *cta_tot;             // forest edges per CTA's chunk range
    uint32_t *giant;               // one bit per vertex: in the largest component (heavy pass)
    uint4 *list;                   // per-warp survivor segments of seg records
    uint32_t *hooked;              // per-warp segments: the roots its records hooked in a round
    uint64_t seg;
    unsigned long long *forest;
    phem_edge *out;
    int32_t *label;                // packed edges: min-id labels (may be null)
    Ctl *ctl;
    Ctl *publish;                  // pinned host copy of the results (null: the host copies them)
    unsigned long long threshold;  // when nothing is selected
    uint64_t light_k, light_k2;    // light edges the threshold aims at: skewed degrees, even ones
    int gather;                    // write the ordered MSF records (kKindMsf)
    int timing;                    // record phase timestamps
};

constexpr int kSolveThreads = 1024;  // most threads per CTA (one CTA per SM); 64 registers each
constexpr int kSolveWarps = kSolveThreads / 32;
constexpr uint32_t kMaxSample = 8192;
constexpr uint32_t kSeenWords = 8192;  // 2^18 bits
constexpr uint32_t kMaxGrid = 1024;

// Survivor records mark in the top bit of each root whether the record's
// offer may have won there; vertex ids leave that bit free up to this n.
constexpr uint32_t kMarkMaxN = 0x80000000u;
constexpr uint32_t kRootMask = 0x7fffffffu;

// An input record takes part in the forest: self-loops never do; packed CC
// edges follow union_find_gpu_COO and only count when u < v
// (CC/ExternalSpanningTree.cu:82).
template <int KIND>
__device__ __forceinline__ bool e0_live(uint32_t u, uint32_t v)
{
    return KIND == kKindMsf ? (u != v) : (u < v);
}

// Key of an edge: (w, id) for weighted edges, id alone for packed CC edges
// (the canonical forest orders edges by index).
template <int KIND>
__device__ __forceinline__ unsigned long long e0_key(uint32_t w, uint32_t id)
{
    return KIND == kKindMsf ? (((unsigned long long)w << 32) | id) : (unsigned long long)id;
}

// ---- shared memory -----------------------------------------------------------

// Offers.  A survivor offers its key to both of its roots' best[] words.
// Most survivors of hub-heavy rounds (and of the heavy pass, whose records
// mostly touch the light phase's giant component) offer to a handful of
// roots, and atomics on one best[] word serialise on its L2 slice; so a root
// first tries the slot hash(t) of a 2048-entry table in the CTA's shared
// memory, claiming it when it is free: offers to a claimed slot are
// shared-memory atomicMins behind a shared read, and the table goes to best[]
// (one atomic per slot) when the CTA's pass ends.  An offer whose slot another
// root holds reads best[t] from L2 first and issues the 64-bit atomicMin only
// when it can still win: the read may be stale but never below the true
// value.  Both roots' reads are issued before either atomic.
constexpr int kOfferSlots = 2048;
constexpr uint32_t kNoTag = 0xffffffffu;

struct OfferCache {
    unsigned long long key[kOfferSlots];
    uint32_t tag[kOfferSlots];
};

constexpr int kEpStages = 2;
constexpr uint32_t kEpStageBytes = 1536;  // 128 records of 12 bytes or 192 packed pairs
constexpr uint32_t kRing = 64;            // survivors staged per warp

struct __align__(16) EpWarp {
    unsigned char stage[kEpStages][kEpStageBytes];
    uint4 ring[kRing];
    unsigned long long bar[kEpStages];
};

struct SolveSmem {
    EpWarp warp[kSolveWarps];   // the select's samples and histogram share this space
    OfferCache oc;
    unsigned long long acc;     // the CTA's contribution to the next barrier's sum
    unsigned long long sum;     // the last barrier's sum over the grid
    unsigned long long red[kSolveWarps];
    uint32_t abort;
    uint32_t fatal;             // a bounded wait of this CTA gave up
    uint32_t scan[kSolveWarps + 1];
    uint32_t pref[kMaxGrid];    // forest edges of the CTA ranges before each (gather)
    uint32_t sel_prefix, sel_rank, sel_or, sel_dup;
};
static_assert(sizeof(EpWarp) * kSolveWarps >= (kMaxSample + kSeenWords) * sizeof(uint32_t),
              "the select's samples, set and histogram fit in the warps' space");

// Grid barrier with a sum: adds the CTAs' `acc`, returns false when the solve
// has to stop (a bounded wait gave up somewhere; the status bit says so).  One
// word per barrier, zeroed with the control block: bits 52.. count arrivals,
// bits 40..51 CTAs that gave up, bits 0..39 the sum, so the sum arrives with
// the release itself.  The fences of thread 0 order the CTA's accesses before
// the arrival and discard its L1 lines after it, so plain loads after the
// barrier see every store made before it on any SM.  1.2 us on 148 CTAs.
constexpr uint32_t kBarSpinCap = 1u << 22;  // about 3 s

template <class Smem>
__device__ __forceinline__ bool grid_sync(Ctl *ctl, Smem &s, uint32_t &seq)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long v = s.acc + ((unsigned long long)s.fatal << 40);
        s.acc = 0;
        __threadfence();
        if (gridDim.x > 1) {
            unsigned long long *word = &ctl->bar[seq];
            v += atomicAdd(word, v + (1ull << 52)) + (1ull << 52);
            uint32_t spins = 0;
            while ((v >> 52) < gridDim.x) {
                if (++spins > kBarSpinCap) {
                    set_err(&ctl->err, kErrLookback);
                    v |= 1ull << 40;
                    break;
                }
                v = ld_relaxed_u64(reinterpret_cast<const uint64_t *>(word));
            }
            __threadfence();
        }
        s.sum = v & ((1ull << 40) - 1);
        s.abort = (uint32_t)(v >> 40) & 0xfffu;
    }
    __syncthreads();
    seq++;
    return s.abort == 0;
}

// Ends a solve's last kernel: the CTA that finishes last writes the results to
// the host's copy and zeroes the block for the next solve, so that neither a
// memset before the launch nor a copy behind it is queued: 222 -> 211 us per
// call at 131,072 vertices and 1,048,576 edges.  Not inlined, or the solve
// spills more (219 us).  A solve that gave up at a barrier never gets here;
// the host sees its copy untouched and reads the block itself.
__device__ __noinline__ inline void publish_ctl(Ctl *ctl, Ctl *host)
{
    __shared__ bool s_last;
    if (!host)
        return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1;
        __threadfence();
    }
    __syncthreads();
    if (!s_last)
        return;
    unsigned long long *src = reinterpret_cast<unsigned long long *>(ctl);
    volatile unsigned long long *dst = reinterpret_cast<volatile unsigned long long *>(host);
    for (uint32_t i = threadIdx.x; i < offsetof(Ctl, stamp) / 8; i += blockDim.x) {
        if (i < offsetof(Ctl, bar) / 8)
            dst[i] = __ldcg(src + i);
        src[i] = 0;
    }
}

// Profiling: one thread of the grid stamps the end of each phase.
struct PhaseClock {
    Ctl *ctl;
    uint32_t marks = 0;
    bool on;
    __device__ PhaseClock(Ctl *c, int timing) : ctl(c), on(timing && blockIdx.x == 0 && threadIdx.x == 0)
    {
        stamp(kKernelCount);  // the start
    }
    __device__ __forceinline__ void stamp(uint32_t phase)
    {
        if (!on || marks >= kMaxPhases)
            return;
        uint64_t t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        ctl->stamp[marks] = t;
        ctl->phase_of[marks] = phase;
        ctl->stamps = ++marks;
    }
};

// parent[] through L1 (weak, never the read-only path: this kernel writes it).
__device__ __forceinline__ uint32_t ld_par(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned long long ld_best(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.global.ca.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}

// Adds a per-lane count to the CTA's contribution to the next barrier.
template <class Smem>
__device__ __forceinline__ void acc_add(Smem &s, uint32_t v)
{
    v = __reduce_add_sync(0xffffffffu, v);
    if (lane_id() == 0 && v)
        atomicAdd(&s.acc, (unsigned long long)v);
}

// True when the offer went to (or lost against) t's shared slot; *may is set
// when it went there below the slot's value.
__device__ __forceinline__ bool table_offer(OfferCache &oc, uint32_t t, unsigned long long k, int *may)
{
    const int slot = (int)((t * 0x9E3779B1u) >> 21);  // 11 bits
    uint32_t tag = *(volatile uint32_t *)&oc.tag[slot];
    if (tag == kNoTag)
        tag = atomicCAS(&oc.tag[slot], kNoTag, t);
    if (tag != kNoTag && tag != t)
        return false;
    // most offers to a hub's slot cannot win: a shared read first avoids the
    // 64-bit shared atomic (a compare-and-swap loop under contention)
    if (k < *(volatile unsigned long long *)&oc.key[slot]) {
        atomicMin(&oc.key[slot], k);
        *may = 1;
    }
    return true;
}

// Returns bit 0 / bit 1 set when the offer at ta / tb may still win.  A
// cleared bit means the key lost there for good: it met a lower value (the
// shared slot's, or best[t]'s in L2), and the final minimum is lower still
// (keys are unique).
__device__ __forceinline__ uint32_t offer_pair(unsigned long long *best, OfferCache &oc, uint32_t ta, uint32_t tb,
                                               unsigned long long key, bool on)
{
    if (!on)
        return 0u;
    int wa = 0, wb = 0;
    const bool da = table_offer(oc, ta, key, &wa), db = table_offer(oc, tb, key, &wb);
    const unsigned long long ga = da ? 0ull : __ldcg(best + ta), gb = db ? 0ull : __ldcg(best + tb);
    if (!da && key < ga) {
        atomicMin(best + ta, key);
        wa = 1;
    }
    if (!db && key < gb) {
        atomicMin(best + tb, key);
        wb = 1;
    }
    return (uint32_t)wa | ((uint32_t)wb << 1);
}

__device__ __forceinline__ uint64_t mix64(uint64_t z)
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Position of sample i of `count` stratified ones over [0, m).
__device__ __forceinline__ uint64_t sample_pos(uint32_t i, uint32_t count, uint64_t m)
{
    const uint64_t lo = (uint64_t)i * m / count, hi = (uint64_t)(i + 1) * m / count;
    return hi > lo ? lo + mix64(0x5EED0000ull + i) % (hi - lo) : lo;
}

// ---- edge pass ---------------------------------------------------------------

// Appends the lanes' survivors (keep) to the ring in lane order.
__device__ __forceinline__ void ring_append(EpWarp &w, uint32_t &filled, bool keep, uint4 rec, uint32_t lane)
{
    const unsigned mask = __ballot_sync(0xffffffffu, keep);
    if (keep)
        w.ring[(filled + __popc(mask & ((1u << lane) - 1u))) & (kRing - 1)] = rec;
    filled += __popc(mask);
}

// Writes the `cnt` (<= 32) oldest ring entries to the warp's list and offers
// them.
template <int KIND>
__device__ __forceinline__ void ring_flush(const SolveArgs &a, SolveSmem &s, unsigned long long *best, uint4 *list,
                                           EpWarp &w, uint32_t &flushed, uint32_t cnt, uint32_t lane)
{
    __syncwarp();  // the lanes' ring writes are visible
    const bool on = lane < cnt;
    const uint4 rec = on ? w.ring[(flushed + lane) & (kRing - 1)] : make_uint4(0, 0, 0, 0);
    const uint32_t may = offer_pair(best, s.oc, rec.x, rec.y, e0_key<KIND>(rec.z, rec.w), on);
    // the hook only looks at the roots where the record may have won
    // (the top bit of a root is free when n <= 2^31)
    uint4 r = rec;
    if (a.n <= kMarkMaxN) {
        r.x |= (may & 1u) << 31;
        r.y |= (may & 2u) << 30;
    }
    if (on)
        list[flushed + lane] = r;
    flushed += cnt;
    __syncwarp();  // the ring slots just read may be written again
}

// Bounded wait of the whole warp for a stage's bulk copy.
__device__ __forceinline__ bool ep_wait(unsigned long long *bar, uint32_t parity, uint32_t *err)
{
    bool ok = mbar_wait(reinterpret_cast<uint64_t *>(bar), parity, err);
    return __all_sync(0xffffffffu, ok);
}

// Per-warp state carried across passes.
struct WarpState {
    uint32_t gw, GW;    // this warp's index and the grid's warp count
    uint32_t len;       // records in the warp's list
    uint32_t parity;    // bit s: phase of stage s's barrier to wait for
    uint32_t hooks;     // roots the warp hooked in this round
    uint4 *list;
    uint32_t *hooked;
};

// One list pass over the warp's own survivors: both roots are relabelled by
// one hop (the compress pointed every root that hooked at its new root),
// records inside one component are dropped and the rest offered and compacted
// in place (a row is written only after the records that fill it were read).
constexpr int kListRows = 4;

template <int KIND>
__device__ __forceinline__ void list_pass(const SolveArgs &a, SolveSmem &s, unsigned long long *best, WarpState &ws)
{
    const uint32_t lane = lane_id();
    EpWarp &w = s.warp[threadIdx.x >> 5];
    const uint32_t rmask = a.n <= kMarkMaxN ? kRootMask : 0xffffffffu;  // drop the last round's marks
    uint32_t filled = 0, flushed = 0;
    for (uint32_t i0 = 0; i0 < ws.len; i0 += 32 * kListRows) {
        uint4 rec[kListRows];
#pragma unroll
        for (int j = 0; j < kListRows; j++) {
            const uint32_t i = i0 + j * 32 + lane;
            rec[j] = i < ws.len ? __ldcg(ws.list + i) : make_uint4(0, 0, 0, 0);
            rec[j].x &= rmask;
            rec[j].y &= rmask;
        }
#pragma unroll
        for (int j = 0; j < kListRows; j++) {
            rec[j].x = ld_par(a.parent + rec[j].x);
            rec[j].y = ld_par(a.parent + rec[j].y);
        }
#pragma unroll
        for (int j = 0; j < kListRows; j++) {
            ring_append(w, filled, i0 + j * 32 + lane < ws.len && rec[j].x != rec[j].y, rec[j], lane);
            if (filled - flushed >= 32)
                ring_flush<KIND>(a, s, best, ws.list, w, flushed, 32, lane);
        }
    }
    if (filled != flushed)
        ring_flush<KIND>(a, s, best, ws.list, w, flushed, filled - flushed, lane);
    ws.len = flushed;
    acc_add(s, lane == 0 ? flushed : 0u);
}

// Hook, over the warp's survivor records: a record whose key is the minimum
// at an endpoint's component is that component's chosen edge (keys are
// unique, so each component finds exactly one).  A component hooks onto the
// far one and marks the edge; when both endpoints chose the same record (a
// mutual pair) the lower id stays root and the higher one hooks
// (new_grafting_edges, MST/src/kernels.cu:73-134).  The roots that stay are
// the lower ends of the mutual pairs -- keys are unique, so the choices of a
// tree of components end in exactly one -- and their next round's best words
// are reset here.
template <int KIND>
__device__ __forceinline__ void hook_pass(const SolveArgs &a, SolveSmem &s, const unsigned long long *best,
                                       unsigned long long *best_next, WarpState &ws)
{
    const uint32_t lane = lane_id(), below = (1u << lane) - 1u;
    uint32_t hooks = 0;
    const bool marks = a.n <= kMarkMaxN;
    const uint32_t rmask = marks ? kRootMask : 0xffffffffu;
    uint32_t choosers = 0;
    for (uint32_t i0 = 0; i0 < ws.len; i0 += 128) {
        uint4 rec[4];
        unsigned long long ka[4], kb[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint32_t i = i0 + q * 32 + lane;
            rec[q] = i < ws.len ? __ldcg(ws.list + i) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            // only the roots where the record's offer may have won (marked by
            // the edge pass; every root when n is too large for marks)
            const bool ma = marks ? (rec[q].x >> 31) != 0 : rec[q].x != rec[q].y;
            const bool mb = marks ? (rec[q].y >> 31) != 0 : rec[q].x != rec[q].y;
            rec[q].x &= rmask;
            rec[q].y &= rmask;
            // cached: the few hub components of late rounds hit in L1
            ka[q] = ma ? ld_best(best + rec[q].x) : kKeyNone;
            kb[q] = mb ? ld_best(best + rec[q].y) : kKeyNone;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const unsigned long long key = e0_key<KIND>(rec[q].z, rec[q].w);
            const bool real = rec[q].x != rec[q].y;
            const bool A = real && ka[q] == key, B = real && kb[q] == key;
            const unsigned won = __ballot_sync(0xffffffffu, A || B);
            if (A || B) {
                uint32_t hk, tgt;
                if (A && B) {
                    hk = max(rec[q].x, rec[q].y);
                    tgt = min(rec[q].x, rec[q].y);
                } else {
                    hk = A ? rec[q].x : rec[q].y;
                    tgt = A ? rec[q].y : rec[q].x;
                }
                const uint32_t id = rec[q].w;
                a.parent[hk] = tgt;
                ws.hooked[hooks + __popc(won & below)] = hk;
                if (A && B)
                    best_next[tgt] = kKeyNone;
                choosers += (uint32_t)A + (uint32_t)B;
                if (KIND == kKindMsf) {
                    atomicOr(a.bitmap + (id >> 5), 1u << (id & 31));
                } else if (a.forest) {
                    a.forest[hk] = __ldg(static_cast<const unsigned long long *>(a.e0) + id);
                }
            }
            hooks += __popc(won);
        }
    }
    ws.hooks = hooks;
    acc_add(s, choosers);
}

// Every root this warp hooked is pointed at its final root.  Only its own
// lane writes a root's pointer, to ever farther ancestors, so long chains
// shorten from all sides; the first steps read through L1 (a stale pointer is
// still an ancestor, and roots are final in this phase), later ones through
// L2, where the other lanes' shortcuts are.
constexpr int kVItems = 4;

__device__ __forceinline__ void compress_pass(uint32_t *parent, uint32_t n, uint32_t *err, const WarpState &ws)
{
    for (uint32_t i0 = lane_id(); i0 < ws.hooks; i0 += 32 * kVItems) {
        uint32_t x[kVItems], y[kVItems];
        bool walking[kVItems];
#pragma unroll
        for (int k = 0; k < kVItems; k++) {
            walking[k] = i0 + 32 * k < ws.hooks;
            x[k] = walking[k] ? __ldcg(ws.hooked + i0 + 32 * k) : 0u;
        }
#pragma unroll
        for (int k = 0; k < kVItems; k++)
            y[k] = walking[k] ? ld_par(parent + x[k]) : 0u;
        for (uint32_t steps = 0;; steps++) {
            uint32_t p[kVItems];
#pragma unroll
            for (int k = 0; k < kVItems; k++)
                p[k] = !walking[k] ? y[k] : (steps < 8 ? ld_par(parent + y[k]) : __ldcg(parent + y[k]));
            bool any = false;
#pragma unroll
            for (int k = 0; k < kVItems; k++) {
                walking[k] = walking[k] && p[k] != y[k];
                if (walking[k])
                    parent[x[k]] = p[k];
                y[k] = p[k];
                any |= walking[k];
            }
            if (!any)
                break;
            if (steps > n) {
                set_err(err, kErrChase);
                break;
            }
        }
    }
}

// Vertices [0, n) pointed at their roots (before the heavy pass, which then
// relabels endpoints in one hop) and the roots' next best words reset (when
// best_next is set); with use_giant also one bit per vertex: in the component
// of root `giant`; with forest also every vertex's forest slot, the edge to
// the parent it had.  CHAINS: the pointers may form chains as long as the
// graph (a path whose every vertex hooked under the one before it), which are
// shortened from all sides as in compress_pass.
template <bool CHAINS = false>
__device__ __forceinline__ void full_compress(uint32_t *parent, uint32_t n, unsigned long long *best_next,
                                              uint32_t *bits_of, uint32_t giant, bool use_giant, uint32_t *err,
                                              unsigned long long *forest = nullptr)
{
    const uint32_t lane = lane_id();
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x * kVItems;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x * kVItems; i0 < n; i0 += step) {
        bool walking[kVItems];
        uint32_t x[kVItems], y[kVItems], y0[kVItems];
        // the vertices' walks advance in lockstep, so their dependent loads
        // are in flight together
#pragma unroll
        for (int k = 0; k < kVItems; k++) {
            const uint64_t i = i0 + k * blockDim.x + threadIdx.x;
            walking[k] = i < n;
            x[k] = walking[k] ? (uint32_t)i : 0u;
        }
#pragma unroll
        for (int k = 0; k < kVItems; k++)
            y0[k] = y[k] = ld_par(parent + x[k]);
        for (uint32_t steps = 0;; steps++) {
            uint32_t p[kVItems];
#pragma unroll
            for (int k = 0; k < kVItems; k++)
                p[k] = !walking[k] ? y[k]
                                   : (CHAINS && steps >= 8 ? __ldcg(parent + y[k]) : ld_par(parent + y[k]));
            bool any = false;
#pragma unroll
            for (int k = 0; k < kVItems; k++) {
                walking[k] = walking[k] && p[k] != y[k];
                if (CHAINS && steps >= 8 && walking[k])
                    parent[x[k]] = p[k];
                y[k] = p[k];
                any |= walking[k];
            }
            if (!any)
                break;
            if (steps > n) {
                set_err(err, kErrChase);
                break;
            }
        }
#pragma unroll
        for (int k = 0; k < kVItems; k++) {
            const uint64_t i = i0 + k * blockDim.x + threadIdx.x;
            if (i < n) {
                if (forest)
                    forest[i] = y0[k] != x[k] ? (unsigned long long)y0[k] << 32 | i : kForestEmpty;
                if (y0[k] != y[k])
                    parent[x[k]] = y[k];
                if (best_next && y[k] == x[k])
                    best_next[x[k]] = kKeyNone;
            }
            if (use_giant) {  // blockDim.x and i0 are multiples of 32
                const unsigned bits = __ballot_sync(0xffffffffu, i < n && y[k] == giant);
                if (lane == 0 && i < n)
                    bits_of[i >> 5] = bits;
            }
        }
    }
}

// Exclusive scan of `count` values into off[], by ranges of `per`: CTA c scans
// range c (offsets within the range) and publishes the range's total; after a
// barrier prefix_totals gives the ranges' offsets.  value(c, i, end) is thread
// i - c's value of a block's step from c (0 where i >= end); whole warps call
// it.
template <class F>
__device__ __forceinline__ void count_scan(SolveSmem &s, uint32_t *off, uint64_t count, uint64_t per,
                                           uint32_t *cta_tot, F value)
{
    const uint64_t c0 = min(blockIdx.x * per, count), c1 = min(c0 + per, count);
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t carry = 0;
    for (uint64_t c = c0; c < c1; c += blockDim.x) {
        const uint64_t i = c + threadIdx.x;
        const uint32_t v = value(c, i, c1);
        uint32_t x = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= (uint32_t)d)
                x += y;
        }
        if (lane == 31)
            s.scan[warp] = x;
        __syncthreads();
        if (warp == 0) {
            const uint32_t t = lane < nw ? s.scan[lane] : 0u;
            uint32_t ti = t;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, ti, d);
                if (lane >= (uint32_t)d)
                    ti += y;
            }
            s.scan[lane] = ti - t;
            if (lane == 31)
                s.scan[kSolveWarps] = ti;
        }
        __syncthreads();
        if (i < c1)
            off[i] = carry + s.scan[warp] + x - v;
        carry += s.scan[kSolveWarps];
        __syncthreads();  // s.scan is reused
    }
    if (threadIdx.x == 0)
        cta_tot[blockIdx.x] = carry;
}

// The ranges' offsets into s.pref (every CTA for itself); returns the total
// in warp 0.
__device__ __forceinline__ uint32_t prefix_totals(SolveSmem &s, const uint32_t *cta_tot)
{
    const uint32_t lane = lane_id();
    uint32_t run = 0;
    if (threadIdx.x < 32) {
        for (uint32_t c0 = 0; c0 < gridDim.x; c0 += 32) {
            const uint32_t c = c0 + lane;
            const uint32_t v = c < gridDim.x ? __ldcg(cta_tot + c) : 0u;
            uint32_t x = v;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= (uint32_t)d)
                    x += y;
            }
            if (c < gridDim.x)
                s.pref[c] = run + x - v;
            run += __shfl_sync(0xffffffffu, x, 31);
        }
    }
    __syncthreads();
    return run;
}

__device__ __forceinline__ void offers_reset(OfferCache &oc)
{
    for (int i = threadIdx.x; i < kOfferSlots; i += blockDim.x) {
        oc.tag[i] = kNoTag;
        oc.key[i] = kKeyNone;
    }
}

// The CTA's offer table to best[], then an empty table for the next pass.
__device__ __forceinline__ void offers_flush(OfferCache &oc, unsigned long long *best)
{
    __syncthreads();
    for (int i = threadIdx.x; i < kOfferSlots; i += blockDim.x) {
        const uint32_t t = oc.tag[i];
        if (t != kNoTag) {
            atomicMin(best + t, oc.key[i]);
            oc.tag[i] = kNoTag;
            oc.key[i] = kKeyNone;
        }
    }
}

}  // namespace phem
