// msf.cu -- minimum spanning forest on sm_100a: Boruvka rounds behind a
// light/heavy edge filter, one persistent launch per solve.
//
// Arithmetic is the reference's device_boruvka (MST/src/kernels.cu:507-689):
// per round every component takes its minimum (weight, edge id) edge, a
// mutual pair keeps the lower id as root and every other chooser hooks onto
// the far component (new_grafting_edges, :73-134), hooks are jumped to roots
// (new_shortcutting_step, :254-271) and edges inside a component are dropped
// (relabelling_step / filtering_step / remove_if, :273-321, :641-649).  The
// order (weight, edge id) is strict, so the forest is the unique MSF that the
// reference's PBBS mst() (MST/src/utils.cu:794-841) returns.
//
// The whole solve is one cooperative launch (solve_kernel): its CTAs go
// through the phases together, with a grid barrier between them.
//   1. Init, and a stratified sample of the weights; every CTA then selects
//      the same weight threshold from it, so that about light_per_vertex * n
//      edges are light: the filtering step of PBBS mst() (approximate k-th
//      smallest, :805-813).
//   2. Light phase.  Round 0 streams the input and keeps the light edges;
//      later rounds walk the (small) survivor lists.  A round is three
//      phases: the edge pass (endpoints to their roots, internal edges
//      dropped, every survivor offered to both roots), the hook (a record
//      whose key won at an endpoint is that component's choice) and the
//      compress (every root that hooked is pointed at its new root).
//   3. When no light edge is left every vertex is pointed at its root and the
//      input is streamed a second time, keeping heavy edges whose endpoints
//      lie in different components (PBBS's second filter, :819-823); Boruvka
//      continues on those survivors.  An edge that is heavy and internal after
//      the light phase closes a cycle of lighter edges, so it is in no MSF:
//      the filter changes the work, not the result.
//   4. The ordered gather writes the MSF records ascending by id.
//
// A component's choice is the minimum key (w << 32 | id) offered to it, kept
// with fire-and-forget 64-bit atomicMin.  The hook runs over the survivor
// records, so the lists may be in any order, and every warp keeps its own: a
// private segment that it alone writes (dense 512-byte rows), compacts in
// place and reads back, with no slot reservation, no list shared between
// warps and no list length in memory.  best[] exists twice, one per round
// parity: the hook resets the next round's words of the components it found,
// so no pass clears them.
//
// Why one launch: the rounds after the first work on lists of a few thousand
// to a million records, where a launch (about 3.5 us of GPU time even when it
// finds nothing to do) and the list's trip through memory cost more than the
// work; a grid barrier costs 1.2 us, and lists private to a warp need no
// reservation.  Against the same phases as separate launches (one per phase
// and round, shared lists): n = 131,101, m = 2^20 uniform 592 -> 287 us; n =
// 262,147 geometric 645 -> 315 us; R-MAT 22 (67 M edges) 1314 -> 1053 us;
// n = 2,003, m = 8,009 312 -> 159 us; the canonical forest of n = 2^20,
// m = 2^23 943 -> 543 us.  Walking parent[] in the edge pass instead of the
// separate compress phase cost 3344 us on R-MAT 22: the path-halving stores
// of every record of a hub hit one word.
#include <algorithm>
#include <cstring>

#include "internal.h"

namespace phem {
namespace {

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
    uint32_t *chunk_cnt;           // MSF edges per 1024 edge ids, then their offsets within a CTA's range
    uint32_t *cta_tot;             // forest edges per CTA's chunk range
    uint32_t *giant;               // one bit per vertex: in the largest component (heavy pass)
    uint4 *list;                   // per-warp survivor segments of seg records
    uint32_t *hooked;              // per-warp segments: the roots its records hooked in a round
    uint64_t seg;
    unsigned long long *forest;
    phem_edge *out;
    Ctl *ctl;
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

// Count words for the chunks of 1024 edge ids (32 bitmap words).
__host__ __device__ inline uint64_t gather_chunks(uint64_t m) { return (m + 1023) / 1024; }

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

__device__ __forceinline__ bool grid_sync(const SolveArgs &a, SolveSmem &s, uint32_t &seq)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long v = s.acc + ((unsigned long long)s.fatal << 40);
        s.acc = 0;
        __threadfence();
        if (gridDim.x > 1) {
            unsigned long long *word = &a.ctl->bar[seq];
            v += atomicAdd(word, v + (1ull << 52)) + (1ull << 52);
            uint32_t spins = 0;
            while ((v >> 52) < gridDim.x) {
                if (++spins > kBarSpinCap) {
                    set_err(&a.ctl->err, kErrLookback);
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
__device__ __forceinline__ void acc_add(SolveSmem &s, uint32_t v)
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

// The sample's rank-th smallest weight (rank = the light edges aimed at, scaled
// to the sample): a three-digit radix select in shared memory, run by every
// CTA on the same sample instead of by one CTA and a further barrier.
//
// How many light edges pay depends on the degrees: the light phase has to
// build the component that filters the heavy edges, which takes well over n/2
// edges when all degrees are alike and far fewer when hubs collect them.  The
// sample tells the two apart: endpoints that repeat (in a hashed set of 2^18)
// several times as often as uniform ones would mean hubs.  us per solve at
// 0.5 / 1 light edges per vertex: R-MAT 22 1065 / 1102; uniform n = 2^20, m =
// 2^23 844 / 542, n = 131,101, m = 2^20 302 / 232; geometric n = 262,147
// 315 / 304.
__device__ __forceinline__ unsigned long long select_threshold(const SolveArgs &a, SolveSmem &s)
{
    uint32_t *samp = reinterpret_cast<uint32_t *>(s.warp);
    uint32_t *hist = samp + kMaxSample;
    const uint32_t S = a.nsamp, tid = threadIdx.x, lane = lane_id();
    if (tid == 0)
        s.sel_prefix = s.sel_or = s.sel_dup = 0;
    uint32_t *seen = hist;  // 2^18 bits, before the histograms
    for (uint32_t i = tid; i < kSeenWords / 4; i += blockDim.x)
        reinterpret_cast<uint4 *>(seen)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    uint32_t orv = 0, dup = 0;
    for (uint32_t i = tid; i < S; i += blockDim.x) {
        const uint32_t x = __ldcg(a.samples + i), v = __ldcg(a.samples + S + i);
        samp[i] = x;
        orv |= x;
        const uint32_t h = (v * 0x9E3779B1u) >> 14, bit = 1u << (h & 31);
        dup += (atomicOr(&seen[h >> 5], bit) & bit) != 0;
    }
    orv = __reduce_or_sync(0xffffffffu, orv);
    dup = __reduce_add_sync(0xffffffffu, dup);
    if (lane == 0) {
        atomicOr(&s.sel_or, orv);
        atomicAdd(&s.sel_dup, dup);
    }
    __syncthreads();
    if (tid == 0) {
        const float even = 0.5f * (float)S * (float)S * (1.f / (32.f * kSeenWords) + 1.f / (float)a.n);
        s.sel_rank = (uint32_t)(((float)s.sel_dup > 4.f * even + 32.f ? a.light_k : a.light_k2) * S / a.m);
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int sh = d == 0 ? 21 : (d == 1 ? 10 : 0), nb = d == 2 ? 10 : 11, hsh = sh + nb;
        __syncthreads();
        // a digit that is zero in every sample (weights below 2^21 leave the
        // top one empty) puts them all in bin 0: the prefix and rank stand
        if ((s.sel_or >> sh) == 0)
            continue;
        for (uint32_t i = tid; i < 2048; i += blockDim.x)
            hist[i] = 0;
        __syncthreads();
        const uint64_t want_hi = (uint64_t)s.sel_prefix >> hsh;
        for (uint32_t i = tid; i < S; i += blockDim.x) {
            const uint32_t x = samp[i];
            if (((uint64_t)x >> hsh) == want_hi)
                atomicAdd(&hist[(x >> sh) & ((1u << nb) - 1)], 1u);
        }
        __syncthreads();
        if (tid < 32) {
            // lane l owns bins l, l + 32, ... of each of 64 rows, row by row
            uint32_t run = 0;
            const uint32_t rank = s.sel_rank;
            for (uint32_t b0 = 0; b0 < 2048; b0 += 128) {
                const uint4 h = reinterpret_cast<const uint4 *>(hist + b0)[lane];
                const uint32_t sum = h.x + h.y + h.z + h.w;
                uint32_t incl = sum;
#pragma unroll
                for (int k = 1; k < 32; k <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, k);
                    if (lane >= (uint32_t)k)
                        incl += y;
                }
                const uint32_t excl = run + incl - sum, total = __shfl_sync(0xffffffffu, incl, 31);
                if (rank >= excl && rank < excl + sum) {
                    uint32_t c = excl, b = 0;
                    const uint32_t q[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
                    for (int k = 0; k < 3; k++)
                        if (b == (uint32_t)k && rank >= c + q[k]) {
                            c += q[k];
                            b = k + 1;
                        }
                    s.sel_prefix |= (b0 + lane * 4 + b) << sh;
                    s.sel_rank = rank - c;
                }
                run += total;
                if (rank < run)
                    break;
            }
        }
        __syncthreads();
    }
    const unsigned long long thr = (unsigned long long)s.sel_prefix << 32;
    fence_proxy_async_smem();  // the samples' space becomes bulk-copy stages
    __syncthreads();
    return thr;
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

// One tile of the caller's records.  A lane takes 4 consecutive records (6
// packed pairs): 48 bytes, read as three 16-byte shared loads (a 48-byte lane
// stride is conflict-free), so a 128-record tile costs 3 load instructions
// instead of 12.  LIGHT keeps key < threshold with the endpoints as roots
// (round 0: every vertex is its own root); otherwise keeps key >= threshold
// between different components: parent[] is fully compressed, so one hop
// reaches the root, and with use_giant a bit per vertex (in the largest
// component) settles most edges before it.
template <int KIND, bool LIGHT>
__device__ __forceinline__ void input_tile(const SolveArgs &a, SolveSmem &s, unsigned long long *best, EpWarp &w,
                                           const unsigned char *stage, bool bulk, uint64_t tbase, uint32_t rem,
                                           unsigned long long thr, bool use_giant, uint4 *list, uint32_t &filled,
                                           uint32_t &flushed, uint32_t lane, bool &any_bad)
{
    constexpr int PER = KIND == kKindMsf ? 4 : 6;
    uint32_t u[PER], v[PER], wt[PER];
    const uint32_t i0 = lane * PER;
    const uint32_t id0 = (uint32_t)tbase + i0;
    if (bulk) {
        const uint4 *q = reinterpret_cast<const uint4 *>(stage) + 3 * lane;
        const uint4 q0 = q[0], q1 = q[1], q2 = q[2];
        if (KIND == kKindMsf) {
            u[0] = q0.x, v[0] = q0.y, wt[0] = q0.z, u[1] = q0.w;
            v[1] = q1.x, wt[1] = q1.y, u[2] = q1.z, v[2] = q1.w;
            wt[2] = q2.x, u[3] = q2.y, v[3] = q2.z, wt[3] = q2.w;
        } else {
            v[0] = q0.x, u[0] = q0.y, v[1] = q0.z, u[1] = q0.w;
            v[2] = q1.x, u[2] = q1.y, v[3] = q1.z, u[3] = q1.w;
            v[PER - 2] = q2.x, u[PER - 2] = q2.y, v[PER - 1] = q2.z, u[PER - 1] = q2.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < PER; j++) {
            u[j] = v[j] = wt[j] = 0;
            if (i0 + j < rem) {
                if (KIND == kKindMsf) {
                    const uint32_t *p = static_cast<const uint32_t *>(a.e0) + 3 * (tbase + i0 + j);
                    u[j] = __ldcs(p);
                    v[j] = __ldcs(p + 1);
                    wt[j] = __ldcs(p + 2);
                } else {
                    const unsigned long long e =
                        __ldcs(static_cast<const unsigned long long *>(a.e0) + tbase + i0 + j);
                    u[j] = (uint32_t)(e >> 32);
                    v[j] = (uint32_t)e;
                }
            }
        }
    }
    uint32_t keep = 0;
#pragma unroll
    for (int j = 0; j < PER; j++) {
        if (KIND != kKindMsf)
            wt[j] = 0;
        const bool live = e0_live<KIND>(u[j], v[j]);  // records past the end read as self-loops
        const bool bad = live && max(u[j], v[j]) >= a.n;
        any_bad |= bad;
        const bool light = e0_key<KIND>(wt[j], id0 + j) < thr;
        keep |= (uint32_t)(live && !bad && (LIGHT ? light : !light)) << j;
    }
    if (!LIGHT) {
        if (use_giant) {
            uint32_t g[PER];
#pragma unroll
            for (int j = 0; j < PER; j++) {
                g[j] = 0;
                if (keep >> j & 1) {
                    const uint32_t gu = ld_par(a.giant + (u[j] >> 5)), gv = ld_par(a.giant + (v[j] >> 5));
                    g[j] = (gu >> (u[j] & 31)) & (gv >> (v[j] & 31)) & 1u;
                }
            }
#pragma unroll
            for (int j = 0; j < PER; j++)
                keep &= ~(g[j] << j);
        }
        // all records' gathers in flight together
#pragma unroll
        for (int j = 0; j < PER; j++)
            if (keep >> j & 1) {
                u[j] = ld_par(a.parent + u[j]);
                v[j] = ld_par(a.parent + v[j]);
            }
#pragma unroll
        for (int j = 0; j < PER; j++)
            if (u[j] == v[j])
                keep &= ~(1u << j);
    }
    if (!__any_sync(0xffffffffu, keep))
        return;
#pragma unroll
    for (int j = 0; j < PER; j++) {
        ring_append(w, filled, keep >> j & 1, make_uint4(u[j], v[j], wt[j], id0 + j), lane);
        if (filled - flushed >= 32)
            ring_flush<KIND>(a, s, best, list, w, flushed, 32, lane);
    }
}

// Streams the caller's records through the warp: it owns tiles gw, gw + GW,
// ... and keeps the copy of the next tile (cp.async.bulk, no multicast) in
// flight while it works on the current one, completion tracked by a
// per-stage mbarrier.  Survivors replace the warp's list.  No CTA barrier.
template <int KIND, bool LIGHT>
__device__ __forceinline__ void input_pass(const SolveArgs &a, SolveSmem &s, unsigned long long *best,
                                        unsigned long long thr, bool use_giant, WarpState &ws)
{
    constexpr uint32_t REC = KIND == kKindMsf ? 12u : 8u;
    constexpr uint32_t TILE = kEpStageBytes / REC;
    const uint32_t lane = lane_id();
    EpWarp &w = s.warp[threadIdx.x >> 5];
    const uint64_t ntiles = (a.m + TILE - 1) / TILE;
    const uint64_t full_tiles = a.m / TILE;  // the partial last tile is read directly
    const uint64_t policy = l2_evict_first();
    const char *src = static_cast<const char *>(a.e0);
    auto issue = [&](uint64_t t, int st) {  // lane 0 only
        mbar_arrive_expect_tx(reinterpret_cast<uint64_t *>(&w.bar[st]), kEpStageBytes);
        bulk_copy_g2s_hint(w.stage[st], src + t * kEpStageBytes, kEpStageBytes,
                           reinterpret_cast<uint64_t *>(&w.bar[st]), policy);
    };
    if (lane == 0 && ws.gw < full_tiles)
        issue(ws.gw, 0);
    uint32_t filled = 0, flushed = 0;  // ring cursors (warp-uniform)
    uint32_t pending = ws.gw < full_tiles ? 1u : 0u;  // bit s: a copy into stage s is in flight
    bool any_bad = false, failed = false;
    int st = 0;
    for (uint64_t t = ws.gw; t < ntiles; t += ws.GW, st ^= 1) {
        // tile t + GW goes into the other stage, which the previous tile left
        // (its reads were fenced against the async proxy before the warp
        // synchronised at the end of that tile)
        const uint64_t t2 = t + ws.GW;
        if (t2 < full_tiles) {
            if (lane == 0)
                issue(t2, st ^ 1);
            pending |= 1u << (st ^ 1);
        }
        const bool bulk = t < full_tiles;
        if (bulk) {
            if (!ep_wait(&w.bar[st], (ws.parity >> st) & 1u, &a.ctl->err)) {
                failed = true;
                break;
            }
            ws.parity ^= 1u << st;
            pending &= ~(1u << st);
        }
        const uint64_t tbase = t * TILE, left = a.m - tbase;
        const uint32_t rem = left < TILE ? (uint32_t)left : TILE;
        input_tile<KIND, LIGHT>(a, s, best, w, w.stage[st], bulk, tbase, rem, thr, use_giant, ws.list, filled,
                                flushed, lane, any_bad);
        fence_proxy_async_smem();  // this lane's reads of the stage precede its refill
        __syncwarp();
    }
    if (failed) {
        // a copy never completed (the status bit is set): wait, bounded, for
        // every copy still in flight into this warp's stages
        for (int q = 0; q < kEpStages; q++)
            if (pending & (1u << q))
                ep_wait(&w.bar[q], (ws.parity >> q) & 1u, &a.ctl->err);
        s.fatal = 1;
    } else if (filled != flushed) {
        ring_flush<KIND>(a, s, best, ws.list, w, flushed, filled - flushed, lane);
    }
    if (LIGHT && __any_sync(0xffffffffu, any_bad) && lane == 0)
        set_err(&a.ctl->err, kErrRange);
    ws.len = flushed;
    acc_add(s, lane == 0 ? flushed : 0u);
}

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
// (new_grafting_edges, MST/src/kernels.cu:73-134).  The next round's best
// word of every chooser is reset here: the components that can still get an
// offer are among them.
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
                if (A)
                    best_next[rec[q].x] = kKeyNone;
                if (B)
                    best_next[rec[q].y] = kKeyNone;
                choosers += (uint32_t)A + (uint32_t)B;
                if (KIND == kKindMsf) {
                    atomicOr(a.bitmap + (id >> 5), 1u << (id & 31));
                    atomicAdd(a.chunk_cnt + (id >> 10), 1u);
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

__device__ __forceinline__ void compress_pass(const SolveArgs &a, const WarpState &ws)
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
            y[k] = walking[k] ? ld_par(a.parent + x[k]) : 0u;
        for (uint32_t steps = 0;; steps++) {
            uint32_t p[kVItems];
#pragma unroll
            for (int k = 0; k < kVItems; k++)
                p[k] = !walking[k] ? y[k] : (steps < 8 ? ld_par(a.parent + y[k]) : __ldcg(a.parent + y[k]));
            bool any = false;
#pragma unroll
            for (int k = 0; k < kVItems; k++) {
                walking[k] = walking[k] && p[k] != y[k];
                if (walking[k])
                    a.parent[x[k]] = p[k];
                y[k] = p[k];
                any |= walking[k];
            }
            if (!any)
                break;
            if (steps > a.n) {
                set_err(&a.ctl->err, kErrChase);
                break;
            }
        }
    }
}

// Every vertex pointed at its root (before the heavy pass, which then
// relabels endpoints in one hop), roots' next best words reset, and the giant
// component's bits.  The giant is the component that most of 32 sampled
// edges' endpoints lie in (a warp per CTA walks them; every CTA finds the
// same one, roots being final here).  Returns whether it is worth testing.
constexpr uint32_t kGiantMinN = 1u << 15;  // below it parent[] itself is served by L1

__device__ __forceinline__ bool full_compress(const SolveArgs &a, SolveSmem &s, unsigned long long *best_next,
                                           bool packed, bool want_giant)
{
    const uint32_t lane = lane_id();
    if (want_giant && threadIdx.x < 32) {
        const uint64_t pos = sample_pos(lane, 32, a.m);
        const uint32_t *e = static_cast<const uint32_t *>(a.e0);
        // endpoints alternate; packed pairs hold u in the high word
        uint32_t x = packed ? __ldg(e + 2 * pos + (lane & 1)) : __ldg(e + 3 * pos + (lane & 1));
        if (x >= a.n)
            x = 0;
        for (uint32_t steps = 0; steps <= a.n; steps++) {
            const uint32_t p = ld_par(a.parent + x);
            if (p == x)
                break;
            x = p;
        }
        const unsigned peers = __match_any_sync(0xffffffffu, x);
        const uint32_t top = __reduce_max_sync(0xffffffffu, ((uint32_t)__popc(peers) << 5) | (31u - lane));
        const uint32_t root = __shfl_sync(0xffffffffu, x, 31 - (top & 31));
        if (lane == 0) {
            s.sel_prefix = root;
            s.sel_rank = top >> 5;
        }
    }
    __syncthreads();
    const uint32_t giant = want_giant ? s.sel_prefix : 0;
    const bool use_giant = want_giant && s.sel_rank >= 8;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x * kVItems;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x * kVItems; i0 < a.n; i0 += step) {
        bool walking[kVItems];
        uint32_t x[kVItems], y[kVItems], y0[kVItems];
        // the vertices' walks advance in lockstep, so their dependent loads
        // are in flight together
#pragma unroll
        for (int k = 0; k < kVItems; k++) {
            const uint64_t i = i0 + k * blockDim.x + threadIdx.x;
            walking[k] = i < a.n;
            x[k] = walking[k] ? (uint32_t)i : 0u;
        }
#pragma unroll
        for (int k = 0; k < kVItems; k++)
            y0[k] = y[k] = ld_par(a.parent + x[k]);
        for (uint32_t steps = 0;; steps++) {
            uint32_t p[kVItems];
#pragma unroll
            for (int k = 0; k < kVItems; k++)
                p[k] = walking[k] ? ld_par(a.parent + y[k]) : y[k];
            bool any = false;
#pragma unroll
            for (int k = 0; k < kVItems; k++) {
                walking[k] = walking[k] && p[k] != y[k];
                y[k] = p[k];
                any |= walking[k];
            }
            if (!any)
                break;
            if (steps > a.n) {
                set_err(&a.ctl->err, kErrChase);
                break;
            }
        }
#pragma unroll
        for (int k = 0; k < kVItems; k++) {
            const uint64_t i = i0 + k * blockDim.x + threadIdx.x;
            if (i < a.n) {
                if (y0[k] != y[k])
                    a.parent[x[k]] = y[k];
                if (y[k] == x[k])
                    best_next[x[k]] = kKeyNone;
            }
            if (use_giant) {  // blockDim.x and i0 are multiples of 32
                const unsigned bits = __ballot_sync(0xffffffffu, i < a.n && y[k] == giant);
                if (lane == 0 && i < a.n)
                    a.giant[i >> 5] = bits;
            }
        }
    }
    return use_giant;
}

// ---- ordered gather ----------------------------------------------------------

// Offsets of the chunks' records.  CTA c scans the counts of its range of
// chunks in place (exclusive, within the range) and publishes the range's
// total; after the barrier every CTA scans the totals for itself.
__device__ __forceinline__ void gather_scan(const SolveArgs &a, SolveSmem &s, uint64_t per)
{
    const uint64_t chunks = gather_chunks(a.m);
    const uint64_t c0 = blockIdx.x * per, c1 = min(c0 + per, chunks);
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t carry = 0;
    for (uint64_t c = c0; c < c1; c += blockDim.x) {
        const uint64_t i = c + threadIdx.x;
        const uint32_t v = i < c1 ? __ldcg(a.chunk_cnt + i) : 0u;
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
            a.chunk_cnt[i] = carry + s.scan[warp] + x - v;
        carry += s.scan[kSolveWarps];
        __syncthreads();  // s.scan is reused
    }
    if (threadIdx.x == 0)
        a.cta_tot[blockIdx.x] = carry;
}

// MSF records ascending by id: every warp takes whole chunks of 1024 edge
// ids, ranks their 32 bitmap words' bits with a warp scan and gathers its
// records (12-byte random reads of the input, four per lane in flight) to
// out[offset + rank]; the total weight is added up on the way.
__device__ __forceinline__ void gather_pass(const SolveArgs &a, SolveSmem &s, uint64_t per)
{
    const uint64_t words = (a.m + 31) / 32, chunks = gather_chunks(a.m);
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (warp == 0) {
        uint32_t run = 0;
        for (uint32_t c0 = 0; c0 < gridDim.x; c0 += 32) {
            const uint32_t c = c0 + lane;
            const uint32_t v = c < gridDim.x ? __ldcg(a.cta_tot + c) : 0u;
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
        if (blockIdx.x == 0 && lane == 0)
            a.ctl->msf_count = run;
    }
    __syncthreads();
    const uint32_t *E = static_cast<const uint32_t *>(a.e0);
    unsigned long long wsum = 0;
    const uint64_t gw = (uint64_t)blockIdx.x * nw + warp, GW = (uint64_t)gridDim.x * nw;
    for (uint64_t c = gw; c < chunks; c += GW) {
        const uint64_t wd = c * 32 + lane;
        uint32_t bits = wd < words ? __ldcg(a.bitmap + wd) : 0u;
        const uint32_t k = __popc(bits);
        uint32_t incl = k;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d)
                incl += y;
        }
        uint32_t pos = __ldcg(a.chunk_cnt + c) + s.pref[c / per] + (incl - k);
        while (bits) {
            uint32_t id[4];
            phem_edge e[4];
            int cnt = 0;
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (bits) {
                    id[q] = (uint32_t)(wd * 32 + (__ffs(bits) - 1));
                    bits &= bits - 1;
                    cnt = q + 1;
                }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (q < cnt) {
                    const uint64_t i3 = (uint64_t)id[q] * 3;
                    e[q].u = __ldg(E + i3);
                    e[q].v = __ldg(E + i3 + 1);
                    e[q].w = __ldg(E + i3 + 2);
                }
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (q < cnt) {
                    if (a.out)
                        a.out[pos] = e[q];
                    pos++;
                    wsum += e[q].w;
                }
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
        wsum += __shfl_xor_sync(0xffffffffu, wsum, d);
    if (lane == 0)
        s.red[warp] = wsum;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (uint32_t i = 0; i < nw; i++)
            t += s.red[i];
        if (t)
            atomicAdd(&a.ctl->msf_total, t);
    }
}

// ---- the solve ---------------------------------------------------------------

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

template <int KIND>
__global__ void __launch_bounds__(kSolveThreads, 1) solve_kernel(const __grid_constant__ SolveArgs a)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    SolveSmem &s = *reinterpret_cast<SolveSmem *>(s_raw);
    Ctl *ctl = a.ctl;
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, nw = blockDim.x >> 5;
    const bool lead = blockIdx.x == 0 && tid == 0;
    uint32_t seq = 0, marks = 0;
    auto stamp = [&](uint32_t phase) {
        if (a.timing && lead && marks < kMaxPhases) {
            uint64_t t;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            ctl->stamp[marks] = t;
            ctl->phase_of[marks] = phase;
            marks++;
            ctl->stamps = marks;
        }
    };
    stamp(kKernelCount);
    // init
    {
        const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + tid, T = (uint64_t)gridDim.x * blockDim.x;
        for (uint64_t i = g; i < a.nsamp; i += T) {
            const uint32_t *e = static_cast<const uint32_t *>(a.e0) + sample_pos((uint32_t)i, a.nsamp, a.m) * 3;
            a.samples[i] = __ldg(e + 2);
            a.samples[a.nsamp + i] = __ldg(e + (i & 1));
        }
        for (uint64_t x = g; x < a.n; x += T) {
            a.parent[x] = (uint32_t)x;
            a.best[x] = kKeyNone;
            if (KIND == kKindPacked && a.forest)
                a.forest[x] = kForestEmpty;
        }
        if (KIND == kKindMsf) {
            const uint64_t words = (a.m + 31) / 32, chunks = gather_chunks(a.m);
            for (uint64_t i = g; i < words; i += T)
                a.bitmap[i] = 0;
            for (uint64_t i = g; i < chunks; i += T)
                a.chunk_cnt[i] = 0;
        }
        if (tid == 0) {
            s.acc = 0;
            s.fatal = 0;
        }
        offers_reset(s.oc);
    }
    if (!grid_sync(a, s, seq))
        return;
    stamp(kKInit);
    unsigned long long thr = a.threshold;
    if (a.nsamp) {
        thr = select_threshold(a, s);
        stamp(kKSelect);
    }
    if (lane == 0) {  // after the select, whose samples shared this space
        for (int q = 0; q < kEpStages; q++)
            mbar_init(reinterpret_cast<uint64_t *>(&s.warp[warp].bar[q]), 1);
        fence_mbar_init();
    }
    __syncwarp();
    WarpState ws;
    ws.gw = blockIdx.x * nw + warp;
    ws.GW = gridDim.x * nw;
    ws.len = 0;
    ws.parity = 0;
    ws.hooks = 0;
    ws.list = a.list + (uint64_t)ws.gw * a.seg;
    ws.hooked = a.hooked + (uint64_t)ws.gw * a.seg;
    uint32_t r = 0, src = kSrcLight, light_rounds = 0;
    bool use_giant = false;
    for (;;) {
        unsigned long long *best = a.best + (r & 1) * a.best_stride, *next = a.best + ((r + 1) & 1) * a.best_stride;
        if (src == kSrcList)
            list_pass<KIND>(a, s, best, ws);
        else if (src == kSrcLight)
            input_pass<KIND, true>(a, s, best, thr, false, ws);
        else
            input_pass<KIND, false>(a, s, best, thr, use_giant, ws);
        offers_flush(s.oc, best);
        if (!grid_sync(a, s, seq))
            return;
        const unsigned long long live = s.sum;
        stamp(kKEdgePass);
        if (lead)
            ctl->m_r[r] = live;
        if (live > 0) {
            hook_pass<KIND>(a, s, best, next, ws);
            if (!grid_sync(a, s, seq))
                return;
            if (lead)
                ctl->n_r[r] = s.sum;
            stamp(kKHook);
            compress_pass(a, ws);
            if (!grid_sync(a, s, seq))
                return;
            stamp(kKCompress);
            src = kSrcList;
        } else {
            if (light_rounds) {  // the heavy phase ran dry
                r++;
                break;
            }
            light_rounds = r + 1;
            if (thr == kKeyNone) {
                r++;
                break;
            }
            use_giant = full_compress(a, s, next, KIND == kKindPacked, a.n >= kGiantMinN);
            if (!grid_sync(a, s, seq))
                return;
            stamp(kKCompress);
            src = kSrcHeavy;
        }
        if (++r >= PHEM_MAX_ROUNDS) {
            if (lead)
                set_err(&ctl->err, kErrRounds);
            break;
        }
    }
    if (lead) {
        ctl->round = r;
        ctl->light_rounds = light_rounds;
        ctl->threshold = thr;
    }
    if (KIND == kKindMsf && a.gather) {
        const uint64_t per = max((gather_chunks(a.m) + gridDim.x - 1) / gridDim.x, (uint64_t)1);
        gather_scan(a, s, per);
        if (!grid_sync(a, s, seq))
            return;
        gather_pass(a, s, per);
        stamp(kKGather);
    }
}

// Light/heavy split: about lpv * n light edges, and only when the input is at
// least filter_min_ratio times that large (0: no split).
uint64_t light_edges(phem_context *ctx, double lpv, uint64_t m, uint64_t n)
{
    const uint64_t k = (uint64_t)(lpv * (double)n);
    return lpv > 0 && (double)m >= ctx->tune_filter_min_ratio * (double)k ? k : 0;
}

// Below this many edges the weighted solve runs unfiltered: a light phase's
// rounds cost their barriers whatever they find.  us per solve without / with
// the filter: m = 100,003 137 / 152, m = 200,000 163 / 188, m = 2^20 276 / 238.
constexpr uint64_t kFilterMinEdges = 240000;

// Sampled weights: enough that the light count is within a few per cent of
// its aim where it matters (a small input's select is part of its latency).
uint32_t sample_count(uint64_t m) { return m >= (1u << 22) ? kMaxSample : 2048; }

// Records of one warp's list segment: what its tiles can hold.
uint64_t seg_records(uint64_t m, uint32_t warps, uint32_t rec_bytes)
{
    const uint64_t tile = kEpStageBytes / rec_bytes, tiles = (m + tile - 1) / tile;
    return (tiles + warps - 1) / warps * tile;
}

template <int KIND>
phem_status setup_kernel(phem_context *ctx)
{
    PHEM_CUDA_TRY(cudaFuncSetAttribute(solve_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(SolveSmem)));
    int per_sm = 0;
    PHEM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, solve_kernel<KIND>,
                                                                kSolveThreads, sizeof(SolveSmem)));
    if (per_sm < 1) {
        set_error("msf: the solve kernel does not fit on an SM");
        return PHEM_ERR_UNSUPPORTED;
    }
    return PHEM_OK;
}

// CTAs and threads of a solve.  A warp gets at least one tile; a small input
// runs more CTAs of fewer warps (more SMs' load queues, and a block barrier
// among fewer warps), a large one needs the warps.  us per solve with 256 /
// 512 / 1024 threads: m = 100,003 137 / 138 / 161; m = 200,000 183 / 163 /
// 198; m = 2^20 250 / 238 / 250; m = 4,000,000 442 / 373 / 361.
struct SolveGrid {
    uint32_t blocks;
    int threads;
};
SolveGrid solve_grid(uint64_t m, uint32_t rec_bytes, int sm_count, int max_groups)
{
    const uint64_t tile = kEpStageBytes / rec_bytes, tiles = (m + tile - 1) / tile;
    const int groups = tiles <= 8 * (uint64_t)sm_count ? 1 : (tiles <= 64 * (uint64_t)sm_count ? 2 : 4);
    SolveGrid g;
    g.threads = 256 * std::min(groups, max_groups);
    const uint64_t warps = (uint64_t)g.threads / 32;
    g.blocks = (uint32_t)std::max<uint64_t>(
        1, std::min({(tiles + warps - 1) / warps, (uint64_t)sm_count, (uint64_t)kMaxGrid}));
    return g;
}

template <int KIND>
phem_status run_impl(phem_context *ctx, MsfPlan &plan)
{
    cudaStream_t st = ctx->stream;
    if (!(ctx->kernels_ready & (1u << KIND))) {
        PHEM_TRY(setup_kernel<KIND>(ctx));
        ctx->kernels_ready |= 1u << KIND;
    }
    SolveArgs a{};
    a.e0 = plan.e0;
    a.m = plan.m;
    a.n = plan.n;
    a.parent = plan.parent;
    a.best = plan.best;
    a.best_stride = plan.best_stride;
    a.samples = plan.samples;
    a.bitmap = plan.bitmap;
    a.chunk_cnt = plan.chunk_cnt;
    a.cta_tot = plan.cta_tot;
    a.giant = plan.giant;
    a.list = plan.list;
    a.hooked = plan.hooked;
    a.forest = reinterpret_cast<unsigned long long *>(plan.forest);
    a.out = plan.out;
    a.gather = plan.gather;
    a.ctl = ctx->ctl;
    a.timing = ctx->profiling;
    // packed edges: the first k by index are light; the canonical forest's
    // slots follow from the rounds, so this rule is the same at every size
    const uint64_t k = KIND == kKindPacked ? canonical_light(ctx, plan.m, plan.n)
                       : plan.m < kFilterMinEdges
                           ? 0
                           : light_edges(ctx, ctx->tune_light_per_vertex, plan.m, plan.n);
    a.light_k = k ? k : plan.m;
    a.light_k2 = light_edges(ctx, 2 * ctx->tune_light_per_vertex, plan.m, plan.n);
    if (!a.light_k2)
        a.light_k2 = a.light_k;
    a.threshold = k && KIND == kKindPacked ? k : kKeyNone;
    a.nsamp = k && KIND == kKindMsf ? sample_count(plan.m) : 0;
    constexpr uint32_t rec_bytes = KIND == kKindMsf ? 12 : 8;
    const SolveGrid g = solve_grid(plan.m, rec_bytes, ctx->sm_count, ctx->tune_edge_ctas);
    a.seg = seg_records(plan.m, g.blocks * (uint32_t)(g.threads / 32), rec_bytes);
    PHEM_CUDA_TRY(cudaMemsetAsync(ctx->ctl, 0, sizeof(Ctl), st));
    void *params[] = {&a};
    KernelScope ks(ctx, kKSolve);
    if (g.blocks == 1)  // one CTA waits for no other
        PHEM_CUDA_TRY(cudaLaunchKernel(solve_kernel<KIND>, dim3(1), dim3(g.threads), params, sizeof(SolveSmem), st));
    else
        PHEM_CUDA_TRY(cudaLaunchCooperativeKernel(solve_kernel<KIND>, dim3(g.blocks), dim3(g.threads), params,
                                                  sizeof(SolveSmem), st));
    return PHEM_OK;
}

}  // namespace

uint64_t canonical_light(phem_context *ctx, uint64_t m, uint64_t n)
{
    return light_edges(ctx, ctx->tune_canonical_light, m, n);
}

// Records all segments may need: every edge plus one tile per warp.
uint64_t list_capacity(uint64_t m, int sm_count)
{
    return m + ((uint64_t)sm_count * kSolveWarps + 1) * (kEpStageBytes / 8);
}

phem_status msf_finish(phem_context *ctx, uint32_t *rounds_out, const char *what)
{
    PHEM_CUDA_TRY(cudaMemcpyAsync(ctx->h_ctl, ctx->ctl, ctx->profiling ? sizeof(Ctl) : offsetof(Ctl, bar),
                                  cudaMemcpyDeviceToHost, ctx->stream));
    PHEM_TRY(stream_wait(ctx));
    const Ctl &h = *ctx->h_ctl;
    if (ctx->profiling)
        for (uint32_t i = 1; i < h.stamps && i < kMaxPhases; i++)
            log_phase(ctx, (int)h.phase_of[i], (float)(h.stamp[i] - h.stamp[i - 1]) * 1e-6f);
    if (rounds_out)
        *rounds_out = h.round;
    return ctl_status(h.err, what);
}

// Workspace of one solve (msf_plan carves in the same order): parent (4n),
// best (2 x 8n), the MSF bitmap (m / 8), the giant bits (n / 8) and the
// survivor segments (16 bytes per record).
static size_t msf_carve(uint64_t m, uint32_t n, int sm_count, char *base, MsfPlan *p)
{
    Carve c;
    const uint64_t stride = ((uint64_t)n + 31) & ~31ull;
    const size_t o_par = c.take<uint32_t>(n), o_best = c.take<unsigned long long>(2 * stride),
                 o_samp = c.take<uint32_t>(2 * kMaxSample), o_bm = c.take<uint32_t>((m + 31) / 32 + 4),
                 o_cnt = c.take<uint32_t>(gather_chunks(m) + 4), o_tot = c.take<uint32_t>(kMaxGrid),
                 o_gi = c.take<uint32_t>(stride / 32 + 4), o_list = c.take<uint4>(list_capacity(m, sm_count)),
                 o_hk = c.take<uint32_t>(list_capacity(m, sm_count));
    if (p) {
        p->parent = reinterpret_cast<uint32_t *>(base + o_par);
        p->best = reinterpret_cast<unsigned long long *>(base + o_best);
        p->best_stride = stride;
        p->samples = reinterpret_cast<uint32_t *>(base + o_samp);
        p->bitmap = reinterpret_cast<uint32_t *>(base + o_bm);
        p->chunk_cnt = reinterpret_cast<uint32_t *>(base + o_cnt);
        p->cta_tot = reinterpret_cast<uint32_t *>(base + o_tot);
        p->giant = reinterpret_cast<uint32_t *>(base + o_gi);
        p->list = reinterpret_cast<uint4 *>(base + o_list);
        p->hooked = reinterpret_cast<uint32_t *>(base + o_hk);
    }
    return c.off;
}

size_t msf_workspace_bytes(uint64_t m, uint32_t n, int sm_count) { return msf_carve(m, n, sm_count, nullptr, nullptr); }

phem_status msf_plan(phem_context *ctx, const void *d_e0, uint64_t m, uint32_t n, size_t extra_bytes, MsfPlan *plan,
                     size_t *extra_off)
{
    Carve c;
    c.off = msf_workspace_bytes(m, n, ctx->sm_count);
    const size_t extra_at = c.take<uint8_t>(extra_bytes);
    PHEM_TRY(ws_reserve(ctx, c.off));
    msf_carve(m, n, ctx->sm_count, static_cast<char *>(ctx->ws), plan);
    plan->e0 = d_e0;
    plan->m = m;
    plan->n = n;
    plan->forest = nullptr;
    plan->out = nullptr;
    plan->gather = 0;
    if (extra_off)
        *extra_off = extra_at;
    return PHEM_OK;
}

phem_status msf_run(phem_context *ctx, int kind, MsfPlan &plan)
{
    return kind == kKindMsf ? run_impl<kKindMsf>(ctx, plan) : run_impl<kKindPacked>(ctx, plan);
}

}  // namespace phem
