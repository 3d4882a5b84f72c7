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
// and round, shared lists), us per call, then with what the comments below
// measure: n = 131,101, m = 2^20 uniform 592 -> 287 -> 211; n = 262,147
// geometric 645 -> 315 -> 273; R-MAT 22 (67 M edges) 1314 -> 1053 -> 980; the
// canonical forest of n = 2^20, m = 2^23 943 -> 543 -> 514.  Walking parent[] in the edge pass instead of the
// separate compress phase cost 3344 us on R-MAT 22: the path-halving stores
// of every record of a hub hit one word.
#include <algorithm>
#include <cstring>

#include "solve.cuh"

namespace phem {
namespace {

// Count words for the chunks of 1024 edge ids (32 bitmap words).
__host__ __device__ inline uint64_t gather_chunks(uint64_t m) { return (m + 1023) / 1024; }

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
    // packed pairs are light by position: each pass reads its side of the list
    const bool split = KIND == kKindPacked && thr != kKeyNone;
    const uint64_t begin = !LIGHT && split ? thr / TILE : 0;
    const uint64_t ntiles = LIGHT && split ? (thr + TILE - 1) / TILE : (a.m + TILE - 1) / TILE;
    const uint64_t full_tiles = min(a.m / TILE, ntiles);  // the partial last tile is read directly
    const uint64_t first = begin + ws.gw;
    const uint64_t policy = l2_evict_first();
    const char *src = static_cast<const char *>(a.e0);
    auto issue = [&](uint64_t t, int st) {  // lane 0 only
        mbar_arrive_expect_tx(reinterpret_cast<uint64_t *>(&w.bar[st]), kEpStageBytes);
        bulk_copy_g2s_hint(w.stage[st], src + t * kEpStageBytes, kEpStageBytes,
                           reinterpret_cast<uint64_t *>(&w.bar[st]), policy);
    };
    if (lane == 0 && first < full_tiles)
        issue(first, 0);
    uint32_t filled = 0, flushed = 0;  // ring cursors (warp-uniform)
    uint32_t pending = first < full_tiles ? 1u : 0u;  // bit s: a copy into stage s is in flight
    bool any_bad = false, failed = false;
    int st = 0;
    for (uint64_t t = first; t < ntiles; t += ws.GW, st ^= 1) {
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
    if ((LIGHT || split) && __any_sync(0xffffffffu, any_bad) && lane == 0)
        set_err(&a.ctl->err, kErrRange);
    ws.len = flushed;
    acc_add(s, lane == 0 ? flushed : 0u);
}

// The giant component's root, for the heavy pass's vertex bits: the component
// that most of 32 sampled edges' endpoints lie in (a warp per CTA walks them
// between rounds, so every CTA finds the same one).  Returns whether the bits
// are worth testing.
constexpr uint32_t kGiantMinN = 1u << 15;  // below it parent[] itself is served by L1

__device__ __forceinline__ bool find_giant(const SolveArgs &a, SolveSmem &s, bool packed, uint32_t *root)
{
    const uint32_t lane = lane_id();
    if (threadIdx.x < 32) {
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
        const uint32_t r = __shfl_sync(0xffffffffu, x, 31 - (top & 31));
        if (lane == 0) {
            s.sel_prefix = r;
            s.sel_rank = top >> 5;
        }
    }
    __syncthreads();
    *root = s.sel_prefix;
    return s.sel_rank >= 8;
}

// ---- ordered gather ----------------------------------------------------------

// MSF records ascending by id: every warp takes whole chunks of 1024 edge
// ids, ranks their 32 bitmap words' bits with a warp scan and gathers its
// records (12-byte random reads of the input, four per lane in flight) to
// out[offset + rank]; the total weight is added up on the way.
__device__ __forceinline__ void gather_pass(const SolveArgs &a, SolveSmem &s, uint64_t per)
{
    const uint64_t words = (a.m + 31) / 32, chunks = gather_chunks(a.m);
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t count = prefix_totals(s, a.cta_tot);
    if (blockIdx.x == 0 && threadIdx.x == 0)
        a.ctl->msf_count = count;
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
        uint32_t pos = __ldcg(a.chunk_off + c) + s.pref[c / per] + (incl - k);
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

// ---- min-id labels (packed edges) ----------------------------------------------
//
// Every vertex to its root, and the smallest id of each component to its
// root's label, which the other vertices then copy.  Lanes hold consecutive
// vertices, so of the lanes that share a root the lowest has the smallest id:
// only it reads the guard (through L1: a stale value is never below the true
// minimum) and offers.  2^20 vertices, 2^23 edges, us per call: as four launches
// behind the solve 528, here 514 (inlined, with more spills, 532).
__device__ __noinline__ void min_ids(const SolveArgs &a, SolveSmem &s)
{
    full_compress(a.parent, a.n, nullptr, nullptr, 0, false, &a.ctl->err);
    uint32_t *mins = reinterpret_cast<uint32_t *>(a.label);
    uint32_t roots = 0;
    // full_compress's own vertices, whose roots this thread wrote
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x * kVItems;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x * kVItems; i0 < a.n; i0 += step) {
        uint32_t r[kVItems], seen[kVItems];
#pragma unroll
        for (int k = 0; k < kVItems; k++) {
            const uint64_t i = i0 + k * blockDim.x + threadIdx.x;
            r[k] = i < a.n ? a.parent[i] : 0xffffffffu;
            roots += i < a.n && r[k] == i;
            const unsigned peers = __match_any_sync(0xffffffffu, r[k]);
            const bool first = i < a.n && (int)lane_id() == __ffs(peers) - 1;
            seen[k] = first ? __ldca(mins + r[k]) : 0u;
        }
#pragma unroll
        for (int k = 0; k < kVItems; k++) {
            const uint32_t i = (uint32_t)(i0 + k * blockDim.x + threadIdx.x);
            if (i < seen[k])
                atomicMin(mins + r[k], i);
        }
    }
    acc_add(s, roots);
}

// ---- the solve ---------------------------------------------------------------

template <int KIND>
__global__ void __launch_bounds__(kSolveThreads, 1) solve_kernel(const __grid_constant__ SolveArgs a)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    SolveSmem &s = *reinterpret_cast<SolveSmem *>(s_raw);
    Ctl *ctl = a.ctl;
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, nw = blockDim.x >> 5;
    const bool lead = blockIdx.x == 0 && tid == 0;
    uint32_t seq = 0;
    PhaseClock clock(ctl, a.timing);
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
            if (KIND == kKindPacked && a.label)
                a.label[x] = -1;  // the largest unsigned id
        }
        if (KIND == kKindMsf) {
            const uint64_t words = (a.m + 31) / 32;
            for (uint64_t i = g; i < words; i += T)
                a.bitmap[i] = 0;
        }
        if (tid == 0) {
            s.acc = 0;
            s.fatal = 0;
        }
        offers_reset(s.oc);
    }
    if (!grid_sync(ctl, s, seq))
        return;
    clock.stamp(kKInit);
    unsigned long long thr = a.threshold;
    if (a.nsamp) {
        thr = select_threshold(a, s);
        clock.stamp(kKSelect);
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
        if (!grid_sync(ctl, s, seq))
            return;
        const unsigned long long live = s.sum;
        clock.stamp(kKEdgePass);
        if (lead)
            ctl->m_r[r] = live;
        if (live > 0) {
            hook_pass<KIND>(a, s, best, next, ws);
            if (!grid_sync(ctl, s, seq))
                return;
            if (lead)
                ctl->n_r[r] = s.sum;
            clock.stamp(kKHook);
            compress_pass(a.parent, a.n, &ctl->err, ws);
            if (!grid_sync(ctl, s, seq))
                return;
            clock.stamp(kKCompress);
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
            uint32_t giant = 0;
            use_giant = a.n >= kGiantMinN && find_giant(a, s, KIND == kKindPacked, &giant);
            full_compress(a.parent, a.n, next, a.giant, giant, use_giant, &ctl->err);
            if (!grid_sync(ctl, s, seq))
                return;
            clock.stamp(kKCompress);
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
        // a chunk's count is its 32 bitmap words' bits: a warp reads its 32
        // lanes' chunks one after the other
        const uint64_t words = (a.m + 31) / 32;
        count_scan(s, a.chunk_off, gather_chunks(a.m), per, a.cta_tot, [&](uint64_t c, uint64_t, uint64_t end) {
            const uint64_t first = c + warp * 32;
            uint32_t mine = 0;
#pragma unroll 8
            for (uint32_t k = 0; k < 32; k++) {
                const uint64_t w = (first + k) * 32 + lane;
                const uint32_t bits = first + k < end && w < words ? __ldcg(a.bitmap + w) : 0u;
                const uint32_t sum = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(bits));
                mine = lane == k ? sum : mine;
            }
            return mine;
        });
        if (!grid_sync(ctl, s, seq))
            return;
        gather_pass(a, s, per);
        clock.stamp(kKGather);
    }
    if (KIND == kKindPacked && a.label) {
        min_ids(a, s);
        if (!grid_sync(ctl, s, seq))
            return;
        if (lead)
            ctl->misc[0] = s.sum;  // components
        const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
        for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + tid; x < a.n; x += step) {
            const uint32_t root = __ldcg(a.parent + x);
            if (root != x)
                a.label[x] = __ldcg(a.label + root);
        }
        clock.stamp(kKCcLabel);
    }
    publish_ctl(ctl, a.publish);
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
    a.chunk_off = plan.chunk_off;
    a.cta_tot = plan.cta_tot;
    a.giant = plan.giant;
    a.list = plan.list;
    a.hooked = plan.hooked;
    a.forest = reinterpret_cast<unsigned long long *>(plan.forest);
    a.out = plan.out;
    a.gather = plan.gather;
    a.label = plan.label;
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
    // a cooperative launch waits until all its CTAs fit at once, and beside a
    // server's other work half of the SMs are free sooner and leave the rest to
    // it: mixed requests at saturation 3026 per second with all SMs, 3057 with
    // half of them (MSF as a launch per phase 2936)
    const int sms = ctx->shares_device ? std::max(1, ctx->sm_count / 2) : ctx->sm_count;
    const SolveGrid g = solve_grid(plan.m, rec_bytes, sms, ctx->tune_edge_ctas);
    a.seg = seg_records(plan.m, g.blocks * (uint32_t)(g.threads / 32), rec_bytes);
    PHEM_TRY(solve_ctl(ctx, &a.ctl, &a.publish));
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

phem_status solve_ctl(phem_context *ctx, Ctl **ctl, Ctl **publish)
{
    // a profiled solve's time stamps stay in the block; and behind a solve that
    // may still publish its own results, these are copied after it
    ctx->publishes = !ctx->profiling && !ctx->unfinished;
    *ctl = ctx->publishes ? ctx->solve_ctl : ctx->ctl;
    *publish = ctx->publishes ? ctx->h_ctl : nullptr;
    if (!ctx->publishes || !ctx->solve_ctl_zero)
        PHEM_CUDA_TRY(cudaMemsetAsync(*ctl, 0, sizeof(Ctl), ctx->stream));
    if (ctx->publishes) {
        ctx->solve_ctl_zero = false;
        ctx->h_ctl->err = kCtlPending;
    }
    return PHEM_OK;
}

phem_status msf_finish(phem_context *ctx, uint32_t *rounds_out, const char *what)
{
    const bool published = ctx->publishes;
    ctx->publishes = false;
    if (!published)
        PHEM_CUDA_TRY(cudaMemcpyAsync(ctx->h_ctl, ctx->ctl, ctx->profiling ? sizeof(Ctl) : offsetof(Ctl, bar),
                                      cudaMemcpyDeviceToHost, ctx->stream));
    PHEM_TRY(stream_wait(ctx));
    const Ctl &h = *ctx->h_ctl;
    if (published) {
        ctx->solve_ctl_zero = h.err != kCtlPending;
        if (!ctx->solve_ctl_zero) {  // gave up at a barrier
            PHEM_CUDA_TRY(cudaMemcpyAsync(ctx->h_ctl, ctx->solve_ctl, offsetof(Ctl, bar), cudaMemcpyDeviceToHost,
                                          ctx->stream));
            PHEM_TRY(stream_wait(ctx));
        }
    }
    if (!published && ctx->profiling)
        for (uint32_t i = 1; i < h.stamps && i < kMaxPhases; i++)
            log_phase(ctx, (int)h.phase_of[i], (float)(h.stamp[i] - h.stamp[i - 1]) * 1e-6f);
    if (rounds_out)
        *rounds_out = h.round;
    return ctl_status(h.err, what);
}

// Workspace of one solve (msf_plan carves in the same order): parent (4n),
// best (8n), the MSF bitmap (m / 8), the giant bits (n / 8) and the survivor
// segments (20 bytes per record), then the caller's extra area.  The second
// best array of a weighted solve lies in the extra area's start, where the
// staged MSF records go (12n): they are written behind the rounds.  The packed
// kind's extra area holds arrays that the rounds write, so it gets its own.
static size_t msf_carve(uint64_t m, uint32_t n, int sm_count, int bests, char *base, MsfPlan *p)
{
    Carve c;
    const uint64_t stride = ((uint64_t)n + 31) & ~31ull;
    const size_t o_par = c.take<uint32_t>(n), o_best = c.take<unsigned long long>(bests * stride),
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
        p->chunk_off = reinterpret_cast<uint32_t *>(base + o_cnt);
        p->cta_tot = reinterpret_cast<uint32_t *>(base + o_tot);
        p->giant = reinterpret_cast<uint32_t *>(base + o_gi);
        p->list = reinterpret_cast<uint4 *>(base + o_list);
        p->hooked = reinterpret_cast<uint32_t *>(base + o_hk);
    }
    return c.off;
}

size_t msf_workspace_bytes(uint64_t m, uint32_t n, int sm_count)
{
    return msf_carve(m, n, sm_count, 1, nullptr, nullptr);
}

phem_status msf_plan(phem_context *ctx, int kind, uint64_t m, uint32_t n, size_t extra_bytes, size_t out_off,
                     MsfPlan *plan, size_t *extra_off)
{
    const int bests = kind == kKindMsf ? 1 : 2;
    const size_t second = bests == 1 ? out_off + 8 * (((size_t)n + 31) & ~size_t(31)) : 0;
    Carve c;
    c.off = msf_carve(m, n, ctx->sm_count, bests, nullptr, nullptr);
    const size_t extra_at = c.take<uint8_t>(std::max(extra_bytes, second));
    PHEM_TRY(ws_reserve(ctx, c.off));
    msf_carve(m, n, ctx->sm_count, bests, static_cast<char *>(ctx->ws), plan);
    if (bests == 1)
        plan->best_stride = (extra_at + out_off - (reinterpret_cast<char *>(plan->best) - static_cast<char *>(ctx->ws))) /
                            sizeof(unsigned long long);
    plan->e0 = nullptr;
    plan->m = m;
    plan->n = n;
    plan->forest = nullptr;
    plan->label = nullptr;
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
