// cc_grid.cu -- connected components + spanning forest of device-resident edges.
//
// Same arithmetic as cc.cu (larger root hooked under the smaller, forest[hooked
// root] = edge, label = root; CC/ExternalSpanningTree.cu:27-116,
// CC/GPUSpanningTree.cu:24-140) and the same schedule -- a prefix of about one
// edge per vertex builds the components, every vertex is pointed at its root,
// the other edges then mostly connect nothing -- but the prefix is united in
// rounds of one cooperative launch instead of by walking: where a giant
// component forms, the walks of concurrent unions chase chains that other
// unions keep extending (half a million edges of a uniform graph, those around
// the critical density, took 127 us; as many before or after it 20-28).
//   round 0   every vertex hooks under its smallest neighbour below it (a
//             fire-and-forget minimum per edge); its forest edge is the one to
//             that parent, so the compress writes the forest slots in order;
//   round r   every edge not yet settled relabels its endpoints by one hop
//             and, if they differ, tries to hook the larger with one CAS; it
//             keeps its record where the CAS lost.  A root that this CTA has
//             tried once is not tried again (it is no root any more), so a
//             root that many edges want to hook costs one CAS per CTA.  (Trying
//             again at once with what the CAS returned read the hubs' words
//             over and over: 851 against 384 us on R-MAT 22.)
//   compress  the roots hooked in the round are pointed at their new roots
//             (those of the last round by the passes over all vertices);
//   the rest  a bit per vertex (in the giant component, read through L1)
//             settles most edges; the others are gathered 32 at a time, their
//             parents read and, where they differ, united with a CAS, as in
//             cc.cu where that loses.
// The labels array is the parent array: the last compress leaves the labels.
//
// us per call, before (cc.cu's launches) -> now: uniform n = 2,000,003, m = 2^23
// 450 -> 273, R-MAT 22 (67 M edges) 444 -> 348.  Bound: the rest's gathers and
// bits (64% L1 hits, 47% of the L2 sector rate, 56% of the issue slots on R-MAT
// 21) and, for uniform graphs, the scattered accesses of the rounds.  Slower than
// before where no giant component forms and the rest still unites much: a mesh of
// 4 x 500,000 in random order 207 -> 228 (its rest 54 -> 80, with 32 warps per SM
// against 60; three blocks per SM 218, but geometric n = 2^19 178 -> 200).
#include <algorithm>

#include "solve.cuh"
#include "uf.cuh"

namespace phem {
namespace {

constexpr uint32_t kCcTile = 128;       // edges per warp step: four per lane
constexpr uint32_t kTriedSlots = 2048;
// Rounds of single tries; the edges left then are united by walking.  What is
// left after four is few edges that meet on one line: us per call with 24 / 4
// rounds, a path of 2^21 vertices in random numbering 208 / 182 (12 rounds), a
// 1448 x 1448 mesh in random order 257 / 257, geometric n = 2^19 199 / 199,
// uniform n = 200,000, m = 3 M 144 / 144.  With at most 16,384 records left at
// any round instead: geometric 177, but uniform 147.
constexpr uint32_t kCcRounds = 4;

struct CcArgs {
    const unsigned long long *edges;
    uint64_t m, s;           // edges, and those of the prefix
    uint32_t n;
    uint32_t *parent;        // the labels
    unsigned long long *forest;
    uint32_t *giant;         // one bit per vertex
    uint4 *list;             // per-warp segments: {root u, root v, u, v}
    uint32_t *hooked;
    uint64_t seg;
    Ctl *ctl;
    Ctl *publish;            // pinned host copy of the results, for the last kernel
    int timing;              // record phase timestamps
};

struct CcSmem {
    uint4 ring[kSolveWarps][kRing];
    uint32_t tried[kTriedSlots];            // roots this CTA has tried to hook
    unsigned long long offered[kTriedSlots];  // vertex << 32 | smallest neighbour offered to it
    unsigned long long acc, sum;
    uint32_t abort, fatal;
    uint32_t giant;
};

// x to its root if that is near, for the giant component's; every block looks
// for itself.  A last round or a rest can leave one chain of hundreds of
// thousands of roots, whose links a walk would take one after the other while
// the passes over all vertices shorten it from all sides: a block that finds no
// root sets no vertex's bit, and the others' bits are still right, because a
// root that is reached is the component's only one.
constexpr uint32_t kNoVertex = 0xffffffffu, kGiantHops = 256;

__device__ __forceinline__ bool near_root(const uint32_t *parent, uint32_t &x)
{
    for (uint32_t steps = 0; steps < kGiantHops; steps++) {
        const uint32_t p = ld_par(parent + x);
        if (p == x)
            return true;
        x = p;
    }
    return false;
}

// Steps of the rest's lockstep walks (uf.cuh), which can start on chains as long.
// us per call without / with the bound, a path of 2^19 vertices 13 times behind a
// component of as many: mean 1050-1870 / 113, slowest of 200 12,500 / 249 (105 as a
// rule: most walks see the chain's links in time); a 4 x 500,000 mesh in random
// order 224 / 230, others the same.
constexpr uint32_t kLockstep = 64;

// Four consecutive edges of tile t (zero -- a self-loop -- past `end`).
__device__ __forceinline__ void load_edges(const unsigned long long *edges, uint64_t first, uint64_t t, uint64_t end,
                                           uint4 (&q)[2])
{
    const uint64_t i = first + t * kCcTile + lane_id() * 4;
    if (i + 4 <= end) {
        const uint4 *p = reinterpret_cast<const uint4 *>(edges + i);
        q[0] = __ldcs(p);
        q[1] = __ldcs(p + 1);
        return;
    }
    unsigned long long e[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
        e[k] = i + k < end ? __ldcs(edges + i + k) : 0ull;
    q[0] = make_uint4((uint32_t)e[0], (uint32_t)(e[0] >> 32), (uint32_t)e[1], (uint32_t)(e[1] >> 32));
    q[1] = make_uint4((uint32_t)e[2], (uint32_t)(e[2] >> 32), (uint32_t)e[3], (uint32_t)(e[3] >> 32));
}

// The lanes' endpoints; bit k of the result: edge k takes part (u < v, in range).
__device__ __forceinline__ uint32_t unpack(const uint4 (&q)[2], uint32_t n, uint32_t (&u)[4], uint32_t (&v)[4],
                                           bool &bad)
{
    v[0] = q[0].x, u[0] = q[0].y, v[1] = q[0].z, u[1] = q[0].w;
    v[2] = q[1].x, u[2] = q[1].y, v[3] = q[1].z, u[3] = q[1].w;
    uint32_t live = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        // union_find_gpu_COO unites u < v (signed; CC/ExternalSpanningTree.cu:82)
        const bool on = (int32_t)u[k] < (int32_t)v[k];
        const bool out = on && ((int32_t)u[k] < 0 || v[k] >= n);
        bad |= out;
        live |= (uint32_t)(on && !out) << k;
    }
    return live;
}

// One try at hooking the larger of two differing ancestors under the smaller.
// Returns the hooked root, or kNotHooked and in x, y the ancestors the edge
// goes on with (equal: settled).
constexpr uint32_t kNotHooked = 0xffffffffu;

__device__ __forceinline__ uint32_t try_hook(const CcArgs &a, CcSmem &s, uint32_t &x, uint32_t &y,
                                             unsigned long long e)
{
    const uint32_t hi = max(x, y), lo = min(x, y);
    if (atomicExch(&s.tried[(hi * 0x9E3779B1u) >> 21], hi) == hi)
        return kNotHooked;  // this CTA tried hi before: it is hooked
    const uint32_t old = atomicCAS(a.parent + hi, hi, lo);
    if (old == hi) {
        if (a.forest)
            a.forest[hi] = e;
        return hi;
    }
    x = lo;
    y = old;
    return kNotHooked;
}

// Appends the lanes' hooked roots to the warp's list of them.
__device__ __forceinline__ void note_hook(WarpState &ws, uint32_t hi, uint32_t below)
{
    const unsigned b = __ballot_sync(0xffffffffu, hi != kNotHooked);
    if (hi != kNotHooked)
        ws.hooked[ws.hooks + __popc(b & below)] = hi;
    ws.hooks += __popc(b);
}

__device__ __forceinline__ void cc_append(uint4 *ring, uint4 *list, uint32_t &filled, uint32_t &flushed, bool keep,
                                          uint4 rec, uint32_t lane, uint32_t below)
{
    const unsigned b = __ballot_sync(0xffffffffu, keep);
    if (keep)
        ring[(filled + __popc(b & below)) & (kRing - 1)] = rec;
    filled += __popc(b);
    if (filled - flushed >= 32) {
        __syncwarp();
        list[flushed + lane] = ring[(flushed + lane) & (kRing - 1)];
        flushed += 32;
        __syncwarp();
    }
}

// The pending edges of a full (or last) ring row: ancestors looked up (the top
// bit of an endpoint says that it is in the giant component, whose root is
// known), and united by walking where they differ.
__device__ __forceinline__ void cc_unite_row(const CcArgs &a, const uint2 *ring, uint32_t giant, uint32_t flushed,
                                             uint32_t cnt, uint32_t lane)
{
    __syncwarp();
    if (lane < cnt) {
        const uint2 r = ring[(flushed + lane) & (kRing - 1)];
        const uint32_t u = r.x & 0x7fffffffu, v = r.y & 0x7fffffffu;
        // from L2: a vertex that an earlier edge attached is seen attached
        uint32_t x = r.x >> 31 ? giant : __ldcg(a.parent + u), y = r.y >> 31 ? giant : __ldcg(a.parent + v);
        const uint32_t hi = max(x, y), lo = min(x, y);
        const unsigned long long e = (unsigned long long)u << 32 | v;
        bool on = x != y;
        // most are a vertex on its own: hooked at once (never the giant's
        // root this way, which every row knows)
        if (on && hi != giant) {
            const uint32_t old = atomicCAS(a.parent + hi, hi, lo);
            if (old == hi) {
                if (a.forest)
                    a.forest[hi] = e;
                on = false;
            } else {
                x = lo;
                y = old;
                on = x != y;
            }
        }
        if (on)
            uf_unite_from<kLockstep>(reinterpret_cast<int32_t *>(a.parent), a.forest, e, (int32_t)x, (int32_t)y,
                                     (int32_t)a.n, &a.ctl->err);
    }
    __syncwarp();
}

// Adds the roots among the vertices this thread compressed (the stride is
// full_compress's) to the block's count and that to the result.
__device__ __forceinline__ void count_roots(const CcArgs &a, unsigned long long *block)
{
    uint32_t roots = 0;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x * kVItems;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x * kVItems; i0 < a.n; i0 += step)
#pragma unroll
        for (int k = 0; k < kVItems; k++) {
            const uint64_t i = i0 + k * blockDim.x + threadIdx.x;
            roots += i < a.n && ld_par(a.parent + i) == (uint32_t)i;
        }
    roots = __reduce_add_sync(0xffffffffu, roots);
    if (lane_id() == 0 && roots)
        atomicAdd(block, (unsigned long long)roots);
    __syncthreads();
    if (threadIdx.x == 0 && *block)
        atomicAdd(&a.ctl->misc[0], *block);
}

__global__ void __launch_bounds__(kSolveThreads, 1) cc_grid_kernel(const __grid_constant__ CcArgs a)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    CcSmem &s = *reinterpret_cast<CcSmem *>(s_raw);
    Ctl *ctl = a.ctl;
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, nw = blockDim.x >> 5;
    const uint32_t below = (1u << lane) - 1u;
    uint32_t seq = 0;
    PhaseClock clock(ctl, a.timing);
    WarpState ws;
    ws.gw = blockIdx.x * nw + warp;
    ws.GW = gridDim.x * nw;
    ws.len = ws.hooks = ws.parity = 0;
    ws.list = a.list + ws.gw * a.seg;
    ws.hooked = a.hooked + ws.gw * a.seg;
    uint4 *ring = s.ring[warp];
    for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + tid; x < a.n; x += (uint64_t)gridDim.x * blockDim.x) {
        a.parent[x] = (uint32_t)x;
    }
    for (uint32_t i = tid; i < kTriedSlots; i += blockDim.x) {
        s.tried[i] = 0xffffffffu;
        s.offered[i] = ~0ull;
    }
    if (tid == 0) {
        s.acc = 0;
        s.fatal = 0;
    }
    if (!grid_sync(ctl, s, seq))
        return;
    clock.stamp(kKCcInit);
    bool bad = false;
    const uint64_t tiles = (a.s + kCcTile - 1) / kCcTile;
    // round 0: every vertex is its own root, and hooks under its smallest
    // neighbour below it: one fire-and-forget minimum per edge.  What the CTA
    // has offered a vertex is remembered, so a vertex that is the larger end
    // of many edges costs few of them.
    {
        uint4 q[2], nq[2];
        load_edges(a.edges, 0, ws.gw, a.s, nq);
        for (uint64_t t = ws.gw; t < tiles; t += ws.GW) {
            q[0] = nq[0], q[1] = nq[1];
            load_edges(a.edges, 0, t + ws.GW, a.s, nq);
            uint32_t u[4], v[4];
            const uint32_t live = unpack(q, a.n, u, v, bad);
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (live >> k & 1) {
                    volatile unsigned long long *seen = &s.offered[(v[k] * 0x9E3779B1u) >> 21];
                    const unsigned long long o = *seen;
                    if ((uint32_t)(o >> 32) != v[k] || u[k] < (uint32_t)o) {
                        *seen = (unsigned long long)v[k] << 32 | u[k];
                        atomicMin(a.parent + v[k], u[k]);
                    }
                }
        }
    }
    if (!grid_sync(ctl, s, seq))
        return;
    clock.stamp(kKCcUnite);
    // a hooked vertex's forest edge is the one to the parent it got; then
    // every vertex to its root
    full_compress<true>(a.parent, a.n, nullptr, nullptr, 0, false, &ctl->err, a.forest);
    if (!grid_sync(ctl, s, seq))
        return;
    clock.stamp(kKCcLabel);
    // round 1, over the edges again
    {
        uint32_t filled = 0, flushed = 0;
        uint4 q[2], nq[2];
        load_edges(a.edges, 0, ws.gw, a.s, nq);
        for (uint64_t t = ws.gw; t < tiles; t += ws.GW) {
            q[0] = nq[0], q[1] = nq[1];
            load_edges(a.edges, 0, t + ws.GW, a.s, nq);
            uint32_t u[4], v[4], x[4], y[4];
            bool again = false;
            const uint32_t live = unpack(q, a.n, u, v, again);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                x[k] = y[k] = 0;
                if (live >> k & 1) {
                    x[k] = ld_par(a.parent + u[k]);
                    y[k] = ld_par(a.parent + v[k]);
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const bool on = x[k] != y[k];
                const uint32_t hi =
                    on ? try_hook(a, s, x[k], y[k], (unsigned long long)u[k] << 32 | v[k]) : kNotHooked;
                note_hook(ws, hi, below);
                cc_append(ring, ws.list, filled, flushed, on && hi == kNotHooked && x[k] != y[k],
                          make_uint4(x[k], y[k], u[k], v[k]), lane, below);
            }
        }
        __syncwarp();
        if (lane < filled - flushed)
            ws.list[flushed + lane] = ring[(flushed + lane) & (kRing - 1)];
        ws.len = filled;
        acc_add(s, lane == 0 ? filled : 0u);
    }
    if (!grid_sync(ctl, s, seq))
        return;
    clock.stamp(kKCcUnite);
    for (uint32_t r = 1; s.sum > 0; r++) {
        compress_pass(a.parent, a.n, &ctl->err, ws);
        ws.hooks = 0;
        if (!grid_sync(ctl, s, seq))
            return;
        clock.stamp(kKCcLabel);
        uint32_t filled = 0, flushed = 0;
        constexpr int ROWS = 4;
        for (uint32_t i0 = 0; i0 < ws.len; i0 += 32 * ROWS) {
            uint4 rec[ROWS];
#pragma unroll
            for (int j = 0; j < ROWS; j++) {
                const uint32_t i = i0 + j * 32 + lane;
                rec[j] = i < ws.len ? __ldcg(ws.list + i) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int j = 0; j < ROWS; j++) {
                rec[j].x = ld_par(a.parent + rec[j].x);
                rec[j].y = ld_par(a.parent + rec[j].y);
            }
#pragma unroll
            for (int j = 0; j < ROWS; j++) {
                const bool on = rec[j].x != rec[j].y;
                uint32_t hi = kNotHooked;
                if (on) {
                    const unsigned long long e = (unsigned long long)rec[j].z << 32 | rec[j].w;
                    if (r < kCcRounds)
                        hi = try_hook(a, s, rec[j].x, rec[j].y, e);
                    else
                        uf_unite_from(reinterpret_cast<int32_t *>(a.parent), a.forest, e, (int32_t)rec[j].x,
                                      (int32_t)rec[j].y, (int32_t)a.n, &ctl->err);
                }
                note_hook(ws, hi, below);
                cc_append(ring, ws.list, filled, flushed,
                          on && hi == kNotHooked && r < kCcRounds && rec[j].x != rec[j].y, rec[j], lane, below);
            }
        }
        __syncwarp();
        if (lane < filled - flushed)
            ws.list[flushed + lane] = ring[(flushed + lane) & (kRing - 1)];
        ws.len = filled;
        acc_add(s, lane == 0 ? filled : 0u);
        if (!grid_sync(ctl, s, seq))
            return;
        clock.stamp(kKCcUnite);
    }
    if (a.s < a.m) {
        // the component that most of 32 sampled endpoints lie in
        if (tid < 32) {
            const uint64_t pos = sample_pos(lane, 32, a.m);
            const unsigned long long e = __ldg(a.edges + pos);
            uint32_t x = (lane & 1) ? (uint32_t)e : (uint32_t)(e >> 32);
            if (x >= a.n)
                x = 0;
            const bool found = __all_sync(0xffffffffu, near_root(a.parent, x));
            const unsigned peers = __match_any_sync(0xffffffffu, x);
            const uint32_t top = __reduce_max_sync(0xffffffffu, ((uint32_t)__popc(peers) << 5) | (31u - lane));
            const uint32_t root = __shfl_sync(0xffffffffu, x, 31 - (top & 31));
            if (lane == 0)
                s.giant = found && top >> 5 >= 8 ? root : kNoVertex;
        }
        __syncthreads();
        full_compress<true>(a.parent, a.n, nullptr, a.giant, s.giant, true, &ctl->err);
        if (blockIdx.x == 0 && tid == 0)
            ctl->misc[3] = s.giant != kNoVertex, ctl->misc[4] = s.giant;
        if (__any_sync(0xffffffffu, bad) && lane == 0)
            set_err(&ctl->err, kErrRange);
        clock.stamp(kKCcLabel);
        return;  // the rest and the labels are launches of their own
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0)
        set_err(&ctl->err, kErrRange);
    full_compress<true>(a.parent, a.n, nullptr, nullptr, 0, false, &ctl->err);
    count_roots(a, &s.acc);
    clock.stamp(kKCcLabel);
    publish_ctl(ctl, a.publish);
}

// The edges behind the prefix.  A lane takes four consecutive edges of a
// 128-edge tile and keeps the next two tiles' loads in flight.
constexpr int kRestThreads = 512, kRestCtasPerSm = 2, kAhead = 2;

__global__ void __launch_bounds__(kRestThreads, kRestCtasPerSm) cc_rest_kernel(const __grid_constant__ CcArgs a, int part)
{
    __shared__ uint2 s_ring[kRestThreads / 32][kRing];
    Ctl *ctl = a.ctl;
    const uint32_t lane = lane_id(), below = (1u << lane) - 1u;
    uint2 *ring = s_ring[threadIdx.x >> 5];
    const bool use_giant = ctl->misc[3] != 0;
    const uint32_t giant = use_giant ? (uint32_t)ctl->misc[part ? 5 : 4] : 0xffffffffu;
    const uint64_t tiles = (a.m - a.s + kCcTile - 1) / kCcTile;
    const uint64_t gw = (uint64_t)blockIdx.x * (kRestThreads / 32) + (threadIdx.x >> 5),
                   GW = (uint64_t)gridDim.x * (kRestThreads / 32);
    uint32_t filled = 0, flushed = 0;
    bool bad = false;
    uint4 nq[kAhead][2];
#pragma unroll
    for (int d = 0; d < kAhead; d++)
        load_edges(a.edges, a.s, gw + d * GW, a.m, nq[d]);
    for (uint64_t t0 = gw; t0 < tiles; t0 += kAhead * GW) {
#pragma unroll
        for (int d = 0; d < kAhead; d++) {
            const uint64_t t = t0 + d * GW;
            uint4 q[2] = {nq[d][0], nq[d][1]};
            load_edges(a.edges, a.s, t + kAhead * GW, a.m, nq[d]);
            uint32_t u[4], v[4];
            uint32_t live = unpack(q, a.n, u, v, bad);
            if (use_giant) {
                uint32_t gu[4], gv[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    gu[k] = gv[k] = 0;
                    if (live >> k & 1) {
                        gu[k] = ld_par(a.giant + (u[k] >> 5)) >> (u[k] & 31);
                        gv[k] = ld_par(a.giant + (v[k] >> 5)) >> (v[k] & 31);
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    live &= ~((gu[k] & gv[k] & 1u) << k);
                    u[k] |= gu[k] << 31;
                    v[k] |= gv[k] << 31;
                }
            }
            if (!__any_sync(0xffffffffu, live))
                continue;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const bool keep = live >> k & 1;
                const unsigned b = __ballot_sync(0xffffffffu, keep);
                if (keep)
                    ring[(filled + __popc(b & below)) & (kRing - 1)] = make_uint2(u[k], v[k]);
                filled += __popc(b);
                if (filled - flushed >= 32) {
                    cc_unite_row(a, ring, giant, flushed, 32, lane);
                    flushed += 32;
                }
            }
        }
    }
    if (filled != flushed)
        cc_unite_row(a, ring, giant, flushed, filled - flushed, lane);
    if (__any_sync(0xffffffffu, bad) && lane == 0)
        set_err(&ctl->err, kErrRange);
}

// Blocks of the passes over all vertices: all resident at once, so that every
// chain is shortened by its own vertices' threads while others walk it.  With
// twice as many blocks the first ones went on to the higher vertices while the
// last ones' vertices, which the chains lead through, had no thread yet: 19 ms for
// a path of 2^20 vertices behind a component of as many, 0.11 now.
constexpr int kVertexBlocksPerSm = 4;

// Between two parts of the rest: every vertex to its root, and the giant
// component's bits again (its root is looked up: it may have been hooked).
__global__ void __launch_bounds__(kBlock, kVertexBlocksPerSm) cc_regroup_kernel(const __grid_constant__ CcArgs a)
{
    __shared__ uint32_t s_giant;
    if (threadIdx.x == 0) {
        uint32_t root = (uint32_t)a.ctl->misc[4];
        const bool found = a.ctl->misc[3] != 0 && near_root(a.parent, root);
        s_giant = found ? root : kNoVertex;
        if (blockIdx.x == 0)
            a.ctl->misc[5] = root;  // or an ancestor of the vertices with a bit, which serves as well
    }
    __syncthreads();
    full_compress<true>(a.parent, a.n, nullptr, a.giant, s_giant, true, &a.ctl->err);
}

// Labels (every vertex to its root) and the number of components.  Bound by
// the walks' L2 latency, so by the warps in flight: two blocks per SM (102
// registers) / four (64), us per call: n = 2^21 282 / 275, R-MAT 22 361 / 355;
// six and eight the same as four.
__global__ void __launch_bounds__(kBlock, kVertexBlocksPerSm) cc_label_count_kernel(const __grid_constant__ CcArgs a)
{
    __shared__ unsigned long long s_roots;
    if (threadIdx.x == 0)
        s_roots = 0;
    __syncthreads();
    full_compress<true>(a.parent, a.n, nullptr, nullptr, 0, false, &a.ctl->err);
    count_roots(a, &s_roots);
    publish_ctl(a.ctl, a.publish);
}

}  // namespace

phem_status cc_grid(phem_context *ctx, const uint64_t *d_edges, int64_t m, int64_t s, int32_t n, int32_t *d_labels,
                    uint64_t *d_forest, void *ws)
{
    if (!(ctx->kernels_ready & kCcGridReady)) {
        PHEM_CUDA_TRY(cudaFuncSetAttribute(cc_grid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)sizeof(CcSmem)));
        ctx->kernels_ready |= kCcGridReady;
    }
    const SolveGrid g = cc_grid_size(m, ctx->sm_count);
    const uint64_t warps = (uint64_t)g.blocks * (g.threads / 32);
    CcArgs a{};
    a.edges = reinterpret_cast<const unsigned long long *>(d_edges);
    a.m = (uint64_t)m;
    a.s = (uint64_t)s;
    a.n = (uint32_t)n;
    a.parent = reinterpret_cast<uint32_t *>(d_labels);
    a.forest = reinterpret_cast<unsigned long long *>(d_forest);
    const uint64_t tiles = ((uint64_t)s + kCcTile - 1) / kCcTile;
    a.seg = (tiles + warps - 1) / warps * kCcTile;
    Carve c;
    char *base = static_cast<char *>(ws);
    a.list = reinterpret_cast<uint4 *>(base + c.take<uint4>(a.seg * warps));
    a.hooked = reinterpret_cast<uint32_t *>(base + c.take<uint32_t>(a.seg * warps));
    a.giant = reinterpret_cast<uint32_t *>(base + c.take<uint32_t>(((uint64_t)n + 31) / 32));
    a.timing = ctx->profiling;
    PHEM_TRY(solve_ctl(ctx, &a.ctl, &a.publish));
    void *params[] = {&a};
    {
        KernelScope ks(ctx, kKCcSolve);
        PHEM_CUDA_TRY(cudaLaunchCooperativeKernel(cc_grid_kernel, dim3(g.blocks), dim3(g.threads), params,
                                                  sizeof(CcSmem), ctx->stream));
    }
    if (s < m) {
        auto rest = [&](uint64_t first, uint64_t end, int part) {
            CcArgs b = a;
            b.s = first;
            b.m = end;
            const uint64_t blocks = ((end - first + kCcTile - 1) / kCcTile + kRestThreads / 32 - 1) / (kRestThreads / 32);
            KernelScope ks(ctx, kKCcUnite);
            cc_rest_kernel<<<(int)std::min<uint64_t>(blocks, (uint64_t)ctx->sm_count * kRestCtasPerSm), kRestThreads, 0,
                             ctx->stream>>>(b, part);
        };
        const int vblocks = (int)std::min<int64_t>(((int64_t)n + kBlock * kVItems - 1) / (kBlock * kVItems),
                                                   (int64_t)ctx->sm_count * kVertexBlocksPerSm);
        // A long rest goes in two parts: the first attaches most of what the
        // prefix left out, and after a second look at the components the
        // bits settle nearly all of the second.  us per solve in one part / cut
        // at 2n: R-MAT 22 (15 n) 370 / 360, uniform 15 n 290 / 237, 7 n 215 /
        // 207, 3.2 n 293 / 295, R-MAT 22 3 n 222 / 240.
        const uint64_t cut = ((uint64_t)s + 2 * (uint64_t)n) & ~3ull;
        if ((uint64_t)(m - s) >= 6 * (uint64_t)n) {
            rest(s, cut, 0);
            {
                KernelScope ks(ctx, kKCcLabel);
                cc_regroup_kernel<<<vblocks, kBlock, 0, ctx->stream>>>(a);
            }
            rest(cut, m, 1);
        } else {
            rest(s, m, 0);
        }
        KernelScope ks(ctx, kKCcLabel);
        cc_label_count_kernel<<<vblocks, kBlock, 0, ctx->stream>>>(a);
        PHEM_CUDA_TRY(cudaGetLastError());
    }
    return PHEM_OK;
}

// Workspace of cc_grid: list and hooked-root segments for the prefix, the bits.
size_t cc_grid_bytes(int64_t m, int64_t s, int32_t n, int sm_count)
{
    const SolveGrid g = cc_grid_size(m, sm_count);
    const uint64_t records = (uint64_t)s + ((uint64_t)g.blocks * (g.threads / 32) + 1) * kCcTile;
    Carve c;
    c.take<uint4>(records);
    c.take<uint32_t>(records);
    c.take<uint32_t>(((uint64_t)n + 31) / 32);
    return c.off;
}

// A warp gets at least one tile of edges.
SolveGrid cc_grid_size(int64_t m, int sm_count)
{
    const uint64_t tiles = ((uint64_t)m + kCcTile - 1) / kCcTile;
    SolveGrid g;
    g.threads = tiles <= 8 * (uint64_t)sm_count ? 256 : (tiles <= 32 * (uint64_t)sm_count ? 512 : 1024);
    const uint64_t warps = (uint64_t)g.threads / 32;
    g.blocks = (uint32_t)std::max<uint64_t>(
        1, std::min({(tiles + warps - 1) / warps, (uint64_t)sm_count, (uint64_t)kMaxGrid}));
    return g;
}

}  // namespace phem
