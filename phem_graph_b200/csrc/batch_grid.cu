// batch_grid.cu -- a batch of graphs as one disjoint union over the whole grid.
//
// The CTA-per-graph kernel (batch.cu) ends with its largest graphs: one SM
// works for milliseconds on a graph of half a million edges while the others
// have run dry.  A batch is also one graph, the disjoint union of its
// graphs: its minimum spanning forest is the union of theirs, and a component
// never leaves its graph.  Here the one-launch solve of msf.cu runs over that
// union.  Every graph's edges are cut into tiles of 128 records (cut on
// 16-byte boundaries of the caller's array, so a graph may start anywhere); a
// descriptor per tile, written by the kernel's first phase, says where the
// tile's records are and which graph they belong to.  An edge's id in the
// union is its position in the tiles, so ids of one graph ascend as its own
// do and ties break alike; vertices are numbered graph after graph.  Every
// graph has its own light/heavy threshold.  At the end the marked ids are
// ranked per tile, written per graph, and labels are the minimum vertex id of
// each component.
//
// Bound: scattered L2 accesses (two offers, a parent store and a bitmap atomic
// per component and round, at 170-290 G/s), not the 12 bytes per edge.
#include <algorithm>

#include "batch.h"
#include "solve.cuh"

namespace phem {
namespace {

// One tile of 128 records: records [base + lo, base + hi) are the graph's.
struct __align__(16) GridTile {
    uint64_t base;
    uint32_t vb, n;      // the graph's first vertex in the union, its vertex count
    uint32_t range;      // lo | hi << 16
    uint32_t item;       // the graph; top bit: connected components
    uint32_t pad[2];
};
static_assert(sizeof(GridTile) == 32, "tile descriptors are two 16-byte loads");

constexpr uint32_t kTileRecs = 128;

struct GridArgs {
    SolveArgs s;         // n is the capacity's vertex count (bounds walks), not the batch's
    const GridHdr *hdr;
    const GridItem *items;
    const phem_edge *edges;
    GridTile *tiles;
    uint32_t *vitem;     // graph of each group of 32 union vertices
    unsigned long long *thr;  // light edge <=> key below its graph's threshold
    uint32_t *ids, *count, *status, *rounds;
    unsigned long long *total;
    int32_t *labels;
    float light_msf, light_cc;
};

// The weight below which about k of the graph's m edges lie: the (k/m)-th of
// 256 stratified samples, by bisection on the value (8 samples per lane).
__device__ __forceinline__ unsigned long long warp_threshold(const phem_edge *e, uint32_t m, uint32_t k)
{
    const uint32_t lane = lane_id();
    uint32_t w[8];
#pragma unroll
    for (int q = 0; q < 8; q++)
        w[q] = __ldg(&e[sample_pos(q * 32 + lane, 256, m)].w);
    const uint32_t rank = (uint32_t)((uint64_t)k * 256 / m);
    uint32_t lo = 0;  // the largest value with at most `rank` samples below it
    for (int b = 31; b >= 0; b--) {
        const uint32_t mid = lo | 1u << b;
        uint32_t below = 0;
#pragma unroll
        for (int q = 0; q < 8; q++)
            below += w[q] < mid;
        if (__reduce_add_sync(0xffffffffu, below) <= rank)
            lo = mid;
    }
    return (unsigned long long)lo << 32;
}

// One tile of the union; as msf.cu's input_tile, with the graph's own vertex
// base, range and threshold.
template <bool LIGHT>
__device__ __forceinline__ void grid_tile(const GridArgs &a, SolveSmem &s, unsigned long long *best, EpWarp &w,
                                          const unsigned char *stage, bool bulk, const GridTile &t, uint32_t id0,
                                          uint4 *list, uint32_t &filled, uint32_t &flushed, uint32_t lane)
{
    constexpr int PER = 4;
    uint32_t u[PER], v[PER], wt[PER];
    const uint32_t i0 = lane * PER, lo = t.range & 0xffffu, hi = t.range >> 16;
    if (bulk) {
        const uint4 *q = reinterpret_cast<const uint4 *>(stage) + 3 * lane;
        const uint4 q0 = q[0], q1 = q[1], q2 = q[2];
        u[0] = q0.x, v[0] = q0.y, wt[0] = q0.z, u[1] = q0.w;
        v[1] = q1.x, wt[1] = q1.y, u[2] = q1.z, v[2] = q1.w;
        wt[2] = q2.x, u[3] = q2.y, v[3] = q2.z, wt[3] = q2.w;
    } else {
#pragma unroll
        for (int j = 0; j < PER; j++) {
            u[j] = v[j] = wt[j] = 0;
            if (i0 + j >= lo && i0 + j < hi) {
                const uint32_t *p = reinterpret_cast<const uint32_t *>(a.edges + t.base + i0 + j);
                u[j] = __ldcs(p);
                v[j] = __ldcs(p + 1);
                wt[j] = __ldcs(p + 2);
            }
        }
    }
    const unsigned long long thr = ld_best(a.thr + (t.item & 0x7fffffffu));
    uint32_t keep = 0;
    bool any_bad = false;
#pragma unroll
    for (int j = 0; j < PER; j++) {
        if (t.item >> 31)
            wt[j] = 0;  // connected components: ordered by id
        const bool in = i0 + j >= lo && i0 + j < hi;
        // every record is checked, self-loops too, as batch.cu does
        const bool bad = in && max(u[j], v[j]) >= t.n;
        any_bad |= bad;
        const unsigned long long key = ((unsigned long long)wt[j] << 32) | (id0 + i0 + j);
        const bool light = key < thr;
        keep |= (uint32_t)(in && !bad && u[j] != v[j] && (LIGHT ? light : !light)) << j;
        u[j] += t.vb;
        v[j] += t.vb;
    }
    if (LIGHT && any_bad)
        atomicOr(a.status + a.items[t.item & 0x7fffffffu].index, kErrRange);
    if (!LIGHT) {
#pragma unroll
        for (int j = 0; j < PER; j++)
            if (keep >> j & 1) {
                u[j] = ld_par(a.s.parent + u[j]);
                v[j] = ld_par(a.s.parent + v[j]);
                if (u[j] == v[j])
                    keep &= ~(1u << j);
            }
    }
    if (!__any_sync(0xffffffffu, keep))
        return;
#pragma unroll
    for (int j = 0; j < PER; j++) {
        ring_append(w, filled, keep >> j & 1, make_uint4(u[j], v[j], wt[j], id0 + i0 + j), lane);
        if (filled - flushed >= 32)
            ring_flush<kKindMsf>(a.s, s, best, list, w, flushed, 32, lane);
    }
}

// Consecutive tiles a warp takes: up to kMaxRun, while a CTA still gets about
// eight blocks (their survivors differ from graph to graph).
constexpr uint32_t kMaxRun = 4;
__device__ __forceinline__ uint32_t tile_run(uint32_t T, uint32_t warps)
{
    return min(max(T / (warps * 8), 1u), kMaxRun);
}

__device__ __forceinline__ GridTile load_tile(const GridTile *tiles, uint32_t t, uint32_t T)
{
    GridTile d;
    if (t >= T) {
        d.range = 0;
        return d;
    }
    const uint4 *q = reinterpret_cast<const uint4 *>(tiles + t);
    const uint4 x = __ldcg(q);
    const uint2 y = __ldcg(reinterpret_cast<const uint2 *>(q + 1));
    d.base = (uint64_t)x.y << 32 | x.x;
    d.vb = x.z;
    d.n = x.w;
    d.range = y.x;
    d.item = y.y;
    return d;
}

// msf.cu's input_pass over the tile descriptors, which are loaded one tile
// further ahead than the records.
template <bool LIGHT>
__device__ __forceinline__ void grid_input_pass(const GridArgs &a, SolveSmem &s, unsigned long long *best, uint32_t T,
                                                WarpState &ws)
{
    const uint32_t lane = lane_id();
    EpWarp &w = s.warp[threadIdx.x >> 5];
    const bool wide = ((uintptr_t)a.edges & 15) == 0;
    const uint64_t policy = l2_evict_first();
    // whole tiles come by bulk copy (lo may be above zero: the records before
    // it are the caller's too, and are skipped)
    auto bulk_of = [&](const GridTile &d) { return wide && (d.range >> 16) == kTileRecs; };
    auto issue = [&](const GridTile &d, int st) {  // lane 0 only
        mbar_arrive_expect_tx(reinterpret_cast<uint64_t *>(&w.bar[st]), kEpStageBytes);
        bulk_copy_g2s_hint(w.stage[st], a.edges + d.base, kEpStageBytes,
                           reinterpret_cast<uint64_t *>(&w.bar[st]), policy);
    };
    // A CTA takes blocks of nw * run consecutive tiles, so the parents and
    // offers of a graph stay with few SMs; a warp's j-th tile:
    const uint32_t nw = blockDim.x >> 5, warp = threadIdx.x >> 5;
    const uint32_t run = tile_run(T, ws.GW);
    auto tile_at = [&](uint32_t j) {
        return ((j / run) * gridDim.x + blockIdx.x) * (nw * run) + warp * run + j % run;
    };
    GridTile cur = load_tile(a.tiles, tile_at(0), T), nxt = load_tile(a.tiles, tile_at(1), T);
    uint32_t filled = 0, flushed = 0, pending = 0;
    bool failed = false;
    int st = 0;
    if (bulk_of(cur)) {
        if (lane == 0)
            issue(cur, 0);
        pending = 1;
    }
    uint32_t t = tile_at(0);
    for (uint32_t j = 0; t < T; t = tile_at(++j), st ^= 1) {  // ascending: past T once, past it for good
        if (bulk_of(nxt)) {
            if (lane == 0)
                issue(nxt, st ^ 1);
            pending |= 1u << (st ^ 1);
        }
        const GridTile after = load_tile(a.tiles, tile_at(j + 2), T);
        const bool bulk = bulk_of(cur);
        if (bulk) {
            if (!ep_wait(&w.bar[st], (ws.parity >> st) & 1u, &a.s.ctl->err)) {
                failed = true;
                break;
            }
            ws.parity ^= 1u << st;
            pending &= ~(1u << st);
        }
        grid_tile<LIGHT>(a, s, best, w, w.stage[st], bulk, cur, t * kTileRecs, ws.list, filled, flushed, lane);
        fence_proxy_async_smem();  // this lane's reads of the stage precede its refill
        __syncwarp();
        cur = nxt;
        nxt = after;
    }
    if (failed) {
        for (int q = 0; q < kEpStages; q++)
            if (pending & (1u << q))
                ep_wait(&w.bar[q], (ws.parity >> q) & 1u, &a.s.ctl->err);
        s.fatal = 1;
    } else if (filled != flushed) {
        ring_flush<kKindMsf>(a.s, s, best, ws.list, w, flushed, filled - flushed, lane);
    }
    ws.len = flushed;
    acc_add(s, lane == 0 ? flushed : 0u);
}

__global__ void __launch_bounds__(kSolveThreads, 1) batch_grid_kernel(const __grid_constant__ GridArgs a)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    SolveSmem &s = *reinterpret_cast<SolveSmem *>(s_raw);
    const uint32_t G = a.hdr->items, T = a.hdr->tiles, V = a.hdr->vertices;
    Ctl *ctl = a.s.ctl;
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, nw = blockDim.x >> 5;
    uint32_t seq = 0;
    WarpState ws;
    ws.gw = blockIdx.x * nw + warp;
    ws.GW = gridDim.x * nw;
    ws.len = ws.hooks = ws.parity = 0;
    const uint32_t run = tile_run(T, ws.GW);
    const uint64_t seg = (uint64_t)((T + ws.GW * run - 1) / (ws.GW * run)) * run * kTileRecs;
    ws.list = a.s.list + ws.gw * seg;
    ws.hooked = a.s.hooked + ws.gw * seg;
    auto give_up = [&]() {  // a bounded wait ran out: every graph of the batch says so
        for (uint32_t i = blockIdx.x * blockDim.x + tid; i < G; i += gridDim.x * blockDim.x)
            atomicOr(a.status + a.items[i].index, kErrLookback);
    };
    // init: vertex state, tile descriptors and thresholds
    if (tid == 0) {
        s.acc = 0;
        s.fatal = 0;
    }
    if (lane == 0) {
        for (int q = 0; q < kEpStages; q++)
            mbar_init(reinterpret_cast<uint64_t *>(&s.warp[warp].bar[q]), 1);
        fence_mbar_init();
    }
    offers_reset(s.oc);
    __syncthreads();
    {
        const uint32_t g = blockIdx.x * blockDim.x + tid, N = gridDim.x * blockDim.x;
        for (uint32_t x = g; x < V; x += N) {
            a.s.parent[x] = x;
            a.s.best[x] = kKeyNone;
        }
        for (uint32_t t = g; t < T; t += N) {
            reinterpret_cast<uint4 *>(a.s.bitmap)[t] = make_uint4(0, 0, 0, 0);
            // the graph whose tiles t is among: the last one with tile0 <= t
            // that has tiles
            uint32_t i = 0;
            for (uint32_t lo = 0, hi = G; lo < hi;) {
                const uint32_t mid = (lo + hi) / 2;
                if (__ldg(&a.items[mid].tile0) <= t)
                    i = mid, lo = mid + 1;
                else
                    hi = mid;
            }
            const GridItem &it = a.items[i];
            const uint32_t q = t - it.tile0, len = it.skip + it.m;
            GridTile d;
            d.base = it.e_off - it.skip + (uint64_t)q * kTileRecs;
            d.vb = it.vb;
            d.n = it.n;
            d.range = (q == 0 ? it.skip : 0u) | min(len - q * kTileRecs, kTileRecs) << 16;
            d.item = i | (it.kind != PHEM_BATCH_MSF ? 0x80000000u : 0u);
            d.pad[0] = d.pad[1] = 0;
            a.tiles[t] = d;
        }
        for (uint32_t q = g; q < V / 32; q += N) {
            uint32_t i = 0;
            for (uint32_t lo = 0, hi = G; lo < hi;) {
                const uint32_t mid = (lo + hi) / 2;
                if (__ldg(&a.items[mid].vb) <= q * 32)
                    i = mid, lo = mid + 1;
                else
                    hi = mid;
            }
            a.vitem[q] = i;
        }
        uint32_t filtered = 0;
        // thresholds: a warp per graph, the graphs spread over the SMs
        for (uint32_t i = warp * gridDim.x + blockIdx.x; i < G; i += ws.GW) {
            const GridItem it = a.items[i];
            const bool cc = it.kind != PHEM_BATCH_MSF;
            const uint32_t k = (uint32_t)((cc ? a.light_cc : a.light_msf) * (float)it.n);
            unsigned long long thr = kKeyNone;
            if (k && it.m >= 2 * (uint64_t)k && it.m >= 1024) {
                thr = cc ? (unsigned long long)it.tile0 * kTileRecs + it.skip + k
                         : warp_threshold(a.edges + it.e_off, it.m, k);
                filtered++;
            }
            if (lane == 0) {
                a.thr[i] = thr;
                a.status[it.index] = 0;
                a.total[it.index] = 0;
            }
        }
        acc_add(s, lane == 0 ? filtered : 0u);
    }
    if (!grid_sync(ctl, s, seq))
        return give_up();
    const bool filter = s.sum > 0;
    uint32_t r = 0, src = kSrcLight;
    bool heavy = false;
    for (;;) {
        unsigned long long *best = a.s.best + (r & 1) * a.s.best_stride,
                           *next = a.s.best + ((r + 1) & 1) * a.s.best_stride;
        if (src == kSrcList)
            list_pass<kKindMsf>(a.s, s, best, ws);
        else if (src == kSrcLight)
            grid_input_pass<true>(a, s, best, T, ws);
        else
            grid_input_pass<false>(a, s, best, T, ws);
        offers_flush(s.oc, best);
        if (!grid_sync(ctl, s, seq))
            return give_up();
        r++;
        if (s.sum > 0) {
            hook_pass<kKindMsf>(a.s, s, best, next, ws);
            if (!grid_sync(ctl, s, seq))
                return give_up();
            compress_pass(a.s.parent, a.s.n, &ctl->err, ws);
            src = kSrcList;
        } else {
            if (heavy || !filter)
                break;
            full_compress(a.s.parent, V, next, nullptr, 0, false, &ctl->err);
            heavy = true;
            src = kSrcHeavy;
        }
        if (!grid_sync(ctl, s, seq))
            return give_up();
        if (r >= PHEM_MAX_ROUNDS) {
            if (blockIdx.x == 0 && tid == 0)
                set_err(&ctl->err, kErrRounds);
            break;
        }
    }
    // every vertex to its root; the roots' words of `mins` start the minimum
    // vertex ids; the tiles' forest counts become offsets
    unsigned long long *mins = a.s.best;
    full_compress(a.s.parent, V, mins, nullptr, 0, false, &ctl->err);
    const uint64_t per = max((T + gridDim.x - 1) / gridDim.x, 1u);
    count_scan(s, a.s.chunk_off, T, per, a.s.cta_tot, [&](uint64_t, uint64_t i, uint64_t end) {
        if (i >= end)
            return 0u;
        const uint4 b = __ldcg(reinterpret_cast<const uint4 *>(a.s.bitmap) + i);
        return (uint32_t)(__popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w));
    });
    if (!grid_sync(ctl, s, seq))
        return give_up();
    const uint32_t all = prefix_totals(s, a.s.cta_tot);
    if (tid == 0)
        s.sel_prefix = all;
    __syncthreads();
    auto offset = [&](uint32_t t) {  // forest edges before tile t
        return t < T ? __ldcg(a.s.chunk_off + t) + s.pref[t / per] : s.sel_prefix;
    };
    // forest ids per graph, ascending, and the totals
    for (uint32_t c = ws.gw; c < (T + 7) / 8; c += ws.GW) {
        const uint32_t t = c * 8 + lane / 4;
        uint32_t bits = t < T ? __ldcg(a.s.bitmap + c * 32 + lane) : 0u;
        uint32_t rank = __popc(bits);
        const uint32_t own = rank;
        for (int d = 1; d < 4; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, rank, d, 4);
            if ((lane & 3) >= (uint32_t)d)
                rank += y;
        }
        rank -= own;
        uint32_t any = bits;  // of the tile's four lanes
        any |= __shfl_xor_sync(0xffffffffu, any, 1);
        any |= __shfl_xor_sync(0xffffffffu, any, 2);
        unsigned long long sum = 0;
        uint32_t index = 0;
        if (any) {
            const GridItem &it = a.items[__ldcg(&a.tiles[t].item) & 0x7fffffffu];
            index = it.index;
            uint32_t pos = offset(t) - offset(it.tile0) + rank;
            const uint32_t id0 = (t - it.tile0) * kTileRecs + (lane & 3) * 32 - it.skip;
            const phem_edge *e = a.edges + it.e_off;
            uint32_t *ids = a.ids + it.v_off;
            const bool weighted = it.kind == PHEM_BATCH_MSF;
            const uint32_t n = it.n;
            while (bits) {
                uint32_t id[4], w[4];
                int cnt = 0;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    w[q] = 0;
                    if (bits) {
                        id[q] = id0 + __ffs(bits) - 1;
                        bits &= bits - 1;
                        cnt = q + 1;
                        if (weighted)
                            w[q] = __ldg(&e[id[q]].w);
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (q < cnt) {
                        if (pos < n)  // a forest has at most n - 1 edges
                            ids[pos] = id[q];
                        else
                            atomicOr(a.status + index, kErrCapacity);
                        pos++;
                        sum += w[q];
                    }
            }
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if ((lane & 3) == 0 && sum)
            atomicAdd(a.total + index, sum);
    }
    // minimum vertex id of each component: among a warp's 32 consecutive
    // vertices of one root the lowest lane has the smallest
    uint32_t *minid = reinterpret_cast<uint32_t *>(mins);
    for (uint32_t q = ws.gw; q < V / 32; q += ws.GW) {
        const uint32_t x = q * 32 + lane;
        const uint32_t root = ld_par(a.s.parent + x);
        const unsigned peers = __match_any_sync(0xffffffffu, root);
        if ((int)lane == __ffs(peers) - 1 && x < __ldcg(minid + 2 * (uint64_t)root))
            atomicMin(minid + 2 * (uint64_t)root, x);
    }
    if (!grid_sync(ctl, s, seq))
        return give_up();
    for (uint32_t q = ws.gw; q < V / 32; q += ws.GW) {
        const GridItem &it = a.items[__ldcg(a.vitem + q)];
        const uint32_t x = q * 32 + lane;
        if (x - it.vb < it.n)
            a.labels[it.v_off + (x - it.vb)] =
                (int32_t)(__ldcg(minid + 2 * (uint64_t)ld_par(a.s.parent + x)) - it.vb);
    }
    for (uint32_t i = blockIdx.x * blockDim.x + tid; i < G; i += gridDim.x * blockDim.x) {
        const GridItem &it = a.items[i];
        const uint32_t nt = it.m ? (it.skip + it.m + kTileRecs - 1) / kTileRecs : 0;
        a.count[it.index] = offset(it.tile0 + nt) - offset(it.tile0);
        if (a.rounds)
            a.rounds[it.index] = r - 1 - (uint32_t)heavy;  // the union's; a phase ends with an empty pass
        const uint32_t err = *(volatile uint32_t *)&ctl->err;
        if (err)
            atomicOr(a.status + it.index, err);
    }
}

}  // namespace

// Capacities of a batch with `records` edges in G graphs over V vertices.
static uint64_t grid_tiles(uint64_t records, uint32_t G) { return records / kTileRecs + 2ull * G + 8; }
static uint64_t grid_vertices(uint32_t V, uint32_t G) { return (uint64_t)V + 32ull * G + 32; }

uint64_t batch_grid_list(uint64_t records, uint32_t G, int sm_count)
{
    return (grid_tiles(records, G) + (uint64_t)sm_count * kSolveWarps * kMaxRun) * kTileRecs;
}

size_t batch_grid_carve(uint32_t G, uint64_t records, uint32_t V, int sm_count, size_t off, char *base, BatchGrid *g)
{
    Carve c;
    c.off = off;
    const uint64_t T = grid_tiles(records, G), N = grid_vertices(V, G), L = batch_grid_list(records, G, sm_count);
    const size_t o_hdr = c.take<GridHdr>(1 + kBatchGroups), o_it = c.take<GridItem>(G ? G : 1),
                 o_ctl = c.take<Ctl>(1), o_t = c.take<GridTile>(T), o_vi = c.take<uint32_t>(N / 32 + 1),
                 o_par = c.take<uint32_t>(N), o_best = c.take<unsigned long long>(2 * N),
                 o_bm = c.take<uint32_t>(4 * T), o_cnt = c.take<uint32_t>(T), o_tot = c.take<uint32_t>(kMaxGrid),
                 o_hk = c.take<uint32_t>(L), o_thr = c.take<unsigned long long>(G ? G : 1);
    if (base) {
        g->hdr = reinterpret_cast<GridHdr *>(base + o_hdr);
        g->items = reinterpret_cast<GridItem *>(base + o_it);
        g->ctl = reinterpret_cast<Ctl *>(base + o_ctl);
        g->tiles = base + o_t;
        g->vitem = reinterpret_cast<uint32_t *>(base + o_vi);
        g->parent = reinterpret_cast<uint32_t *>(base + o_par);
        g->best = reinterpret_cast<unsigned long long *>(base + o_best);
        g->best_stride = N;
        g->bitmap = reinterpret_cast<uint32_t *>(base + o_bm);
        g->tile_off = reinterpret_cast<uint32_t *>(base + o_cnt);
        g->cta_tot = reinterpret_cast<uint32_t *>(base + o_tot);
        g->hooked = reinterpret_cast<uint32_t *>(base + o_hk);
        g->thr = reinterpret_cast<unsigned long long *>(base + o_thr);
    }
    return c.off;
}

GridHdr batch_grid_items(const BatchItem *items, uint32_t G, GridItem *out)
{
    GridHdr h{G, 0, 0, 0};
    for (uint32_t i = 0; i < G; i++) {
        const BatchItem &x = items[i];
        GridItem &g = out[i];
        g.e_off = x.e_off;
        g.m = x.m;
        g.n = x.n;
        g.v_off = x.v_off;
        g.kind = x.kind;
        g.index = x.index;
        g.tile0 = h.tiles;
        g.vb = h.vertices;
        g.skip = (uint32_t)(x.e_off & 3);
        if (x.m)
            h.tiles += (uint32_t)(((uint64_t)g.skip + x.m + kTileRecs - 1) / kTileRecs);
        h.vertices += (x.n + 31) & ~31u;
    }
    return h;
}

// Which kernel takes a batch: the one whose time, from these measured rates,
// is shorter.  The CTA-per-graph kernel ends with its largest graph (4.5 ns per
// edge or vertex with the state in shared memory, 10 ns without) or when the
// SMs have worked everything off (6 ns per SM and edge or vertex of a graph with
// its state in shared memory, 9 ns otherwise, 12.5 us per graph); that is with
// 1024 threads per CTA, and what 512 and 256 change is in the table.  The grid
// pays its barriers once and 55 ps per edge or vertex.  us, CTA per graph / grid:
// 256 graphs of up to 65,536 vertices (16.7 M edges and vertices) 5608 / 1117, of
// up to 8192 566 / 353, of up to 4096 215 / 282; 4 of up to 20,000 468 / 182; 2048
// of up to 8192 1033 / 1144; 4096 of up to 128 451 / 196, of up to 4096 1143 /
// 1198, of up to 16,384 3829 / 3270, of up to 65,536 (215 M) 15,045 / 9618.  512,
// 256 threads / grid: 256 of up to 8192 862, 1467 / 343; 2048 of up to 8192 1474,
// 2340 / 1172; 4096 of up to 4096 889, 1294 / 1271, of up to 128 188, 115 / 203.
bool batch_takes_grid(const BatchLayout &L, const BatchLaunch &l, int sm_count)
{
    // one graph's time, all graphs' work and all graphs' number, against 1024 threads
    static constexpr double kFactors[3][3] = {{1.0, 1.0, 1.0}, {1.6, 0.75, 0.27}, {2.7, 1.0, 0.06}};
    const double *f = kFactors[l.block >= 1024 ? 0 : l.block >= 512 ? 1 : 2];
    double all = 0, cta = 0, largest = 0;
    uint64_t verts = 0;
    for (const BatchItem &x : L.items) {
        if (x.kind == kBatchPairs)
            return false;
        const double work = (double)x.m + x.n;
        const bool smem = x.n <= l.smem_vertices;
        all += work;
        cta += f[1] * work * (smem ? 6.0 : 9.0) + f[2] * 12.5e3;
        largest = std::max(largest, f[0] * work * (smem ? 4.5 : 10.0));
        verts += ((uint64_t)x.n + 31) & ~31ull;
    }
    const uint64_t tiles = L.wl_records / kTileRecs + 2ull * L.items.size();
    if (tiles * kTileRecs >= (1ull << 32) - (1u << 24) || verts >= (1ull << 31))
        return false;  // union ids and vertices are 32-bit
    const double cta_ns = 25e3 + std::max(largest, cta / sm_count);
    const double grid_ns = 190e3 + 0.055 * all;
    return grid_ns < cta_ns;
}

uint32_t batch_grid_ctas(int sm_count) { return std::min((uint32_t)sm_count, kMaxGrid); }

phem_status batch_grid_launch(cudaStream_t stream, int sm_count, const BatchGrid &g, uint32_t group, uint32_t first,
                              const phem_edge *edges, uint4 *list, const BatchArgs &b, float light_msf,
                              float light_cc)
{
    PHEM_CUDA_TRY(cudaFuncSetAttribute(batch_grid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(SolveSmem)));
    GridArgs a{};
    a.s.n = (uint32_t)g.best_stride;
    a.s.parent = g.parent;
    a.s.best = g.best;
    a.s.best_stride = g.best_stride;
    a.s.bitmap = g.bitmap;
    a.s.chunk_off = g.tile_off;
    a.s.cta_tot = g.cta_tot;
    a.s.list = list;
    a.s.hooked = g.hooked;
    a.s.ctl = g.ctl;
    a.hdr = g.hdr + group;
    a.items = g.items + first;
    a.edges = edges;
    a.tiles = static_cast<GridTile *>(g.tiles);
    a.vitem = g.vitem;
    a.thr = g.thr;
    a.ids = b.msf_ids;
    a.count = b.msf_count;
    a.total = b.msf_total;
    a.labels = b.labels;
    a.status = b.status;
    a.rounds = b.rounds;
    a.light_msf = light_msf;
    a.light_cc = light_cc;
    PHEM_CUDA_TRY(cudaMemsetAsync(g.ctl, 0, sizeof(Ctl), stream));
    void *params[] = {&a};
    PHEM_CUDA_TRY(cudaLaunchCooperativeKernel(batch_grid_kernel, dim3(batch_grid_ctas(sm_count)), dim3(kSolveThreads),
                                              params, sizeof(SolveSmem), stream));
    return PHEM_OK;
}

}  // namespace phem
