// tiny.cu -- solves of small graphs by one CTA, all state on the SM.
//
// A graph of a few thousand edges is latency: the grid solve's barriers and L2
// round trips (105-150 us per call) and the union-find path's six launches
// are the time, not the work.  Here one CTA of 1024 threads holds the graph:
// every thread keeps K edge records in registers for the whole solve (record
// k * 1024 + thread, so its id is implied and a record never moves), and the
// per-vertex state lives in shared memory.  Host inputs are read in place from
// pinned memory (the caller's, or staging for a pageable array) and results are
// written to it, so a host call queues no copy of its own; the control block's
// results go straight to its pinned mirror.
//
// Bound: shared-memory gathers.  A live record costs four per round (its two
// parents, their best weights), about four cycles a warp each with random
// banks, so the edge pass of 8,192 records takes 2 us; the records that may
// still win (marked in registers) are the only ones the other passes look at.
// us per call, grid solve -> this: n = 2,003, m = 8,009 152 -> 56 (326 with
// one launch per phase); n = 1,021, m = 4,093 from host memory 146 -> 51; CC
// n = 3,001, m = 9,001 72 -> 33.  64-bit minima in shared memory (a
// compare-and-swap loop) instead of weight, then id: 64 against 61.
#include <algorithm>
#include <cstring>

#include "tiny.h"

namespace phem {
namespace {

constexpr int kTinyThreads = 1024;
constexpr int kTinyWarps = kTinyThreads / 32;

struct TinyArgs {
    const void *e0;
    uint32_t m, n;
    unsigned long long light;  // kKindPacked: edges below this id first (all ones: one phase)
    phem_edge *out;
    uint64_t *d_count_total;
    int32_t *labels;
    unsigned long long *forest;
    Ctl *res;                  // pinned host memory
};

struct TinySmem {
    uint32_t cnt[16][kTinyWarps];  // forest records per (record row, warp), then their offsets
    uint32_t row[17];
    uint32_t live[2], choosers;
    unsigned long long total;
    uint32_t err, comps;
};

// The input into shared memory (coalesced 16-byte reads; 4-byte ones from an
// unaligned pointer).
__device__ __forceinline__ void stage_input(const void *src, uint32_t bytes, unsigned char *dst)
{
    if (((uintptr_t)src & 15) == 0) {
        const uint4 *q = static_cast<const uint4 *>(src);
        uint4 *d = reinterpret_cast<uint4 *>(dst);
        for (uint32_t i = threadIdx.x; i < bytes / 16; i += kTinyThreads)
            d[i] = __ldcs(q + i);
    }
    const uint32_t done = ((uintptr_t)src & 15) == 0 ? bytes / 16 * 4 : 0;
    const uint32_t *q = static_cast<const uint32_t *>(src);
    uint32_t *d = reinterpret_cast<uint32_t *>(dst);
    for (uint32_t i = done + threadIdx.x; i < bytes / 4; i += kTinyThreads)
        d[i] = __ldcs(q + i);
}

// Boruvka rounds as in msf.cu, on registers and shared memory.  parent[x] is
// x's root as of the last compress; hook[] is the hooking forest over roots
// (a round's hooks never touch parent[], so the pass that looks for winners
// can still read every record's roots from it).
template <int KIND, int K>
__global__ void __launch_bounds__(kTinyThreads, 1) tiny_msf_kernel(const TinyArgs a)
{
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ TinySmem s;
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, n = a.n;
    uint32_t *best_w = reinterpret_cast<uint32_t *>(dyn), *best_id = best_w + n;
    uint16_t *parent = reinterpret_cast<uint16_t *>(dyn + 8 * (size_t)n), *hook = parent + n;
    if (tid == 0) {
        s.live[0] = s.live[1] = s.choosers = s.err = s.comps = 0;
        s.total = 0;
    }
    stage_input(a.e0, a.m * (KIND == kKindMsf ? 12u : 8u), dyn);
    __syncthreads();
    uint32_t uv[K], w[KIND == kKindMsf ? K : 1], live = 0, heavy = 0, mine = 0;
    const uint32_t *e = reinterpret_cast<const uint32_t *>(dyn);
#pragma unroll
    for (int k = 0; k < K; k++) {
        const uint32_t id = k * kTinyThreads + tid;
        uv[k] = 0;
        if (KIND == kKindMsf)
            w[k] = 0;
        if (id >= a.m)
            continue;
        const uint32_t u = KIND == kKindMsf ? e[3 * id] : e[2 * id + 1], v = KIND == kKindMsf ? e[3 * id + 1] : e[2 * id];
        if (KIND == kKindMsf)
            w[k] = e[3 * id + 2];
        if (KIND == kKindMsf ? u == v : u >= v)
            continue;
        if (max(u, v) >= n) {
            atomicOr(&s.err, kErrRange);
            continue;
        }
        uv[k] = u | v << 16;
        if (KIND == kKindMsf || id < a.light)
            live |= 1u << k;
        else
            heavy |= 1u << k;
    }
    __syncthreads();
    for (uint32_t x = tid; x < n; x += kTinyThreads) {
        best_w[x] = best_id[x] = 0xffffffffu;
        parent[x] = hook[x] = (uint16_t)x;
        if (KIND == kKindPacked && a.forest)
            a.forest[x] = kForestEmpty;
    }
    __syncthreads();
    uint32_t r = 0, light_rounds = 0;
    for (;; r++) {
        // edge pass; a record is only looked at again where its key was not
        // above the minimum it met (may: bit 2k for its first root, 2k + 1)
        uint32_t may = 0;
#pragma unroll
        for (int k = 0; k < K; k++)
            if (live >> k & 1) {
                const uint32_t ru = parent[uv[k] & 0xffffu], rv = parent[uv[k] >> 16];
                if (ru == rv) {
                    live &= ~(1u << k);
                } else {
                    const uint32_t x = KIND == kKindMsf ? w[KIND == kKindMsf ? k : 0] : k * kTinyThreads + tid;
                    const uint32_t bu = *(volatile uint32_t *)(best_w + ru), bv = *(volatile uint32_t *)(best_w + rv);
                    if (x < bu)
                        atomicMin(best_w + ru, x);
                    if (x < bv)
                        atomicMin(best_w + rv, x);
                    may |= ((uint32_t)(x <= bu) | (uint32_t)(x <= bv) << 1) << 2 * k;
                }
            }
        {
            const uint32_t c = __reduce_add_sync(0xffffffffu, __popc(live));
            if (lane == 0 && c)
                atomicAdd(&s.live[r & 1], c);
        }
        __syncthreads();
        const uint32_t m_r = s.live[r & 1];
        if (tid == 0) {
            a.res->m_r[r] = m_r;
            a.res->n_r[r] = 0;
        }
        if (m_r == 0) {
            if (light_rounds == 0)
                light_rounds = r + 1;
            else {
                r++;
                break;
            }
            if (a.light == kKeyNone) {
                r++;
                break;
            }
            live = heavy;
            if (tid == 0)
                s.live[(r + 1) & 1] = 0;
            __syncthreads();
            continue;
        }
        if (KIND == kKindMsf) {
            // ties: the lowest id among the records of a root's lowest weight
#pragma unroll
            for (int k = 0; k < K; k++)
                if (may >> 2 * k & 3) {
                    const uint32_t id = k * kTinyThreads + tid, x = w[KIND == kKindMsf ? k : 0];
                    if (may >> 2 * k & 1) {
                        const uint32_t ru = parent[uv[k] & 0xffffu];
                        if (best_w[ru] == x)
                            atomicMin(best_id + ru, id);
                        else
                            may &= ~(1u << 2 * k);
                    }
                    if (may >> 2 * k & 2) {
                        const uint32_t rv = parent[uv[k] >> 16];
                        if (best_w[rv] == x)
                            atomicMin(best_id + rv, id);
                        else
                            may &= ~(2u << 2 * k);
                    }
                }
            __syncthreads();
        }
        // hook
        uint32_t ch = 0;
#pragma unroll
        for (int k = 0; k < K; k++)
            if (may >> 2 * k & 3) {
                const uint32_t ru = parent[uv[k] & 0xffffu], rv = parent[uv[k] >> 16];
                const uint32_t id = k * kTinyThreads + tid;
                const uint32_t *won = KIND == kKindMsf ? best_id : best_w;
                const bool A = (may >> 2 * k & 1) && won[ru] == id, B = (may >> 2 * k & 2) && won[rv] == id;
                if (A || B) {
                    uint32_t hk = A ? ru : rv, tgt = A ? rv : ru;
                    if (A && B) {
                        hk = max(ru, rv);
                        tgt = min(ru, rv);
                    }
                    hook[hk] = (uint16_t)tgt;
                    mine |= 1u << k;
                    live &= ~(1u << k);
                    ch += (uint32_t)A + (uint32_t)B;
                    if (KIND == kKindPacked && a.forest)
                        a.forest[hk] = (unsigned long long)(uv[k] & 0xffffu) << 32 | uv[k] >> 16;
                }
            }
        ch = __reduce_add_sync(0xffffffffu, ch);
        if (lane == 0 && ch)
            atomicAdd(&s.choosers, ch);
        if (tid == 0)
            s.live[(r + 1) & 1] = 0;
        __syncthreads();
        if (tid == 0) {
            a.res->n_r[r] = s.choosers;
            s.choosers = 0;
        }
        // compress: every vertex to its root, by halving over the hooks (no
        // hook is made here, so every pointer written is an ancestor)
        for (uint32_t x = tid; x < n; x += kTinyThreads) {
            volatile uint16_t *h = hook;
            uint32_t y = parent[x], p = h[y], steps = 0;
            while (p != y) {
                const uint32_t g = h[p];
                if (g == p) {
                    y = p;
                    break;
                }
                h[y] = (uint16_t)g;
                y = g;
                p = h[y];
                if (++steps > n) {
                    atomicOr(&s.err, kErrChase);
                    break;
                }
            }
            parent[x] = (uint16_t)y;
            best_w[x] = best_id[x] = 0xffffffffu;
        }
        __syncthreads();
        if (r + 1 >= PHEM_MAX_ROUNDS) {
            if (tid == 0)
                s.err |= kErrRounds;
            r++;
            break;
        }
    }
    // results
    uint32_t count = 0;
    if (KIND == kKindMsf) {
        // records ascending by id: rank by (row, warp, lane)
        unsigned long long sum = 0;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const unsigned b = __ballot_sync(0xffffffffu, mine >> k & 1);
            if (lane == 0)
                s.cnt[k][warp] = __popc(b);
            if (mine >> k & 1)
                sum += w[KIND == kKindMsf ? k : 0];
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
            sum += __shfl_xor_sync(0xffffffffu, sum, d);
        if (lane == 0 && sum)
            atomicAdd(&s.total, sum);
        __syncthreads();
        if (warp < K) {
            const uint32_t c = s.cnt[warp][lane];
            uint32_t inc = c;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= (uint32_t)d)
                    inc += y;
            }
            s.cnt[warp][lane] = inc - c;
            if (lane == 31)
                s.row[warp] = inc;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < K; k++) {
            const unsigned b = __ballot_sync(0xffffffffu, mine >> k & 1);
            if ((mine >> k & 1) && a.out) {
                phem_edge x;
                x.u = uv[k] & 0xffffu;
                x.v = uv[k] >> 16;
                x.w = w[KIND == kKindMsf ? k : 0];
                a.out[count + s.cnt[k][warp] + __popc(b & ((1u << lane) - 1u))] = x;
            }
            count += s.row[k];
        }
    } else {
        // minimum vertex id of each component
        uint32_t *minid = reinterpret_cast<uint32_t *>(dyn);
        for (uint32_t x = tid; x < n; x += kTinyThreads)
            minid[x] = 0xffffffffu;
        __syncthreads();
        uint32_t roots = 0;
        for (uint32_t x = tid; x < n; x += kTinyThreads) {
            atomicMin(minid + parent[x], x);
            roots += parent[x] == x;
        }
        roots = __reduce_add_sync(0xffffffffu, roots);
        if (lane == 0 && roots)
            atomicAdd(&s.comps, roots);
        __syncthreads();
        for (uint32_t x = tid; x < n; x += kTinyThreads)
            a.labels[x] = (int32_t)minid[parent[x]];
    }
    if (tid == 0) {
        Ctl *c = a.res;
        c->err = s.err;
        c->round = r;
        c->light_rounds = light_rounds;
        c->threshold = a.light;
        c->msf_count = count;
        c->msf_total = s.total;
        c->misc[0] = s.comps;
        c->misc[1] = n - s.comps;
        if (a.d_count_total) {
            a.d_count_total[0] = count;
            a.d_count_total[1] = s.total;
        }
    }
}

// Root of x in shared memory, by halving (ids fall towards the root, so the
// writes are atomic mins, as in uf.cuh).
__device__ __forceinline__ uint32_t tiny_find(volatile uint32_t *parent, uint32_t x, uint32_t n, uint32_t *err)
{
    for (uint32_t steps = 0; steps <= n; steps++) {
        const uint32_t p = parent[x];
        if (p == x)
            return x;
        const uint32_t g = parent[p];
        if (g == p)
            return p;
        atomicMin((uint32_t *)parent + x, g);
        x = g;
    }
    atomicOr(err, kErrChase);
    return x;
}

// Connected components: union-find as in cc.cu with the parent array in
// shared memory.
__global__ void __launch_bounds__(kTinyThreads, 1) tiny_cc_kernel(const TinyArgs a)
{
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ uint32_t s_err, s_comps;
    uint32_t *parent = reinterpret_cast<uint32_t *>(dyn);
    const uint32_t tid = threadIdx.x, n = a.n;
    if (tid == 0)
        s_err = s_comps = 0;
    for (uint32_t x = tid; x < n; x += kTinyThreads) {
        parent[x] = x;
        if (a.forest)
            a.forest[x] = kForestEmpty;
    }
    __syncthreads();
    const bool wide = ((uintptr_t)a.e0 & 15) == 0;
    const uint32_t pairs = wide ? a.m / 2 : 0;
    auto unite = [&](unsigned long long e) {
        uint32_t u = (uint32_t)(e >> 32), v = (uint32_t)e;
        if ((int32_t)u >= (int32_t)v)
            return;  // union_find_gpu_COO only unites u < v (CC/ExternalSpanningTree.cu:82)
        if ((int32_t)u < 0 || v >= n) {
            atomicOr(&s_err, kErrRange);
            return;
        }
        for (uint32_t retry = 0; retry < kUnionRetryCap; retry++) {
            u = tiny_find(parent, u, n, &s_err);
            v = tiny_find(parent, v, n, &s_err);
            if (u == v)
                return;
            const uint32_t hi = max(u, v), lo = min(u, v);
            const uint32_t old = atomicCAS(parent + hi, hi, lo);
            if (old == hi) {
                if (a.forest)
                    a.forest[hi] = e;
                return;
            }
            u = old;
            v = lo;
        }
        atomicOr(&s_err, kErrRetry);
    };
    const uint4 *q = static_cast<const uint4 *>(a.e0);
    const unsigned long long *q1 = static_cast<const unsigned long long *>(a.e0);
    for (uint32_t i0 = tid; i0 < pairs; i0 += 4 * kTinyThreads) {
        uint4 x[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
            x[k] = i0 + k * kTinyThreads < pairs ? __ldcs(q + i0 + k * kTinyThreads) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            unite((unsigned long long)x[k].y << 32 | x[k].x);
            unite((unsigned long long)x[k].w << 32 | x[k].z);
        }
    }
    for (uint32_t i = 2 * pairs + tid; i < a.m; i += kTinyThreads)
        unite(__ldcs(q1 + i));
    __syncthreads();
    uint32_t roots = 0;
    for (uint32_t x = tid; x < n; x += kTinyThreads) {
        const uint32_t r = tiny_find(parent, x, n, &s_err);
        a.labels[x] = (int32_t)r;
        roots += r == x;
    }
    roots = __reduce_add_sync(0xffffffffu, roots);
    if (lane_id() == 0 && roots)
        atomicAdd(&s_comps, roots);
    __syncthreads();
    if (tid == 0) {
        Ctl *c = a.res;
        c->err = s_err;
        c->round = 0;
        c->misc[0] = s_comps;
        c->misc[1] = n - s_comps;
    }
}

template <class F>
phem_status launch(phem_context *ctx, F *kernel, uint32_t bit, const TinyArgs &a, size_t smem)
{
    if (!(ctx->tiny_ready & (1u << bit))) {
        PHEM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTinyDynSmem));
        ctx->tiny_ready |= 1u << bit;
    }
    kernel<<<1, kTinyThreads, smem, ctx->stream>>>(a);
    PHEM_CUDA_TRY(cudaGetLastError());
    return PHEM_OK;
}

// The smallest K that holds the records.
template <int KIND>
phem_status launch_msf(phem_context *ctx, const TinyArgs &a)
{
    constexpr uint32_t rec = KIND == kKindMsf ? 12 : 8;
    const size_t smem = std::max<size_t>((size_t)a.n * 12, (size_t)a.m * rec) + 16;
    KernelScope ks(ctx, kKSolve);
    if (a.m <= 4 * kTinyThreads)
        return launch(ctx, tiny_msf_kernel<KIND, 4>, KIND * 3, a, smem);
    if (a.m <= 8 * kTinyThreads)
        return launch(ctx, tiny_msf_kernel<KIND, 8>, KIND * 3 + 1, a, smem);
    return launch(ctx, tiny_msf_kernel<KIND, 16>, KIND * 3 + 2, a, smem);
}

}  // namespace

phem_status tiny_host(phem_context *ctx, char **buf)
{
    if (!ctx->tiny_host && cudaMallocHost(&ctx->tiny_host, kTinyHostBytes) != cudaSuccess) {
        cudaGetLastError();
        ctx->tiny_host = nullptr;
        set_error("small solve: cannot allocate %zu bytes of pinned staging", kTinyHostBytes);
        return PHEM_ERR_NOMEM;
    }
    *buf = static_cast<char *>(ctx->tiny_host);
    return PHEM_OK;
}

phem_status tiny_input(phem_context *ctx, const void *p, size_t bytes, size_t word, void *ws, const void **in)
{
    *in = p;
    if (!bytes)
        return PHEM_OK;
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
        cudaGetLastError();
        attr.type = cudaMemoryTypeUnregistered;
    }
    const bool fits = (uintptr_t)p % word == 0;
    if (attr.type == cudaMemoryTypeDevice && attr.device == ctx->device && fits)
        return PHEM_OK;
    if (attr.type == cudaMemoryTypeHost && attr.devicePointer && fits) {
        *in = attr.devicePointer;
        return PHEM_OK;
    }
    if (attr.type == cudaMemoryTypeUnregistered && !ctx->tiny_busy) {
        char *buf = nullptr;
        PHEM_TRY(tiny_host(ctx, &buf));
        std::memcpy(buf, p, bytes);
        ctx->tiny_busy = ctx->stream;
        *in = buf;
        return PHEM_OK;
    }
    *in = ws;
    PHEM_CUDA_TRY(cudaMemcpyAsync(ws, p, bytes, cudaMemcpyDefault, ctx->stream));
    return PHEM_OK;
}

bool tiny_msf_fits(uint64_t m, uint64_t n) { return m <= kTinyMaxEdges && n <= kTinyMaxVertices; }
bool tiny_cc_fits(int64_t m, int64_t n) { return m <= kTinyCcMaxEdges && n <= kTinyCcMaxVertices; }

phem_status tiny_msf(phem_context *ctx, const phem_edge *d_edges, uint32_t m, uint32_t n, phem_edge *d_out,
                     uint64_t *d_count_total)
{
    TinyArgs a{};
    a.e0 = d_edges;
    a.m = m;
    a.n = n;
    a.light = kKeyNone;
    a.out = d_out;
    a.d_count_total = d_count_total;
    a.res = ctx->h_ctl;
    return launch_msf<kKindMsf>(ctx, a);
}

phem_status tiny_canonical(phem_context *ctx, const uint64_t *d_edges, uint32_t m, uint32_t n, uint64_t light,
                           int32_t *d_labels, uint64_t *d_forest)
{
    TinyArgs a{};
    a.e0 = d_edges;
    a.m = m;
    a.n = n;
    a.light = light;
    a.labels = d_labels;
    a.forest = reinterpret_cast<unsigned long long *>(d_forest);
    a.res = ctx->h_ctl;
    return launch_msf<kKindPacked>(ctx, a);
}

phem_status tiny_cc(phem_context *ctx, const uint64_t *d_edges, uint32_t m, uint32_t n, int32_t *d_labels,
                    uint64_t *d_forest)
{
    TinyArgs a{};
    a.e0 = d_edges;
    a.m = m;
    a.n = n;
    a.labels = d_labels;
    a.forest = reinterpret_cast<unsigned long long *>(d_forest);
    a.res = ctx->h_ctl;
    KernelScope ks(ctx, kKCcSolve);
    return launch(ctx, tiny_cc_kernel, 6, a, (size_t)n * 4 + 16);
}

}  // namespace phem
