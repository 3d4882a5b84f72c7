// csr.cu -- symmetrised CSR -> packed COO (or {u, v, w} records) on sm_100a.
//
// csr_to_coo (CC/graph.cu:149-196) walks rows in order and emits (i << 32 | col)
// for every entry with i < col.  Here the entries are cut into segments of 256
// consecutive entries, each handled by one warp on its own -- no block
// barrier anywhere -- with eight consecutive entries per lane:
//   1. csr_seg_rows_kernel writes for every segment the row that holds its
//      first entry, so no segment searches the offsets;
//   2. csr_pass_kernel<kCount>: a warp marks, in its shared memory, where each
//      row inside its segment starts, resolves the row of every entry from the
//      marks and counts the entries with row < col;
//   3. csr_scan_kernel turns the counts into offsets: every block scans a group
//      of 4096 segments and the last block to finish scans the groups' totals
//      (no block waits for another);
//   4. csr_pass_kernel<kPairs or kRecords> resolves the rows again and writes
//      the kept entries in order: group offset + segment offset + the lanes
//      before.  The record form fuses the MSF CSR input's packing: the
//      kept entry at position p becomes {row, col, w[p]}; a warp's pairs or
//      records are put together in shared memory and leave as 16-byte stores
//      (pairs by 8-byte stores from the lanes, four times the L2 sectors:
//      R-MAT 20 212 us per call against 177).
// Every entry keeps its place in the reference's row walk, so the output order
// (and therefore the edge numbering) is exactly the reference's.  The next
// segment's columns and row range are loaded while the current one is worked
// on.
//
// R-MAT 20 (33.5 M entries; 134 MB read by pass 2, 402 MB moved by pass 4), us
// of passes 1-4: 18 / 50 / 10 / 103 (13 / 72 / 9 / 148 with a block per 2048
// entries, two block barriers each and 4-byte stores).  Bound: the latency of
// the offsets' loads (without the marks pass 2 takes 31), above all in the
// segments at the end that span up to 2,000 nearly empty rows.  A decoupled
// look-back over 740 running blocks instead of passes 2 and 3: 2480.
#include <algorithm>

#include "internal.h"

namespace phem {
namespace {

constexpr int kCsrThreads = 256;
constexpr int kCsrWarps = kCsrThreads / 32;
constexpr int kCsrItems = 8;           // entries per lane
constexpr int kCsrSeg = 32 * kCsrItems;
// Blocks per SM: the write passes hold more registers and staging.
constexpr int csr_blocks_per_sm(int mode) { return mode == 0 ? 5 : 4; }
constexpr int kAhead = 4;              // rows per lane whose offsets are loaded together
constexpr int kScanBlock = 1024;
constexpr int kScanItems = 4;
constexpr int kScanGroup = kScanBlock * kScanItems;  // segments per block of pass 3

enum CsrMode : int { kCount = 0, kPairs, kRecords };

// seg_rows[t] = the row i with offsets[i] <= t * kCsrSeg < offsets[i + 1].
// A row of many segments is written by its whole warp.  Malformed offsets
// leave segments unwritten; the conversion clamps what it reads.
__global__ void __launch_bounds__(kBlock) csr_seg_rows_kernel(const int64_t *offsets, int32_t n, uint32_t nseg,
                                                              uint32_t *seg_rows, unsigned long long *ticket)
{
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *ticket = 0;  // of the scan, two launches on
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const uint32_t lane = lane_id();
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x; i0 < n; i0 += stride) {
        const int64_t i = i0 + threadIdx.x;
        int64_t t = 0, t1 = -1;
        if (i < n) {
            const int64_t a = std::max<int64_t>(__ldg(offsets + i), 0), b = __ldg(offsets + i + 1);
            if (a < b) {
                t = (a + kCsrSeg - 1) / kCsrSeg;
                t1 = std::min<int64_t>((b - 1) / kCsrSeg, (int64_t)nseg - 1);
            }
        }
        const bool wide = t1 - t >= 8;
        if (!wide)
            for (; t <= t1; t++)
                seg_rows[t] = (uint32_t)i;
        for (unsigned todo = __ballot_sync(0xffffffffu, wide); todo; todo &= todo - 1) {
            const int src = __ffs(todo) - 1;
            const int64_t from = __shfl_sync(0xffffffffu, t, src), to = __shfl_sync(0xffffffffu, t1, src);
            const uint32_t row = (uint32_t)(i - (int64_t)lane + src);
            for (int64_t q = from + lane; q <= to; q += 32)
                seg_rows[q] = row;
        }
    }
}

// The columns of this lane's entries of segment t (zero past the end: below no
// row).  `wide`: cols is 16-byte aligned.
__device__ __forceinline__ void load_cols(const uint32_t *cols, int64_t nnz, uint32_t t, uint32_t nseg, bool wide,
                                          uint32_t (&c)[kCsrItems])
{
    if (t >= nseg)
        return;
    const int64_t j0 = (int64_t)t * kCsrSeg + lane_id() * kCsrItems;
    if (wide && j0 + kCsrItems <= nnz) {
        const uint4 *p = reinterpret_cast<const uint4 *>(cols + j0);
        const uint4 a = __ldcs(p), b = __ldcs(p + 1);
        c[0] = a.x, c[1] = a.y, c[2] = a.z, c[3] = a.w;
        c[4] = b.x, c[5] = b.y, c[6] = b.z, c[7] = b.w;
        return;
    }
#pragma unroll
    for (int k = 0; k < kCsrItems; k++)
        c[k] = j0 + k < nnz ? __ldcs(cols + j0 + k) : 0u;
}

// The rows holding the first entry of segment t and of the next one, clamped
// to [0, n).
__device__ __forceinline__ void load_row_range(const uint32_t *seg_rows, int32_t n, uint32_t t, uint32_t nseg,
                                               int32_t &row0, int32_t &row1)
{
    if (t >= nseg)
        return;
    row0 = (int32_t)min(__ldg(seg_rows + t), (uint32_t)(n - 1));
    row1 = max(row0, t + 1 < nseg ? (int32_t)min(__ldg(seg_rows + t + 1), (uint32_t)(n - 1)) : n - 1);
}

// Rows of this lane's entries and their keep flags (bit k: entry k has
// row < col).  mark[o - first] = r for every non-empty row r > row0 that starts
// inside the segment.  Rows ascend, so an entry's row is the largest mark up to
// it: a running maximum over the lane's eight marks and one scan over the
// lanes.  Marks are never cleared: a warp's segments ascend, so what an earlier
// one left is at most this one's row0.
__device__ __forceinline__ uint32_t resolve_rows(const int64_t *offsets, int64_t first, int64_t end, int32_t row0,
                                                 int32_t row1, uint32_t *mark, const uint32_t (&col)[kCsrItems],
                                                 uint32_t (&row)[kCsrItems])
{
    const uint32_t lane = lane_id();
    __syncwarp();  // the last segment's marks are read
    {
        const int64_t r = (int64_t)row0 + 1 + lane;
        if (r <= row1) {
            const int64_t o = __ldg(offsets + r), on = __ldg(offsets + r + 1);
            if (o > first && o < end && on > o)
                mark[o - first] = (uint32_t)r;
        }
    }
    // a segment of nearly empty rows spans thousands of them: kAhead rows' loads
    // per lane in flight together
    for (int64_t r0 = (int64_t)row0 + 33 + lane; r0 <= row1; r0 += 32 * kAhead) {
        int64_t o[kAhead], on[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; q++) {
            const int64_t r = min(r0 + 32 * q, (int64_t)row1);
            o[q] = __ldg(offsets + r);
            on[q] = __ldg(offsets + r + 1);
        }
#pragma unroll
        for (int q = 0; q < kAhead; q++)
            if (r0 + 32 * q <= row1 && o[q] > first && o[q] < end && on[q] > o[q])
                mark[o[q] - first] = (uint32_t)(r0 + 32 * q);
    }
    __syncwarp();
    const uint4 a = reinterpret_cast<const uint4 *>(mark)[2 * lane], b = reinterpret_cast<const uint4 *>(mark)[2 * lane + 1];
    row[0] = max(a.x, (uint32_t)row0);
    row[1] = max(row[0], a.y);
    row[2] = max(row[1], a.z);
    row[3] = max(row[2], a.w);
    row[4] = max(row[3], b.x);
    row[5] = max(row[4], b.y);
    row[6] = max(row[5], b.z);
    row[7] = max(row[6], b.w);
    uint32_t before = row[7];  // the largest mark up to this lane's end ...
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, before, d);
        if (lane >= (uint32_t)d)
            before = max(before, y);
    }
    before = __shfl_up_sync(0xffffffffu, before, 1);  // ... up to the lane before
    if (lane == 0)
        before = (uint32_t)row0;
    uint32_t keep = 0;
#pragma unroll
    for (int k = 0; k < kCsrItems; k++) {
        row[k] = max(row[k], before);
        keep |= (uint32_t)(row[k] < col[k]) << k;
    }
    return keep;
}

// Passes 2 and 4.  kCount: counts[t] = kept entries of segment t.  kRecords:
// {row, col, w[p]} to rec_out[p] for p < cap; kPairs: packed pairs to out.
template <int MODE>
__global__ void __launch_bounds__(kCsrThreads, csr_blocks_per_sm(MODE))
    csr_pass_kernel(const int64_t *offsets, const uint32_t *cols, int32_t n, int64_t nnz, const uint32_t *seg_rows,
                    uint32_t *counts, const uint32_t *prefix, const uint32_t *group_off, unsigned long long *out,
                    const uint32_t *w, phem_edge *rec_out, uint64_t cap)
{
    __shared__ __align__(16) uint32_t s_mark[kCsrWarps][kCsrSeg];
    __shared__ __align__(16) uint32_t s_out[kCsrWarps][MODE == kRecords ? kCsrSeg * 3 + 4 : MODE == kPairs ? kCsrSeg * 2 + 4 : 4];
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    const bool wide = ((uintptr_t)cols & 15) == 0;
    const uint32_t nseg = (uint32_t)((nnz + kCsrSeg - 1) / kCsrSeg);
    const uint32_t GW = gridDim.x * kCsrWarps;
    uint32_t *mark = s_mark[warp];
    for (uint32_t i = lane; i < kCsrSeg; i += 32)
        mark[i] = 0;
    uint32_t t = blockIdx.x * kCsrWarps + warp;
    uint32_t nc[kCsrItems];
    int32_t nrow0 = 0, nrow1 = 0;
    load_row_range(seg_rows, n, t, nseg, nrow0, nrow1);
    load_cols(cols, nnz, t, nseg, wide, nc);
    for (; t < nseg; t += GW) {
        uint32_t col[kCsrItems], row[kCsrItems];
#pragma unroll
        for (int k = 0; k < kCsrItems; k++)
            col[k] = nc[k];
        const int32_t row0 = nrow0, row1 = nrow1;
        // in flight while this segment is worked on (no overflow: nseg < 2^24)
        load_row_range(seg_rows, n, t + GW, nseg, nrow0, nrow1);
        load_cols(cols, nnz, t + GW, nseg, wide, nc);
        const uint64_t base = MODE == kCount ? 0 : (uint64_t)__ldg(prefix + t) + __ldg(group_off + t / kScanGroup);
        const int64_t first = (int64_t)t * kCsrSeg;
        const uint32_t keep = resolve_rows(offsets, first, min(first + kCsrSeg, nnz), row0, row1, mark, col, row);
        if (MODE == kCount) {
            const uint32_t kept = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(keep));
            if (lane == 0)
                counts[t] = kept;
            continue;
        }
        uint32_t at = __popc(keep);  // place of the lane's first kept entry
        const uint32_t own = at;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, at, d);
            if (lane >= (uint32_t)d)
                at += y;
        }
        uint32_t total = __shfl_sync(0xffffffffu, at, 31);
        at -= own;
        if (MODE == kPairs) {
            // as the records below, in 16-byte stores of two pairs
            const uint32_t shift = (uint32_t)((reinterpret_cast<uintptr_t>(out) >> 3) + base) & 1u;
            unsigned long long *so = reinterpret_cast<unsigned long long *>(s_out[warp]);
#pragma unroll
            for (int k = 0; k < kCsrItems; k++)
                if (keep >> k & 1)
                    so[shift + at++] = ((unsigned long long)row[k] << 32) | col[k];
            __syncwarp();
            const uint32_t end = shift + total;
            unsigned long long *g = out + base - shift;
            for (uint32_t c = lane * 2; c < end; c += 64) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(so + c);
                if (c >= shift && c + 2 <= end) {
                    __stcs(reinterpret_cast<ulonglong2 *>(g + c), v);
                } else {
                    if (c >= shift)
                        g[c] = v.x;
                    if (c + 1 >= shift && c + 1 < end)
                        g[c + 1] = v.y;
                }
            }
            continue;
        }
        if (base + total > cap)  // a wrong entry count: only the first cap records are written
            total = base < cap ? (uint32_t)(cap - base) : 0u;
        // at the output's own offset from a 16-byte boundary; the weights of
        // the segment's records are contiguous
        const uint32_t shift = (uint32_t)(base * 3) & 3u;
        uint32_t *so = s_out[warp] + shift;
        const uint32_t *wp = w + base;
        for (uint32_t i = lane; i < total; i += 64) {
            const uint32_t x = __ldcs(wp + i), y = i + 32 < total ? __ldcs(wp + i + 32) : 0u;
            so[3 * i + 2] = x;
            if (i + 32 < total)
                so[3 * i + 98] = y;
        }
#pragma unroll
        for (int k = 0; k < kCsrItems; k++)
            if (keep >> k & 1) {
                so[3 * at] = row[k];
                so[3 * at + 1] = col[k];
                at++;
            }
        __syncwarp();
        const uint32_t end = shift + 3 * total;
        uint32_t *g = reinterpret_cast<uint32_t *>(rec_out) + (base * 3 - shift);
        for (uint32_t c = lane * 4; c < end; c += 128) {
            const uint4 v = *reinterpret_cast<const uint4 *>(s_out[warp] + c);
            if (c >= shift && c + 4 <= end) {
                __stcs(reinterpret_cast<uint4 *>(g + c), v);
            } else {
                const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int x = 0; x < 4; x++)
                    if (c + x >= shift && c + x < end)
                        g[c + x] = q[x];
            }
        }
        // (the next segment's resolve_rows synchronises before so is rewritten)
    }
}

// Pass 3: prefix[t] = kept entries before segment t within its group of
// kScanGroup (one block per group, kScanItems segments per thread); the
// last block to finish scans the group totals into group_off[] and writes
// the whole count to *kept and to the host's pinned *host_kept.
__global__ void __launch_bounds__(kScanBlock) csr_scan_kernel(const uint32_t *counts, uint32_t nseg,
                                                              uint32_t *prefix, uint32_t *group_tot,
                                                              uint32_t *group_off, unsigned long long *kept,
                                                              unsigned long long *host_kept,
                                                              unsigned long long *ticket)
{
    __shared__ uint32_t s_w[kScanBlock / 32 + 1];
    __shared__ bool s_last;
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    // exclusive scan of one value per thread over the block; *total = the sum
    auto block_scan = [&](uint32_t x, uint32_t *total) {
        uint32_t inc = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= (uint32_t)d)
                inc += y;
        }
        if (lane == 31)
            s_w[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            const uint32_t a = s_w[lane];
            uint32_t z = a;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, z, d);
                if (lane >= (uint32_t)d)
                    z += y;
            }
            s_w[lane] = z - a;
            if (lane == 31)
                s_w[32] = z;
        }
        __syncthreads();
        *total = s_w[32];
        const uint32_t r = s_w[warp] + inc - x;
        __syncthreads();  // s_w is reused
        return r;
    };
    const uint64_t i0 = (uint64_t)blockIdx.x * kScanGroup + (uint64_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems], sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        v[k] = i0 + k < nseg ? counts[i0 + k] : 0u;
        sum += v[k];
    }
    uint32_t total;
    uint32_t run = block_scan(sum, &total);
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
        if (i0 + k < nseg) {
            prefix[i0 + k] = run;
            run += v[k];
        }
    if (threadIdx.x == 0) {
        group_tot[blockIdx.x] = total;
        __threadfence();
        s_last = atomicAdd(ticket, 1ull) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    uint64_t carry = 0;
    for (uint32_t g0 = 0; g0 < gridDim.x; g0 += kScanBlock) {
        const uint32_t g = g0 + threadIdx.x;
        const uint32_t x = g < gridDim.x ? __ldcg(group_tot + g) : 0u;
        uint32_t s;
        const uint32_t ex = block_scan(x, &s);
        if (g < gridDim.x)
            group_off[g] = (uint32_t)carry + ex;
        carry += s;
    }
    if (threadIdx.x == 0)
        *kept = *host_kept = carry;
}

}  // namespace

size_t csr_scratch_bytes(int64_t nnz)
{
    const size_t segs = (size_t)((nnz + kCsrSeg - 1) / kCsrSeg);
    const size_t groups = (segs + kScanGroup - 1) / kScanGroup;
    return align256((3 * segs + 1 + 2 * groups) * sizeof(uint32_t));
}

phem_status csr_launch_to_coo(phem_context *ctx, const int64_t *offsets, const uint32_t *cols, int32_t n,
                              int64_t nnz, uint32_t *scratch, uint64_t *out, const uint32_t *w, phem_edge *records,
                              uint64_t cap)
{
    if (nnz < 0 || (uint64_t)nnz >= (1ull << 32)) {
        set_error("csr: %lld entries (must be < 2^32)", (long long)nnz);
        return PHEM_ERR_INVALID;
    }
    const uint64_t segs = ((uint64_t)nnz + kCsrSeg - 1) / kCsrSeg;
    if (segs == 0 || n <= 0) {
        PHEM_CUDA_TRY(cudaMemsetAsync(&ctx->ctl->misc[2], 0, sizeof(unsigned long long), ctx->stream));
        *ctx->h_kept = 0;
        return PHEM_OK;
    }
    const uint64_t groups = (segs + kScanGroup - 1) / kScanGroup;
    uint32_t *seg_rows = scratch, *counts = scratch + segs + 1, *prefix = counts + segs;
    uint32_t *group_tot = prefix + segs, *group_off = group_tot + groups;
    auto *o = reinterpret_cast<unsigned long long *>(out);
    auto pass = [&](auto kernel, int mode) {
        KernelScope k(ctx, kKCsrCoo);
        const int blocks = (int)std::min<uint64_t>((segs + kCsrWarps - 1) / kCsrWarps,
                                                   (uint64_t)ctx->sm_count * csr_blocks_per_sm(mode));
        kernel<<<blocks, kCsrThreads, 0, ctx->stream>>>(offsets, cols, n, nnz, seg_rows, counts, prefix, group_off, o, w,
                                                        records, cap);
    };
    {
        KernelScope k(ctx, kKCsrCoo);
        const int rblocks = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)n + kBlock - 1) / kBlock,
                                                                         (int64_t)ctx->sm_count * 8));
        csr_seg_rows_kernel<<<rblocks, kBlock, 0, ctx->stream>>>(offsets, n, (uint32_t)segs, seg_rows,
                                                                &ctx->ctl->misc[3]);
    }
    pass(csr_pass_kernel<kCount>, kCount);
    {
        KernelScope k(ctx, kKCsrCoo);
        csr_scan_kernel<<<(unsigned)groups, kScanBlock, 0, ctx->stream>>>(counts, (uint32_t)segs, prefix, group_tot,
                                                                         group_off, &ctx->ctl->misc[2],
                                                                         reinterpret_cast<unsigned long long *>(ctx->h_kept),
                                                                         &ctx->ctl->misc[3]);
    }
    if (records)
        pass(csr_pass_kernel<kRecords>, kRecords);
    else if (out)
        pass(csr_pass_kernel<kPairs>, kPairs);
    PHEM_CUDA_TRY(cudaGetLastError());
    return PHEM_OK;
}

}  // namespace phem
