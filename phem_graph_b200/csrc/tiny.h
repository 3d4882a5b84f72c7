// tiny.h -- solves of small graphs by one CTA (tiny.cu).
#pragma once

#include "internal.h"

namespace phem {

// Limits: 16 records per thread in registers; 12 bytes of shared memory per
// vertex (MSF) or 4 (CC), and the staged input, within one CTA's 227 KB.  At
// the limits one CTA still wins, us per call against the grid's: MSF n = 4003,
// m = 16384 104 / 200, n = 15000 128 / 247; canonical n = 15000 116 / 183; CC
// n = 20000, m = 32768 63 / 72 (m = 65536, n = 32768 it loses, 93 / 76).
constexpr uint32_t kTinyMaxEdges = 16384, kTinyMaxVertices = 16384;
constexpr uint32_t kTinyCcMaxEdges = 32768, kTinyCcMaxVertices = 32768;
static_assert(kTinyCcMaxEdges * 8 >= kTinyMaxEdges * 12, "the staging buffer's input part holds either kind");
constexpr size_t kTinyDynSmem = 16384 * 12 + 16;

// The context's pinned staging buffer: a small solve's pageable input at 0, its
// host output records at kTinyHostOut.
constexpr size_t kTinyHostOut = kTinyCcMaxEdges * 8, kTinyHostBytes = kTinyHostOut + kTinyMaxVertices * 12;
phem_status tiny_host(phem_context *ctx, char **buf);

// The pointer the kernel reads a small input from: device memory of the
// context's device and pinned host memory in place, so in stream order like
// everything else that earlier work on the stream may write; pageable memory
// through the pinned buffer, unless a launch that reads the buffer may still be
// queued (a call that timed out); anything else through `ws` (device workspace,
// `bytes` large).  In place only on a multiple of `word`, the kernel's narrowest
// reads (4 bytes of {u, v, w} records, 8 of packed pairs).
phem_status tiny_input(phem_context *ctx, const void *p, size_t bytes, size_t word, void *ws, const void **in);

bool tiny_msf_fits(uint64_t m, uint64_t n);
bool tiny_cc_fits(int64_t m, int64_t n);

// Each queues one launch on the context stream; the pointers are device (or
// mapped pinned host) memory.  Results: err, round, light_rounds, threshold,
// m_r, n_r, msf_count and msf_total (MSF) or misc[0] = components, misc[1] =
// forest edges (CC) in ctx->h_ctl once the stream has been waited for.
phem_status tiny_msf(phem_context *ctx, const phem_edge *d_edges, uint32_t m, uint32_t n, phem_edge *d_out,
                     uint64_t *d_count_total);
phem_status tiny_canonical(phem_context *ctx, const uint64_t *d_edges, uint32_t m, uint32_t n, uint64_t light,
                           int32_t *d_labels, uint64_t *d_forest);
phem_status tiny_cc(phem_context *ctx, const uint64_t *d_edges, uint32_t m, uint32_t n, int32_t *d_labels,
                    uint64_t *d_forest);

}  // namespace phem
