// batch.h -- device layout and launch plumbing of the batched engine.
#pragma once

#include <vector>

#include "internal.h"

namespace phem {

// Internal kind: a CC graph whose edges are packed pairs (u << 32 | v) in
// BatchArgs::pairs at e_off (the serving loop's CC requests).
constexpr uint32_t kBatchPairs = 2;

// One graph as the kernel sees it, in queue order (largest first).  Scratch
// offsets are the host's exclusive prefix sums, so graphs whose caller edge
// ranges overlap or leave gaps still get private scratch.
struct BatchItem {
    uint64_t e_off;   // first input record (caller's edge_offset)
    uint64_t wl_off;  // first survivor-list record (prefix sum of m)
    uint32_t m, n;
    uint32_t v_off;   // caller's vertex_offset: outputs and global vertex state
    uint32_t kind;    // PHEM_BATCH_MSF, PHEM_BATCH_CC or kBatchPairs
    uint32_t bm_off;  // first word of the graph's forest bitmap (prefix sum of ceil(m / 32))
    uint32_t index;   // caller's graph index: per-graph outputs
};
static_assert(sizeof(BatchItem) == 40, "BatchItem layout");

struct BatchArgs {
    const BatchItem *items;
    const uint32_t *num_graphs;  // device word, so one captured launch serves any batch size
    uint32_t *queue;             // next item to take (zeroed before each launch)
    const phem_edge *edges;
    const unsigned long long *pairs;  // kBatchPairs graphs' input (may be null otherwise)
    uint4 *wl;                   // sum of m records
    uint32_t *bitmap;            // sum of ceil(m / 32) words
    unsigned long long *g_best;  // vertex state of graphs too large for shared memory
    uint32_t *g_parent;
    uint32_t *g_aux;
    uint32_t *g_roots;
    uint32_t *msf_ids;           // vertex-indexed: graph g's forest at [vertex_offset, + count)
    uint32_t *msf_count;         // per graph
    unsigned long long *msf_total;
    int32_t *labels;             // vertex-indexed
    uint32_t *status;            // per graph error bits
    uint32_t *rounds;            // per graph Boruvka rounds (may be null)
    uint32_t smem_vertices;      // set by batch_launch
    float compact_ratio;         // compact a list pass when live <= ratio * length
};

// One graph as the grid kernel (batch_grid.cu) sees it.
struct GridItem {
    uint64_t e_off;   // first input record
    uint32_t m, n;
    uint32_t v_off;   // caller's vertex_offset: outputs
    uint32_t kind, index;
    uint32_t tile0;   // the graph's first tile of the union
    uint32_t vb;      // the graph's first vertex of the union (a multiple of 32)
    uint32_t skip;    // records between the first tile's aligned start and e_off
};
// Sizes of one launch of it (device memory, so one captured launch serves any
// batch).
struct GridHdr {
    uint32_t items, tiles, vertices, pad;
};
// Its device buffers.
struct BatchGrid {
    GridHdr *hdr = nullptr;  // one per launch: the whole batch's, then the groups'
    GridItem *items = nullptr;
    Ctl *ctl = nullptr;
    void *tiles = nullptr;
    uint32_t *vitem = nullptr, *parent = nullptr, *bitmap = nullptr, *tile_off = nullptr, *cta_tot = nullptr,
             *hooked = nullptr;
    unsigned long long *best = nullptr, *thr = nullptr;
    uint64_t best_stride = 0;
};

struct BatchLaunch {
    const void *kernel = nullptr;
    int block = 0, items = 0, grid = 0;
    size_t dyn_smem = 0;
    uint32_t smem_vertices = 0;
};

// Device buffers of one batch (context workspace or plan memory).
struct BatchBuffers {
    BatchItem *items;
    uint32_t *num_graphs, *queue;
    phem_edge *edges;
    uint4 *wl;
    uint32_t *bitmap, *g_parent, *g_aux, *g_roots;
    unsigned long long *g_best;
    uint32_t *msf_ids, *msf_count;
    unsigned long long *msf_total;
    int32_t *labels;
    uint32_t *status, *rounds;
};

// A large batch whose edges are in host memory is copied in kBatchGroups
// chunks on the copy stream; the graphs whose edges are complete after chunk
// k form launch k, which waits only for that chunk's copy, so the copies and
// the solves overlap.
constexpr int kBatchGroups = 4;
constexpr uint64_t kBatchOverlapMinEdges = 1ull << 22;
struct BatchGroups {
    int k = 0;                           // launches; 0: one launch after one copy
    uint64_t bound[kBatchGroups + 1];    // edge chunk boundaries
    uint32_t start[kBatchGroups] = {};   // first item of each launch (queue order)
    uint32_t count[kBatchGroups] = {};   // items of each launch
};

// Validated work items in queue order (largest graphs first, so the longest
// solves start early and the persistent grid finishes together), with the
// private scratch offsets of every graph.
struct BatchLayout {
    std::vector<BatchItem> items;
    uint64_t wl_records = 0;
    uint64_t bm_words = 0;
};

// Validates caller graphs (ranges, kinds, non-overlapping vertex ranges) and
// builds the queue-ordered items with private scratch offsets.
phem_status build_items(const phem_batch_graph *graphs, uint32_t G, uint64_t total_edges, uint32_t total_vertices,
                        BatchLayout *L);
// Carves every buffer for the given capacities out of `base` (null: sizing
// only); returns the bytes needed.
size_t batch_carve(uint32_t G, uint64_t E, uint64_t wl, uint64_t bm, uint32_t V, bool edges_inline, char *base,
                   BatchBuffers *b);
BatchArgs make_args(const BatchBuffers &b, const phem_edge *edges, float ratio);

// ---- one union over the whole grid (batch_grid.cu) ----
constexpr float kGridLightMsf = 1.f;  // light edges per vertex of a weighted graph
// The CTAs it launches.
uint32_t batch_grid_ctas(int sm_count);
// True when the batch goes to the grid kernel rather than to configuration l of
// the other one.
bool batch_takes_grid(const BatchLayout &L, const BatchLaunch &l, int sm_count);
// List records its survivor segments need.
uint64_t batch_grid_list(uint64_t records, uint32_t G, int sm_count);
// Carves its buffers behind `off` (base null: sizing only); returns the end.
size_t batch_grid_carve(uint32_t G, uint64_t records, uint32_t V, int sm_count, size_t off, char *base, BatchGrid *g);
// The grid form of `items` (one launch's), and its sizes.
GridHdr batch_grid_items(const BatchItem *items, uint32_t G, GridItem *out);
// Queues launch `group` (its header) over the items from `first` on.
phem_status batch_grid_launch(cudaStream_t stream, int sm_count, const BatchGrid &g, uint32_t group, uint32_t first,
                              const phem_edge *edges, uint4 *list, const BatchArgs &b, float light_msf,
                              float light_cc);

// Resolves the kernel for (block, items), sets its shared-memory attribute and
// sizes the persistent grid from the occupancy API.
phem_status batch_launch_config(int device, int sm_count, int block, int items, BatchLaunch *out);
phem_status batch_launch(cudaStream_t stream, const BatchLaunch &l, BatchArgs args);

}  // namespace phem

struct phem_batch_plan {
    phem_context *ctx = nullptr;
    uint32_t max_graphs = 0, max_vertices = 0;
    uint64_t max_edges = 0, max_wl = 0, max_bm = 0;
    void *mem = nullptr;
    phem::BatchBuffers buf{};
    phem::BatchLaunch launch{};
    float ratio = 0.5f;
    // the grid kernel's part, made when a batch first goes to it
    bool may_grid = false;               // (never in a serving slot's plan)
    bool on_grid = false;                // the uploaded batch is the grid kernel's
    void *grid_mem = nullptr;
    uint4 *grid_list = nullptr;
    phem::BatchGrid grid{};
    phem::GridItem *h_grid = nullptr;    // pinned staging of its items
    phem::GridHdr *h_hdr = nullptr;
    float light_cc = 0.f;                // the context's tuning when the plan was made
    cudaGraph_t grid_graph = nullptr;
    cudaGraphExec_t grid_exec = nullptr;
    phem::BatchItem *h_items = nullptr;  // pinned staging of the work items
    uint32_t *h_num = nullptr;     // pinned batch size
    uint32_t *h_status = nullptr;  // pinned per-graph status
    cudaEvent_t staged = nullptr;  // the pinned staging has been consumed
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    uint32_t num_graphs = 0, total_vertices = 0;
};

namespace phem {
// (Re)captures the plan's CTA-per-graph launch, with `pairs` as the input of
// kBatchPairs graphs.
phem_status batch_plan_capture(phem_batch_plan *p, const unsigned long long *pairs);
// phem_batch_plan_create; with `grid` the plan can also route a batch to the
// grid kernel (a serving slot's plan cannot: its launches overlap on the
// device, and a cooperative launch waits for every SM).
phem_status batch_plan_create(phem_context *ctx, uint32_t max_graphs, uint64_t max_edges, uint32_t max_vertices,
                              bool grid, phem_batch_plan **out);
}  // namespace phem
