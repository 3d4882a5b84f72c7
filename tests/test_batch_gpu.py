"""GPU parity of the batched engine (many graphs, one persistent launch)
against the oracle: per graph, the forest edge ids (ascending), count and
uint64 total equal the (w, id) Kruskal restatement for MSF graphs and the
index-order Kruskal (the canonical forest) for CC graphs; labels equal the
oracle's min-id labels.  Every kernel configuration the autotuner can pick
gives the same results."""
import numpy as np
import pytest

import oracle
from phem_graph_b200 import _lib, gen
from phem_graph_b200._lib import PhemError

pytestmark = pytest.mark.gpu
TUNING = ("batch.block_size", "batch.items", "batch.compact_ratio")


def _pack(e):
    u = e[:, 0].astype(np.uint64)
    v = e[:, 1].astype(np.uint64)
    lo, hi = np.minimum(u, v), np.maximum(u, v)
    return (lo << np.uint64(32)) | hi


def expected(batch, g):
    """(ids, total, labels) of graph g from the oracle."""
    r = batch.graphs[g]
    n, kind = int(r["num_vertices"]), int(r["kind"])
    e = batch.graph_edges(g)
    if n == 0:
        return np.empty(0, np.uint32), 0, np.empty(0, np.int32)
    if kind == gen.PHEM_BATCH_MSF:
        flags, _, total = oracle.msf_kruskal(e, n)
    else:
        z = e.copy()
        z[:, 2] = 0  # Kruskal under edge index order
        flags, _, _ = oracle.msf_kruskal(z, n)
        total = 0
    keep = e[:, 0] != e[:, 1]
    labels, _ = oracle.cc_solve(_pack(e[keep]), n)
    return np.nonzero(flags)[0].astype(np.uint32), total, labels


def check_batch(batch, res, graphs=None):
    for g in (range(batch.num_graphs) if graphs is None else graphs):
        ids, total, labels = expected(batch, g)
        np.testing.assert_array_equal(res.forest(batch, g), ids, err_msg=f"graph {g} {batch.names[g]}")
        assert int(res.count[g]) == len(ids)
        assert int(res.total[g]) == total, f"graph {g}"
        if res.labels is not None:
            np.testing.assert_array_equal(res.graph_labels(batch, g), labels, err_msg=f"graph {g}")


def small_mixed(num=64, seed=9, n_lo=16, n_hi=12000, kind=gen.PHEM_BATCH_MSF):
    return gen.mixed_batch(num, seed, n_lo=n_lo, n_hi=n_hi, kind=kind, threads=8)


def edge_case_batch():
    """Empty, single-vertex, self-loop-only, duplicate/tie, reversed (u > v)
    and disconnected graphs, MSF and CC kinds."""
    rng = np.random.default_rng(5)
    parts = [("empty_n0", 0, np.empty((0, 3), np.uint32), gen.PHEM_BATCH_MSF),
             ("single", 1, np.empty((0, 3), np.uint32), gen.PHEM_BATCH_MSF),
             ("loops", 4, np.array([[0, 0, 5], [3, 3, 1]], np.uint32), gen.PHEM_BATCH_MSF),
             ("isolated", 50, np.array([[1, 2, 7]], np.uint32), gen.PHEM_BATCH_CC)]
    ties = rng.integers(0, 40, (400, 2)).astype(np.uint32)
    parts.append(("ties", 40, np.column_stack([ties, np.full(400, 3, np.uint32)]), gen.PHEM_BATCH_MSF))
    rev = rng.integers(0, 300, (900, 2)).astype(np.uint32)
    parts.append(("reversed", 300, np.column_stack([rev, rng.integers(1, 4, 900).astype(np.uint32)]),
                  gen.PHEM_BATCH_MSF))
    parts.append(("reversed_cc", 300, np.column_stack([rev, np.zeros(900, np.uint32)]), gen.PHEM_BATCH_CC))
    blocks = np.concatenate([rng.integers(0, 100, (300, 2)), rng.integers(100, 200, (300, 2))]).astype(np.uint32)
    parts.append(("two_blocks", 200, np.column_stack([blocks, rng.integers(1, 1 << 20, 600).astype(np.uint32)]),
                  gen.PHEM_BATCH_MSF))
    return gen.batch_from(parts)


def test_mixed_batch_matches_oracle(ctx):
    b = small_mixed()
    res = ctx.batch_solve(b)
    assert res.stats["max_rounds"] >= 1
    check_batch(b, res)


def test_caller_output_arrays(ctx):
    """Results written into caller arrays (pinned, and larger than needed)
    equal the ones the call allocates; a wrong dtype is refused."""
    import torch
    b = small_mixed(24, seed=7)
    want = ctx.batch_solve(b)
    V, G = b.total_vertices, b.num_graphs
    out = {"ids": torch.empty(V + 5, dtype=torch.int32).pin_memory().numpy().view(np.uint32),
           "count": torch.empty(G, dtype=torch.int32).pin_memory().numpy().view(np.uint32),
           "total": torch.empty(G + 1, dtype=torch.int64).pin_memory().numpy().view(np.uint64),
           "labels": torch.empty(V, dtype=torch.int32).pin_memory().numpy()}
    for _ in range(2):
        got = ctx.batch_solve(b, out=out)
        np.testing.assert_array_equal(got.count, want.count)
        np.testing.assert_array_equal(got.total, want.total)
        np.testing.assert_array_equal(got.labels, want.labels)
        for g in range(G):
            np.testing.assert_array_equal(got.forest(b, g), want.forest(b, g))
    with pytest.raises(ValueError):
        ctx.batch_solve(b, out={"count": np.empty(G, np.int64)})


def test_cc_kind_canonical_forest(ctx):
    b = small_mixed(32, seed=3, kind=gen.PHEM_BATCH_CC)
    res = ctx.batch_solve(b)
    check_batch(b, res)
    assert np.all(res.total == 0)


def test_edge_cases(ctx):
    b = edge_case_batch()
    check_batch(b, ctx.batch_solve(b))


def test_empty_batch(ctx):
    res = ctx.batch_solve(gen.batch_from([]))
    assert len(res.count) == 0


@pytest.mark.parametrize("block", [256, 512, 1024])
@pytest.mark.parametrize("items", [1, 2, 4])
def test_every_configuration(ctx, block, items):
    b = small_mixed(24, seed=11, n_lo=16, n_hi=20000)
    saved = [ctx.get_tuning(k) for k in TUNING]
    try:
        for ratio in (0.0, 0.5, 1.0):
            ctx.set_tuning("batch.block_size", block)
            ctx.set_tuning("batch.items", items)
            ctx.set_tuning("batch.compact_ratio", ratio)
            res = ctx.batch_solve(b)
            assert res.stats["block_size"] == block and res.stats["items"] == items
            check_batch(b, res)
    finally:
        for k, v in zip(TUNING, saved):
            ctx.set_tuning(k, v)


def test_large_graphs_use_global_state(ctx):
    """Graphs above the shared-memory capacity keep their state in HBM."""
    b = small_mixed(6, seed=21, n_lo=30000, n_hi=65536)
    res = ctx.batch_solve(b)
    assert int(b.graphs["num_vertices"].min()) > res.stats["smem_vertices"]
    check_batch(b, res)


def test_plan_replay_two_batches(ctx):
    a = small_mixed(40, seed=1)
    c = small_mixed(70, seed=2, n_hi=5000)
    with ctx.batch_plan(128, max(a.total_edges, c.total_edges), max(a.total_vertices, c.total_vertices)) as p:
        for b in (a, c, a):
            p.upload(b)
            p.run()
            check_batch(b, p.download())
        assert all(v for v in p.device().values())


def test_large_host_batch_overlapped_launches(ctx):
    """A batch of host edges past the overlap size is copied in chunks and
    solved by one launch per chunk group (graphs straddling chunk ends go
    to the later group); every graph's forest, count, total and labels equal
    the single-launch result of a plan, twice in a row."""
    b = gen.mixed_batch(160, 21, n_lo=64, n_hi=65536, threads=8)
    assert b.total_edges >= 1 << 22
    with ctx.batch_plan(b.num_graphs, b.total_edges, b.total_vertices) as p:
        p.upload(b)
        p.run()
        want = p.download(labels=True)
    for _ in range(2):
        got = ctx.batch_solve(b)
        np.testing.assert_array_equal(got.count, want.count)
        np.testing.assert_array_equal(got.total, want.total)
        np.testing.assert_array_equal(got.labels, want.labels)
        for g in range(b.num_graphs):
            np.testing.assert_array_equal(got.forest(b, g), want.forest(b, g))


def test_plan_rejects_oversized_batch(ctx):
    a = small_mixed(8, seed=4)
    with ctx.batch_plan(4, a.total_edges, a.total_vertices) as p:
        with pytest.raises(PhemError) as e:
            p.upload(a)
        assert e.value.status == _lib.PHEM_ERR_INVALID


def test_invalid_inputs_are_rejected(ctx):
    bad = gen.batch_from([("oob", 5, np.array([[0, 9, 1]], np.uint32), gen.PHEM_BATCH_MSF)])
    with pytest.raises(PhemError) as e:
        ctx.batch_solve(bad)
    assert e.value.status == _lib.PHEM_ERR_INVALID
    one = np.array([[0, 1, 1]], np.uint32)
    ov = gen.batch_from([("a", 10, one, 0), ("b", 10, one, 0)])
    ov.graphs["vertex_offset"][1] = 5  # overlaps graph 0
    with pytest.raises(PhemError) as e:
        ctx.batch_solve(ov)
    assert e.value.status == _lib.PHEM_ERR_INVALID
    b = edge_case_batch()  # the context stays usable
    check_batch(b, ctx.batch_solve(b))


def test_autotune_picks_a_grid_point(ctx):
    b = small_mixed(48, seed=13)
    saved = [ctx.get_tuning(k) for k in TUNING]
    try:
        best = ctx.batch_autotune(b, reps=1)
        assert best["block_size"] in (256, 512, 1024) and best["items"] in (1, 2, 4)
        assert best["compact_ratio"] in (0.25, 0.5, 1.0) and best["device_ms"] > 0
        assert ctx.get_tuning("batch.block_size") == best["block_size"]
        check_batch(b, ctx.batch_solve(b))
    finally:
        for k, v in zip(TUNING, saved):
            ctx.set_tuning(k, v)


def test_batch_equals_one_graph_path(ctx):
    """A graph's batched forest equals phem_msf_solve's on that graph alone."""
    b = small_mixed(12, seed=17, n_lo=1000, n_hi=40000)
    res = ctx.batch_solve(b)
    for g in range(b.num_graphs):
        n = int(b.graphs[g]["num_vertices"])
        one = ctx.msf_solve(b.graph_edges(g), n)
        np.testing.assert_array_equal(b.graph_edges(g)[res.forest(b, g)], one.edges)
        assert one.total == int(res.total[g])


@pytest.mark.slow
def test_full_workload_sampled(ctx):
    """The 4096-graph workload: every graph's forest size agrees with its
    labels, and a sample of graphs matches the oracle exactly."""
    b = gen.mixed_batch(4096, 4)
    res = ctx.batch_solve(b)
    for g in range(b.num_graphs):
        n = int(b.graphs[g]["num_vertices"])
        assert int(res.count[g]) == n - len(np.unique(res.graph_labels(b, g)))
    rng = np.random.default_rng(0)
    check_batch(b, res, graphs=sorted(rng.choice(b.num_graphs, 96, replace=False).tolist()))


@pytest.mark.parametrize("device", [0, 1, 2])
@pytest.mark.parametrize("kind", [gen.PHEM_BATCH_MSF, gen.PHEM_BATCH_CC])
def test_grid_batch_shapes(ctx, device, kind):
    """A batch with one graph large enough for the grid kernel, beside empty,
    one-vertex, one-edge and tile-sized ones whose edges start at every offset
    mod 4, with gaps and shared edge ranges, from host memory and from device
    memory at 16- and 4-byte alignment."""
    sizes = [(60000, 300001), (0, 0), (1, 0), (2, 1), (33, 127), (40, 128), (41, 129), (500, 1023), (7, 3), (3000, 9000)]
    parts = []
    for i, (n, m) in enumerate(sizes):
        p = gen.er(n, m + m // 8 + 8, 50 + i)[:m] if m else np.zeros(0, np.uint64)
        parts.append((f"g{i}", n, gen.msf_edges(p, gen.weights(len(p), i, bits=5)), kind))
    b = gen.batch_from(parts)
    # the second 127-edge graph reads the first one's records; vertex ranges get gaps
    b.graphs[7]["edge_offset"] = b.graphs[4]["edge_offset"]
    b.graphs[7]["num_edges"] = 127
    b.graphs["vertex_offset"] += np.arange(len(sizes), dtype=np.uint32) * 5
    b.total_vertices += 5 * len(sizes)
    host = b.edges
    if device:
        import torch
        t = torch.from_numpy(np.concatenate([host[:device - 1], host]).view(np.int32)).cuda()
        torch.cuda.synchronize()
        b.edges = t[device - 1:]
    r = ctx.batch_solve(b)
    for g in range(len(sizes)):
        q = b.graphs[g]
        o, m, n = int(q["edge_offset"]), int(q["num_edges"]), int(q["num_vertices"])
        E = host[o:o + m].copy()
        if kind == gen.PHEM_BATCH_CC:
            E[:, 2] = 0
        flags, cnt, tot = oracle.msf_kruskal(E, n) if n else (np.zeros(0), 0, 0)
        assert (int(r.count[g]), int(r.total[g])) == (cnt, tot)
        np.testing.assert_array_equal(r.forest(b, g), np.nonzero(flags)[0])
        if n:
            labels, _ = oracle.cc_solve((E[:, 0].astype(np.uint64) << np.uint64(32)) | E[:, 1], n)
            np.testing.assert_array_equal(r.graph_labels(b, g), labels)


def test_plan_replays_both_kernels(ctx):
    """One plan, a batch for the CTA-per-graph kernel, one for the grid, and
    the first again; a bad endpoint in the grid batch is reported."""
    small, large = gen.mixed_batch(12, 5, 64, 300), gen.mixed_batch(6, 6, 20000, 40000)
    with ctx.batch_plan(16, max(small.total_edges, large.total_edges), max(small.total_vertices, large.total_vertices)) as p:
        for b in (small, large, small):
            p.upload(b)
            p.run()
            r = p.download()
            for g in range(b.num_graphs):
                E, n = b.graph_edges(g), int(b.graphs[g]["num_vertices"])
                flags, cnt, tot = oracle.msf_kruskal(E, n)
                assert (int(r.count[g]), int(r.total[g])) == (cnt, tot)
                np.testing.assert_array_equal(r.forest(b, g), np.nonzero(flags)[0])
        large.edges[int(large.graphs[1]["edge_offset"]) + 3, 1] = 70000
        p.upload(large)
        p.run()
        with pytest.raises(PhemError):
            p.download()


def test_large_graphs_without_room_for_the_grid():
    """Device memory that holds a batch but not the grid kernel's arrays: the
    CTA-per-graph kernel solves it."""
    import phem_graph_b200 as P
    import torch
    n = 200000
    p = gen.er(n, 3_000_000, 5)
    b = gen.batch_from([("", n, gen.msf_edges(p, gen.weights(len(p), 1)), gen.PHEM_BATCH_MSF)])
    host = b.edges
    b.edges = torch.from_numpy(host.view(np.int32)).cuda()
    torch.cuda.synchronize()
    with P.Context(0) as c:
        small = gen.mixed_batch(4, 5, 64, 300)
        c.batch_solve(small)  # its kernel is loaded
        c.trim()
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (80 << 20), dtype=torch.uint8, device="cuda")
        try:
            r = c.batch_solve(b)
        finally:
            del hog
            torch.cuda.empty_cache()
    flags, cnt, tot = oracle.msf_kruskal(host, n)
    assert (int(r.count[0]), int(r.total[0])) == (cnt, tot)
    np.testing.assert_array_equal(r.forest(b, 0), np.nonzero(flags)[0])


def test_plan_takes_the_grid_when_needed(ctx):
    """A plan of small graphs holds nothing for the grid kernel; a batch for
    it gets its buffers at upload, and the other kernel while there is no room
    for them."""
    import torch
    small, large = gen.mixed_batch(12, 5, 64, 300), gen.mixed_batch(6, 6, 20000, 40000)

    def check(p, b):
        p.upload(b)
        p.run()
        r = p.download()
        for g in range(b.num_graphs):
            flags, cnt, tot = oracle.msf_kruskal(b.graph_edges(g), int(b.graphs[g]["num_vertices"]))
            assert (int(r.count[g]), int(r.total[g])) == (cnt, tot)
            np.testing.assert_array_equal(r.forest(b, g), np.nonzero(flags)[0])

    ctx.batch_solve(large)  # the kernels are loaded
    ctx.batch_solve(small)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with ctx.batch_plan(16, small.total_edges, small.total_vertices) as p:
        assert free - torch.cuda.mem_get_info()[0] < 16 << 20
        check(p, small)
    with ctx.batch_plan(16, large.total_edges, large.total_vertices) as p:
        check(p, small)
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (16 << 20), dtype=torch.uint8, device="cuda")
        try:
            check(p, large)
        finally:
            del hog
            torch.cuda.empty_cache()
        for b in (large, small, large):
            check(p, b)


def test_rounds_of_chains(ctx):
    """Paths with ascending weights hook into one chain each and are done in
    one round: every vertex's pointer is at its root when the round ends."""
    n = 5000
    u = np.arange(n - 1, dtype=np.uint32)
    E = np.ascontiguousarray(np.stack([u, u + 1, u + 1], axis=1))
    b = gen.batch_from([(f"p{i}", n, E, gen.PHEM_BATCH_MSF) for i in range(16)])
    for _ in range(20):
        r = ctx.batch_solve(b)
        assert r.stats["smem_vertices"] > n and r.stats["max_rounds"] == 1
        assert (r.count == n - 1).all() and not r.labels.any()


@pytest.mark.parametrize("block,items", [(256, 1), (256, 4), (512, 2), (1024, 4)])
def test_cta_kernel_takes_every_batch_when_asked(ctx, block, items):
    """With batch.grid 0 a batch that the grid kernel would take runs in the
    tuned configuration, graphs above the shared-memory capacity among them,
    through a call and through a plan."""
    b = small_mixed(12, seed=21, n_lo=500, n_hi=40000)
    assert ctx.batch_solve(b).stats["smem_vertices"] == 0
    saved = [ctx.get_tuning(k) for k in TUNING]
    try:
        ctx.set_tuning("batch.grid", 0)
        ctx.set_tuning("batch.block_size", block)
        ctx.set_tuning("batch.items", items)
        res = ctx.batch_solve(b)
        assert 0 < res.stats["smem_vertices"] < int(b.graphs["num_vertices"].max())
        check_batch(b, res)
        with ctx.batch_plan(b.num_graphs, b.total_edges, b.total_vertices) as p:
            p.upload(b)
            p.run()
            check_batch(b, p.download())
    finally:
        ctx.set_tuning("batch.grid", 1)
        for k, v in zip(TUNING, saved):
            ctx.set_tuning(k, v)


@pytest.mark.parametrize("grid", [0, 1])
def test_stats_of_both_kernels(ctx, grid):
    """A path with ascending weights joins in one round, and so do many; the
    statistics say which kernel ran."""
    n = 60000
    u = np.arange(n - 1, dtype=np.uint32)
    b = gen.batch_from([("path", n, np.ascontiguousarray(np.stack([u, u + 1, u + 1], axis=1)), gen.PHEM_BATCH_MSF)])
    try:
        ctx.set_tuning("batch.grid", grid)
        st = ctx.batch_solve(b).stats
    finally:
        ctx.set_tuning("batch.grid", 1)
    assert st["max_rounds"] == 1
    assert (st["smem_vertices"] == 0) == bool(grid) and st["device_ms"] > 0
    if grid:
        import torch
        assert st["grid"] == torch.cuda.get_device_properties(0).multi_processor_count
