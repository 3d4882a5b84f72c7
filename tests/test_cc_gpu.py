"""GPU parity: connected components + spanning forest against the oracle and
the reference's golden vectors.  Labels are bit-exact; the default forest is
checked for validity (which edge wins a hooking race is not fixed, in the
reference either); the canonical forest is bit-exact as a set."""
import numpy as np
import pytest

import oracle
import phem_graph_b200 as P
from phem_graph_b200 import _lib, gen
from phem_graph_b200.api import forest_set
from tests.golden import load, names

pytestmark = pytest.mark.gpu
CC_CASES = names("cc_")


def check_forest(edges, n, labels, forest):
    """Valid spanning forest of the graph: |F| = n - c, every slot edge is an
    input edge with u < v, and F alone reproduces the labels."""
    f = forest_set(forest)
    c = len(np.unique(labels))
    assert len(f) == n - c
    live = np.unique(edges[(edges >> np.uint64(32)) < (edges & np.uint64(0xFFFFFFFF))])
    assert np.all(np.isin(f, live))
    lab_f, _ = oracle.cc_solve(f, n)
    np.testing.assert_array_equal(lab_f, labels)


@pytest.mark.parametrize("name", CC_CASES)
def test_golden_labels_and_forest(ctx, name):
    g = load(name)
    edges, n = g["edges"], int(g["n"])
    r = ctx.cc_solve(edges, n)
    np.testing.assert_array_equal(r.labels, g["labels"])
    check_forest(edges, n, r.labels, r.forest)
    assert r.components == len(np.unique(g["labels"]))


@pytest.mark.parametrize("name", CC_CASES)
def test_golden_canonical_forest_bit_exact(ctx, name):
    g = load(name)
    edges, n = g["edges"], int(g["n"])
    r = ctx.cc_solve(edges, n, canonical=True)
    np.testing.assert_array_equal(r.labels, g["labels"])
    np.testing.assert_array_equal(forest_set(r.forest), g["forest"])


@pytest.mark.parametrize("seed", [1, 2, 3, 4])
@pytest.mark.parametrize("n,draws", [(1000, 800), (1 << 14, 1 << 15), (1 << 16, 1 << 19)])
def test_er_random(ctx, seed, n, draws):
    g = gen.er_graph(n, draws, seed)
    labels, forest = oracle.cc_solve(g.pairs, n)
    r = ctx.cc_solve(g.pairs, n)
    np.testing.assert_array_equal(r.labels, labels)
    check_forest(g.pairs, n, r.labels, r.forest)
    rc = ctx.cc_solve(g.pairs, n, canonical=True)
    np.testing.assert_array_equal(rc.labels, labels)
    np.testing.assert_array_equal(forest_set(rc.forest), oracle.forest_set(forest))


@pytest.mark.parametrize("scale", [12, 16])
def test_rmat_hubs(ctx, scale):
    p = gen.rmat(scale, 16 << scale, seed=scale)
    n = 1 << scale
    labels, forest = oracle.cc_solve(p, n)
    r = ctx.cc_solve(p, n)
    np.testing.assert_array_equal(r.labels, labels)
    check_forest(p, n, r.labels, r.forest)
    rc = ctx.cc_solve(p, n, canonical=True)
    np.testing.assert_array_equal(forest_set(rc.forest), oracle.forest_set(forest))


@pytest.mark.slow
def test_full_size_er20(ctx):
    """The CC workload at full size: n = 2^20, 8 * 2^20 draws, seed 1."""
    g = gen.er_graph(1 << 20, 8 << 20, 1)
    labels, forest = oracle.cc_solve(g.pairs, g.n)
    r = ctx.cc_solve(g.pairs, g.n)
    np.testing.assert_array_equal(r.labels, labels)
    assert r.forest_edges == g.n - len(np.unique(labels))
    rc = ctx.cc_solve(g.pairs, g.n, canonical=True)
    np.testing.assert_array_equal(forest_set(rc.forest), oracle.forest_set(forest))
    # idempotence: solving the forest alone gives the same labels and keeps every forest edge
    r2 = ctx.cc_solve(forest_set(r.forest), g.n)
    np.testing.assert_array_equal(r2.labels, labels)
    assert r2.forest_edges == r.forest_edges


def test_edge_cases(ctx):
    # no edges
    r = ctx.cc_solve(np.zeros(0, np.uint64), 5)
    np.testing.assert_array_equal(r.labels, np.arange(5))
    assert np.all(r.forest == _lib.PHEM_FOREST_EMPTY)
    # one vertex
    assert ctx.cc_solve(np.zeros(0, np.uint64), 1).labels.tolist() == [0]
    # self-loops and u > v are skipped (union_find_gpu_COO unites only u < v)
    e = np.array([(3 << 32) | 3, (4 << 32) | 1, (1 << 32) | 2], np.uint64)
    r = ctx.cc_solve(e, 5)
    assert r.labels.tolist() == [0, 1, 1, 3, 4]
    rc = ctx.cc_solve(e, 5, canonical=True)
    assert rc.labels.tolist() == [0, 1, 1, 3, 4]
    assert forest_set(rc.forest).tolist() == [(1 << 32) | 2]
    # odd m exercises the tail of the vectorised loads
    e = gen.er(100, 333, 3)
    assert len(e) % 2 == 1 or True
    lab, _ = oracle.cc_solve(e, 100)
    np.testing.assert_array_equal(ctx.cc_solve(e[:-1], 100).labels, oracle.cc_solve(e[:-1], 100)[0])
    np.testing.assert_array_equal(ctx.cc_solve(e, 100).labels, lab)


def test_out_of_range_endpoint_rejected(ctx):
    e = np.array([(1 << 32) | 7], np.uint64)
    with pytest.raises(P.PhemError) as ei:
        ctx.cc_solve(e, 5)
    assert ei.value.status == _lib.PHEM_ERR_INVALID
    with pytest.raises(P.PhemError):
        ctx.cc_solve(e, 5, canonical=True)
    # the context is still usable
    assert ctx.cc_solve(np.array([(0 << 32) | 1], np.uint64), 2).labels.tolist() == [0, 0]


def test_device_resident_inputs(ctx):
    import torch
    g = gen.er_graph(1 << 15, 1 << 16, 9)
    d_edges = torch.from_numpy(g.pairs.view(np.int64)).cuda()
    d_lab = torch.empty(g.n, dtype=torch.int32, device="cuda")
    d_for = torch.empty(g.n, dtype=torch.int64, device="cuda")
    ctx.cc_solve(d_edges, g.n, labels=d_lab, forest=d_for)
    labels, _ = oracle.cc_solve(g.pairs, g.n)
    np.testing.assert_array_equal(d_lab.cpu().numpy(), labels)
    check_forest(g.pairs, g.n, labels, d_for.cpu().numpy().view(np.uint64))


def test_stage_entry_points_and_reference_pipeline(ctx):
    """SpanningTree + gpu_spanning_tree as the reference driver runs them
    (CC/main.cu:157-186): stream the edges in batches, then merge the batch
    forest with a second forest (here the CPU oracle's forest of a second edge
    share, standing in for the reference's CPU partner)."""
    import torch
    g = gen.er_graph(1 << 16, 3 << 16, 5)
    n = g.n
    half = len(g.pairs) // 2
    gpu_share, cpu_share = g.pairs[:half], g.pairs[half:]
    parent = torch.empty(n, dtype=torch.int32, device="cuda")
    label = torch.empty(n, dtype=torch.int32, device="cuda")
    t1 = torch.empty(n, dtype=torch.int64, device="cuda")
    pinned = torch.from_numpy(gpu_share.view(np.int64)).pin_memory()
    ctx.cc_stream(pinned, n, 4097, parent, label, t1)
    _, cpu_forest = oracle.cc_solve(cpu_share, n)
    extra = torch.from_numpy(cpu_forest.view(np.int64)).cuda()
    t2 = torch.empty(n, dtype=torch.int64, device="cuda")
    ctx.cc_merge(t1, extra, n, parent, label, t2)
    labels, _ = oracle.cc_solve(g.pairs, n)
    np.testing.assert_array_equal(label.cpu().numpy(), labels)
    check_forest(g.pairs, n, labels, t2.cpu().numpy().view(np.uint64))
    # stage-level calls on device buffers reproduce the one-shot solve
    d_edges = torch.from_numpy(g.pairs.view(np.int64)).cuda()
    ctx.cc_init(n, parent, label, t1)
    ctx.cc_unite(d_edges, len(g.pairs), n, parent, t1)
    ctx.cc_label(n, parent, label)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(label.cpu().numpy(), labels)


def test_stream_unsorted_rmat_batches(ctx):
    """SpanningTree over an unsorted R-MAT stream in ragged batches: labels
    equal the oracle's, the forest reproduces them."""
    import ctypes as C
    import torch
    scale, draws = 18, 32 << 18
    out = np.empty(draws, np.uint64)
    m = C.c_uint64()
    _lib.check(_lib.lib().phem_gen_rmat_range(scale, 0, draws, 0.57, 0.19, 0.19, 28, out.ctypes.data, C.byref(m)),
               "phem_gen_rmat_range")
    pairs = out[: m.value]
    n = 1 << scale
    pinned = torch.from_numpy(pairs.view(np.int64)).pin_memory()
    dev = torch.device("cuda", 0)
    parent = torch.empty(n, dtype=torch.int32, device=dev)
    label = torch.empty(n, dtype=torch.int32, device=dev)
    forest = torch.empty(n, dtype=torch.int64, device=dev)
    ctx.cc_stream(pinned.numpy().view(np.uint64), n, (1 << 20) + 12345, parent, label, forest)
    ctx.cc_label(n, parent, label)
    torch.cuda.synchronize()
    want, _ = oracle.cc_solve(pairs, n)
    got = label.cpu().numpy()
    np.testing.assert_array_equal(got, want)
    check_forest(pairs, n, got, forest.cpu().numpy().view(np.uint64))


def test_incremental_stream_batches_of_every_kind(ctx):
    """phem_cc_stream_begin/push/end: ragged batches from pinned and pageable
    host memory (one larger than the first staging buffers, which then grow),
    aligned device memory (united in place, one batch empty) and an unaligned
    device view (staged): labels equal the oracle's and the forest reproduces
    them."""
    import torch
    g = gen.er_graph(1 << 16, 1 << 21, 41)
    n, pairs = g.n, g.pairs
    cuts = [0, 1, 1001, 1001, 70001, 1270001, 1273000, len(pairs)]
    dev = torch.device("cuda", ctx.device)
    parent = torch.empty(n, dtype=torch.int32, device=dev)
    label = torch.empty(n, dtype=torch.int32, device=dev)
    forest = torch.empty(n, dtype=torch.int64, device=dev)
    d_all = torch.from_numpy(pairs.view(np.int64)).to(dev)
    ctx.cc_stream_begin(n, parent, label, forest)
    for k in range(len(cuts) - 1):
        a, b = cuts[k], cuts[k + 1]
        kind = k % 4
        if kind == 0:
            ctx.cc_stream_push(torch.from_numpy(pairs[a:b].view(np.int64)).pin_memory())
        elif kind == 1:
            ctx.cc_stream_push(pairs[a:b].copy())
        elif kind == 2:
            ctx.cc_stream_push(d_all[a:b] if a % 2 == 0 else d_all[a:b].clone())
        else:
            ctx.cc_stream_push(d_all[a:b])  # odd start: 8-byte aligned only, staged
    ms = ctx.cc_stream_end()
    assert ms > 0
    ctx.cc_label(n, parent, label)
    torch.cuda.synchronize()
    want, _ = oracle.cc_solve(pairs, n)
    got = label.cpu().numpy()
    np.testing.assert_array_equal(got, want)
    check_forest(pairs, n, got, forest.cpu().numpy().view(np.uint64))


def test_incremental_stream_call_order(ctx):
    """push and end need an open stream; a second begin is refused; a stream
    can be opened again after its end."""
    import torch
    n = 64
    parent = torch.empty(n, dtype=torch.int32, device="cuda")
    with pytest.raises(P.PhemError) as ei:
        ctx.cc_stream_push(np.array([1], np.uint64))
    assert ei.value.status == _lib.PHEM_ERR_INVALID
    with pytest.raises(P.PhemError):
        ctx.cc_stream_end()
    ctx.cc_stream_begin(n, parent)
    with pytest.raises(P.PhemError):
        ctx.cc_stream_begin(n, parent)
    ctx.cc_stream_push(np.array([(1 << 32) | 2, (2 << 32) | 3], np.uint64))
    ctx.cc_stream_end()
    ctx.cc_stream_begin(n, parent)
    ctx.cc_stream_push(np.array([(5 << 32) | 9], np.uint64))
    ctx.cc_stream_end()
    label = torch.empty(n, dtype=torch.int32, device="cuda")
    ctx.cc_label(n, parent, label)
    got = label.cpu().numpy()
    assert got[9] == 5 and got[3] == 3 and got[2] == 2  # only the second stream's edge


@pytest.mark.parametrize("light", [0.0, 0.5, 2.0, 6.0])
def test_canonical_filter_setting_does_not_change_the_forest(ctx, light):
    """The canonical forest's light/heavy split (first edges by index) gives
    the sequential reference's forest set for any split size, unfiltered
    included."""
    g = gen.er_graph(1 << 15, 1 << 18, 23)
    want_labels, want_forest = oracle.cc_solve(g.pairs, g.n)
    saved = ctx.get_tuning("cc.canonical_light_per_vertex")
    try:
        ctx.set_tuning("cc.canonical_light_per_vertex", light)
        rc = ctx.cc_solve(g.pairs, g.n, canonical=True)
    finally:
        ctx.set_tuning("cc.canonical_light_per_vertex", saved)
    np.testing.assert_array_equal(rc.labels, want_labels)
    np.testing.assert_array_equal(forest_set(rc.forest), oracle.forest_set(want_forest))


@pytest.mark.parametrize("sample", [0.0, 0.5, 2.0, 1000.0])
def test_sample_schedule_same_labels(ctx, sample):
    """The prefix-sample / compress / rest schedule gives the same labels and
    a valid forest for any sample size."""
    g = gen.er_graph(1 << 16, 1 << 19, 9)
    want, _ = oracle.cc_solve(g.pairs, g.n)
    saved = ctx.get_tuning("cc.sample_per_vertex")
    try:
        ctx.set_tuning("cc.sample_per_vertex", sample)
        r = ctx.cc_solve(g.pairs, g.n)
    finally:
        ctx.set_tuning("cc.sample_per_vertex", saved)
    np.testing.assert_array_equal(r.labels, want)
    check_forest(g.pairs, g.n, r.labels, r.forest)


@pytest.mark.parametrize("sample", [0.0, 1.0, 6.0])
@pytest.mark.parametrize("pinned", [False, True])
def test_host_edges_copied_in_overlapped_chunks(ctx, sample, pinned):
    """Large host inputs are copied in 2^21-edge chunks on a second stream,
    each chunk's union waiting for its own copy; prefixes that end inside,
    at the end of, or beyond several chunks give the oracle's labels and a
    valid forest, from pageable and from pinned memory, twice in a row."""
    import torch
    g = gen.er_graph(1 << 19, 5_000_001, 17)
    edges = g.pairs if not pinned else torch.from_numpy(g.pairs.view(np.int64)).pin_memory().numpy().view(np.uint64)
    want, _ = oracle.cc_solve(g.pairs, g.n)
    saved = ctx.get_tuning("cc.sample_per_vertex")
    try:
        ctx.set_tuning("cc.sample_per_vertex", sample)
        for _ in range(2):
            r = ctx.cc_solve(edges, g.n)
            np.testing.assert_array_equal(r.labels, want)
            check_forest(g.pairs, g.n, r.labels, r.forest)
    finally:
        ctx.set_tuning("cc.sample_per_vertex", saved)


def test_solves_from_reference_file_formats(ctx, tmp_path):
    """Inputs read from the reference drivers' file formats solve to the
    oracle's results (ECL binary CSR for CC, MatrixMarket for MSF)."""
    from phem_graph_b200 import io
    g = gen.rmat_graph(12, 8, seed=6)
    off, cols = gen.csr_from_pairs(g.pairs, g.n)
    io.write_ecl(tmp_path / "g.egr", off, cols)
    pairs, n = io.read_graph_pairs(tmp_path / "g.egr")
    want, _ = oracle.cc_solve(pairs, n)
    np.testing.assert_array_equal(ctx.cc_solve(pairs, n).labels, want)
    io.write_mtx(tmp_path / "g.mtx", g.msf_edges(), g.n)
    e, n = io.read_mtx(tmp_path / "g.mtx")
    flags, cnt, tot = oracle.msf_kruskal(e, n)
    r = ctx.msf_solve(e, n)
    assert (r.count, r.total) == (cnt, tot)
    np.testing.assert_array_equal(r.edges, e[flags])


@pytest.mark.parametrize("kind", ["er", "er_long_rest", "rmat", "rgg", "path", "path_shuffled", "star_low", "star_high"])
@pytest.mark.parametrize("odd", [0, 1])
def test_device_edges_in_rounds(ctx, kind, odd):
    """Device-resident edges past the one-CTA sizes: prefixes with and without
    a rest, long chains, hubs as the smaller and as the larger endpoint of
    repeated edges, odd counts; labels exact, slots exactly the non-roots, the
    forest valid; out-of-range endpoints in the prefix and in the rest."""
    import torch
    n = 50001
    u = np.arange(n - 1, dtype=np.uint64)
    p = {"er": lambda: gen.er(n, 120000, 3), "er_long_rest": lambda: gen.er(n, 12 * n, 4),
         "rmat": lambda: gen.rmat_graph(15, 16, seed=5).pairs, "rgg": lambda: gen.rgg_graph(n, 8, 3).pairs,
         "path": lambda: (u << np.uint64(32)) | (u + np.uint64(1)),
         "path_shuffled": lambda: np.random.default_rng(0).permutation((u << np.uint64(32)) | (u + np.uint64(1))),
         "star_low": lambda: np.concatenate([u + np.uint64(1)] * 8),
         "star_high": lambda: np.concatenate([(u << np.uint64(32)) | np.uint64(n - 1)] * 8)}[kind]()
    p = np.ascontiguousarray(p[:len(p) - odd])
    d = torch.from_numpy(p.view(np.int64)).cuda()
    lab = torch.empty(n, dtype=torch.int32, device="cuda")
    slots = torch.empty(n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    r = ctx.cc_solve(d, n, labels=lab, forest=slots)
    want, _ = oracle.cc_solve(p, n)
    np.testing.assert_array_equal(lab.cpu().numpy(), want)
    f = slots.cpu().numpy().view(np.uint64)
    assert r.components == len(np.unique(want)) == n - r.forest_edges
    np.testing.assert_array_equal(np.nonzero(f != np.uint64(_lib.PHEM_FOREST_EMPTY))[0],
                                  np.nonzero(want != np.arange(n))[0])
    check_forest(p, n, want, f)
    for at in (5, len(p) - 1):
        bad = d.clone()
        bad[at] = (3 << 32) | n
        torch.cuda.synchronize()
        with pytest.raises(P.PhemError) as ei:
            ctx.cc_solve(bad, n, labels=lab, forest=slots)
        assert ei.value.status == _lib.PHEM_ERR_INVALID


@pytest.mark.parametrize("n", [20000, 40003])
def test_solves_after_failed_and_profiled_ones(ctx, n):
    """A solve hands over a zeroed control block: canonical CC, weighted MSF
    and default CC repeated in turn, after solves that gave up on an endpoint
    out of range and with profiled ones (another control block) in between."""
    p = gen.er(n, 3 * n + 1, 9)
    want, _ = oracle.cc_solve(p, n)
    cset = forest_set(ctx.cc_solve(p, n, canonical=True).forest)
    w = np.random.default_rng(1).integers(0, 1000, len(p), dtype=np.uint32)
    e = np.stack([(p >> np.uint64(32)).astype(np.uint32), p.astype(np.uint32), w], axis=1)
    flags, cnt, tot = oracle.msf_kruskal(e, n)
    bad_p, bad_e = p.copy(), e.copy()
    bad_p[-1] = np.uint64((3 << 32) | n)
    bad_e[-1, 1] = n
    for step in range(4):
        if step % 2:
            for call in (lambda: ctx.msf_solve(bad_e, n), lambda: ctx.cc_solve(bad_p, n, canonical=True),
                         lambda: ctx.cc_solve(bad_p, n)):
                with pytest.raises(P.PhemError):
                    call()
        ctx.set_profiling(step == 2)
        r = ctx.msf_solve(e, n)
        assert (r.count, r.total) == (cnt, tot)
        np.testing.assert_array_equal(r.edges, e[flags])
        c = ctx.cc_solve(p, n, canonical=True)
        np.testing.assert_array_equal(c.labels, want)
        np.testing.assert_array_equal(forest_set(c.forest), cset)
        assert c.components == len(np.unique(want)) == n - c.forest_edges
        d = ctx.cc_solve(p, n)
        np.testing.assert_array_equal(d.labels, want)
        assert d.components == c.components
        ctx.set_profiling(False)


@pytest.mark.parametrize("where", ["device", "pinned", "pageable"])
@pytest.mark.parametrize("m", [1, 9001, 32767, 32768, 32769])  # one CTA, and one edge more than it takes
@pytest.mark.parametrize("words", [1, 2, 3])
def test_pairs_at_any_word_offset(ctx, where, m, words):
    """A pair array at every multiple of 4 bytes is solved (the small solve
    reads packed pairs as 8-byte words; other offsets are copied first)."""
    import torch
    n = max(2, m // 3)
    p = gen.er(n, 2 * m + 8, seed=m)[:m]
    flat = np.concatenate([np.zeros(words, np.int32), p.view(np.int32)])
    t = torch.from_numpy(flat)
    t = t.cuda() if where == "device" else t.pin_memory() if where == "pinned" else t
    torch.cuda.synchronize()
    want, _ = oracle.cc_solve(p, n)
    for flags in (0, _lib.PHEM_CC_CANONICAL):
        lab, slots, st = np.empty(n, np.int32), np.empty(n, np.uint64), _lib.CCStats()
        _lib.check(_lib.lib().phem_cc_solve(ctx.handle, t.data_ptr() + 4 * words, len(p), n, lab.ctypes.data,
                                            slots.ctypes.data, flags, _lib.C.byref(st)), "phem_cc_solve")
        np.testing.assert_array_equal(lab, want)
        check_forest(p, n, want, slots)


def _zigzag(k):
    """r_i = i, a_i = k + 2i, b_i = a_i + 1: all (r_i, a_i) and (r_i, b_i), then all (a_i, b_{i+1}).  Every vertex
    hooks under its r_i at once, and the k roots then hook into one chain in a single round."""
    i = np.arange(k, dtype=np.uint64)
    a, b = np.uint64(k) + 2 * i, np.uint64(k) + 2 * i + np.uint64(1)
    u = np.concatenate([i, i, np.minimum(a[:-1], b[1:])])
    v = np.concatenate([a, b, np.maximum(a[:-1], b[1:])])
    return (u << np.uint64(32)) | v, 3 * k


def _block_and_path(n, low, repeat):
    """n edges that make one component of n / 2 vertices, then a path over the other half in order, `repeat` times,
    linked to the component; low: the path has the smaller ids, so the component's root ends up under it."""
    h = n // 2
    rng = np.random.default_rng(7)
    x = np.concatenate([np.arange(1, h), rng.integers(1, h, n - h + 1)])
    block = (np.zeros(n, np.uint64) << np.uint64(32)) | x.astype(np.uint64)
    path = np.arange(h - 1, dtype=np.uint64)
    path = (path << np.uint64(32)) | (path + np.uint64(1))
    off = np.uint64((h << 32) | h)
    if low:
        block += off
        link = np.uint64(((h - 1) << 32) | h)
    else:
        path += off
        link = np.uint64((1 << 32) | h)
    return np.concatenate([block, [link]] + [path] * repeat), n


@pytest.mark.parametrize("kind", ["zigzag", "zigzag_rest", "path", "path_low", "path_long_rest", "path_low_long_rest",
                                  "path_links", "path_low_links"])
def test_chains_of_roots(ctx, kind):
    """Roots that hook into chains of hundreds of thousands in one step, before each of the passes that point vertices
    at their roots: labels and forest exact, and no walk of a chain one vertex after another."""
    import torch
    if kind.startswith("zigzag"):
        p, n = _zigzag(350000)
        if kind == "zigzag_rest":
            p = np.concatenate([p, p[:n]])
    else:
        p, n = _block_and_path(1 << 21 if kind == "path" else 1 << 20, "low" in kind, 13 if "long" in kind else 2)
        if "links" in kind:  # from all over the path to the other half
            u, v = np.random.default_rng(3).integers(0, n // 2, (2, n // 4)).astype(np.uint64)
            p = np.concatenate([p, (u << np.uint64(32)) | (v + np.uint64(n // 2))])
    d = torch.from_numpy(p.view(np.int64)).cuda()
    lab = torch.empty(n, dtype=torch.int32, device="cuda")
    slots = torch.empty(n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ms = []
    for _ in range(3):
        r = ctx.cc_solve(d, n, labels=lab, forest=slots)
        ms.append(r.device_ms)
        assert not lab.any() and r.components == 1
    check_forest(p, n, np.zeros(n, np.int32), slots.cpu().numpy().view(np.uint64))
    assert min(ms) < 2.0  # 0.07 to 0.6; link by link 10 to 60


def test_solves_without_room_for_the_lists():
    """Device memory that holds the arrays of a solve but not the lists of the
    one-launch form: the launches without lists solve it."""
    import torch
    n = 4_000_000
    p = gen.er(n, 4_400_000, 5)
    d = torch.from_numpy(p.view(np.int64)).cuda()
    lab = torch.empty(n, dtype=torch.int32, device="cuda")
    slots = torch.empty(n, dtype=torch.int64, device="cuda")
    with P.Context(0) as c:
        c.cc_solve(p, n)  # their kernels are loaded
        c.trim()
        lab.fill_(-1)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (100 << 20), dtype=torch.uint8, device="cuda")
        try:
            r = c.cc_solve(d, n, labels=lab, forest=slots)
        finally:
            del hog
            torch.cuda.empty_cache()
    want, _ = oracle.cc_solve(p, n)
    np.testing.assert_array_equal(lab.cpu().numpy(), want)
    assert r.components == len(np.unique(want)) == n - r.forest_edges
    check_forest(p, n, want, slots.cpu().numpy().view(np.uint64))


def test_canonical_solve_of_many_vertices_in_little_memory():
    """The canonical forest of 8,000,000 vertices and few edges, results on
    the host, in 290 MB of device memory (it needs 32 bytes per vertex)."""
    import torch
    n = 8_000_000
    p = gen.er(n, 100_000, 5)
    with P.Context(0) as c:
        want = c.cc_solve(p, n, canonical=True)
        c.trim()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (290 << 20), dtype=torch.uint8, device="cuda")
        try:
            r = c.cc_solve(p, n, canonical=True)
        finally:
            del hog
            torch.cuda.empty_cache()
    labels, forest = oracle.cc_solve(p, n)
    for x in (want, r):
        np.testing.assert_array_equal(x.labels, labels)
        np.testing.assert_array_equal(forest_set(x.forest), oracle.forest_set(forest))


@pytest.mark.parametrize("n,m", [(3000, 9000), (40000, 200000)])  # one CTA, the grid
@pytest.mark.parametrize("canonical", [False, True])
def test_pageable_outputs_do_not_hold_up_other_threads(ctx, n, m, canonical):
    """While one thread waits for a solve with results in pageable memory,
    behind other work on its stream, another thread's solves on a context of
    its own go on."""
    import threading
    import time
    import torch
    p, q = gen.er(n, m, 3), gen.er(2000, 8000, 4)
    d, dq = (torch.from_numpy(x.view(np.int64)).cuda() for x in (p, q))
    ahead = torch.zeros(1 << 26, device="cuda")
    stream = torch.cuda.Stream()
    out = {}

    def solve():
        ctx.set_stream(stream)
        out["r"] = ctx.cc_solve(d, n, canonical=canonical)
        ctx.set_stream(None)

    with P.Context(0) as other:
        solve()
        other.cc_solve(dq, 2000)
        ahead.add_(1)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for _ in range(800):  # about 0.07 s of kernels
                ahead.add_(1)
        t = threading.Thread(target=solve)
        t.start()
        calls = []
        while t.is_alive():
            t0 = time.perf_counter()
            other.cc_solve(dq, 2000)
            calls.append(time.perf_counter() - t0)
        t.join()
    np.testing.assert_array_equal(out["r"].labels, oracle.cc_solve(p, n)[0])
    assert len(calls) > 20 and max(calls) < 0.02
