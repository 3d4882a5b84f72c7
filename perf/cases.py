"""Performance cases: whole calls of the public API over the sizes it is used at.

A case names an entry point (`call`), a graph family and its size.  Families:

* er    Erdos-Renyi pairs in draw order, duplicates kept (the connected-components workload);
* rmat  R-MAT pairs sorted row-major as a symmetrised CSR lists them (the minimum-spanning-forest workload);
* rgg   2-D random geometric 8-nearest-neighbour graphs with distance weights (road-like: high diameter,
        many Boruvka rounds).

Weights of er and rmat are uniform in [1, 2^20].  All cases share one Context, as a program that solves many graphs
does.  Every output is an integer and has to be reproduced exactly, so there is no floating-point reference.  The
default connected-components forest is whichever edges won the hooking races (two runs differ), so those cases return
the labels and the counts; the canonical case returns its forest slots too.
"""
from __future__ import annotations

import ctypes as C
import random
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from phem_graph_b200 import Context, _lib, gen

_context = None


def _ctx() -> Context:
    """The program's one solver handle."""
    global _context
    if _context is None:
        _context = Context(torch.cuda.current_device())
    return _context


def listed():
    return [
        # the smallest solves: a served request of about 2^13 edges, device-resident and from pageable host memory,
        # where launches, round trips and synchronisations are the time
        {"name": "msf_er_2k", "call": "msf", "family": "er", "n": 2003, "m": 8009},
        {"name": "msf_host_er_1k", "call": "msf_host", "family": "er", "n": 1021, "m": 4093},
        # an ordinary graph of about a million edges with an odd size (a large served request)
        {"name": "msf_er_131k", "call": "msf", "family": "er", "n": 131101, "m": 1048573},
        # a road-like graph: many rounds over short lists
        {"name": "msf_rgg_262k", "call": "msf", "family": "rgg", "n": 262147, "m": 1209000},
        # the headline workload: R-MAT scale 22, edge factor 16, device-resident records
        {"name": "msf_rmat_22", "call": "msf", "family": "rmat", "n": 1 << 22, "m": 1 << 26},
        # the same family given as a symmetrised CSR with one weight per edge
        {"name": "msf_csr_rmat_20", "call": "msf_csr", "family": "rmat", "n": 1 << 20, "m": 1 << 24},
        # end to end: pinned host records in, host records out
        {"name": "msf_host_rmat_19", "call": "msf_host", "family": "rmat", "n": 1 << 19, "m": 1 << 23},
        # connected components: a small request, the Erdos-Renyi workload (8 M edges), the largest R-MAT
        {"name": "cc_er_3k", "call": "cc", "family": "er", "n": 3001, "m": 9001},
        {"name": "cc_er_2m", "call": "cc", "family": "er", "n": 2000003, "m": 1 << 23},
        {"name": "cc_rmat_22", "call": "cc", "family": "rmat", "n": 1 << 22, "m": 1 << 26},
        # the deterministic forest (minimum spanning forest under edge order)
        {"name": "cc_canonical_er_1m", "call": "cc_canonical", "family": "er", "n": 1 << 20, "m": 1 << 23},
        # many small graphs in one call: 256 of the mixed er / rgg workload, n log-uniform in [64, 65536]
        {"name": "batch_256", "call": "batch", "family": "mixed", "graphs": 256, "n_lo": 64, "n_hi": 65536},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    call = rng.choice(["msf", "msf", "msf", "msf_host", "msf_csr", "cc", "cc", "cc_canonical", "batch"])
    if call == "batch":
        n_hi = _log_uniform(rng, 256, 65536)
        return {"call": call, "family": "mixed", "graphs": _log_uniform(rng, 16, 256), "n_lo": 64, "n_hi": n_hi}
    family = rng.choice(["er", "er", "rmat", "rmat"] + ([] if call == "cc" else ["rgg"]))
    if family == "rgg":
        n = _log_uniform(rng, 500, 1 << 18)
        return {"call": call, "family": family, "n": n, "m": int(4.6 * n)}
    if family == "rmat":
        m = _log_uniform(rng, 1 << 10, 1 << 26 if call in ("msf", "cc") else 1 << 23)
        n = 1 << min(22, max(6, (int(m / rng.uniform(4, 32)) + 1).bit_length() - 1))
    else:
        m = _log_uniform(rng, 1 << 10, 1 << 24 if call in ("msf", "cc") else 1 << 23)
        # edges per vertex; components are only of interest below the density where a graph is one component
        n = int(m / rng.uniform(0.5, 0.28 * np.log(m))) if call == "cc" else max(16, int(m / rng.uniform(1, 16)))
    return {"call": call, "family": family, "n": n, "m": m}


def _pairs(case, seed):
    """Packed pairs (u << 32 | v), u < v, and the graph's own weights if it has any, on the GPU."""
    n, m, dev = case["n"], case["m"], torch.device("cuda")
    if case["family"] == "rgg":
        p, w = gen.rgg(n, 8, seed)
        return torch.from_numpy(p.view(np.int64)).to(dev), torch.from_numpy(w.view(np.int32)).to(dev)
    if case["family"] == "rmat":
        out = torch.empty(m, dtype=torch.int64, device=dev)
        torch.cuda.synchronize()
        k = gen.rmat_range_device(_ctx(), n.bit_length() - 1, 0, m, seed, out)
        return torch.sort(out[:k]).values, None
    g = torch.Generator(device=dev).manual_seed(seed)
    a = torch.randint(0, n, (m,), generator=g, device=dev)
    b = torch.randint(0, n - 1, (m,), generator=g, device=dev)
    b += b >= a  # no self-loops
    return (torch.minimum(a, b) << 32) | torch.maximum(a, b), None


def _mixed(case, seed):
    """Batch of er (mean degree uniform in [2, 16]) and rgg graphs in turn, n log-uniform; the sizes belong to the
    case, the edges to the seed."""
    sizes = random.Random(4)
    parts = []
    for i in range(case["graphs"]):
        n, degree = _log_uniform(sizes, case["n_lo"], case["n_hi"]), sizes.uniform(2, 16)
        parts.append((n, int(n * degree / 2) if i % 2 == 0 else 0, seed * 1000003 + i))

    def graph(part):
        n, draws, gs = part
        pairs, w = (gen.er(n, draws, gs), None) if draws else gen.rgg(n, 8, gs)
        return "", n, gen.msf_edges(pairs, gen.weights(len(pairs), gs + 7) if w is None else w), gen.PHEM_BATCH_MSF

    with ThreadPoolExecutor(16) as pool:
        return gen.batch_from(pool.map(graph, parts))


def _weights(count, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 1000)
    return torch.randint(1, (1 << gen.WEIGHT_BITS) + 1, (count,), generator=g, device="cuda", dtype=torch.int32)


def _records(pairs, w):
    """{u, v, w} records."""
    return torch.stack(((pairs >> 32).to(torch.int32), (pairs & 0xffffffff).to(torch.int32), w), dim=1).contiguous()


def prepare(case, seed):
    ctx, call = _ctx(), case["call"]
    s = {"ctx": ctx, "call": call}
    if call == "batch":
        b = _mixed(case, seed)
        b.edges = torch.from_numpy(b.edges.view(np.int32)).cuda()
        s["batch"] = b
        pinned = lambda k, dt: torch.empty(k, dtype=dt).pin_memory().numpy()  # noqa: E731
        s["out"] = {"ids": pinned(b.total_vertices, torch.int32).view(np.uint32),
                    "count": pinned(b.num_graphs, torch.int32).view(np.uint32),
                    "total": pinned(b.num_graphs, torch.int64).view(np.uint64),
                    "labels": pinned(b.total_vertices, torch.int32)}
        s["forests"] = np.zeros(b.total_vertices, np.uint32)
        return s
    n = s["n"] = case["n"]
    pairs, w = _pairs(case, seed)
    s["m"] = pairs.numel()
    if call in ("cc", "cc_canonical"):
        s["edges"] = pairs
        s["labels"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["forest"] = torch.empty(n, dtype=torch.int64, device="cuda")
        return s
    w = _weights(s["m"], seed) if w is None else w
    if call == "msf_csr":
        rows, cols = pairs >> 32, pairs & 0xffffffff
        order = torch.sort(pairs).indices  # weights follow the row-major entry order
        both = torch.sort(torch.cat((pairs, (cols << 32) | rows))).values
        s["offsets"] = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        s["offsets"][1:] = torch.cumsum(torch.bincount(both >> 32, minlength=n), 0)
        s["cols"] = (both & 0xffffffff).to(torch.int32)
        s["weights"] = w[order].contiguous()
        s["out"] = torch.zeros((n, 3), dtype=torch.int32, device="cuda")
        return s
    rec = _records(pairs, w)
    if call == "msf":
        s["edges"], s["out"] = rec, torch.zeros((n, 3), dtype=torch.int32, device="cuda")
    elif s["m"] >= 1 << 20:  # large host inputs and outputs are pinned, small ones plain arrays
        s["edges"] = rec.cpu().pin_memory().numpy().view(np.uint32)
        s["out"] = torch.zeros((n, 3), dtype=torch.int32).pin_memory().numpy().view(np.uint32)
    else:
        s["edges"], s["out"] = rec.cpu().numpy().view(np.uint32), np.zeros((n, 3), np.uint32)
    return s


def run(s):
    ctx, call = s["ctx"], s["call"]
    if call == "msf":
        r = ctx.msf_solve_device(s["edges"], s["m"], s["n"], s["out"])
        return {"edges": s["out"], "count": r.count, "total": r.total}
    if call == "msf_host":
        r = ctx.msf_solve(s["edges"], s["n"], out=s["out"])
        return {"edges": s["out"], "count": r.count, "total": r.total}
    if call == "msf_csr":
        cnt, tot = C.c_uint64(), C.c_uint64()
        _lib.check(_lib.lib().phem_msf_solve_csr(ctx.handle, s["offsets"].data_ptr(), s["cols"].data_ptr(), s["n"],
                                                 s["weights"].data_ptr(), s["m"], s["out"].data_ptr(), C.byref(cnt),
                                                 C.byref(tot), None), "phem_msf_solve_csr")
        return {"edges": s["out"], "count": cnt.value, "total": tot.value}
    if call == "batch":
        b = s["batch"]
        r = ctx.batch_solve(b, out=s["out"])
        np.concatenate([r.forest(b, g) for g in range(b.num_graphs)], out=s["forests"][:int(r.count.sum())])
        return {"forests": s["forests"], "count": r.count, "total": r.total, "labels": r.labels}
    r = ctx.cc_solve(s["edges"], s["n"], canonical=call == "cc_canonical", labels=s["labels"], forest=s["forest"])
    out = {"labels": s["labels"], "components": r.components, "forest_edges": r.forest_edges}
    if call == "cc_canonical":
        out["forest"] = s["forest"]
    return out


def work(case):
    """Each input read once and each output written once (integer work: no floating-point operations)."""
    call = case["call"]
    if call == "batch":
        v = case["graphs"] * (case["n_hi"] - case["n_lo"]) / max(1e-9, np.log(case["n_hi"] / case["n_lo"]))
        return {"bytes": float(v * (12 * 4.5 + 8)), "flops": 0}
    n, m = case["n"], case["m"]
    if call in ("cc", "cc_canonical"):
        return {"bytes": 8 * m + 12 * n, "flops": 0}
    read = 4 * 2 * m + 8 * (n + 1) + 4 * m if call == "msf_csr" else 12 * m
    return {"bytes": read + 12 * min(n - 1, m), "flops": 0}
