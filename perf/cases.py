"""The calls whose speed this framework is judged by, over the sizes it is used at.

A case is one call of a public entry point on inputs of one family: a single
graph (``canon`` / ``canon_rows``), a batch in host memory (``canon_batch``) or
a batch resident on the device (``gcl_canon_batch_device_async``); the case of
isomorphism pairs checks a short list of them (``is_isomorphic``).  Families and sizes are those of the
benchmark workloads (``graphs.py``): trees of maximum degree 4 with a few extra
edges, Erdos-Renyi graphs, random regular graphs, toroidal grids, unions of
identical components, and dense coloured graphs up to 64 vertices.

``listed()`` gives the named cases, ``draw(rng)`` another one of the same
ranges, ``prepare`` the inputs, ``run`` one call and its results, ``work`` the
bytes a call cannot do without: the CSR arena read once and the results
written once.  There are no floating-point operations.

Results are whole numbers.  A batch returns forms, labelings, statistics and
statuses, all of which the sequential order defines.  A single graph above 64
vertices returns its canonical form alone: its labeling is one of several
equivalent ones and its statistics depend on the order in which warps finish.

A case fixes the sizes (and, in a batch, which graphs are relabelings of
others); the seed draws the graphs.
"""
import importlib
import math

import numpy as np
import torch

PKG = importlib.import_module("gpu-canonical-labeling_b200")
API = importlib.import_module("gpu-canonical-labeling_b200.api")
G = PKG.graphs

MAX_AUT = 10000  # automorphisms kept per search, the workloads' setting
MOLECULE = 24    # vertices of the small seeded component beside a torus


def listed():
    return [
        # the command line and the drop-in call on a small molecule-like
        # graph: one launch, latency is everything
        {"name": "one_tree_24", "call": "one", "family": "tree", "n": 24},
        # the two-graph check: candidate pairs one after the other, each an
        # Erdos-Renyi graph beside a relabeling of it or a copy with an edge moved
        {"name": "pairs_er_256", "call": "pairs", "family": "er", "n": 256, "degree": 12.8,
         "count": 12},
        # the throughput workload: 10,000 small graphs already on the device
        {"name": "device_small_10000", "call": "device", "family": "tree", "count": 10000,
         "lo": 10, "hi": 64},
        # the same family from host memory, as a pipeline stage calls it
        {"name": "host_small_4000", "call": "host", "family": "tree", "count": 4000,
         "lo": 10, "hi": 64},
        # dense and coloured small graphs, matrices out as bytes
        {"name": "host_dense_colored_2000", "call": "host", "family": "dense", "count": 2000,
         "lo": 2, "hi": 64},
        # the serving loop's middle class: trees just above the small kernel
        {"name": "host_trees_256", "call": "host", "family": "tree", "count": 512,
         "lo": 65, "hi": 256},
        # ... and its large class: few graphs, long searches
        {"name": "host_trees_1000", "call": "host", "family": "tree", "count": 48,
         "lo": 257, "hi": 1000},
        # the mixed-size batch: four families, sizes log-uniform
        {"name": "host_mixed_256", "call": "host", "family": "mixed", "count": 160,
         "lo": 64, "hi": 256},
        # single symmetric or rigid graphs, each spread over the whole GPU
        {"name": "one_regular_4096", "call": "one", "family": "regular", "n": 4096, "degree": 3},
        {"name": "one_torus_64x64", "call": "one", "family": "torus", "n": 4120, "k": 64},
        {"name": "one_union_4x64", "call": "one", "family": "union", "n": 256, "k": 4,
         "degree": 4},
        # the largest graphs: a sparse random graph of 20,000 vertices
        {"name": "one_er_20000", "call": "one", "family": "er", "n": 20000, "degree": 8.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one_small", "pairs", "device", "host", "dense", "mid", "long", "mixed",
                       "regular", "torus", "union", "er"])
    if kind == "one_small":
        return {"call": "one", "family": "tree", "n": rng.randint(6, 64)}
    if kind == "pairs":
        return {"call": "pairs", "family": "er", "n": _log_int(rng, 30, 600),
                "degree": round(rng.uniform(6.0, 16.0), 2), "count": rng.randint(8, 16)}
    if kind in ("device", "host"):
        lo = rng.randint(2, 32)
        return {"call": kind, "family": "tree",
                "count": _log_int(rng, 20, 10000 if kind == "device" else 4000),
                "lo": lo, "hi": rng.randint(max(lo, 24), 64)}
    if kind == "dense":
        return {"call": "host", "family": "dense", "count": _log_int(rng, 20, 2000), "lo": 2,
                "hi": rng.randint(16, 64)}
    if kind == "mid":
        lo = rng.randint(40, 128)
        return {"call": "host", "family": "tree", "count": _log_int(rng, 20, 512), "lo": lo,
                "hi": rng.randint(lo, 256)}
    if kind == "long":
        hi = _log_int(rng, 300, 1000)
        return {"call": "host", "family": "tree", "count": _log_int(rng, 4, 48), "lo": 257,
                "hi": hi}
    if kind == "mixed":
        return {"call": "host", "family": "mixed", "count": _log_int(rng, 16, 160), "lo": 64,
                "hi": rng.randint(96, 256)}
    if kind == "regular":
        return {"call": "one", "family": "regular", "n": 2 * _log_int(rng, 40, 2048),
                "degree": rng.choice([3, 3, 4])}
    if kind == "torus":
        k = _log_int(rng, 9, 64)
        k2 = max(8, int(k * rng.uniform(0.7, 1.0)))
        return {"call": "one", "family": "torus", "n": k * k2 + MOLECULE, "k": k}
    if kind == "union":
        k = rng.choice([2, 3, 4])
        return {"call": "one", "family": "union", "n": k * rng.randint(34, 64), "k": k,
                "degree": 4}
    return {"call": "one", "family": "er", "n": _log_int(rng, 600, 20000),
            "degree": round(rng.uniform(6.0, 10.0), 2)}


def _sparse_er(n, degree, rng):
    """An Erdos-Renyi graph of the given mean degree from sampled pairs (the
    all-pairs generator of graphs.py would hold n * n / 2 of them)."""
    m = int(rng.binomial(n * (n - 1) // 2, min(1.0, degree / max(n - 1, 1))))
    a = rng.integers(0, n, int(m * 1.2) + 16)
    b = rng.integers(0, n, int(m * 1.2) + 16)
    keep = a != b
    key = np.unique(np.minimum(a, b)[keep] * n + np.maximum(a, b)[keep])
    key = rng.permutation(key)[:m]
    return G.from_edges(n, np.stack([key // n, key % n], axis=1))


def _one(case, rng):
    n, fam = case["n"], case["family"]
    if fam == "tree":
        return G.tree_plus_edges(n, rng)
    if fam == "er":
        return _sparse_er(n, case["degree"], rng)
    if fam == "regular":
        return G.random_regular(n, case["degree"], rng)
    if fam == "torus":
        # beside a small random component, so that every seed has its own form
        t, mol = G.torus(case["k"], (n - MOLECULE) // case["k"]), G.tree_plus_edges(MOLECULE, rng)
        return G.random_relabel(
            G.from_edges(n, np.concatenate([t.edges(), mol.edges() + t.n])), rng)
    return G.random_relabel(
        G.disjoint_union(G.random_regular(n // case["k"], case["degree"], rng), case["k"]), rng)


def _mixed(i, n, shape, rng):
    """Graph i of the mixed batch: four families in turn.  Unions have two or
    three components (the search grows exponentially in their number)."""
    if i % 4 == 0:
        return _sparse_er(n, 8.0, rng)
    if i % 4 == 1:
        d = int(shape.choice([3, 4, 6]))
        return G.random_regular(n + (n * d) % 2, d, rng)
    if i % 4 == 2:
        k = max(3, int(round(math.sqrt(n) * shape.uniform(0.7, 1.3))))
        return G.random_relabel(G.torus(k, max(3, round(n / k))), rng)
    k = int(shape.choice([2, 3]))
    c = n // k
    return G.random_relabel(G.disjoint_union(G.random_regular(c, 4 if c % 2 else 3, rng), k), rng)


def _batch(case, rng):
    count, lo, hi, fam = case["count"], case["lo"], case["hi"], case["family"]
    shape = np.random.default_rng(count)  # what the case fixes, whatever the seed
    out = []
    for i in range(count):
        if fam == "mixed":
            n = int(round(math.exp(shape.uniform(math.log(lo), math.log(hi)))))
            out.append(_mixed(i, n, shape, rng))
            continue
        n = int(shape.integers(lo, hi + 1))
        if fam == "dense":  # any density, every second graph coloured
            g = G.erdos_renyi(n, float(rng.uniform(0.1, 0.9)), rng)
            if i % 2:
                g.color = rng.integers(0, 4, n).astype(np.int32)
            out.append(g)
        elif i and shape.random() < 0.2:  # a fifth are relabelings of earlier graphs
            out.append(G.random_relabel(out[int(shape.integers(i))], rng))
        else:
            out.append(G.tree_plus_edges(n, rng))
    return out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    ctx = PKG.default_context()
    call = case["call"]
    if call == "one":
        return {"call": call, "ctx": ctx, "graph": _one(case, rng), "small": case["n"] <= 64}
    if call == "pairs":
        pairs = []
        for _ in range(case["count"]):
            g = _one(case, rng)
            h = g if rng.random() < 0.5 else G.move_one_edge(g, rng)
            pairs.append((g, G.random_relabel(h, rng)))
        return {"call": call, "ctx": ctx, "pairs": pairs}
    arena = G.pack(_batch(case, rng))
    if call == "host":
        return {"call": call, "ctx": ctx, "arena": arena, "dense": case["family"] == "dense"}
    # device-resident: arena and result buffers that the program keeps
    roff = API.rows_offsets(arena)
    dev = {k: torch.from_numpy(v).cuda() for k, v in (
        ("voff", arena.voff), ("eoff", arena.eoff), ("rowptr", arena.rowptr),
        ("col", arena.col if arena.col.size else np.zeros(1, np.int32)), ("roff", roff))}
    out = {"rows": torch.zeros(max(int(roff[-1]), 1), dtype=torch.int64, device="cuda"),
           "label": torch.zeros(max(int(arena.voff[-1]), 1), dtype=torch.int32, device="cuda"),
           "stats": torch.zeros(2 * arena.count, dtype=torch.int64, device="cuda"),
           "status": torch.zeros(arena.count, dtype=torch.int32, device="cuda")}
    torch.cuda.synchronize()
    return {"call": call, "ctx": ctx, "count": arena.count, "max_n": int(arena.sizes().max()),
            "max_m2": int(np.diff(arena.eoff).max()), "dev": dev, "out": out}


def run(s):
    ctx, call = s["ctx"], s["call"]
    if call == "one":
        if s["small"]:
            r = PKG.canon(s["graph"], MAX_AUT, ctx)
            return {"matrix": r.matrix, "nodes": r.nodes, "num_aut": r.num_aut}
        return {"rows": API.canon_rows(s["graph"], MAX_AUT, ctx)[0].view(np.int64)}
    if call == "pairs":
        return {"isomorphic": np.array([PKG.is_isomorphic(a, b, MAX_AUT, ctx)
                                        for a, b in s["pairs"]], dtype=np.uint8)}
    if call == "host":
        r = PKG.canon_batch(s["arena"], MAX_AUT, ctx, dense=s["dense"], rows=not s["dense"])
        return {"form": r.dense if s["dense"] else r.rows.view(np.int64), "label": r.label,
                "stats": r.stats, "status": r.status}
    d, o = s["dev"], s["out"]
    rc = ctx.lib.gcl_canon_batch_device_async(
        ctx.handle, s["count"], d["voff"].data_ptr(), d["eoff"].data_ptr(),
        d["rowptr"].data_ptr(), d["col"].data_ptr(), None, MAX_AUT, s["max_n"], s["max_m2"],
        None, None, o["rows"].data_ptr(), d["roff"].data_ptr(), o["label"].data_ptr(),
        o["stats"].data_ptr(), o["status"].data_ptr())
    if rc != 0:
        raise API.GclError(rc, "gcl_canon_batch_device_async")
    ctx.sync()  # the call only enqueues; its results may be read after this
    return o


def work(case):
    fam = case["family"]
    if case["call"] in ("one", "pairs"):
        sizes = [(float(case["n"]), 1.0 if case["call"] == "one" else 2.0 * case["count"])]
    elif fam == "mixed":  # log-uniform sizes
        pts = np.exp(np.linspace(math.log(case["lo"]), math.log(case["hi"]), 65))
        sizes = [(float(p), case["count"] / 65.0) for p in pts]
    else:  # uniform sizes
        span = range(case["lo"], case["hi"] + 1)
        sizes = [(float(p), case["count"] / len(span)) for p in span]
    total = 0.0
    for n, k in sizes:
        if fam == "tree":
            m2 = 2.0 * (n + 2.0)
        elif fam == "dense":
            m2 = 0.5 * n * (n - 1.0)
        elif fam == "torus":
            m2 = 4.0 * n
        elif fam == "mixed":
            m2 = 5.0 * n
        else:
            m2 = n * case["degree"]
        read = 4.0 * (n + 1.0) + 4.0 * m2
        if fam == "dense":
            read += 2.0 * n  # colours of every second graph
        if case["call"] == "pairs":
            wrote = 0.5
        elif fam == "dense" or (case["call"] == "one" and n <= 64):
            wrote = n * n
        else:
            wrote = 8.0 * n * math.ceil(n / 64.0)
        if case["call"] in ("host", "device"):
            read += 24.0           # offsets
            wrote += 4.0 * n + 20  # labeling, statistics, status
        total += k * (read + wrote)
    return {"bytes": total, "flops": 0.0}
