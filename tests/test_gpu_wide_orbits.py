"""Orbits in the wide search: target cells at the sizes where their merging
changes (two members, the lanes of a warp, more), beside many stored
automorphisms that fix the sequence and move no member of the cell."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _broom(G, leaves, rng):
    """A path whose vertex i carries leaves[i] leaves, and a tail that makes its
    ends differ: the leaves of a vertex are one cell, its automorphisms fix every
    other cell."""
    edges, n = [], len(leaves) + 3
    edges += [(i, i + 1) for i in range(n - 1)]
    for i, k in enumerate(leaves):
        edges += [(i, n + j) for j in range(k)]
        n += k
    return G.random_relabel(G.from_edges(n, np.asarray(edges)), rng)


@pytest.mark.parametrize("gate", [0, 1])
@pytest.mark.parametrize("leaves", [[2] * 40, [3, 2, 31, 2, 4], [2, 32, 3, 2], [33, 2, 2, 3],
                                    [2, 2, 65, 2]])
def test_cells(pkg, G, oracle_mod, leaves, gate):
    g = _broom(G, leaves, np.random.default_rng(len(leaves)))
    ctx = pkg.Context(0, wide_min_n=1)
    ctx.set_option(pkg.api.GCL_OPT_WIDE_GATE, gate)
    r = pkg.canon(g, ctx=ctx)
    assert np.array_equal(r.matrix, oracle_mod.canon(g)[0])
    assert pkg.api.group_order(g, ctx) == math.prod(math.factorial(k) for k in leaves)


def test_idle_entries_cost_a_test(pkg, G):
    """A tree: each of some 255 stored automorphisms swaps a few vertices, and the
    others' target cells need none of it.  Tested, not merged, they leave the
    orbits at 4.0 times the refinement's cycles; merged, they took 9.0 times.  The
    line lies at the geometric mean."""
    g = G.tree_plus_edges(2100, np.random.default_rng(7))
    ctx = pkg.Context(0)
    ctx.set_option(pkg.api.GCL_OPT_COUNTERS, 1)
    rows = pkg.api.canon_rows(g, 10000, ctx)[0]
    c = ctx.wide_counters()
    assert c["auts_first"] > 200, c
    assert c["orbit_cycles"] < 6 * c["refine_cycles"], c
    batch = pkg.canon_batch([g], max_aut=10000, ctx=pkg.Context(0), dense=False, rows=True)
    assert np.array_equal(rows.ravel(), batch.rows[: rows.size])


@pytest.mark.parametrize("leaves", [[2, 32, 3], [33, 2, 2], [64, 2, 65], [3, 96, 40, 2], [129, 2]])
def test_cells_in_a_batch(pkg, G, oracle_mod, leaves):
    # ... and the ring's search, also where the ring wraps
    rng = np.random.default_rng(len(leaves))
    gs = [_broom(G, leaves, rng) for _ in range(2)] + [G.random_relabel(G.torus(9, 8), rng)]
    for max_aut in (10000, 20):
        res = pkg.canon_batch(gs, max_aut=max_aut, rows=True)
        out, ooff, na, nd = oracle_mod.canon_batch(res.arena, max_aut=max_aut)
        assert (res.status == 0).all()
        assert np.array_equal(res.dense[: ooff[-1]], out[: ooff[-1]])
        assert np.array_equal(res.stats[:, 0], na) and np.array_equal(res.stats[:, 1], nd)


def test_large_cells_join_their_members_together(pkg, G):
    """A star: every stored automorphism swaps two of up to 100 members."""
    g = G.from_edges(101, np.array([(0, i) for i in range(1, 101)]))
    ctx = pkg.Context(0)
    ctx.set_option(pkg.api.GCL_OPT_COUNTERS, 1)
    pkg.api.canon_rows(g, 10000, ctx)
    c = ctx.wide_counters()
    assert c["auts_first"] == 99, c
    assert c["orbit_cycles"] < 160000 * c["nodes"], c
