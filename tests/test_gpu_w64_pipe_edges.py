"""Edge families of up to 64 vertices in batches of more than 64 graphs, which run
on the pipelined launch: root partitions handed over (coloured, discrete, regular),
rings that wrap, complete, empty, star and bipartite graphs, unions, tori.  (Fewer
graphs get a block each, test_gpu_w64_edges.py.)  Each graph is there relabeled
too; forms, automorphism counts and node counts equal the oracle's."""
import numpy as np
import pytest

from test_gpu_w64_edges import graphs as edge_graphs

pytestmark = pytest.mark.gpu


def _symmetric(G, rng):
    out = [G.torus(k) for k in (3, 5, 8)] + [G.cfi_graph(4, rng), G.cfi_graph(6, rng, twist=True)]
    out += [G.disjoint_union(G.random_regular(8, 3, rng), k) for k in (2, 4, 8)]
    return [g for g in out if g.n <= 64]


def _colored(G, g, rng):
    return G.from_edges(g.n, g.edges(), rng.integers(-3, 4, g.n))


@pytest.mark.parametrize("max_aut", [3, 40, 300, 10000])
@pytest.mark.parametrize("sizes", [(1, 2, 3, 33), (31, 32), (63, 64)])
def test_edges(pkg, G, oracle_mod, sizes, max_aut):
    rng = np.random.default_rng(sum(sizes))
    pool = _symmetric(G, rng)
    for n in sizes:
        # a short store hardly prunes the empty and the complete graph
        pool += edge_graphs(G, n, rng)[0 if max_aut >= 40 else 2:]
    pool += [G.random_relabel(g, rng) for g in pool] + [_colored(G, g, rng) for g in pool]
    gs = [pool[i % len(pool)] for i in range(max(len(pool), 65))]
    assert len(gs) > 64
    res = pkg.canon_batch(gs, max_aut=max_aut, rows=True)
    out, ooff, na, nd = oracle_mod.canon_batch(res.arena, max_aut=max_aut)
    assert (res.status == 0).all()
    assert np.array_equal(res.dense[: ooff[-1]], out[: ooff[-1]])
    assert np.array_equal(res.stats[:, 0], na) and np.array_equal(res.stats[:, 1], nd)
    # the same graphs a few at a time
    for i in range(0, len(gs), 48):
        few = pkg.canon_batch(gs[i: i + 48], max_aut=max_aut, rows=True)
        a, b = res.roff[i], res.roff[i + few.arena.count]
        assert np.array_equal(few.rows[: b - a], res.rows[a:b])
        assert np.array_equal(few.label, res.label[res.arena.voff[i]: res.arena.voff[i] + len(few.label)])
        assert np.array_equal(few.stats, res.stats[i: i + few.arena.count])
