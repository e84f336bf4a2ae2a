"""Orbit pruning of the batched search above 64 vertices (sp_orbits,
csrc/canon_sparse.cuh) where its forms change: target cells of up to and above
32 vertices, ring entries across 32-bit words, a ring that wraps, levels deeper
than one pass held before.  Forms, automorphism counts and node counts equal
the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stars(G, k, leaves):
    n = k * (leaves + 1)
    e = [(i, i + 1) for i in range(k - 1)]
    e += [(i, k + i * leaves + j) for i in range(k) for j in range(leaves)]
    return G.from_edges(n, e)


@pytest.mark.parametrize("max_aut", [1, 2, 31, 32, 33, 64, 65, 300, 10000])
def test_orbits_vs_oracle(pkg, G, oracle_mod, max_aut):
    rng = np.random.default_rng(7)
    ctx = pkg.Context(0, wide_min_n=pkg.api.GCL_MAX_N + 1)
    cyc = G.from_edges(5, [(i, (i + 1) % 5) for i in range(5)])
    gs = [stars(G, 34, 2), stars(G, 3, 31), stars(G, 3, 32), stars(G, 2, 33), stars(G, 2, 65),
          G.tree_plus_edges(330, rng), G.tree_plus_edges(200, rng), G.torus(8, 9)]
    if max_aut >= 31:  # a short store prunes these too little
        gs.append(G.disjoint_union(cyc, 14))
    res = pkg.canon_batch(gs, max_aut=max_aut, ctx=ctx)
    out, ooff, na, nd = oracle_mod.canon_batch(res.arena, max_aut=max_aut)
    assert (res.status == 0).all()
    assert np.array_equal(res.dense[: ooff[-1]], out[: ooff[-1]])
    assert np.array_equal(res.stats[:, 0], na) and np.array_equal(res.stats[:, 1], nd)
