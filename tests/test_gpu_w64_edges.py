"""The warp kernel for graphs of up to 64 vertices at the edges of its 32-lane
halves: target cells of up to and above 32 members, rings that wrap and that
reach past 32 entries, rows of every length.  Forms, automorphism counts and
node counts equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graphs(G, n, rng):
    out = [G.from_edges(n, []),
           G.from_edges(n, [(i, j) for i in range(n) for j in range(i + 1, n)])]
    if n >= 3:
        out.append(G.from_edges(n, [(i, (i + 1) % n) for i in range(n)]))
        out.append(G.from_edges(n, [(0, i) for i in range(1, n)]))
        out.append(G.from_edges(n, [(i, j) for i in range(n // 2) for j in range(n // 2, n)]))
    for p in (0.05, 0.3, 0.5, 0.95):
        g = G.erdos_renyi(n, p, rng)
        out.append(g)
        out.append(G.from_edges(n, g.edges(), rng.integers(-3, 4, n)))
    if n >= 12 and n % 2 == 0:
        out.append(G.random_regular(n, 3, rng))
        out.append(G.disjoint_union(G.random_regular(n // 2 - (n // 2) % 2, 3, rng), 2))
    return out


@pytest.mark.parametrize("max_aut", [1, 3, 40, 10000])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 63, 64])
def test_sizes(pkg, G, oracle_mod, n, max_aut):
    gs = graphs(G, n, np.random.default_rng(100 * n))
    if max_aut < 40:  # a short store hardly prunes the empty and the complete graph
        gs = gs[2:]
    res = pkg.canon_batch(gs, max_aut=max_aut)
    out, ooff, na, nd = oracle_mod.canon_batch(res.arena, max_aut=max_aut)
    assert (res.status == 0).all()
    assert np.array_equal(res.dense[: ooff[-1]], out[: ooff[-1]])
    assert np.array_equal(res.stats[:, 0], na) and np.array_equal(res.stats[:, 1], nd)
