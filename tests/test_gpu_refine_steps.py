"""The sparse kernels' refinement steps at the sizes where they change: words and
summary words of the bitmaps, one or four words per lane in the hash fold,
splitters of 32 and more members or edges, cells of 32 and more vertices,
neighbour counts of 64 and more, shared-memory and device-memory state.
Bit-exact against the oracle, through the batched search (form and
statistics) and the search of one graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def star(G, k, leaves):
    """k stars of `leaves` leaves whose centres form a path."""
    n = k * (leaves + 1)
    e = [(i, i + 1) for i in range(k - 1)]
    e += [(i, k + i * leaves + j) for i in range(k) for j in range(leaves)]
    return G.from_edges(n, e)


def bipartite(G, a, b, p, rng):
    m = np.argwhere(rng.random((a, b)) < p)
    return G.from_edges(a + b, np.stack([m[:, 0], a + m[:, 1]], axis=1))


def graphs(G, n, rng):
    out = [G.tree_plus_edges(n, rng),
           G.erdos_renyi(n, min(1.0, 6.0 / n), rng),
           G.erdos_renyi(n, min(0.5, 60.0 / n), rng)]
    g = G.erdos_renyi(n, min(1.0, 6.0 / n), rng)
    # many colours: every byte of the colour sort
    out.append(G.from_edges(n, g.edges(), rng.integers(-70000, 70000, n)))
    out.append(G.from_edges(n, g.edges(), rng.integers(0, 300, n)))
    return out


def check(pkg, oracle_mod, gs, **opts):
    seq = pkg.Context(0, wide_min_n=pkg.api.GCL_MAX_N + 1)
    one = pkg.Context(0, wide_min_n=1)
    for c in (seq, one):
        for k, v in opts.items():
            c.set_option(getattr(pkg.api, k), v)
    res = pkg.canon_batch(gs, ctx=seq)
    out, ooff, na, nd = oracle_mod.canon_batch(res.arena)
    assert (res.status == 0).all()
    assert np.array_equal(res.dense[: ooff[-1]], out[: ooff[-1]])
    assert np.array_equal(res.stats[:, 0], na) and np.array_equal(res.stats[:, 1], nd)
    for i, g in enumerate(gs):
        assert np.array_equal(pkg.canon(g, ctx=one).matrix, res.matrix(i)), (i, g.n)


@pytest.mark.parametrize("n", [65, 95, 96, 97, 127, 128, 129, 255, 256, 257])
def test_sizes(pkg, G, oracle_mod, n):
    check(pkg, oracle_mod, graphs(G, n, np.random.default_rng(n)))


@pytest.mark.parametrize("n", [1023, 1024, 1025, 1057])
def test_large_sparse(pkg, G, oracle_mod, n):
    rng = np.random.default_rng(n)
    gs = [G.erdos_renyi(n, 9.0 / n, rng)]
    check(pkg, oracle_mod, gs)
    check(pkg, oracle_mod, gs, GCL_OPT_SMEM_STAGE=0)


@pytest.mark.parametrize("leaves", [15, 16, 31, 32, 33, 70])
def test_stars_and_large_cells(pkg, G, oracle_mod, leaves):
    rng = np.random.default_rng(leaves)
    gs = [star(G, 3, leaves), bipartite(G, 40, leaves + 30, 0.5, rng),
          bipartite(G, 100, 2 * leaves, 0.9, rng), G.torus(9, 11)]
    check(pkg, oracle_mod, gs)
    check(pkg, oracle_mod, gs, GCL_OPT_SMEM_STAGE=0)


@pytest.mark.parametrize("n", [130, 300])
def test_few_touched_vertices_of_large_cells(pkg, G, oracle_mod, n):
    rng = np.random.default_rng(n)
    gs = [G.random_regular(n, 3, rng), G.random_regular(n, 5, rng),
          G.disjoint_union(G.random_regular(n // 2 - (n // 2) % 2, 4, rng), 2)]
    check(pkg, oracle_mod, gs)
    check(pkg, oracle_mod, gs, GCL_OPT_SMEM_STAGE=0)
