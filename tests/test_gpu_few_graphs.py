"""Batches around the size up to which every graph of up to 64 vertices gets a
block of its own (w64_few_kernel), and around the eighths of the size ordering:
equal to the oracle and to the same graphs in a large batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_aut", [2, 300, 10000])
@pytest.mark.parametrize("count", [1, 2, 63, 64, 65, 2047, 2049, 4097])
def test_counts(pkg, G, oracle_mod, count, max_aut):
    pool = G.small_batch(200, seed=count, n_lo=1, n_hi=64) + [G.from_edges(0, []), G.torus(3)]
    gs = [pool[i % len(pool)] for i in range(count)]
    res = pkg.canon_batch(gs, max_aut=max_aut, rows=True)
    out, ooff, na, nd = oracle_mod.canon_batch(res.arena, max_aut=max_aut)
    assert (res.status == 0).all()
    assert np.array_equal(res.dense[: ooff[-1]], out[: ooff[-1]])
    assert np.array_equal(res.stats[:, 0], na) and np.array_equal(res.stats[:, 1], nd)
    big = pkg.canon_batch(gs + pool, max_aut=max_aut, rows=True)
    assert np.array_equal(res.label[: res.arena.voff[-1]], big.label[: res.arena.voff[-1]])
    assert np.array_equal(res.rows[: res.roff[-1]], big.rows[: res.roff[-1]])


def test_bad_graph_among_few(pkg, G):
    bad = G.torus(4)
    bad = G.Graph(bad.n, bad.rowptr, np.where(np.arange(bad.col.size) == 3, 40, bad.col).astype(np.int32))
    res = pkg.canon_batch([G.torus(5), bad, G.torus(4)], per_graph_errors=True)
    assert res.status.tolist() == [0, 3, 0]
    assert np.array_equal(res.matrix(2), pkg.canon(G.torus(4)).matrix)


def test_packed_and_direct_copies_agree(pkg, G):
    # 13,000 graphs with dense output pass the size up to which a call's arrays
    # are packed into one copy; halves of it do not
    pool = G.small_batch(250, seed=9, n_lo=20, n_hi=60)
    gs = pool * 52
    whole = pkg.canon_batch(gs, rows=True)
    half = pkg.canon_batch(gs[: len(gs) // 4], rows=True)
    assert whole.arena.out_offsets()[-1] > 16 << 20 and (whole.status == 0).all()
    assert np.array_equal(whole.dense[: half.ooff[-1]], half.dense[: half.ooff[-1]])
    assert np.array_equal(whole.rows[: half.roff[-1]], half.rows[: half.roff[-1]])
    assert np.array_equal(whole.stats[: len(half.stats)], half.stats)
    assert np.array_equal(whole.dense[-half.ooff[-1]:], half.dense[: half.ooff[-1]])
