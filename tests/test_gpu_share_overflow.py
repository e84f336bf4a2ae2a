"""Work sharing when a warp's orbit representatives outgrow their room: warps that
wait for a handed-over subtree see that status (kAutOverflow, 1) and end, and the
call falls back to the sequential search."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _complete(G, n):
    return G.from_edges(n, np.array([(i, j) for i in range(n) for j in range(i)]))


def _star(G, n):
    return G.from_edges(n, np.array([(0, i) for i in range(1, n)]))


# 140 vertices: target cells of 139 + 138 + ... members, room for 64 of 142
@pytest.mark.parametrize("gate", [0, 1, 2])
@pytest.mark.parametrize("make", [_complete, _star])
def test_overflow_ends_the_waits(pkg, G, oracle_mod, make, gate):
    g = make(G, 140)
    ctx = pkg.Context(0)
    ctx.set_option(pkg.api.GCL_OPT_WIDE_SHARE, 1)
    ctx.set_option(pkg.api.GCL_OPT_WIDE_GATE, gate)
    want = oracle_mod.canon(g)
    assert np.array_equal(pkg.canon(g, ctx=ctx).matrix, want[0])
