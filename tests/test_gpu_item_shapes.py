"""The wide search's launch shapes for graphs of which fewer than four warps' state
fits a block's shared memory: item counts on both sides of the line between them
give the form that a search from device memory gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(G, n, k, rng):
    """A cubic component of k vertices -- k - 1 items -- beside a sparse random
    rest, which the root refinement makes (all but) discrete."""
    a, b = G.random_regular(k, 3, rng), n - k
    e = np.sort(rng.integers(0, b, (4 * b, 2)), axis=1)
    e = np.unique(e[e[:, 0] != e[:, 1]], axis=0)
    return G.random_relabel(G.from_edges(n, np.concatenate([a.edges(), e + k])), rng)


# n, then the line's item count at 148 SMs: 8 per warp, 3 / 2 / 1 warps per SM
@pytest.mark.parametrize("n,line", [(8200, 3552), (11000, 2368), (17000, 1184)])
def test_both_sides_of_the_line(pkg, G, n, line):
    rng = np.random.default_rng(n)
    staged, device = pkg.Context(0), pkg.Context(0)
    device.set_option(pkg.api.GCL_OPT_SMEM_STAGE, 0)
    for k in (40, line - 40, line + 40):
        g = _graph(G, n, k, rng)
        a = pkg.api.canon_rows(g, 10000, staged)[0]
        h = G.random_relabel(g, rng)
        assert np.array_equal(a, pkg.api.canon_rows(h, 10000, staged)[0])
        assert np.array_equal(a, pkg.api.canon_rows(h, 10000, device)[0])
