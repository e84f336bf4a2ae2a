"""The branch-free cell lookup of the sparse kernels for up to 1,024 vertices
(cell_of_1k, csrc/canon_sparse.cuh), restated in Python: bounds equal a direct
search and every word it reads lies among the bitmap's words of positions."""
import random

import pytest

M = 0xffffffff


def clz(x):
    return 32 - x.bit_length()


def ffs(x):
    return (x & -x).bit_length()


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 96, 127, 128, 129, 500, 992, 1023, 1024])
def test_cell_bounds(n):
    rng = random.Random(n)
    nwd, words = (n + 31) // 32, 2 * ((n + 63) // 64 + 1)
    for _ in range(40):
        density = rng.random() ** 3
        starts = {0, n} | {i for i in range(n) if rng.random() < density}
        st = [0] * words
        for q in starts:
            st[q >> 5] |= 1 << (q & 31)
        some = sum(1 << w for w in range(nwd) if st[w])
        for p in rng.sample(range(n), min(n, 40)):
            w, sh = p >> 5, p & 31
            lo, hi = st[w] & (M >> (31 - sh)), st[w] & (0xfffffffe << sh & M)
            below, above = some & ((1 << w) - 1), some & (0xfffffffe << w & M)
            wl = w if lo or not below else 31 - clz(below)
            wh = w if hi or not above else ffs(above) - 1
            assert 0 <= wl < nwd and 0 <= wh < nwd
            y, z = lo or st[wl], hi or st[wh]
            a = wl * 32 + 31 - clz(y)
            e = min(n, wh * 32 + ffs(z) - 1) if hi or above else n
            assert a == max(q for q in starts if q <= p) and e == min(q for q in starts if q > p)
