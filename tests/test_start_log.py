"""Backtracking by the log of cell starts (csrc/canon_sparse.cuh) against
reconstruct_at_level (partition_refinement.cpp:541-604): the reference keeps an
in_level per cell and merges every maximal run of cells created below the
target level with the cell after it; the kernel clears the starts logged since
that level's child was made.  Random searches on the CPU: splits give every
fragment but the last the new level, backtracks go to any level above."""
import random

import pytest


def reconstruct(starts, inlev, level):
    """The cell starts that survive, and their in_levels."""
    order = sorted(starts)
    keep, lev, run = set(), {}, None
    for p in order:
        if run is None:
            run = p
        if inlev[p] <= level:  # closes the run: the merged cell starts at `run`
            keep.add(run)
            lev[run] = inlev[p]
            run = None
    assert run is None
    return keep, lev


@pytest.mark.parametrize("n", [2, 3, 31, 64, 65, 200])
def test_start_log_equals_reconstruct_at_level(n):
    rng = random.Random(n)
    for _ in range(60):
        starts = {0} | {rng.randrange(n) for _ in range(rng.randrange(3))}
        inlev = {p: 0 for p in starts}
        log, mark, level = [], {}, 1
        for _ in range(40):
            if len(starts) < n and (level == 1 or rng.random() < 0.7):
                mark[level] = len(log)
                for step in range(rng.randrange(1, 5)):  # individualize, then refine
                    cells = [(p, q) for p, q in zip(sorted(starts), sorted(starts)[1:] + [n])
                             if q - p > 1]
                    if not cells:
                        break
                    c, e = rng.choice(cells)
                    new = sorted(rng.sample(range(c + 1, e),
                                            1 if step == 0 else rng.randrange(1, e - c)))
                    old = inlev[c]
                    for f in [c] + new[:-1]:
                        inlev[f] = level + 1
                    inlev[new[-1]] = old
                    starts |= set(new)
                    log += new
                level += 1
            elif level > 1:
                level = rng.randrange(1, level)
                keep, lev = reconstruct(starts, inlev, level)
                starts -= set(log[mark[level]:])
                del log[mark[level]:]
                assert starts == keep
                inlev = lev
            assert len(log) <= n
