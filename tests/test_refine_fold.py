"""The sparse kernels' hash fold over a bitmap of fragment starts (sp_fold,
csrc/canon_sparse.cuh), restated in Python and checked on the CPU against the
serial chain mash(l, i) = ((l ^ 065435) + i) & 077777
(partition_refinement.h:9-19): an item per set position, the position plus its
count, folded one bit of the running value at a time over all positions, with
words of 32 positions spread over 32 lanes."""
import random

import pytest

C, M = 0o65435, 0o77777


def serial(lc, valid, cnt):
    for p in range(len(valid)):
        if valid[p]:
            lc = ((lc ^ C) + p + cnt[p]) & M
    return lc


def parity(x):
    return bin(x).count("1") & 1


def fold_dense(lc, base, words, kw, cnt):
    """One chunk: lane l holds words l*kw .. l*kw+kw-1 of 32 positions from
    word `base` on; returns the value after the chunk's items."""
    full = 0xffffffff
    pat = [0xaaaaaaaa, 0xcccccccc, 0xf0f0f0f0, 0xff00ff00, 0xffff0000]
    kb = [[0] * len(words) for _ in range(6)]
    for w, v in enumerate(words):
        for b in range(32):
            if v >> b & 1:
                k = cnt.get((base + w) * 32 + b, 0)
                for j in range(6):
                    kb[j][w] |= (k >> j & 1) << b
    carry, cp, out = [0] * len(words), [0] * len(words), 0
    for j in range(15):
        cm = full if C >> j & 1 else 0
        vj, inc = [0] * len(words), [0] * len(words)
        for w, v in enumerate(words):
            pj = pat[j] if j < 5 else (full if ((base + w) * 32) >> j & 1 else 0)
            kj = kb[j][w] if j < 6 else 0
            vj[w] = pj ^ kj ^ cp[w]
            cp[w] = (pj & kj) | (cp[w] & (pj ^ kj))
            f = v & (cm ^ vj[w] ^ carry[w])
            for s in (1, 2, 4, 8, 16):
                f ^= f << s & full
            inc[w] = f
        lanes = [0] * 32
        for w in range(len(words)):
            lanes[w // kw] ^= inc[w] >> 31
        x0 = lc >> j & 1
        for lane in range(32):
            run = x0 ^ (sum(lanes[:lane]) & 1)
            for w in range(lane * kw, lane * kw + kw):
                y = (full if run else 0) ^ (inc[w] << 1 & full) ^ cm
                carry[w] = (y & vj[w]) | (carry[w] & (y ^ vj[w]))
                run ^= inc[w] >> 31
        out |= (x0 ^ (sum(lanes) & 1)) << j
    return out


@pytest.mark.parametrize("kw", [1, 4])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 1023, 1024, 1025, 4096, 4097, 40000])
def test_fold_over_positions_equals_serial_chain(n, kw):
    rng = random.Random(n * 8 + kw)
    for density in (0.01, 0.3, 1.0):
        valid = [rng.random() < density for _ in range(n)]
        cnt = {p: rng.randrange(64) for p in range(n) if rng.random() < 0.05}
        lc0 = rng.randrange(1 << 17)
        lc, words = lc0, []
        for wi in range((n + 31) // 32):
            words.append(sum(valid[p] << (p - 32 * wi) for p in range(32 * wi, min(n, 32 * wi + 32))))
        for base in range(0, len(words), 32 * kw):
            chunk = words[base:base + 32 * kw]
            lc = fold_dense(lc, base, chunk + [0] * (32 * kw - len(chunk)), kw, cnt)
        full = [cnt.get(p, 0) for p in range(n)]
        assert lc & M == serial(lc0, valid, full) & M
