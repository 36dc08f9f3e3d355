"""The rule the lane-split band kernel rests on, on the CPU: a band computed with more
columns than it has, and more rows and reference positions than the pair has, gives the
band's own result when the extra cells never match -- over the scorings at the edge of
what the dispatch accepts."""
import random

import numpy as np
import pytest

NEG = -1_000_000


def padded_sw(q, r, band, extra, match, mis, go, ge):
    """Smith-Waterman over columns [0, 2*band + extra], rows [0, len(q) + extra): cells
    outside the band or the matrix never match, none are skipped but ri < 0."""
    goe, w = go + ge, 2 * band + 1 + extra
    h = [0] * w
    best = (0, 0, 0)
    for qi in range(len(q) + extra):
        left, e, cur = 0, NEG, []
        for j in range(w):
            ri = qi - band + j
            real = j <= 2 * band and 0 <= ri < len(r) and qi < len(q)
            sub = match if real and q[qi] == r[ri] else mis
            e = max(e + ge, (h[j + 1] if j + 1 < w else 0) + goe)
            v = max(h[j] + sub, e, left + goe, 0)
            if v > best[0]:
                best = (v, qi, ri)
            cur.append(v)
            left = v
        h = cur
    return best


def padded_nw(q, r, band, extra, match, mis, go, ge):
    goe, w = go + ge, 2 * band + 1 + extra
    h = [NEG if j < band or j > 2 * band else 0 if j == band else go + (j - band) * ge
         for j in range(w)]
    for qi in range(len(q)):
        left, cur = NEG, []
        for j in range(w):
            ri = qi - band + j
            if ri < 0:
                cur.append(NEG)
                left = NEG
                continue
            real = j <= 2 * band and ri < len(r)
            sub = match if real and q[qi] == r[ri] else mis
            left = max(h[j] + sub, (h[j + 1] if j + 1 < w else NEG) + goe, left + goe)
            cur.append(left)
        h = cur
    fo = len(r) - len(q) + band
    return h[fo] if 0 <= fo <= 2 * band else NEG


def _pair(rng):
    n = rng.randint(1, 24)
    q = [rng.randrange(4) for _ in range(n)]
    if rng.random() < 0.6:
        r = list(q)
        for _ in range(rng.randint(0, 5)):
            p = rng.randrange(len(r) + 1)
            if rng.random() < 0.5:
                r.insert(p, rng.randrange(4))
            elif p < len(r) and len(r) > 1:
                del r[p]
    else:
        r = [rng.randrange(4) for _ in range(rng.randint(1, 30))]
    return q, r


def _batch(seqs):
    from genomics_b200 import SequenceBatch
    return SequenceBatch.from_strings(["".join("ACGT"[c] for c in s) for s in seqs]).arrays()


# gap_open, gap_extend, mismatch: mismatch down to go + ge, ge up to 0
@pytest.mark.parametrize("sc", [(2, -4, -4, -2), (2, -6, -4, -2), (1, -1, 0, -1), (3, -5, -5, 0),
                                (1, 0, 0, 0), (5, -1, -1, 0), (2, -3, -5, -2)])
def test_smith_waterman_padding(oracle, sc):
    rng = random.Random(hash(sc) & 0xFFFF)
    pairs = [_pair(rng) for _ in range(150)]
    (qp, _, qo, ql), (rp, _, ro, rl) = _batch([p[0] for p in pairs]), _batch([p[1] for p in pairs])
    for band in (0, 1, 3, 7):
        want = oracle.sw_batch(qp, qo, ql, rp, ro, rl, *sc, band)
        for i, (q, r) in enumerate(pairs):
            got = padded_sw(q, r, band, rng.randint(0, 9), *sc)
            assert got == tuple(int(c[i]) for c in want), (sc, band, q, r)


# mismatch down to 2 * (go + ge)
@pytest.mark.parametrize("sc", [(2, -4, -4, -2), (2, -12, -4, -2), (1, -2, 0, -1), (3, 1, -5, 0),
                                (1, 0, 0, 0), (2, -3, -5, -2)])
def test_needleman_wunsch_padding(oracle, sc):
    rng = random.Random(hash(sc) & 0xFFFF)
    pairs = [_pair(rng) for _ in range(150)]
    (qp, _, qo, ql), (rp, _, ro, rl) = _batch([p[0] for p in pairs]), _batch([p[1] for p in pairs])
    for band in (0, 1, 3, 7):
        want = np.asarray(oracle.nw_batch(qp, qo, ql, rp, ro, rl, *sc, band))
        for i, (q, r) in enumerate(pairs):
            assert padded_nw(q, r, band, rng.randint(0, 9), *sc) == int(want[i]), (sc, band, q, r)
