"""The one-thread-per-pair Smith-Waterman kernel (bands 16 and 32, scores to 511) against the
oracle where it can go wrong: lengths from 0 to the score limit, references shorter and
longer than the query, gap terms of 0 and 255, mismatch equal to the gap cost, a last warp of
one pair, ragged lengths (queued) and equal ones.  Integers: equal or wrong."""
import numpy as np
import pytest

from genomics_b200 import AlignConfig
from test_gpu_split import _pack, _pairs, _rows, _sw, _tile

pytestmark = pytest.mark.gpu

SCORES = [(2, -4, -4, -2), (1, -1, -1, 0), (3, -6, -6, 0), (1, 0, -1, -1), (5, -250, -255, 0),
          (100, -155, -100, -155), (255, 0, 0, 0), (0, -3, -3, -1)]


@pytest.mark.parametrize("band", [16, 32])
@pytest.mark.parametrize("sc", SCORES)
def test_scores_to_the_limit(device, oracle, band, sc):
    rng = np.random.default_rng(band + sc[0])
    longest = min(511 // max(sc[0], 1) - 1, 160)
    q, r = _pairs(rng, 400, 0, max(longest, 0), pad=band // 2)
    # _mutate may lengthen a query: keep the ones within the limit, in a last warp of one
    ql = q.arrays()[3]
    keep = np.nonzero(ql <= longest)[0][:321]
    (qp, qm, qo, _), (rp, rm, ro, rl) = q.arrays(), r.arrays()
    q = type(q).from_arrays(qp, qm, qo[keep], ql[keep])
    r = type(r).from_arrays(rp, rm, ro[keep], rl[keep])
    want = _sw(oracle, q, r, sc, band)
    cfg = AlignConfig(*sc, band)
    for times in (1, 201):
        for batched in (True, False):
            got = _rows(device.sw_banded(_tile(q, times), _tile(r, times), cfg, batched=batched))
            np.testing.assert_array_equal(got, np.tile(want, (times, 1)))


@pytest.mark.parametrize("band", [16, 32])
@pytest.mark.parametrize("qlen,rlen", [(1, 1), (15, 17), (16, 16), (17, 15), (31, 64), (33, 32),
                                       (48, 20), (20, 150), (150, 150), (150, 182), (182, 150)])
def test_equal_lengths(device, oracle, band, qlen, rlen):
    rng = np.random.default_rng(qlen * 200 + rlen)
    qs, rs = [], []
    for _ in range(97):
        t = rng.integers(0, 4, max(qlen, rlen)).astype(np.uint64)
        s = t.copy()
        flip = rng.random(s.size) < 0.06
        s[flip] = rng.integers(0, 4, int(flip.sum()))
        qs.append(s[:qlen])
        rs.append(np.roll(t, int(rng.integers(0, 4)))[:rlen])
    q, r = _pack(qs), _pack(rs)
    want = _sw(oracle, q, r, (2, -4, -4, -2), band)
    for times in (1, 641):
        got = _rows(device.sw_banded(_tile(q, times), _tile(r, times), AlignConfig(2, -4, -4, -2, band)))
        np.testing.assert_array_equal(got, np.tile(want, (times, 1)))
