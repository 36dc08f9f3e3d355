"""How inputs and results travel: a pair per call at the lengths around a word and around
the limit of the single-copy upload (2^21 bases), and batches large enough to run in parts
(2^18 pairs and more), against the oracle.  Integers: equal or wrong."""
import numpy as np
import pytest

from genomics_b200 import AlignConfig, SequenceBatch, WFAConfig

pytestmark = pytest.mark.gpu

SC = (2, -4, -4, -2)


def _batch(lens, rng, like=None):
    """Random sequences, or ones that follow those of `like` except for a base in forty."""
    lens = np.asarray(lens, np.int64)
    words = (lens + 31) // 32
    offs = np.concatenate(([0], np.cumsum(words)[:-1])).astype(np.int64)
    flat = rng.integers(0, 4, max(int(words.sum()), 1) * 32).astype(np.uint64)
    if like is not None:
        m = min(flat.size, like.size)
        keep = rng.random(m) > 0.025
        flat[:m][keep] = like[:m][keep]
    codes = flat.copy()
    for o, w, l in zip(offs, words, lens):
        flat[o * 32 + l:(o + w) * 32] = 0
    shift = (62 - 2 * np.arange(32)).astype(np.uint64)
    packed = np.bitwise_or.reduce(flat.reshape(-1, 32) << shift, axis=1)
    return SequenceBatch.from_arrays(packed, np.zeros_like(packed), offs, lens), codes


LIMIT = 1 << 21


@pytest.mark.parametrize("qlen,rlen", [(0, 0), (0, 1), (1, 0), (1, 1), (31, 32), (32, 33), (33, 31),
                                       (64, 65), (1000, 1003), (LIMIT, LIMIT), (LIMIT + 1, 7),
                                       (7, LIMIT + 1)])
def test_pair_calls(device, oracle, qlen, rlen):
    rng = np.random.default_rng(qlen * 7 + rlen)
    r, codes = _batch([rlen], rng)
    q, _ = _batch([qlen], rng, codes)
    qp, _, qo, ql = q.arrays()
    rp, _, ro, rl = r.arrays()
    cfg = AlignConfig(*SC, 5)
    want = np.stack(oracle.sw_batch(qp, qo, ql, rp, ro, rl, *SC, 5), 1)[0]
    got = device.sw_pair(qp, qlen, rp, rlen, cfg)
    assert [int(v) for v in got] == [int(v) for v in want]
    wcfg = WFAConfig(4, 6, 2, 400)
    want = oracle.wfa_batch(qp, qo, ql, rp, ro, rl, 4, 6, 2, 400)[0][0]
    assert device.wfa_pair(qp, qlen, rp, rlen, wcfg) == int(want)


@pytest.mark.parametrize("bands", [False, True])
@pytest.mark.parametrize("n", [(1 << 18) - 1, 1 << 18, 300001])
def test_batches_in_parts(device, oracle, n, bands):
    rng = np.random.default_rng(n)
    m = 500
    lens = rng.integers(0, 60, m)
    r, codes = _batch(lens + rng.integers(0, 9, m), rng)
    q, _ = _batch(lens, rng, codes)
    qp, qm, qo, ql = q.arrays()
    rp, rm, ro, rl = r.arrays()
    b = rng.integers(0, 20, m).astype(np.int32) if bands else None
    idx = np.arange(n) % m
    tile = lambda p, k, o, l: SequenceBatch.from_arrays(p, k, o[idx], l[idx])
    Q, R = tile(qp, qm, qo, ql), tile(rp, rm, ro, rl)
    B = b[idx] if bands else None
    cfg = AlignConfig(*SC, 12)
    sw = np.stack(oracle.sw_batch(qp, qo, ql, rp, ro, rl, *SC, 12, bands=b), 1)[idx]
    got = device.sw_banded(Q, R, cfg, bands=B).view(np.int32).reshape(-1, 3)
    np.testing.assert_array_equal(got, sw)
    nw = oracle.nw_batch(qp, qo, ql, rp, ro, rl, *SC, 12, bands=b)[idx]
    np.testing.assert_array_equal(device.nw_banded(Q, R, cfg, bands=B)["score"], nw)
