"""The lane-split band kernel (Smith-Waterman and Needleman-Wunsch, any band) against the
oracle at the sizes where it can go wrong: bands at and around the column counts of its
shapes, batches small and large enough for every shape, lengths around the 16-row blocks,
scores that move the values' base up and down, per-pair bands, layouts at the limits of
its 16-bit range.  Integers: equal or wrong."""
import numpy as np
import pytest

from genomics_b200 import AlignConfig, SequenceBatch
from genomics_b200._lib import FLAG_INT32

pytestmark = pytest.mark.gpu

READS = (2, -4, -4, -2)


def _pack(seqs):
    """SequenceBatch of code arrays, one after another."""
    lens = np.array([len(s) for s in seqs], np.int64)
    words = (lens + 31) // 32
    offs = np.concatenate(([0], np.cumsum(words)[:-1])).astype(np.int64)
    flat = np.zeros(max(int(words.sum()), 1) * 32, np.uint64)
    for s, o in zip(seqs, offs):
        flat[o * 32:o * 32 + len(s)] = s
    shift = (62 - 2 * np.arange(32)).astype(np.uint64)
    packed = np.bitwise_or.reduce(flat.reshape(-1, 32) << shift, axis=1)
    return SequenceBatch.from_arrays(packed, np.zeros_like(packed), offs, lens)


def _mutate(rng, s, rate):
    out = []
    for c, u in zip(s.tolist(), rng.random(len(s)).tolist()):
        if u < rate * 0.2:
            continue
        out.append((c + int(rng.integers(1, 4))) & 3 if u < rate * 0.7 else c)
        if u > 1 - rate * 0.3:
            out.append(int(rng.integers(0, 4)))
    return np.array(out, np.uint64)


def _pairs(rng, n, lo, hi, pad=12):
    qs, rs = [], []
    for _ in range(n):
        L = int(rng.integers(lo, hi + 1))
        t = rng.integers(0, 4, L + 2 * pad).astype(np.uint64)
        if rng.random() < 0.2:
            q = rng.integers(0, 4, L).astype(np.uint64)
        else:
            q = _mutate(rng, t[pad:pad + L], 0.1)
        qs.append(q)
        rs.append(t)
    return _pack(qs), _pack(rs)


def _tile(b, times):
    """The same sequences `times` over (they share their words)."""
    p, m, o, l = b.arrays()
    return SequenceBatch.from_arrays(p, m, np.tile(o, times), np.tile(l, times))


def _sw(O, q, r, sc, band, bands=None):
    qp, _, qo, ql = q.arrays()
    rp, _, ro, rl = r.arrays()
    return np.stack(O.sw_batch(qp, qo, ql, rp, ro, rl, *sc, band, bands=bands), 1)


def _rows(res):
    return res.view(np.int32).reshape(-1, 3)


@pytest.mark.parametrize("band", [2, 8, 12, 13, 17, 20, 24, 28, 33, 40, 49, 57, 66, 79, 99, 131,
                                  159, 271, 543])
def test_sw_bands_of_every_shape(device, oracle, band):
    """250 pairs once (the shapes with the most lanes) and repeated to 60,000 (those with
    the most columns per lane), in input order and queued by length."""
    rng = np.random.default_rng(band)
    q, r = _pairs(rng, 250, 0, 90)
    want = _sw(oracle, q, r, READS, band)
    cfg = AlignConfig(*READS, band)
    for times in (1, 12, 240):
        qq, rr = _tile(q, times), _tile(r, times)
        for batched in (True, False):
            got = _rows(device.sw_banded(qq, rr, cfg, batched=batched))
            assert (got.reshape(times, -1, 3) == want).all(), (band, times, batched)


@pytest.mark.parametrize("sc", [(2, -6, -4, -2), (3, -5, -5, 0), (1, 0, 0, 0), (100, -100, -60, -40)])
def test_sw_scorings_at_the_edge(device, oracle, sc):
    rng = np.random.default_rng(sc[0])
    q, r = _pairs(rng, 400, 0, 35)
    for band in (5, 32, 50):
        got = _rows(device.sw_banded(q, r, AlignConfig(*sc, band)))
        assert (got == _sw(oracle, q, r, sc, band)).all(), (sc, band)


@pytest.mark.parametrize("length", [1, 15, 16, 17, 31, 32, 33, 47, 48, 49])
def test_sw_lengths_around_the_blocks(device, oracle, length):
    rng = np.random.default_rng(length)
    q, r = _pairs(rng, 60, length, length)
    q2, r2 = _pairs(rng, 60, length, length, pad=0)
    for qq, rr in ((q, r), (q2, r2), (r, q)):
        for band in (3, 32, 70):
            got = _rows(device.sw_banded(qq, rr, AlignConfig(*READS, band)))
            assert (got == _sw(oracle, qq, rr, READS, band)).all(), band


def test_sw_long_scores_move_the_base(device, oracle):
    """Pairs whose scores pass 4,094 and fall again: matching stretches, unrelated ones
    (the score decays to 0 and the base with it), sequences that end early on either
    side, repeats (equal maxima), and a second, larger stretch after a decay."""
    rng = np.random.default_rng(12)
    rnd = lambda n: rng.integers(0, 4, n).astype(np.uint64)
    qs, rs = [], []
    for k in range(24):
        a, b = rnd(2600 + 150 * k), rnd(1500 + 200 * (k % 5))
        x, y = rnd(1800 + 300 * (k % 4)), rnd(1800 + 300 * (k % 4))
        qs += [np.concatenate(s) for s in ((a, x, b), (a, x, b, a), (b, x, a), (a,), (a, b))]
        rs += [np.concatenate(s) for s in ((a, y, b), (a, y, b, a), (b, y, a), (a, b, x), (a,))]
    unit = rnd(37)
    for k in range(6):
        qs.append(np.tile(unit, 90 + k))
        rs.append(np.tile(unit, 85 + 2 * k))
    qs = [_mutate(rng, s, 0.02) if i % 3 else s for i, s in enumerate(qs)]
    q, r = _pack(qs), _pack(rs)
    for band in (16, 32, 40, 128):
        want = _sw(oracle, q, r, READS, band)
        assert (want[:, 0] > 4094).any()
        cfg = AlignConfig(*READS, band)
        for batched in (True, False):
            assert (_rows(device.sw_banded(q, r, cfg, batched=batched)) == want).all(), band
        if band != 40:
            assert (_rows(device.sw_banded(q, r, cfg, flags=FLAG_INT32)) == want).all(), band
        # many of them: the shapes with more columns per lane
        got = _rows(device.sw_banded(_tile(q, 40), _tile(r, 40), cfg))
        assert (got.reshape(40, -1, 3) == want).all(), band


def test_sw_scores_past_what_the_base_can_follow(device, oracle):
    """Penalties so large that the band's spread does not fit the 16-bit window: long
    pairs take the int32 or literal kernel, short ones of the same call do not."""
    rng = np.random.default_rng(3)
    sc = (20, -60, -50, -20)
    q, r = _pairs(rng, 120, 20, 900)
    for band in (32, 45, 128):
        assert (_rows(device.sw_banded(q, r, AlignConfig(*sc, band)))
                == _sw(oracle, q, r, sc, band)).all(), band


def test_sw_any_band_per_pair(device, oracle):
    rng = np.random.default_rng(4)
    q, r = _pairs(rng, 600, 0, 300)
    for top in (3, 64, 128, 600):  # above 543: those pairs take the literal kernel
        bands = rng.integers(0, top + 1, 600).astype(np.int32)
        bands[:3] = 0, top, top
        want = _sw(oracle, q, r, READS, 32, bands=bands)
        for batched in (True, False):
            got = _rows(device.sw_banded(q, r, AlignConfig(*READS, 32), bands=bands,
                                         batched=batched))
            assert (got == want).all(), top
        got = _rows(device.sw_banded(_tile(q, 30), _tile(r, 30), AlignConfig(*READS, 32),
                                     bands=np.tile(bands, 30)))
        assert (got.reshape(30, -1, 3) == want).all(), top


def _nw(O, q, r, sc, band, bands=None):
    qp, _, qo, ql = q.arrays()
    rp, _, ro, rl = r.arrays()
    return np.stack((O.nw_batch(qp, qo, ql, rp, ro, rl, *sc, band, bands=bands), ql - 1, rl - 1), 1)


@pytest.mark.parametrize("band", [0, 2, 8, 12, 13, 17, 24, 33, 49, 66, 131, 271, 543, 544])
def test_nw_bands_of_every_shape(device, oracle, band):
    rng = np.random.default_rng(band + 1)
    q, r = _pairs(rng, 250, 0, 90, pad=3)
    want = _nw(oracle, q, r, READS, band)
    cfg = AlignConfig(*READS, band)
    for times in (1, 12, 240 if band < 544 else 2):
        got = _rows(device.nw_banded(_tile(q, times), _tile(r, times), cfg))
        assert (got.reshape(times, -1, 3) == want).all(), (band, times)


@pytest.mark.parametrize("sc", [(2, -12, -4, -2), (1, -2, 0, -1), (3, 1, -5, 0), (1, 0, 0, 0),
                                (0, -255, -120, -80), (2, -13, -4, -2)])
def test_nw_scorings_and_lengths(device, oracle, sc):
    """Scorings at the edge of the padding rule (the last one outside it), lengths around
    the 16-row blocks, whole-matrix bands, per-pair bands."""
    rng = np.random.default_rng(abs(sc[1]))
    q, r = _pairs(rng, 500, 0, 70, pad=1)
    for band in (1, 4, 32, 80):
        assert (_rows(device.nw_banded(q, r, AlignConfig(*sc, band)))
                == _nw(oracle, q, r, sc, band)).all(), (sc, band)
    bands = rng.integers(0, 90, 500).astype(np.int32)
    assert (_rows(device.nw_banded(q, r, AlignConfig(*sc, 0), bands=bands))
            == _nw(oracle, q, r, sc, 0, bands=bands)).all(), sc


def test_nw_up_to_and_past_the_16_bit_range(device, oracle):
    """Pairs of up to 7,000 (inside) and 9,000 bases (int32 or literal kernels) at +2/-4."""
    rng = np.random.default_rng(8)
    for hi in (6500, 9000):
        qs, rs = [], []
        for k in range(12):
            t = rng.integers(0, 4, hi - 37 * k).astype(np.uint64)
            qs.append(_mutate(rng, t, 0.02) if k % 2 else (t + 1) & 3)
            rs.append(t)
        q, r = _pack(qs), _pack(rs)
        for band in (16, 60):
            assert (_rows(device.nw_banded(q, r, AlignConfig(*READS, band)))
                    == _nw(oracle, q, r, READS, band)).all(), (hi, band)
