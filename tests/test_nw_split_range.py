"""The 16-bit range of the lane-split Needleman-Wunsch kernel: large gap costs, whose
re-centring must not wrap the floor that stands for cells outside the matrix, and positive
mismatch scores, which make cells left of the reference start climb from it.

On the CPU the kernel's arithmetic (nw_split_model.cpp, with the library's own admission
rule) against the oracle; on the GPU the calls themselves.  Whether a case runs on the
lane-split kernel is asked of the rule for every shape, so a call that falls back cannot
pass for one that does not.  Integers: equal or wrong."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT
from genomics_b200 import AlignConfig, SequenceBatch

REGS = (5, 9, 13, 17, 21, 25, 29, 33)


@pytest.fixture(scope="session")
def model(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("model") / "libnwmodel.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", so,
                           "-I" + os.path.join(PKG, "csrc"),
                           os.path.join(ROOT, "tests", "nw_split_model.cpp")])
    lib = ctypes.CDLL(so)
    lib.nw_fits.argtypes = [ctypes.c_int64] * 7 + [ctypes.c_int] * 2
    lib.nw_model.argtypes = [ctypes.c_char_p, ctypes.c_int32, ctypes.c_char_p] + \
        [ctypes.c_int32] * 6 + [ctypes.c_int] * 3
    return lib


def _shapes(band):
    """(registers, log2 lanes) of every shape that holds the band."""
    out = []
    for regs in REGS:
        lg = next((g for g in range(6) if 2 * regs << g >= 2 * band + 1), None)
        if lg is not None:
            out.append((regs, lg))
    return out


def _fits(model, sc, band, qmax, rmax):
    """Per shape, whether the library runs the call on the lane-split kernel."""
    return [bool(model.nw_fits(*sc, band, qmax, rmax, regs, lg)) for regs, lg in _shapes(band)]


def _pairs(rng, qlen, n, band, odd=2):
    """n pairs: queries of qlen bases, references a few bases off, near and unrelated."""
    qs, rs = [], []
    for i in range(n):
        t = rng.integers(0, 4, qlen + 2 * odd)
        q = t[odd:odd + qlen].copy()
        hit = rng.random(qlen) < (0.05, 0.3, 1.0)[i % 3]
        q[hit] = rng.integers(0, 4, int(hit.sum()))
        r = t[int(rng.integers(0, 2 * odd + 1)):]
        qs.append(q.astype(np.uint8))
        rs.append(r[:max(1, qlen - band, len(r) - int(rng.integers(0, odd + 1)))].astype(np.uint8))
    return qs, rs


def _batch(seqs):
    return SequenceBatch.from_strings(["".join("ACGT"[c] for c in s) for s in seqs])


def _want(O, q, r, sc, band, bands=None):
    qp, _, qo, ql = q.arrays()
    rp, _, ro, rl = r.arrays()
    return np.asarray(O.nw_batch(qp, qo, ql, rp, ro, rl, *sc, band, bands=bands))


def _model_scores(model, qs, rs, sc, band, regs, lg, wrapping=0):
    return [model.nw_model(q.tobytes(), len(q), r.tobytes(), len(r), *sc, band, regs, lg, wrapping)
            for q, r in zip(qs, rs)]


# match, mismatch, gap open, gap extend: g = -(open + extend) on both sides of 55, up to which
# the floor of -31000 less 32g fits 16 bits; and mismatches above 0
GAPS = [(2, -4, -50, -4), (2, -4, -50, -5), (2, -4, -54, -2), (5, -4, -60, -1), (2, -4, -60, -10),
        (20, -60, -50, -20), (10, -40, -40, -16), (10, -20, -100, -10), (1, 0, -150, 0)]
GAINS = [(5, 2, -4, -2), (20, 10, -4, -2), (70, 60, -2, -1), (150, 120, -2, -1), (255, 255, 0, 0),
         (60, 30, -58, -2)]


@pytest.mark.parametrize("sc", GAPS + GAINS)
def test_model_is_exact_where_the_rule_admits(model, oracle, sc):
    rng = np.random.default_rng(abs(sc[1]) + abs(sc[2]))
    admitted = 0
    for band in (0, 1, 4, 16, 32, 64, 131, 400):
        for qlen in (1, 15, 16, 17, 33, 70, 150):
            qs, rs = _pairs(rng, qlen, 9, band, odd=min(2, band))
            fits = _fits(model, sc, band, qlen, max(len(r) for r in rs))
            if not any(fits):
                continue
            want = _want(oracle, _batch(qs), _batch(rs), sc, band).tolist()
            for ok, (regs, lg) in zip(fits, _shapes(band)):
                if ok and (band < 131 or regs % 8 == 1):
                    admitted += 1
                    got = _model_scores(model, qs, rs, sc, band, regs, lg)
                    assert got == want, (sc, band, qlen, regs, lg)
    assert admitted >= 20, (sc, admitted)


def test_model_of_short_references(model, oracle):
    """Queries much longer than their references inside a wide band: the most rows of cells
    left of the reference start, with gains for mismatches."""
    rng = np.random.default_rng(5)
    seen = {True: 0, False: 0}
    for band in (100, 250, 400, 543):
        for sc in GAINS + [(2, -4, -4, -2), (2, -4, -4, -60)]:
            qs = [rng.integers(0, 4, 100 + int(rng.integers(0, band))).astype(np.uint8)
                  for _ in range(4)]
            rs = [rng.integers(0, 4, 100).astype(np.uint8) for _ in range(4)]
            want = _want(oracle, _batch(qs), _batch(rs), sc, band).tolist()
            fits = _fits(model, sc, band, max(map(len, qs)), 100)
            for ok, (regs, lg) in zip(fits, _shapes(band)):
                seen[ok] += 1
                if ok:
                    assert _model_scores(model, qs, rs, sc, band, regs, lg) == want
    assert min(seen.values()) >= 10, seen


def test_a_floor_that_wraps_is_seen(model, oracle):
    """The model finds both faults: a floor that wraps at g = 56, and a climb that the rule
    refuses."""
    rng = np.random.default_rng(1)
    qs, rs = _pairs(rng, 40, 9, 4)
    sc = (2, -4, -54, -2)
    want = _want(oracle, _batch(qs), _batch(rs), sc, 4).tolist()
    assert _model_scores(model, qs, rs, sc, 4, 5, 0) == want
    assert _model_scores(model, qs, rs, sc, 4, 5, 0, wrapping=1) != want
    sc = (150, 120, -2, -1)
    qs = [rng.integers(0, 4, 420).astype(np.uint8)]
    rs = [rng.integers(0, 4, 100).astype(np.uint8)]
    want = _want(oracle, _batch(qs), _batch(rs), sc, 400).tolist()
    assert not any(_fits(model, sc, 400, 420, 100))
    assert _model_scores(model, qs, rs, sc, 400, 13, 5) != want


def _gpu_check(device, oracle, qs, rs, sc, band):
    q, r = _batch(qs), _batch(rs)
    want = _want(oracle, q, r, sc, band)
    got = device.nw_banded(q, r, AlignConfig(*sc, band))["score"]
    assert (got == want).all(), (sc, band, np.nonzero(got != want)[0][:5])
    bands = np.full(q.count, band, np.int32)
    bands[::3] = band // 2
    want = _want(oracle, q, r, sc, 0, bands)
    got = device.nw_banded(q, r, AlignConfig(*sc, 0), bands=bands)["score"]
    assert (got == want).all(), (sc, "per pair up to", band)


# calls that run on the lane-split kernel, whichever shape the batch takes
ADMITTED = [(sc, band, qlen) for sc in ((2, -4, -50, -5), (2, -4, -54, -2), (2, -4, -60, -10))
            for band in (4, 16, 32, 64) for qlen in (16, 17, 33, 150)
            if (sc[2], band) != (-60, 64)] + [
    ((2, -4, -20, -5), 131, 33), ((10, -40, -40, -16), 16, 60), ((5, -4, -60, -1), 32, 150),
    ((10, -20, -100, -10), 4, 60)]
ADMITTED_GAINS = [((20, 10, -4, -2), 64, 150), ((20, 10, -4, -2), 400, 33),
                  ((5, 2, -4, -2), 400, 150), ((60, 30, -58, -2), 16, 60)]


def test_the_cases_of_the_lane_split_kernel_are_its_own(model):
    for sc, band, qlen in ADMITTED + ADMITTED_GAINS:
        assert all(_fits(model, sc, band, qlen, qlen + 4)), (sc, band, qlen)


@pytest.mark.gpu
@pytest.mark.parametrize("sc,band,qlen", ADMITTED + ADMITTED_GAINS)
def test_gpu_cases_of_the_lane_split_kernel(device, oracle, model, sc, band, qlen):
    """Few pairs and many (the shapes with the most lanes, and with the most columns)."""
    rng = np.random.default_rng(band + qlen)
    qs, rs = _pairs(rng, qlen, 60, band)
    assert all(_fits(model, sc, band, qlen, max(len(r) for r in rs)))
    for times in (1, 100):
        _gpu_check(device, oracle, qs * times, rs * times, sc, band)


@pytest.mark.gpu
@pytest.mark.parametrize("band,qlen", [(1, 17), (4, 33), (16, 33), (32, 150), (64, 33)])
def test_gpu_largest_gap_costs(device, oracle, model, band, qlen):
    """The largest gap cost that every shape admits, that any does, and the one after it
    (which falls back), at +2/-4."""
    rng = np.random.default_rng(band)
    qs, rs = _pairs(rng, qlen, 60, band, odd=min(2, band))
    rmax = max(len(r) for r in rs)
    fits = {g: _fits(model, (2, -4, -(g - 2), -2), band, qlen, rmax) for g in range(3, 256)}
    every = max(g for g in fits if all(fits[g]))
    some = max(g for g in fits if any(fits[g]))
    assert every > 55 or band >= 64, (every, some)
    for g in sorted({every, every + 1, some, some + 1}):
        _gpu_check(device, oracle, qs * 40, rs * 40, (2, -4, -(g - 2), -2), band)


@pytest.mark.gpu
def test_gpu_positive_mismatch_in_a_wide_band(device, oracle, model):
    """Queries longer than their references by most of the band: refused by the rule where
    cells left of the reference start could pass real ones, exact either way."""
    rng = np.random.default_rng(9)
    qs = [rng.integers(0, 4, 420 - i).astype(np.uint8) for i in range(40)]
    rs = [rng.integers(0, 4, 100).astype(np.uint8) for _ in range(40)]
    for sc, admitted in (((150, 120, -2, -1), False), ((5, 2, -4, -2), True)):
        assert all(f == admitted for f in _fits(model, sc, 400, 420, 100)), sc
        _gpu_check(device, oracle, qs, rs, sc, 400)
