"""Where a WFA batch starts -- eight, four or one warp per pair, or eight lanes -- changes
with the number of pairs as long as the longest: the same costs on both sides of each line,
for even and ragged lengths, and batches between the lines of few launches."""
import numpy as np
import pytest

from genomics_b200 import SequenceBatch, WFAConfig

pytestmark = pytest.mark.gpu


def _pairs(rng, n, lo, hi):
    qs, rs = [], []
    for i in range(n):
        t = rng.integers(0, 4, hi if i == 0 else int(rng.integers(lo, hi + 1)))
        q = t.copy()
        hit = rng.random(len(q)) < (0.02, 0.1, 1.0)[i % 3]
        q[hit] = rng.integers(0, 4, int(hit.sum()))
        cut = int(rng.integers(0, len(q)))
        qs.append("".join("ACGT"[c] for c in np.delete(q, slice(cut, cut + i % 4))))
        rs.append("".join("ACGT"[c] for c in t))
    return SequenceBatch.from_strings(qs), SequenceBatch.from_strings(rs)


def _copies(b, n):
    """n sequences with words of their own: the batch's over and over."""
    p, m, o, ln = b.arrays()
    times = -(-n // len(ln))
    offs = np.concatenate([o + k * p.size for k in range(times)])
    return SequenceBatch.from_arrays(np.tile(p, times), np.tile(m, times), offs[:n],
                                     np.tile(ln, times)[:n])


@pytest.mark.parametrize("lo,hi", [(150, 150), (1, 512), (300, 700)])
@pytest.mark.parametrize("per_sm", [1.4, 4.0, 100.0])
def test_costs_on_both_sides_of_a_line(device, oracle, lo, hi, per_sm):
    rng = np.random.default_rng(lo + hi)
    q, r = _pairs(rng, 60, lo, hi)
    qp, _, qo, ql = q.arrays()
    rp, _, ro, rl = r.arrays()
    cfg = WFAConfig(4, 6, 2, 900)
    want, _ = oracle.wfa_batch(qp, qo, ql, rp, ro, rl, 4, 6, 2, 900, envelope=True)
    alike = (np.mean(rl) / rl.max()) ** 1.5 if per_sm < 100 else 1.0
    line = int(148 * per_sm / alike)
    for n in (line - 3, line + 3):
        got = device.wfa_affine(_copies(q, n), _copies(r, n), cfg)
        assert (got == np.resize(want, n)).all(), n


def test_lengths_count_no_further_than_max_error_lets_them(device, oracle):
    """1,200 pairs of 100-3,000 bases, few of them long: with a small max_error they are as
    good as alike, and one warp per pair is all that is launched."""
    rng = np.random.default_rng(3)
    qs, rs = [], []
    for i in range(60):
        t = rng.integers(0, 4, int(100 * 30 ** (i / 59)))
        q = t.copy()
        hit = rng.random(len(q)) < 0.1
        q[hit] = rng.integers(0, 4, int(hit.sum()))
        qs.append("".join("ACGT"[c] for c in q))
        rs.append("".join("ACGT"[c] for c in t))
    q, r = SequenceBatch.from_strings(qs), SequenceBatch.from_strings(rs)
    qp, _, qo, ql = q.arrays()
    rp, _, ro, rl = r.arrays()
    want, _ = oracle.wfa_batch(qp, qo, ql, rp, ro, rl, 4, 6, 2, 200, envelope=True)
    seen = set()
    for batched in (True, False):
        dq, dr = device.upload_batch(_copies(q, 1200)), device.upload_batch(_copies(r, 1200))
        try:
            device.stats_reset()
            got = device.wfa_affine(dq, dr, WFAConfig(4, 6, 2, 200), batched=batched)
            assert (got == np.resize(want, 1200)).all()
            seen.add((batched, device.stats()["launches"]))
        finally:
            dq.close()
            dr.close()
    # (three kernels order a batched call's pairs)
    assert seen == {(True, 4), (False, 1)}, seen


@pytest.mark.parametrize("pen", [(1, 0, 31), (31, 0, 31), (1, 1, 30), (2, 1, 30)])
def test_penalties_of_many_slots_keep_the_one_warp_tier(device, oracle, pen):
    """Up to 96 wavefront rows: the one-warp tier's window is 64 diagonals at least, beside
    sequence copies that then hold no more than some 4,000 bases."""
    rng = np.random.default_rng(pen[1])
    q, r = _pairs(rng, 60, 100, 200)
    lq, lr = _pairs(rng, 4, 4300, 4500)
    both = []
    for a, b in ((q, lq), (r, lr)):
        p, m, o, ln = a.arrays()
        p2, m2, o2, ln2 = b.arrays()
        both.append(SequenceBatch.from_arrays(np.concatenate((p, p2)), np.concatenate((m, m2)),
                                              np.concatenate((o, o2 + p.size)),
                                              np.concatenate((ln, ln2))))
    for (a, b), times in (((q, r), 42), (both, 40)):
        qp, _, qo, ql = a.arrays()
        rp, _, ro, rl = b.arrays()
        n = len(ql) * times
        for me in (100, 400, 3000):
            want, _ = oracle.wfa_batch(qp, qo, ql, rp, ro, rl, *pen, me, envelope=True)
            got = device.wfa_affine(_copies(a, n), _copies(b, n), WFAConfig(*pen, me))
            assert (got == np.resize(want, n)).all(), (pen, me)


def test_reads_at_many_slots_start_on_one_warp(device):
    """100 steps leave the one-warp tier's 64 diagonals, not the four-warp one's: two
    launches, where one means that the first was left out."""
    rng = np.random.default_rng(4)
    q, r = _pairs(rng, 60, 150, 150)
    dq, dr = device.upload_batch(_copies(q, 2500)), device.upload_batch(_copies(r, 2500))
    try:
        device.stats_reset()
        device.wfa_affine(dq, dr, WFAConfig(1, 0, 31, 100), batched=False)
        assert device.stats()["launches"] == 2
    finally:
        dq.close()
        dr.close()


def test_a_small_batch_of_reads_starts_on_one_warp_per_pair(device):
    """2,500 reads: one launch, without the eight-lane kernel and its second one."""
    rng = np.random.default_rng(1)
    q, r = _pairs(rng, 60, 150, 150)
    dq, dr = device.upload_batch(_copies(q, 2500)), device.upload_batch(_copies(r, 2500))
    try:
        device.stats_reset()
        device.wfa_affine(dq, dr, WFAConfig(4, 6, 2, 100), batched=False)
        assert device.stats()["launches"] == 1
    finally:
        dq.close()
        dr.close()
