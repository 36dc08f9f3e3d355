"""The tiered WFA kernels where their storage and bookkeeping have edges, against the
oracle: sequence copies at a tier's capacity, windows that fill up and move on with and
without pruning, targets far off diagonal 0 on either side, penalty lattices with steps
that have no source.  Each batch runs small (eight warps per pair first), and repeated so
that the one-warp and four-warp tiers come first.  Integers: equal or wrong."""
import numpy as np
import pytest

from genomics_b200 import SequenceBatch, WFAConfig
from genomics_b200._lib import FLAG_NO_PRUNE

pytestmark = pytest.mark.gpu


def _pack(seqs):
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


def _rnd(rng, n):
    return rng.integers(0, 4, n).astype(np.uint64)


def _copies(b, times):
    """The sequences `times` over, each with words of its own (the batch's words then show
    its mean length)."""
    p, m, o, l = b.arrays()
    offs = np.concatenate([o + k * p.size for k in range(times)])
    return SequenceBatch.from_arrays(np.tile(p, times), np.tile(m, times), offs, np.tile(l, times))


def _check(device, oracle, q, r, cfg, copies, flags=(0,)):
    qp, _, qo, ql = q.arrays()
    rp, _, ro, rl = r.arrays()
    want, _ = oracle.wfa_batch(qp, qo, ql, rp, ro, rl, cfg.x, cfg.o, cfg.e, cfg.max_error,
                               envelope=True)
    for times in copies:
        qq, rr = _copies(q, times), _copies(r, times)
        for fl in flags:
            for batched in (True, False):
                got = device.wfa_affine(qq, rr, cfg, batched=batched, flags=fl)
                bad = np.nonzero((got.reshape(times, -1) != want).any(0))[0]
                assert bad.size == 0, (cfg, times, fl, batched, bad[:5], ql[bad[:5]], rl[bad[:5]])
    return want


@pytest.mark.parametrize("cap", [6144, 12288, 16384, 32768])
def test_lengths_at_the_copies_capacity(device, oracle, cap):
    rng = np.random.default_rng(cap)
    qs, rs = [], []
    for d in (-33, -32, -1, 0, 1, 31, 32, 33):
        t = _rnd(rng, cap + d)
        q = _mutate(rng, t, 0.004)
        qs += [q, t]
        rs += [t, q]
    q, r = _pack(qs), _pack(rs)
    _check(device, oracle, q, r, WFAConfig(4, 6, 2, 2000), (1, 40, 70) if cap < 20000 else (1, 30))


@pytest.mark.parametrize("pen", [(4, 6, 2), (3, 5, 2), (7, 1, 3), (1, 30, 1), (5, 0, 5), (9, 4, 6),
                                 (2, 28, 3), (31, 0, 1), (1, 0, 1)])
def test_penalty_lattices(device, oracle, pen):
    """Steps that have no source, es > 1, many slots (narrow windows); length differences
    of both signs; the pruning bound on (a sequence of over 1,024 bases) and off."""
    rng = np.random.default_rng(sum(pen))
    qs, rs = [_rnd(rng, 1100)], []
    rs.append(_mutate(rng, qs[0], 0.05))
    for k in range(60):
        t = _rnd(rng, int(rng.integers(1, 500)))
        q = _mutate(rng, t, float(rng.choice([0.01, 0.05, 0.2])))
        if k % 3 == 1:
            q = q[len(q) // 3:]
        elif k % 3 == 2:
            t = t[:2 * len(t) // 3 + 1]
        if k % 10 == 9:
            q = _rnd(rng, len(q) + 1)
        qs.append(q)
        rs.append(t)
    q, r = _pack(qs), _pack(rs)
    cover = 2 * max(pen[0] * 1200, pen[1] + pen[2] * 1200)
    for me in (cover, 90):
        _check(device, oracle, q, r, WFAConfig(*pen, me), (1, 8, 60), flags=(0, FLAG_NO_PRUNE))


def test_targets_far_off_the_main_diagonal(device, oracle):
    """Long pairs whose lengths differ by hundreds to thousands, either way: the bound
    closes on a target far from diagonal 0 while the other side still grows."""
    rng = np.random.default_rng(5)
    qs, rs = [], []
    for d in (0, 1, 57, 300, 700, 1500, 2600):
        t = _rnd(rng, 2800)
        for rate in (0.02, 0.15):
            q = _mutate(rng, t, rate)
            qs += [q[d:], t, np.concatenate((q[:900], q[900 + min(d, 1800):]))]
            rs += [t, q[d:], t]
    q, r = _pack(qs), _pack(rs)
    want = _check(device, oracle, q, r, WFAConfig(4, 6, 2, 12000), (1, 12, 40),
                  flags=(0, FLAG_NO_PRUNE))
    assert want.max() > 4000
    _check(device, oracle, q, r, WFAConfig(2, 3, 1, 2500), (1, 40))


def test_empty_and_tiny_pairs(device, oracle):
    rng = np.random.default_rng(6)
    qs = [_rnd(rng, n) for n in (0, 0, 1, 1, 2, 31, 32, 33, 64, 5, 200, 0)]
    rs = [_rnd(rng, n) for n in (0, 1, 0, 1, 3, 32, 31, 33, 64, 200, 5, 200)]
    q, r = _pack(qs), _pack(rs)
    for me in (0, 3, 8, 400, 1200):
        _check(device, oracle, q, r, WFAConfig(4, 6, 2, me), (1, 30, 400))


@pytest.mark.parametrize("pen", [(4, 6, 2), (3, 5, 2), (7, 1, 3), (5, 0, 5), (1, 0, 1), (9, 4, 6),
                                 (10, 20, 9), (2, 28, 3)])
def test_short_pairs(device, oracle, pen):
    """Batches of at most 512 bases: eight lanes per pair.  Reads, unrelated pairs whose
    intervals outgrow the window (the one-warp tier starts them over), one-sided length
    differences, and the longest that qualify beside one base more (which do not)."""
    rng = np.random.default_rng(pen[0] * 100 + pen[2])
    qs, rs = [], []
    for k in range(150):
        t = _rnd(rng, int(rng.integers(0, 160)) if k % 5 else int(rng.integers(300, 513)))
        q = _mutate(rng, t, float(rng.choice([0.0, 0.02, 0.06, 0.3])))[:512]
        if k % 7 == 3:
            q = _rnd(rng, len(t))
        elif k % 7 == 5:
            q = q[len(q) // 2:]
        elif k % 7 == 6:
            t = t[:len(t) // 3]
        qs.append(q)
        rs.append(t)
    q, r = _pack(qs), _pack(rs)
    for me in (2 * max(pen[0] * 512, pen[1] + 512 * pen[2]), 200, 17, 0):
        _check(device, oracle, q, r, WFAConfig(*pen, me), (100,))
    q, r = _pack(qs + [_rnd(rng, 513)]), _pack(rs + [_rnd(rng, 500)])
    _check(device, oracle, q, r, WFAConfig(*pen, 300), (100,))


@pytest.mark.parametrize("pen", [(4, 6, 2), (3, 5, 2), (7, 1, 3), (5, 0, 5), (1, 0, 1), (9, 4, 6)])
def test_cigars_of_the_pruned_history(device, oracle, pen):
    """The CIGAR pass visits only diagonals that can finish within the known cost, in a
    record sized from the cost: the strings, ties included, are the reference's, over
    repeats (many equal alignments), one-sided length differences, unrelated pairs and
    costs many times the lengths."""
    rng = np.random.default_rng(pen[0] + 10 * pen[2])
    unit = _rnd(rng, 7)
    qs, rs = [], []
    for k in range(60):
        t = _rnd(rng, int(rng.integers(0, 90)))
        if k % 4 == 1:
            t = np.tile(unit, int(rng.integers(1, 13)))
        q = _mutate(rng, t, float(rng.choice([0.02, 0.1, 0.3])))
        if k % 6 == 2:
            q = q[len(q) // 2:]
        elif k % 6 == 3:
            t = t[:len(t) // 3]
        elif k % 6 == 4:
            q = _rnd(rng, int(rng.integers(0, 60)))
        qs.append(q)
        rs.append(t)
    letters = ["".join("ACGT"[c] for c in s) for s in qs], ["".join("ACGT"[c] for c in s) for s in rs]
    q, r = _pack(qs), _pack(rs)
    for me in (900, 60):
        expect = [oracle.wfa_cigar(a, b, *pen, me) for a, b in zip(*letters)]
        for copies in (1, 40):
            cost, cig = device.wfa_cigar(_copies(q, copies), _copies(r, copies),
                                         WFAConfig(*pen, me))
            for i, want in enumerate(expect):
                for j in (i, i + (copies - 1) * len(qs)):
                    assert (int(cost[j]), cig[j]) == want, (pen, me, letters[0][i], letters[1][i])
