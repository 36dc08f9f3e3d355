"""Smith-Waterman calls whose highest scores leave the lane-split kernel's range for the wide
bands only: which kernels are launched beside it, and that every pair gets its result."""
import numpy as np
import pytest

from genomics_b200 import AlignConfig, SequenceBatch
from genomics_b200._lib import FLAG_INT32

pytestmark = pytest.mark.gpu

# 16-bit values follow scores past 4,094 up to band 64 (96 and more do not fit)
SCORES = (5, -4, -10, -1)


@pytest.fixture(scope="module")
def pairs():
    rng = np.random.default_rng(21)
    qs, rs = [], []
    for i in range(24):
        t = rng.integers(0, 4, 1200 if i % 2 else 300)
        q = t[10:-10].copy()
        hit = rng.random(len(q)) < 0.04
        q[hit] = rng.integers(0, 4, int(hit.sum()))
        qs.append("".join("ACGT"[c] for c in q))
        rs.append("".join("ACGT"[c] for c in t))
    return SequenceBatch.from_strings(qs), SequenceBatch.from_strings(rs)


# three planning kernels, the lane-split kernel's shapes (up to five), and for the bands past
# 64 the int32 kernel of band 128 and the literal one
@pytest.mark.parametrize("top,only,launches", [(64, None, 8), (16, 16, 8), (128, 128, 10),
                                               (600, None, 10)])
def test_launches_beside_the_lane_split_kernel(device, oracle, pairs, top, only, launches):
    q, r = pairs
    rng = np.random.default_rng(top)
    bands = np.full(24, only, np.int32) if only else rng.integers(0, top + 1, 24).astype(np.int32)
    bands[0], bands[1] = top, top
    qp, _, qo, ql = q.arrays()
    rp, _, ro, rl = r.arrays()
    want = np.stack(oracle.sw_batch(qp, qo, ql, rp, ro, rl, *SCORES, 32, bands=bands), 1)
    assert want[:, 0].max() > 4094
    dq, dr = device.upload_batch(q), device.upload_batch(r)
    try:
        for _ in range(2):
            device.stats_reset()
            got = device.sw_banded(dq, dr, AlignConfig(*SCORES, 32), bands=bands)
            assert (got.view(np.int32).reshape(-1, 3) == want).all()
            assert device.stats()["launches"] <= launches, top
    finally:
        dq.close()
        dr.close()


@pytest.mark.parametrize("band", [16, 64, 65, 128, 543, 544, 600])
@pytest.mark.parametrize("scores", [SCORES, (2, -4, -4, -2), (1, -8, -2, -1)])
def test_one_band_of_ragged_pairs(device, oracle, pairs, band, scores):
    """Every pair is taken by some kernel: bands on both sides of the lane-split kernel's
    widest, scores inside and past its range, and a scoring that no packed kernel takes."""
    q, r = pairs
    qp, _, qo, ql = q.arrays()
    rp, _, ro, rl = r.arrays()
    want = np.stack(oracle.sw_batch(qp, qo, ql, rp, ro, rl, *scores, band), 1)
    out = np.full(24 * 3, -77, np.int32).view([("score", "<i4"), ("query_end", "<i4"),
                                               ("ref_end", "<i4")])
    for flags in (0, FLAG_INT32):
        for batched in (True, False):
            dq, dr = device.upload_batch(q), device.upload_batch(r)
            got = device.sw_banded(dq, dr, AlignConfig(*scores, band), batched=batched,
                                   flags=flags, out=out)
            assert (got.view(np.int32).reshape(-1, 3) == want).all(), (band, flags, batched)
            dq.close()
            dr.close()
