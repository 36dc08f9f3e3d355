"""One pair of chromosome-sized sequences: the tier whose rings lie in global memory takes a
region per pair it can hold at once, not one per SM."""
import numpy as np
import pytest

from genomics_b200 import SequenceBatch, WFAConfig

pytestmark = pytest.mark.gpu

N = 20_000_000
AT = (11, 9_000_000, N - 5)  # single substitutions


@pytest.fixture(scope="module")
def pair():
    rng = np.random.default_rng(2)
    t = rng.integers(0, 4, N).astype(np.uint64)
    q = t.copy()
    q[list(AT)] = (q[list(AT)] + 1) & 3
    shift = (62 - 2 * np.arange(32)).astype(np.uint64)
    out = []
    for s in (q, t):
        packed = np.bitwise_or.reduce(s.reshape(-1, 32) << shift, axis=1)
        out.append(SequenceBatch.from_arrays(packed, np.zeros_like(packed),
                                             np.zeros(1, np.int64), np.array([N], np.int64)))
    return out


def test_cost_and_cigar(device, pair):
    q, r = pair
    cfg = WFAConfig(4, 6, 2, 40)
    cost, cigars = device.wfa_cigar(q, r, cfg)
    runs, at = "", 0
    for k in AT:
        runs += f"{k - at}=1X"
        at = k + 1
    assert cost.tolist() == [12] and cigars == [runs + f"{N - at}="]
    assert device.wfa_affine(q, r, cfg).tolist() == [12]
    assert device.wfa_affine(q, r, WFAConfig(4, 6, 2, 11)).tolist() == [-1]
