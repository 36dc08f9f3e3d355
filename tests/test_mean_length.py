"""Kernels are chosen by the mean length of a call's pairs.  It must not depend on how the
batch lays its words out (sequences that share words, gaps), on how many of the batch's
pairs the call takes, or on the parts a large call runs in."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG
from genomics_b200 import SequenceBatch, WFAConfig

SHIM = """
#include "seq_view.cuh"
extern "C" double mean_of_part(int64_t words, int64_t bases, int64_t count, int64_t n, int64_t p0,
                               int64_t m, int64_t longest)
{
    const gb2::SeqView v{nullptr, nullptr, nullptr, 0, words, gb2::bases_share(bases, n, count)};
    return gb2::mean_length(gb2::part_of(v, p0, m, n), m, longest);
}
"""


def test_mean_of_a_part(tmp_path):
    src, so = str(tmp_path / "shim.cpp"), str(tmp_path / "shim.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-o", so,
                           "-I" + os.path.join(PKG, "csrc"), src])
    mean = ctypes.CDLL(so).mean_of_part
    mean.restype = ctypes.c_double
    mean.argtypes = [ctypes.c_int64] * 7
    # 400,000 pairs of 1,050 bases on average, 2,000 at most, in four parts
    bases = 400_000 * 1050
    for words in (400_000 * 34, 10, 400_000 * 300):  # own words, shared ones, gaps
        for n in (400_000, 300_000):
            per = (n + 3) // 4
            for k in range(4):
                m = min(per, n - k * per)
                got = mean(words, bases, 400_000, n, k * per, m, 2000)
                assert got == pytest.approx(1050, rel=1e-4)
    assert mean(1, 0, 5, 5, 0, 5, 0) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("batched", [True, False])
def test_wfa_of_shared_words_runs_like_its_copy(device, batched):
    """All against all of 60 sequences: the same launches and costs whether the 3,600 pairs
    share the sequences' words or have their own; and for the half of them."""
    rng = np.random.default_rng(0)
    seqs = ["".join("ACGT"[c] for c in rng.integers(0, 4, int(rng.integers(500, 900))))
            for _ in range(60)]
    i, j = np.divmod(np.arange(3600), 60)
    p, m, o, ln = SequenceBatch.from_strings(seqs).arrays()
    own = [SequenceBatch.from_strings([seqs[k] for k in idx]) for idx in (i, j)]
    shared = [SequenceBatch.from_arrays(p, m, o[idx], ln[idx]) for idx in (i, j)]
    cfg = WFAConfig(4, 6, 2, 3000)
    seen = {}
    for name, (qh, rh) in (("own", own), ("shared", shared)):
        q, r = device.upload_batch(qh), device.upload_batch(rh)
        try:
            for n in (3600, 1800):
                device.stats_reset()
                cost = device.wfa_affine(q, r, cfg, n_pairs=n, batched=batched)
                seen[name, n] = device.stats()["launches"], cost.tolist()
        finally:
            q.close()
            r.close()
    for n in (3600, 1800):
        assert seen["own", n][1] == seen["shared", n][1]
        assert seen["own", n][0] == seen["shared", n][0], n
