"""The work list's order (prep kernels) over the haplotype-length classes a batch can
have: one class, fewer than a scan round, around 1,024-class rounds, at the cap of
4,096 classes and past it.  Every pair must appear exactly once, whatever the order:
a lost or doubled item leaves a score unset, so the scores are compared with the
FP64 oracle (parity tolerance, conftest)."""
import numpy as np
import pytest

import gpupairhmm_b200 as g
import oracle
from conftest import assert_log10_close
from gpupairhmm_b200.synth import ACGT, _Builder

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_hap", [1, 2, 3, 4, 1022, 1023, 1024, 1025, 2047, 2048, 4094, 4095, 4096, 5000])
@pytest.mark.parametrize("mode", ["engine", "plain"])
def test_every_pair_scored_over_haplotype_classes(mode, max_hap, engine, plain_engine):
    rng = np.random.default_rng(max_hap)
    b = _Builder()
    for i in range(5):  # reads of two buckets, haplotype lengths spread over the classes and at both ends
        L = np.array([17, 40, 41][: 1 + i % 3])
        H = np.r_[max_hap, 1, rng.integers(1, max_hap + 1, size=3)]
        n = int(L.sum())
        b.add_concat(L, ACGT[rng.integers(0, 4, size=n)], rng.integers(5, 41, size=n).astype(np.uint8),
                     np.full(n, 40, np.uint8), np.full(n, 40, np.uint8), H, ACGT[rng.integers(0, 4, size=int(H.sum()))])
    batch = b.build()
    want = oracle.batch_log10(batch)
    out = np.full(batch.num_pairs, np.float32(7.0))
    got = (engine if mode == "engine" else plain_engine).compute(batch, out=out)
    ok = want > -60.0 if mode == "plain" else np.ones(len(want), bool)  # the plain form is FP32 only
    assert_log10_close(got[ok], want[ok], what=f"max_hap {max_hap} {mode}")
    assert not np.any(got == np.float32(7.0))
