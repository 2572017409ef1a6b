"""Which pairs single precision keeps: scores near the low end of its range, on engines
with and without the FP64 pass, in both gap modes."""
import numpy as np
import pytest

import gpupairhmm_b200 as g
import oracle
from conftest import assert_log10_close
from test_gpu_flat import ladder

pytestmark = pytest.mark.gpu

LENGTHS = [20, 40, 70, 101, 120, 150, 151, 200, 250, 300, 330, 500, 700]


@pytest.mark.parametrize("gcp", [False, True])
@pytest.mark.parametrize("gaps", [40, (30, 45), (60, 93)])
def test_engine_without_fp64_keeps_the_range(gaps, gcp, plain_engine):
    """fp64_rescue off: scores are what single precision gives, and between 1e-72 and 1e-79
    its denormal range sets the error by the scale of the values.  The plain engine's padded
    kernels have the scale the engine's have to have (gcp quality 10 is the default mode's
    eps and beta), so errors against the oracle are alike; a factor of 3 covers other orders
    of rounding.  On exact tiles they were 10 times as large at gap quality 40, and scores of
    reads with gap qualities 60-93 were off by 0.07 or -inf."""
    batch = ladder(2, LENGTHS * 3, gaps, rates=(0.02, 0.5))
    batch.gcp_quals[:] = 10
    want = oracle.batch_log10(batch)
    plain = plain_engine.compute(batch).astype(np.float64)
    with g.Engine(fp64_rescue=False, gcp=gcp) as e:
        got = e.compute(batch).astype(np.float64)
        assert e.stats().rescued <= len(want) // 100   # none but pairs that overflow
    low = (want > -79.0) & (want <= -72.0)
    assert low.sum() >= 30
    assert np.isfinite(got[low]).all()
    rms = lambda x: float(np.sqrt(np.mean((x[low] - want[low]) ** 2)))
    assert rms(got) <= 3.0 * rms(plain), (rms(got), rms(plain))
    kept = want > -72.0
    assert_log10_close(got[kept], want[kept], what=f"gaps {gaps} gcp {gcp}")
