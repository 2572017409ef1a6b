"""Which pairs single precision keeps: scores near the low end of its range, on engines
with and without the FP64 pass, in both gap modes."""
import numpy as np
import pytest

import gpupairhmm_b200 as g
import oracle
from conftest import assert_log10_close
from test_gpu_flat import ladder

pytestmark = pytest.mark.gpu


def pair_lengths(batch):
    """Read and haplotype length of every score."""
    R, H = batch.reads_per_record, batch.haps_per_record
    first = np.cumsum(H) - H
    return (np.repeat(batch.read_lengths, np.repeat(H, R)).astype(np.float64),
            np.concatenate([np.tile(batch.hap_lengths[f:f + n], r) for f, n, r in zip(first, H, R)]).astype(np.float64))


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


@pytest.mark.parametrize("quality", [1, 2, 4])
def test_gcp_threshold_counts_the_reads_own_beta(quality):
    """Single precision keeps a pair down to 3*L*H*2^-127 of a sum that carries the read's
    beta = 1 - p(gcp) (FLT_MAX/16 = 2^124 the boundary's scale): every pair below that is
    recomputed in double, also where low gcp qualities make beta small."""
    # lengths at which unrelated reads score about there
    lengths = {1: range(640, 800, 8), 2: range(300, 380, 4), 4: range(150, 230, 4)}[quality]
    batch = ladder(3, lengths, 20, rates=(0.1, 0.75))
    batch.gcp_quals[:] = quality
    want = oracle.batch_log10(batch, gcp=True)
    L, H = pair_lengths(batch)
    beta = 1.0 - 10.0 ** (-quality / 10.0)
    below = want < np.log10(3.0 * L * H / beta) - (127 + 124) * np.log10(2.0) - 1e-3
    default = want < np.log10(3.0 * L * H / 0.9) - (127 + 124) * np.log10(2.0) - 1e-3
    assert below.sum() > default.sum()
    with g.Engine(gcp=True) as e:
        got = e.compute(batch)
        assert e.stats().rescued >= below.sum()
    assert_log10_close(got, want)


@pytest.mark.parametrize("few", [True, False])
def test_long_reads_are_counted_beyond_the_same_length(few):
    """LONG_READ is where the engine's tables begin to count pairs as multi-tile, on the table
    for few pairs and on the one for many."""
    batch = ladder(4, [640, 641, g.LONG_READ - 1, g.LONG_READ, g.LONG_READ + 1, 1500], 40,
                   rates=(0.0, 0.02), reads=4 if few else 1200, haps=1 if few else 2)
    L, _ = pair_lengths(batch)
    with g.Engine() as e:
        e.compute(batch)
        assert e.stats().multi_tile_pairs == (L > g.LONG_READ).sum()
