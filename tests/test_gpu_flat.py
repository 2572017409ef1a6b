"""The allocation-free flat list (noalloc.cu) where its two forms meet: pairs near the low
end of the single-precision range, which the exact tiles leave to the general form."""
import numpy as np
import pytest

import gpupairhmm_b200 as g
import oracle
from gpupairhmm_b200.synth import ACGT, _Builder

pytestmark = pytest.mark.gpu


def ladder(seed, lengths, gaps, rates=(0.02, 0.4), reads=16, haps=4):
    """One record per length: reads cut from the haplotypes' common start with substitution
    rates spread over `rates`, so that scores fall from near zero to below the FP32 range.
    gaps: one gap quality, or (lo, hi) drawn per position."""
    rng = np.random.default_rng(seed)
    b = _Builder()
    for L in lengths:
        H = L + rng.integers(20, 200, size=haps)
        base = ACGT[rng.integers(0, 4, size=int(H.max()))]
        rs = []
        for rate in np.linspace(*rates, reads):
            r = base[:L].copy()
            m = rng.random(L) < rate
            r[m] = ACGT[rng.integers(0, 4, size=int(m.sum()))]
            rs.append(r)
        n = reads * L
        q = [np.full(n, gaps) if np.isscalar(gaps) else rng.integers(gaps[0], gaps[1] + 1, size=n) for _ in range(2)]
        b.add_concat(np.full(reads, L), np.concatenate(rs), rng.integers(30, 42, size=n).astype(np.uint8),
                     q[0].astype(np.uint8), q[1].astype(np.uint8), H, np.concatenate([base[:h] for h in H]))
    return b.build()


def pair_list(batch):
    """(read, haplotype) pairs in the engine's score order."""
    pairs, r0, h0 = [], 0, 0
    for nr, nh in zip(batch.reads_per_record, batch.haps_per_record):
        pairs += [(batch.read_offsets[i], batch.hap_offsets[j], batch.read_lengths[i], batch.hap_lengths[j])
                  for i in range(r0, r0 + nr) for j in range(h0, h0 + nh)]
        r0, h0 = r0 + nr, h0 + nh
    return np.array(pairs, dtype=g.PAIR_DTYPE)


def flat_call(batch):
    """A function scoring a pair list over the batch's arrays."""
    import torch
    dev = torch.device("cuda:0")
    d = [torch.from_numpy(np.ascontiguousarray(getattr(batch, k))).to(dev)
         for k in ("read_bases", "base_quals", "ins_quals", "del_quals", "hap_bases")]

    def call(pairs, stream=None):
        dpairs = torch.from_numpy(np.ascontiguousarray(pairs).view(np.uint8)).to(dev)
        scores = torch.full((len(pairs),), 7.0, dtype=torch.float32, device=dev)
        g.forward_pairs_noalloc(0, *d, dpairs, len(pairs), int(batch.hap_lengths.max()), scores, stream)
        torch.cuda.synchronize(dev)
        return scores.cpu().numpy()

    return call


@pytest.mark.parametrize("gaps", [40, (30, 45), 48])
def test_low_end_of_the_range_is_kept(gaps, plain_engine):
    """Between 1e-74 and 1e-80 a score loses digits in the denormal range, and how many is
    set by the scale of the values.  The general form has the scale of the padded kernels
    that the plain engine runs (boundary value FLT_MAX/16 over the haplotype's length), so
    its errors against the oracle are alike; a factor of 3 covers the different order of
    roundings.  With every pair on the tiles, whose values lie up to 1/delta lower, errors
    were 10 times as large."""
    batch = ladder(1, [40, 70, 101, 120, 150, 151, 200, 250, 300, 330, 700] * 3, gaps)
    want = oracle.batch_log10(batch)
    plain = plain_engine.compute(batch).astype(np.float64)
    got = flat_call(batch)(pair_list(batch)).astype(np.float64)
    low = (want > -80.0) & (want <= -74.0)
    assert low.sum() >= 30
    assert np.isfinite(got[low]).all()
    rms = lambda x: float(np.sqrt(np.mean((x[low] - want[low]) ** 2)))
    assert rms(got) <= 3.0 * rms(plain), (rms(got), rms(plain))


def test_score_does_not_depend_on_the_list():
    """Pairs of the same shapes with ordinary and with very high gap qualities, scores from
    near zero to below the range: in list order, many times over and shuffled (a warp then
    takes several pairs at a time and mixes the two), and in short lists (one pair a warp
    at a time), bitwise the same pair by pair."""
    lengths = [30, 101, 103, 150, 152, 200, 250, 330, 650, 700]
    from gpupairhmm_b200 import synth
    batch = synth.concat([ladder(5, lengths, 40, haps=3), ladder(6, lengths, (80, 127), haps=3),
                          ladder(7, lengths, (30, 93), haps=3)])
    pairs = pair_list(batch)
    call = flat_call(batch)
    want = call(pairs)
    assert np.isfinite(want).mean() > 0.3 and (want == -np.inf).any()
    rng = np.random.default_rng(9)
    many = np.tile(np.arange(len(pairs)), 50)   # 72,000 pairs: 8 at a time
    for order in (many, rng.permutation(many), rng.permutation(many)):
        np.testing.assert_array_equal(call(pairs[order]), want[order])
    for part in np.array_split(rng.permutation(len(pairs))[:600], 40):
        np.testing.assert_array_equal(call(pairs[part]), want[part])


def test_calls_of_different_sizes_follow_one_another():
    """Every call starts from its own empty queue: lists from one pair to some 70,000, one
    after another on one stream, each scored whole; and a call captured in a graph, whose
    replays come between other calls."""
    import torch
    batch = ladder(3, [9, 40, 100, 151, 250, 700], (30, 45), reads=8, haps=3)
    pairs = pair_list(batch)
    call = flat_call(batch)
    want = call(pairs)
    assert not np.any(want == np.float32(7.0))
    rng = np.random.default_rng(4)
    dev = torch.device("cuda:0")
    d = [torch.from_numpy(np.ascontiguousarray(getattr(batch, k))).to(dev)
         for k in ("read_bases", "base_quals", "ins_quals", "del_quals", "hap_bases")]
    order = rng.integers(0, len(pairs), size=5000)
    dpairs = torch.from_numpy(pairs[order].view(np.uint8)).to(dev)
    scores = torch.empty(len(order), dtype=torch.float32, device=dev)
    side = torch.cuda.Stream(dev)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        g.forward_pairs_noalloc(0, *d, dpairs, len(order), int(batch.hap_lengths.max()), scores, side)
    for n in (70000, 1, 3, 20000, 64, 2, 40000, 500):
        pick = rng.integers(0, len(pairs), size=n)
        np.testing.assert_array_equal(call(pairs[pick]), want[pick])
        scores.fill_(7.0)
        torch.cuda.synchronize(dev)
        graph.replay()
        torch.cuda.synchronize(dev)
        np.testing.assert_array_equal(scores.cpu().numpy(), want[order])
