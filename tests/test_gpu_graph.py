"""Batches that repeat are launched as one graph from the ninth on: scores against the same
batches launched kernel by kernel, bitwise, with inputs, lengths and batch sizes that change
from call to call within the classes, and calls of other shapes in between."""
import numpy as np
import pytest

import gpupairhmm_b200 as g
from gpupairhmm_b200 import synth
from gpupairhmm_b200.synth import ACGT, _Builder

pytestmark = pytest.mark.gpu


def _batch(rng, lengths, reads, haps):
    """One record per length; half of the reads unrelated, so that the FP64 pass has work."""
    b = _Builder()
    for L in lengths:
        H = L + rng.integers(20, 120, size=haps)
        base = ACGT[rng.integers(0, 4, size=int(H.max()))]
        seqs = [base[:L] if i % 2 else ACGT[rng.integers(0, 4, size=L)] for i in range(reads)]
        n = reads * L
        b.add_concat(np.full(reads, L), np.concatenate(seqs), rng.integers(20, 42, size=n).astype(np.uint8),
                     np.full(n, 40, np.uint8), np.full(n, 40, np.uint8), H, np.concatenate([base[:h] for h in H]))
    return b.build()


@pytest.mark.parametrize("classes", [[100], [36, 100, 148], [40, 70, 100, 150, 200, 250]])
def test_repeated_batches_as_graphs(classes):
    rng = np.random.default_rng(len(classes))
    other = synth.config0(seed=2, records=3)
    with g.Engine(use_graphs=True) as a, g.Engine(use_graphs=False) as c:
        for call in range(30):
            # lengths move within their class (multiples of 32 positions apart for few pairs)
            lengths = [(L - 1) // 32 * 32 + int(rng.integers(1, 33)) for L in classes]
            b = _batch(rng, lengths, reads=2 + call % 3 * 4, haps=3)
            got, want = a.compute(b), c.compute(b)
            np.testing.assert_array_equal(got, want, err_msg=f"call {call}")
            sa, sc = a.stats(), c.stats()
            assert (sa.rescued, sa.rescued_ext, sa.launches) == (sc.rescued, sc.rescued_ext, sc.launches)
            assert sa.device_ms > 0 and sa.prep_ms > 0 and sa.fp32_ms > 0 and sa.fp64_ms > 0
            if call in (12, 13, 20):   # another shape: launched kernel by kernel, the graph kept
                np.testing.assert_array_equal(a.compute(other), c.compute(other))


def test_repeated_device_batches_as_graphs():
    import torch
    rng = np.random.default_rng(5)
    with g.Engine(use_graphs=True) as a, g.Engine(use_graphs=False) as c:
        for call in range(20):
            b = _batch(rng, [int(rng.integers(97, 129)), int(rng.integers(129, 161))], reads=6 + call, haps=4)
            dev = b.to_device()
            scores = torch.full((b.num_pairs,), 7.0, dtype=torch.float32, device="cuda")
            a.compute_device(dev, scores, stream=torch.cuda.current_stream(), max_read_length=160,
                             max_hap_length=int(b.hap_lengths.max()))
            torch.cuda.synchronize()
            np.testing.assert_array_equal(scores.cpu().numpy(), c.compute(b), err_msg=f"call {call}")
