"""Host calls around the size up to which inputs and index go up in one gathered copy
(384 KB: about 27 of these records), from pageable and page-locked arrays, with the
records' bytes starting at an odd offset of the arrays: bitwise the scores of one
large call."""
import numpy as np
import pytest

import gpupairhmm_b200 as g
from gpupairhmm_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gcp", [False, True])
@pytest.mark.parametrize("records", [1, 2, 24, 26, 27, 28, 30, 60])
def test_gathered_and_staged_uploads_agree(records, gcp):
    b = synth.config0(seed=9, records=64)
    # one byte in front of everything: absolute offsets are odd
    for name in ("read_bases", "base_quals", "ins_quals", "del_quals", "gcp_quals", "hap_bases"):
        setattr(b, name, np.r_[np.uint8(30), getattr(b, name)])
    b.read_offsets, b.hap_offsets = b.read_offsets + 1, b.hap_offsets + 1
    with g.Engine(gcp=gcp) as e:
        want = e.compute(b)
        part = b.select_records(3, 3 + records)
        got = e.compute(part)
        pinned = e.compute(part.pin())
    np.testing.assert_array_equal(got, want[3 * 128:(3 + records) * 128])
    np.testing.assert_array_equal(pinned, got)
