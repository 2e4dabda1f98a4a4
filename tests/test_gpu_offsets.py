"""Images whose mean is thousands of times their contrast, against the oracle.

The FP32 cross term is summed about a constant of the block, so a common offset
leaves no cancellation in it, in every search form.  Best, second and argmax equal
the FP64 oracle's exactly.
"""
import numpy as np
import pytest

import mirorr_b200 as mb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [1000.0, 4000.0, 20000.0])
@pytest.mark.parametrize("bw,nw,bgap,gap", [
    (4, 5, 1, 2), (4, 5, 1, 1), (4, 7, 1, 2), (4, 9, 1, 2), (4, 7, 1, 20), (5, 11, 1, 3),
    (3, 5, 1, 2), (3, 5, 2, 2), (2, 5, 1, 2), (8, 5, 1, 3)])
def test_common_offset(ctx, bw, nw, bgap, gap, offset):
    rng = np.random.default_rng(7)
    base, search = (rng.random((2, 24, 30, 41)).astype(np.float32) + np.float32(offset))
    m = mb.BlockMatcher(ctx)
    m.SetBlockWidth(bw)
    m.SetBlockGap(bgap)
    m.SetNhoodWidth(nw)
    m.SetNhoodGap(gap)
    m.SetBaseImage(base)
    m.SetSearchImage(search)
    ref = O.match_blocks(base, search, None, None, O.BMParams(bw, bgap, gap, nw, 1.0))
    m.GetOffsets()
    mi, best, second, _ = m.BlockResults()
    m.close()
    np.testing.assert_array_equal(best, ref.best)
    np.testing.assert_array_equal(second, ref.second)
    np.testing.assert_array_equal(mi, ref.match)
