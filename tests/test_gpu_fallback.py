"""The full FP64 re-scoring of blocks whose candidate list overflows.

Sparse masks leave a few voxels of a block inside both masks, so that many
candidates score nearly alike and the block is re-scored entirely: from a staged
window (up to 21 voxels a side) or from global memory, at several block widths,
gaps and window sizes.  Equal to the FP64 oracle exactly.
"""
import numpy as np
import pytest

import mirorr_b200 as mb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bw,nw,bgap,shape", [
    (4, 7, 1, (16, 18, 26)), (4, 9, 1, (15, 17, 23)), (2, 5, 1, (12, 13, 17)),
    (5, 11, 1, (18, 19, 24)), (8, 3, 1, (17, 18, 20)), (3, 5, 4, (22, 21, 25)),
    (3, 7, 4, (30, 29, 31)), (4, 6, 2, (17, 19, 22))])
@pytest.mark.parametrize("share", [0.03, 0.2])
def test_sparse_masks(ctx, bw, nw, bgap, shape, share):
    rng = np.random.default_rng(bw * 10 + nw)
    base, search = rng.random((2, *shape)).astype(np.float32)
    bm = (rng.random(shape) < share).astype(np.uint8) * 255
    sm = (rng.random(shape) < 0.9).astype(np.uint8)
    search[: shape[0] // 2, :5] = 0.75  # a constant region: equal scores
    m = mb.BlockMatcher(ctx)
    m.SetBlockWidth(bw)
    m.SetBlockGap(bgap)
    m.SetNhoodWidth(nw)
    m.SetNhoodGap(3)
    m.SetBaseImage(base)
    m.SetSearchImage(search)
    m.SetBaseMask(bm)
    m.SetSearchMask(sm)
    prm = O.BMParams(bw, bgap, 3, nw, 1.0)
    ref = O.match_blocks(base, search, bm, sm, prm)
    try:
        m.GetOffsets()
    except mb.MirorrError as e:
        assert e.name == "ENOBLOCKS"
    mi, best, second, status = m.BlockResults()
    overflowed = m.LastDiagnostics()[1]
    m.close()
    if share < 0.1 and bw in (2, 4) and bgap == 1:
        assert overflowed > 0
    s = ref.status == 1
    np.testing.assert_array_equal(best[s], ref.best[s])
    np.testing.assert_array_equal(second[s], ref.second[s])
    np.testing.assert_array_equal(mi[s], ref.match[s])
