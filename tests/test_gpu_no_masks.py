"""A call without masks equals the same call with masks of 255 everywhere.

Without masks the window-AND, the masked searches and most mask reads are left
out; every search form (general, per-x-lane, per-warp, tensor-core, direct) has
to return the same bytes either way, and a mask on one side only is a mask.
"""
import numpy as np
import pytest

import mirorr_b200 as mb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,bw,nw,bgap,keep", [
    ("f32", 4, 5, 1, 1.0), ("f32", 4, 7, 1, 1.0), ("f32", 4, 9, 1, 0.5), ("f32", 5, 11, 1, 1.0),
    ("f32", 3, 5, 1, 1.0), ("f32", 4, 5, 2, 1.0), ("bf16", 4, 7, 1, 1.0), ("f16", 4, 9, 1, 1.0),
    ("f16", 5, 11, 1, 0.3)])
def test_equals_full_masks(ctx, storage, bw, nw, bgap, keep):
    rng = np.random.default_rng(4)
    base, search = rng.random((2, 26, 29, 37)).astype(np.float32)
    base[:8] = 0.5  # flat blocks too
    ones = np.full(base.shape, 255, np.uint8)
    got = []
    for bm, sm in ((None, None), (ones, ones), (ones, None), (None, ones)):
        m = mb.BlockMatcher(ctx)
        m.SetStorage(storage)
        m.SetBlockWidth(bw)
        m.SetBlockGap(bgap)
        m.SetNhoodWidth(nw)
        m.SetNhoodGap(3)
        m.SetBlockKeep(keep)
        m.SetBaseImage(base)
        m.SetSearchImage(search)
        m.SetBaseMask(bm)
        m.SetSearchMask(sm)
        got.append((*m.GetOffsets(), *m.BlockResults()))
        m.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            np.testing.assert_array_equal(a, b)
