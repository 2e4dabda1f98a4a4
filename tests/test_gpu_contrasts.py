"""Search images of low contrast beside large values, and large common offsets.

The FP32 cross term is summed about a constant (the mean of the block's own
candidate; zero in the general search), and its roundings grow with a candidate's
distance from it over its contrast.  The refinement list allows for that, so best,
second and argmax equal the FP64 oracle's exactly in every search form; images of
ordinary contrast are not sent to the FP64 fallback by it.
"""
import numpy as np
import pytest

import mirorr_b200 as mb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPE = (24, 30, 41)
FORMS = [(4, 5, 1, 2), (4, 5, 1, 1), (4, 7, 1, 2), (4, 9, 1, 2), (4, 7, 1, 20), (5, 11, 1, 3),
         (3, 5, 1, 2), (3, 5, 2, 2), (2, 5, 1, 2), (8, 5, 1, 3)]


def _check(ctx, form, base, search, bm=None, sm=None):
    bw, nw, bgap, gap = form
    m = mb.BlockMatcher(ctx)
    m.SetBlockWidth(bw)
    m.SetBlockGap(bgap)
    m.SetNhoodWidth(nw)
    m.SetNhoodGap(gap)
    m.SetBaseImage(base)
    m.SetSearchImage(search)
    m.SetBaseMask(bm)
    m.SetSearchMask(sm)
    ref = O.match_blocks(base, search, bm, sm, O.BMParams(bw, bgap, gap, nw, 1.0))
    try:
        m.GetOffsets()
    except mb.MirorrError as e:
        assert e.name == "ENOBLOCKS"
    mi, best, second, _ = m.BlockResults()
    overflowed = m.LastDiagnostics()[1]
    m.close()
    np.testing.assert_array_equal(best, ref.best)
    np.testing.assert_array_equal(second, ref.second)
    np.testing.assert_array_equal(mi, ref.match)
    return overflowed


@pytest.mark.parametrize("offset", [0.0, 1000.0, 4000.0, 20000.0])
@pytest.mark.parametrize("form", FORMS)
def test_common_offset(ctx, form, offset):
    rng = np.random.default_rng(7)
    base, search = rng.random((2, *SHAPE)).astype(np.float32) + np.float32(offset)
    overflowed = _check(ctx, form, base, search)
    if offset == 0.0:
        assert overflowed == 0


@pytest.mark.parametrize("ramp", [False, True])
@pytest.mark.parametrize("dark", [1.0, 0.03, 0.001, 1e-5])
@pytest.mark.parametrize("form", FORMS)
def test_dark_side(ctx, form, dark, ramp):
    # half of the search image at 1,000 to 1,300, half at 0 to `dark`; smooth base
    # blocks (whose partial sums grow most) or random ones
    rng = np.random.default_rng(8)
    base, search = rng.random((2, *SHAPE))
    if ramp:
        base = base * 0.05 + np.linspace(0, 3, SHAPE[0])[:, None, None] ** 2
    search = search * 300 + 1000
    search[:, : SHAPE[1] // 2] = rng.random((SHAPE[0], SHAPE[1] // 2, SHAPE[2])) * dark
    _check(ctx, form, base.astype(np.float32), search.astype(np.float32))


@pytest.mark.parametrize("form", [(4, 5, 1, 1), (4, 7, 1, 2), (4, 9, 1, 2), (5, 11, 1, 3)])
def test_dark_side_behind_a_mask_edge(ctx, form):
    rng = np.random.default_rng(9)
    base, search = rng.random((2, *SHAPE))
    search = search * 300 + 1000
    search[:, : SHAPE[1] // 2] = rng.random((SHAPE[0], SHAPE[1] // 2, SHAPE[2])) * 0.01
    sm = np.full(SHAPE, 255, np.uint8)
    sm[:, :, SHAPE[2] // 2: SHAPE[2] // 2 + 3] = 0
    sm[: 3] = 0
    _check(ctx, form, base.astype(np.float32), search.astype(np.float32), None, sm)
