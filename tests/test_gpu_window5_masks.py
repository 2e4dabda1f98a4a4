"""Window 5 with masks on the register-blocked searches (10,000 blocks and more).

Masks bring the window-AND, the masked-window search of one warp per block and
the base-mask search of ten blocks per CTA into the call.  Best, second, argmax
and points equal the FP64 oracle's exactly; masks of 255 everywhere give what no
masks give.
"""
import numpy as np
import pytest

import mirorr_b200 as mb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _run(ctx, base, search, bm, sm, gap, keep):
    m = mb.BlockMatcher(ctx)
    m.SetNhoodWidth(5)
    m.SetNhoodGap(gap)
    m.SetBlockKeep(keep)
    m.SetBaseImage(base)
    m.SetSearchImage(search)
    m.SetBaseMask(bm)
    m.SetSearchMask(sm)
    out = (*m.GetOffsets(), *m.BlockResults())
    d = m.LastDiagnostics()
    m.close()
    return out, d


def _volumes(shape, seed):
    rng = np.random.default_rng(seed)
    base, search = rng.random((2, *shape)).astype(np.float32)
    base[:, : shape[1] // 4] = 0.5  # flat blocks and candidates
    search[: shape[0] // 5] = 0.25
    z, y, x = np.ogrid[: shape[0], : shape[1], : shape[2]]
    r = ((z / shape[0] - .5) ** 2 + (y / shape[1] - .5) ** 2 + (x / shape[2] - .5) ** 2) ** .5
    bm = (r < 0.45).astype(np.uint8)
    sm = ((r < 0.55) & (rng.random(shape) < 0.995)).astype(np.uint8) * 255
    return base, search, bm, sm


@pytest.mark.parametrize("keep", [1.0, 0.4])
@pytest.mark.parametrize("sides", ["search", "base", "both"])
@pytest.mark.parametrize("shape,gap", [((27, 30, 41), 1), ((44, 47, 63), 2)])
def test_matches_oracle(ctx, shape, gap, sides, keep):
    base, search, bm, sm = _volumes(shape, 3)
    bm = bm if sides != "search" else None
    sm = sm if sides != "base" else None
    (bp, mp, mi, best, second, status), d = _run(ctx, base, search, bm, sm, gap, keep)
    prm = O.BMParams(4, 1, gap, 5, keep)
    ref = O.match_blocks(base, search, bm, sm, prm)
    assert d[3] >= 10000 and d[4] > 0
    if sides != "search":
        assert d[5] > 0
    s = ref.status == 1
    np.testing.assert_array_equal(status & 1, ref.status)
    np.testing.assert_array_equal(best[s], ref.best[s])
    np.testing.assert_array_equal(second[s], ref.second[s])
    np.testing.assert_array_equal(mi[s], ref.match[s])
    ob, om, _ = O.emit_points(ref, O.Image(base), prm)
    np.testing.assert_array_equal(bp, ob)
    np.testing.assert_array_equal(mp, om)


def test_equals_full_masks(ctx):
    base, search, _, _ = _volumes((27, 30, 41), 4)
    ones = np.full(base.shape, 255, np.uint8)
    got = [_run(ctx, base, search, bm, sm, 1, 1.0)[0]
           for bm, sm in ((None, None), (ones, ones), (ones, None), (None, ones))]
    for other in got[1:]:
        for a, b in zip(got[0], other):
            np.testing.assert_array_equal(a, b)
