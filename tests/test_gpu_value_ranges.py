"""The float32 search over the amplitudes of its images, against the oracle.

Scores do not change when an image is scaled, so neither may the route to them:
the FP32 filter keeps its bound while sums of squares lie in a wide middle range,
and blocks that see sums outside it are re-scored in FP64.  Both images alike and
one image alone are scaled, up and down to where squares leave the float range and
values are subnormal, in every search form.  Best, second and argmax equal the
FP64 oracle's exactly; ordinary small and large amplitudes stay with the filter.
"""
import numpy as np
import pytest

import mirorr_b200 as mb
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# block width, window, block gap, spacing, shape (z, y, x)
FORMS = {
    "general_w5": (4, 5, 1, 3, (15, 17, 19)),
    "xlane_w5": (4, 5, 1, 1, (24, 30, 41)),
    "xlane_w7": (4, 7, 1, 3, (15, 17, 33)),
    "xlane_w9": (4, 9, 1, 3, (15, 17, 33)),
    "warp_w7": (4, 7, 1, 20, (33, 29, 99)),
    "warp_w9": (4, 9, 1, 25, (33, 30, 99)),
    "warp_bw5": (5, 11, 1, 3, (18, 19, 24)),
    "general_bw3": (3, 5, 1, 3, (15, 17, 19)),
    "general_gap2": (3, 5, 2, 2, (17, 18, 19)),
}
# amplitudes of the base and of the search image
SMALL = [(1e-10, 1e-10), (1e-11, 1e-11), (3e-12, 3e-12), (3e9, 3e9), (1e-11, 1e3)]
SCALES = SMALL + [(1.0, 1e-20), (1.0, 2e-20), (1.0, 5e-21), (2e-20, 1.0), (0.1, 8e18),
                  (1.0, 1e-24), (1e-24, 1.0), (1e-20, 1e-20), (1.0, 1e-40), (1e-40, 1e-40),
                  (1e19, 1e19), (1e-30, 1e30), (1e37, 1.0)]


def _masks(rng, shape):
    out = []
    for _ in range(2):
        m = np.full(shape, 255, np.uint8)
        z, y, x = (int(rng.integers(2, s - 4)) for s in shape)
        m[z: z + 3, y: y + 4] = 0
        m[:, :, x: x + 2] = 0
        out.append(m)
    return out


def _check(ctx, form, base, search, bm, sm):
    bw, nw, bgap, gap, shape = form
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
    return overflowed, best.size


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("scale", SCALES, ids=lambda s: f"{s[0]:g}x{s[1]:g}")
@pytest.mark.parametrize("form", FORMS)
def test_scaled_images(ctx, form, scale, masked):
    shape = FORMS[form][4]
    rng = np.random.default_rng(11)
    base, search = rng.random((2, *shape))
    with np.errstate(under="ignore"):
        base = (base * scale[0]).astype(np.float32)
        search = (search * scale[1]).astype(np.float32)
    bm, sm = _masks(rng, shape) if masked else (None, None)
    overflowed, blocks = _check(ctx, FORMS[form], base, search, bm, sm)
    if scale in SMALL and not masked:
        assert overflowed < blocks / 10


@pytest.mark.parametrize("level", [2.0 ** -80, 2.0 ** -40, 2.0 ** 70])
@pytest.mark.parametrize("form", FORMS)
def test_two_levels(ctx, form, level):
    # footprint means that are floats, so that no rounding residual keeps the FP32
    # sum of squares away from zero, and flat footprints among the others
    shape = FORMS[form][4]
    rng = np.random.default_rng(12)
    base = rng.random(shape).astype(np.float32)
    search = ((rng.random(shape) < 0.5) * level).astype(np.float32)
    search[:, : shape[1] // 3] = 0
    search[:, -shape[1] // 3:] = level
    _check(ctx, FORMS[form], base, search, None, None)
