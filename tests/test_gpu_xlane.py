"""The per-x-lane search over its windows, spacings and volume edges.

Block width 4 with windows 7 and 9, and 5 from 10,000 blocks on, takes the
per-x-lane kernel at every block spacing whose union window fits; spacings above
4 use the run-time row pitch.  Odd and even volumes (statistics rows padded to an even pitch), volumes
smaller than a window, flat regions (degenerate candidates) and fewer blocks
than one tile are where its tiles end.  Best, second, argmax and points equal
the FP64 oracle's exactly, as for every other search kernel.
"""
import numpy as np
import pytest

import mirorr_b200 as mb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(ctx, base, search, nw, gap):
    m = mb.BlockMatcher(ctx)
    m.SetNhoodWidth(nw)
    m.SetNhoodGap(gap)
    m.SetBaseImage(base)
    m.SetSearchImage(search)
    prm = O.BMParams(4, 1, gap, nw, 1.0)
    ref = O.match_blocks(base, search, None, None, prm)
    ob, om, _ = O.emit_points(ref, O.Image(base), prm)
    try:
        bp, mp = m.GetOffsets()
    except mb.MirorrError as e:
        assert e.name == "ENOBLOCKS" and len(ob) == 0
        bp, mp = ob, om
    mi, best, second, status = m.BlockResults()
    m.close()
    np.testing.assert_array_equal(best, ref.best)
    np.testing.assert_array_equal(second, ref.second)
    np.testing.assert_array_equal(mi, ref.match)
    np.testing.assert_array_equal(bp, ob)
    np.testing.assert_array_equal(mp, om)


def _volume(shape, seed, flat):
    rng = np.random.default_rng(seed)
    v = rng.random(shape).astype(np.float32)
    if flat:  # constant slabs: blocks and candidates with no variance
        v[:, : shape[1] // 2, :] = 0.25
        v[: shape[0] // 3] = 0.25
    return v


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("shape", [(13, 17, 40), (20, 11, 33), (4, 6, 5), (9, 21, 62)])
@pytest.mark.parametrize("nw,gap", [(5, 2), (5, 1), (5, 7), (7, 3), (7, 5), (9, 4), (9, 6)])
def test_matches_oracle(ctx, nw, gap, shape, flat):
    _check(ctx, _volume(shape, 1, flat), _volume(shape, 2, flat), nw, gap)


@pytest.mark.parametrize("nw", [5, 7, 9])
def test_wide_value_ranges(ctx, nw):
    # a large common offset (the shifted cross term), and tiny magnitudes whose
    # sums of squares leave the float range downwards
    rng = np.random.default_rng(5)
    a, b = rng.random((2, 10, 14, 30)).astype(np.float32)
    _check(ctx, a + np.float32(4000.0), b + np.float32(4000.0), nw, 3)
    _check(ctx, a * np.float32(1e-20), b * np.float32(1e-20), nw, 3)


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("shape,gap", [((24, 30, 41), 1), ((43, 44, 62), 2), ((27, 25, 30), 1)])
def test_window_5_on_both_sides_of_its_limit(ctx, shape, gap, flat):
    # 20,000 to 22,000 blocks, and 13,700; the smaller volumes above stay below
    _check(ctx, _volume(shape, 1, flat), _volume(shape, 2, flat), 5, gap)


def test_window_5_wide_value_ranges(ctx):
    rng = np.random.default_rng(5)
    a, b = rng.random((2, 24, 30, 41)).astype(np.float32)
    _check(ctx, a + np.float32(4000.0), b + np.float32(4000.0), 5, 1)
    _check(ctx, a * np.float32(1e-20), b * np.float32(1e-20), 5, 1)
