"""LTS fits of pairs that hold NaN or infinities.

A fit with a non-finite residual has no finite cut-off: it ends, with NaN
transforms, in every form of the launch (one CTA, one cluster, the whole grid).
"""
import numpy as np
import pytest

import mirorr_b200 as mb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, -np.nan])
@pytest.mark.parametrize("n", [3000, 9000, 20000])
def test_fit_of_non_finite_pairs(ctx, n, value, symmetric):
    rng = np.random.default_rng(1)
    x = rng.uniform(-60, 60, size=(n, 3))
    y = x + rng.normal(0, 1, (n, 3))
    y[: 2 * n // 3, 1] = value
    t = [mb.Transform.make(mb.AFFINE, [1, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0], [0, 0, 0])
         for _ in range(3)]
    if symmetric:
        mb.lts_symmetric(ctx, *t, x, y, 0.5)
    else:
        mb.lts_classic(ctx, t[0], x, y, 0.5)
    assert np.isnan(t[0].M).any()
