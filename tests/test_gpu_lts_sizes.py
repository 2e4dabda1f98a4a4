"""The LTS fit where its launch and its selection change form, against the oracle.

* pair counts around one CTA's limit (4,096 pairs), one cluster's (16,384) and
  a CTA's thread and candidate counts, down to a handful;
* residuals below, inside and above the first histogram's range
  ([2^-12, 2^20) mm^2), so the cut-off falls into its open end bins;
* more equal residuals than the final ranking holds.

Tolerances are those of the other fits: matrices 1e-9, offsets 1e-8, the same
number of inner iterations.
"""
import numpy as np
import pytest

import mirorr_b200 as mb
from mirorr_b200.phantom import random_rotation
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _to_mb(t):
    return mb.Transform.make(mb.RIGID if t.kind == "rigid" else mb.AFFINE, t.params(), t.c)


def _fit_both(ctx, kind, x, y, symmetric):
    t = O.Tfm(kind)
    if symmetric:
        f, b = O.compute_half_space(t)
        tg, fg, bg = _to_mb(t), _to_mb(f), _to_mb(b)
        it_o = O.lts_symmetric(t, f, b, x, y, 0.5)
        it_g = mb.lts_symmetric(ctx, tg, fg, bg, x, y, 0.5)
        pairs = [(tg, t), (fg, f), (bg, b)]
    else:
        tg = _to_mb(t)
        it_o = O.lts_classic(t, x, y, 0.5)
        it_g = mb.lts_classic(ctx, tg, x, y, 0.5)
        pairs = [(tg, t)]
    assert it_g == it_o
    for a, o in pairs:
        np.testing.assert_allclose(a.M, o.M, atol=1e-9)
        np.testing.assert_allclose(a.off, o.off, atol=1e-8)


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("kind", ["rigid", "affine"])
@pytest.mark.parametrize("n", [40, 511, 4096, 4097, 16384, 16385, 33000])
def test_pair_counts(ctx, n, kind, symmetric):
    rng = np.random.default_rng(n)
    x = rng.uniform(-60, 60, size=(n, 3))
    y = x @ random_rotation(rng, 4.0).T + rng.uniform(-4, 4, 3) + rng.normal(0, 0.3, (n, 3))
    k = n // 4
    y[:k] += rng.normal(0, 10, size=(k, 3))
    _fit_both(ctx, kind, x, y, symmetric)


@pytest.mark.parametrize("n", [2500, 20000])
@pytest.mark.parametrize("noise,outliers,spread", [(1e-4, 0.25, 3.0), (3.0, 0.7, 4000.0)])
def test_residual_ranges(ctx, n, noise, outliers, spread):
    # residuals of about 1e-8 mm^2 with the cut-off among them, and a cut-off
    # among outliers of about 1e7 mm^2
    rng = np.random.default_rng(7)
    x = rng.uniform(-60, 60, size=(n, 3))
    y = x @ random_rotation(rng, 2.0).T + rng.normal(0, noise, (n, 3))
    k = int(outliers * n)
    y[:k] += rng.normal(0, spread, size=(k, 3))
    _fit_both(ctx, "affine", x, y, False)


@pytest.mark.parametrize("n", [8 * 700, 8 * 2500])
def test_equal_residuals(ctx, n):
    # eight pairs, each many times over: the cut-off's bucket holds more equal
    # residuals than are ranked
    rng = np.random.default_rng(3)
    c = np.array([[a, b, d] for a in (-40., 41.) for b in (-30., 33.) for d in (-20., 25.)])
    m = c @ random_rotation(rng, 3.0).T + rng.normal(0, 1.5, (8, 3))
    pick = rng.permutation(np.repeat(np.arange(8), n // 8))
    _fit_both(ctx, "rigid", c[pick], m[pick], False)
