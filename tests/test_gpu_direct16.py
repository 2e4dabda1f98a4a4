"""The direct 16-bit search where its tiles and routes change, against the oracle.

Strip lengths (windows 3 to 13 at block width 4, 11 and 12 at width 5, which
have one thread per strip or several), windows clipped by the volume, blocks
and windows across mask edges (the listed candidates), flat blocks (written
without a search) and selections (whole warps culled).  The oracle runs on the
stored 16-bit values; scores within 1e-4, argmax equal wherever best and second
differ by more, the bars of the 16-bit storage tests.
"""
import numpy as np
import pytest

import mirorr_b200 as mb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _mask(shape, seed):
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*(np.linspace(-1, 1, n) for n in shape), indexing="ij")
    m = (z * z + y * y + x * x < rng.uniform(0.9, 1.6)).astype(np.uint8) * 255
    m[rng.random(shape) < 0.01] = 0
    return m


@pytest.mark.parametrize("kind", ["plain", "masked", "flat", "selected"])
@pytest.mark.parametrize("dtype", ["bf16", "f16"])
@pytest.mark.parametrize("bw,nw", [(4, 3), (4, 7), (4, 9), (4, 13), (5, 5), (5, 11), (5, 12)])
def test_matches_oracle(ctx, bw, nw, dtype, kind):
    shape = (19, 22, 31)
    rng = np.random.default_rng(bw * 100 + nw)
    base, search = rng.random((2, *shape)).astype(np.float32)
    if kind == "flat":
        base[:, :12] = 0.5
        search[:9] = 0.25
    bm, sm = (_mask(shape, 1), _mask(shape, 2)) if kind == "masked" else (None, None)
    keep = 0.3 if kind == "selected" else 1.0
    base, search = (mb.from_storage(mb.to_storage(v, dtype), dtype) for v in (base, search))
    prm = O.BMParams(bw, 1, 3, nw, keep)
    ref = O.match_blocks(base, search, bm, sm, prm)
    m = mb.BlockMatcher(ctx)
    m.SetStorage(dtype)
    m.SetBlockWidth(bw)
    m.SetNhoodWidth(nw)
    m.SetNhoodGap(3)
    m.SetBlockKeep(keep)
    m.SetBaseImage(base)
    m.SetSearchImage(search)
    if bm is not None:
        m.SetBaseMask(bm)
        m.SetSearchMask(sm)
    m.GetOffsets()
    mi, best, second, status = m.BlockResults()
    m.close()
    np.testing.assert_array_equal((status & 1).astype(np.uint8), ref.status)
    s = ref.status == 1
    np.testing.assert_allclose(best[s], ref.best[s], atol=1e-4)
    np.testing.assert_allclose(second[s], ref.second[s], atol=1e-4)
    clear = s & (ref.best - ref.second > 1e-4)
    np.testing.assert_array_equal(mi[clear], ref.match[clear])
