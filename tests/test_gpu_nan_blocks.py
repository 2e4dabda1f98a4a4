"""Base blocks that hold NaN: no candidate scores, so the candidate list is empty,
and the candidates still count as evaluated.
"""
import numpy as np
import pytest

import mirorr_b200 as mb
from mirorr_b200.phantom import make_phantom

pytestmark = pytest.mark.gpu


def test_evaluated_candidates_are_counted(ctx):
    ph = make_phantom((48, 44, 40), n_gauss=12, seed=3)
    p = mb.reg_params(symmetric=False, kind="rigid", levels=1, iterations=2)
    per_call = []
    for nan in (False, True):
        moving = ph.moving.copy()
        if nan:
            moving[: moving.shape[0] // 2] = np.nan
        _, st = mb.register(ctx, ph.fixed, moving, p)
        assert st.matcher_calls > 0
        assert st.block_ncc_evaluated % st.matcher_calls == 0
        per_call.append(st.block_ncc_evaluated // st.matcher_calls)
    assert per_call[0] == per_call[1]
