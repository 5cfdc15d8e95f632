"""Poll limits at which waits of the panels and of the bulge chase run out here and there: a solve
ends with DVR3D_ERR_NOCONV or with its levels, and the context solves on."""
from __future__ import annotations

import numpy as np
import pytest

import dvr3d_b200
from dvr3d_b200 import AUTOCM, configs, parse_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [dvr3d_b200.DVR3D_PREC_FP64, dvr3d_b200.DVR3D_PREC_MIXED_DAVIDSON])
def test_every_limit_ends_the_solve(ctx, precision):
    w = configs.jacobi_h3p_like(14, 14, 24, 50000.0, 45000.0, 150, title="limits")
    d = parse_deck(w.deck)
    ctx.set_pes(w.pes)
    ref = ctx.solve(d, 0, precision=precision).eval

    def same_levels():
        assert np.abs(ctx.solve(d, 0, precision=precision).eval - ref).max() * AUTOCM <= 1e-6

    gave_up = 0
    try:
        for limit in (1, 3, 10, 30, 100, 300, 1000, 3000):
            ctx.set_wait_limit(limit)
            for _ in range(3):
                try:
                    same_levels()
                except dvr3d_b200.DVR3DError as e:
                    assert e.code == -5  # DVR3D_ERR_NOCONV
                    gave_up += 1
    finally:
        ctx.set_wait_limit(0)
    assert gave_up >= 3
    same_levels()
