"""Shift-invert solves whose Cholesky factorisation ends in leaves of every kind (orders of 1, 31,
32, 33, 63 and 64 in the last one: the 32- and the 64-row kernel, full and ragged) and whose Krylov
blocks take the 32-row kernel: the levels agree with the default form."""
from __future__ import annotations

import numpy as np
import pytest

import dvr3d_b200
from dvr3d_b200 import AUTOCM, configs, parse_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("last", [1, 31, 32, 33, 63, 64])
def test_levels_with_last_leaf_of(ctx, last):
    n = 704 + last
    w = configs.jacobi_h3p_like(18, 16, 30, 45000.0, 0.0, 40, max3d=n)
    d = parse_deck(w.deck.replace("ZCUT=.TRUE.", "ZCUT=.FALSE."))
    ctx.set_pes(w.pes)
    plain = ctx.solve(d, 0)
    got = ctx.solve(d, 0, precision=dvr3d_b200.DVR3D_PREC_MIXED_DAVIDSON)
    assert got.extra["path"] == dvr3d_b200.DVR3D_PATH_SHIFT_INVERT
    assert plain.nham3 == got.nham3 == n
    assert np.abs(got.eval - plain.eval).max() * AUTOCM <= 1e-3  # the bar of the iterative path
