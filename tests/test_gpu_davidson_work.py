"""Davidson solves whose products H3 V split more than sixteen ways (bases of a few hundred to
about 2300 functions): the partial sums have to fit their buffer, and the levels agree with the
default form."""
from __future__ import annotations

import numpy as np
import pytest

import dvr3d_b200
from dvr3d_b200 import AUTOCM, configs, parse_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nlevels", [(300, 31), (850, 31), (850, 8), (1500, 32), (2240, 24)])
def test_levels_below_2300_functions(ctx, n, nlevels):
    w = configs.jacobi_h3p_like(26, 23, 52, 45000.0, 0.0, nlevels, max3d=n)
    d = parse_deck(w.deck.replace("ZCUT=.TRUE.", "ZCUT=.FALSE."))
    ctx.set_pes(w.pes)
    plain = ctx.solve(d, 0)
    got = ctx.solve(d, 0, precision=dvr3d_b200.DVR3D_PREC_MIXED_DAVIDSON)
    assert plain.nham3 == got.nham3 == n
    assert np.abs(got.eval - plain.eval).max() * AUTOCM <= 1e-3
