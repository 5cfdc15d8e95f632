"""The two-stage dense eigensolve of the default precision form (reduction to a band of
half-bandwidth 32, then the bulge chase) at orders around its panel and tile edges, levels and
vectors against LAPACK on the assembled matrix that the solve returns."""
from __future__ import annotations

import numpy as np
import pytest

import dvr3d_b200
from dvr3d_b200 import configs

pytestmark = pytest.mark.gpu


# the smallest orders, panels of 32 with 0, 1, 2 rows left, the 64-row tiles, the first panels with
# more than one block a warp (over 7680 rows: config 4 in test_gpu_parity.py)
@pytest.mark.parametrize("n", [3, 4, 31, 32, 33, 34, 63, 64, 65, 66, 95, 97, 127, 129, 161, 513, 545, 1027])
def test_levels_and_vectors(ctx, n):
    w = configs.radau_water_like(16, 24, 0.0, min(n, 40), zcut=False, max3d=n)
    d = dvr3d_b200.parse_deck(w.deck)
    ctx.set_pes(w.pes)
    r = ctx.solve(d, 0, want_vectors=True, want_h3=True, want_resid=True)
    assert r.nham3 == n
    h = np.tril(r.h3) + np.tril(r.h3, -1).T
    ref = np.linalg.eigvalsh(h)[:len(r.eval)]
    # backward error of both sides: a modest multiple of eps ||H||
    tol = 40 * np.finfo(float).eps * max(n, 10) ** 0.5 * np.abs(h).sum(1).max()
    assert np.abs(r.eval - ref).max() <= tol
    z = r.evec
    assert np.abs(h @ z - z * r.eval).max() <= 10 * tol
    assert np.abs(z.T @ z - np.eye(z.shape[1])).max() <= 1e-9
    assert r.max_resid <= 20 * tol
