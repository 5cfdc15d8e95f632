"""Eigenvectors of the dense two-stage solve for every slab width of the chase's back-transformation
(1, 2, 4 and 8 columns a CTA on 148 SMs, the last slab ragged), against the matrix itself."""
from __future__ import annotations

import numpy as np
import pytest

import dvr3d_b200
from dvr3d_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nev", [41, 201, 401, 797])
def test_vectors(ctx, nev):
    n = 997
    w = configs.radau_water_like(16, 24, 0.0, nev, zcut=False, max3d=n)
    d = dvr3d_b200.parse_deck(w.deck)
    ctx.set_pes(w.pes)
    r = ctx.solve(d, 0, want_vectors=True, want_h3=True)
    assert r.nham3 == n and len(r.eval) == nev
    h = np.tril(r.h3) + np.tril(r.h3, -1).T
    # backward error: a modest multiple of eps ||H||
    tol = 40 * np.finfo(float).eps * n ** 0.5 * np.abs(h).sum(1).max()
    z = r.evec
    assert np.abs(r.eval - np.linalg.eigvalsh(h)[:nev]).max() <= tol
    assert np.abs(h @ z - z * r.eval).max() <= 10 * tol
    assert np.abs(z.T @ z - np.eye(nev)).max() <= 1e-9
