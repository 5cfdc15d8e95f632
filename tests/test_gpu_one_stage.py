"""The one-stage dense reduction, which serves orders below three and eigenvectors of more than 22000
rows: its levels against the two-stage reduction's (which takes that order without vectors), its
vectors against the matrix, and the bounded waits of its grid barriers."""
from __future__ import annotations

import numpy as np
import pytest

import dvr3d_b200
from dvr3d_b200 import AUTOCM, configs, parse_deck

pytestmark = pytest.mark.gpu

NEV = 24


@pytest.fixture(scope="module")
def large(ctx):
    """The k = 0 block of the H/C/N workload with its basis chosen by count, at an odd order just
    beyond the limit of the two-stage vectors."""
    n = 22003
    w = configs.config5()
    w.deck = w.deck.replace("ZCUT=.TRUE.", "ZCUT=.FALSE.")
    lines = w.deck.splitlines()
    c3 = lines[2]
    assert c3[10:15] == " 1000" and c3[25:30] == "40000"  # NEVAL, MAX3D
    lines[2] = c3[:10] + f"{NEV:5d}" + c3[15:25] + f"{n:5d}" + c3[30:]
    d = parse_deck("\n".join(lines) + "\n")
    ctx.set_pes(w.pes)
    return n, d


def test_large_order_with_vectors(ctx, large):
    n, d = large
    two = ctx.solve(d, 0)
    one = ctx.solve(d, 0, want_vectors=True, want_resid=True)
    assert two.nham3 == one.nham3 == n and len(one.eval) == NEV
    assert one.extra["dom_kernel"] == "dense_panel_kernel" != two.extra["dom_kernel"]
    assert np.abs(one.eval - two.eval).max() * AUTOCM <= 1e-6  # the bar of the default form
    assert one.max_resid < 1e-9
    z = one.evec
    assert np.abs(z.T @ z - np.eye(NEV)).max() <= 1e-9


def test_grid_barriers_run_out(ctx, large):
    _, d = large
    try:
        ctx.set_wait_limit(1)
        with pytest.raises(dvr3d_b200.DVR3DError) as e:
            ctx.solve(d, 0, want_vectors=True)
        assert e.value.code == -5  # DVR3D_ERR_NOCONV
    finally:
        ctx.set_wait_limit(0)


@pytest.mark.parametrize("n", [1, 2])
def test_smallest_orders(ctx, n):
    w = configs.radau_water_like(16, 24, 0.0, n, zcut=False, max3d=n)
    ctx.set_pes(w.pes)
    r = ctx.solve(parse_deck(w.deck), 0, want_vectors=True, want_h3=True, want_resid=True)
    assert r.nham3 == n
    h = np.tril(r.h3) + np.tril(r.h3, -1).T
    tol = 40 * np.finfo(float).eps * np.abs(h).sum(1).max()
    assert np.abs(r.eval - np.linalg.eigvalsh(h)[:len(r.eval)]).max() <= tol
    assert np.abs(h @ r.evec - r.evec * r.eval).max() <= 10 * tol
