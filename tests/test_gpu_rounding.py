"""How far eigenvalues and vectors are from the true ones of the same matrix, beyond what a 64-bit
eigensolver can tell: first-order corrections from residuals whose products are exact where they
matter (operands in slices of 19 bits, so that sums of up to 2^15 products of two slices are exact)."""
from __future__ import annotations

import numpy as np
import pytest

import dvr3d_b200
from dvr3d_b200 import configs, parse_deck

pytestmark = pytest.mark.gpu


def _slices(x, dim):
    """Three leading slices of x, scaled by its rows' (dim 1) or columns' (dim 0) largest, and the rest."""
    import torch

    out = []
    for _ in range(3):
        unit = torch.exp2(torch.ceil(torch.log2(x.abs().amax(dim=dim, keepdim=True).clamp_min(1e-300))) + 34)
        out.append((x + unit) - unit)
        x = x - out[-1]
    return out + [x]


def _residual(h, z, w):
    """H z - w z for all columns."""
    hs, zs = _slices(h, 1), _slices(z, 0)
    p = z * w
    zh = (134217729.0 * z) - (134217729.0 * z - z)
    wh = (134217729.0 * w) - (134217729.0 * w - w)
    low = ((zh * wh - p) + zh * (w - wh) + (z - zh) * wh) + (z - zh) * (w - wh)  # z w - p
    r = hs[0] @ zs[0] - p
    r = (r + hs[0] @ zs[1]) + hs[1] @ zs[0]
    rest = hs[0] @ (zs[2] + zs[3]) + hs[1] @ (z - zs[0]) + (hs[2] + hs[3]) @ z
    return (r - low) + rest


def test_levels_of_the_dense_solve(ctx):
    """Root mean square error of 300 levels of order 3984: a numpy restatement of the two stages in 64
    bits, each update rounded once an element, has 0.5e-16 hartree in the reduction to the band and
    1.4e-16 in the chase, so no more than 1.5e-16."""
    import torch

    w = configs.config2()
    ctx.set_pes(w.pes)
    r = ctx.solve(parse_deck(w.deck), 0, want_vectors=True, want_h3=True)
    h = torch.tensor(np.tril(r.h3), device="cuda")
    h = h + torch.tril(h, -1).T
    z = torch.tensor(np.ascontiguousarray(r.evec), device="cuda")
    err = (z * _residual(h, z, torch.tensor(r.eval, device="cuda"))).sum(0) / (z * z).sum(0)
    assert r.nham3 == 3984 and err.square().mean().sqrt().item() <= 1.5e-16
