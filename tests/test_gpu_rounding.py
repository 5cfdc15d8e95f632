"""How far eigenvalues and vectors are from the true ones of the same matrix, beyond what a 64-bit
eigensolver can tell: first-order corrections from residuals whose products are exact where they
matter (operands in slices of 19 bits, so that sums of up to 2^15 products of two slices are exact)."""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import pytest

import dvr3d_b200
from dvr3d_b200 import _abi, configs, parse_deck

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


def _dvr_block(n, k):
    """A sinc-DVR Hamiltonian: kinetic energy, Morse well, ripple."""
    import torch

    i = torch.arange(n)
    x, d = 12.0 / (n + 1) * (i + 1.0).double(), (i[:, None] - i[None, :]).double()
    t = (1.0 - 2.0 * (d.abs() % 2)) / torch.where(d == 0, 1.0, d) ** 2
    t.fill_diagonal_(math.pi ** 2 / 6)
    v = (4 + k % 5) * (1 - torch.exp(-(0.5 + 0.01 * k) * (x - 2.0))) ** 2 + 0.3 * torch.cos((1 + 0.05 * k) * x)
    return (t * ((n + 1) / 12.0) ** 2 + torch.diag(v)).cuda()


def _errors(h, z, w):
    """Squared errors of the vectors (to first order) and squared residuals by the norm."""
    r = _residual(h, z, w)
    p = z.t() @ r
    gap = (w + p.diagonal())[None, :] - (w + p.diagonal())[:, None]
    q = p / gap.fill_diagonal_(1.0)
    return q.fill_diagonal_(0.0).square().sum(0).mean().item(), (r.square().sum(0).mean() / w.abs().max() ** 2).item()


@pytest.fixture(scope="module", params=[(160, 13), (470, 9)], ids=["160_to_459", "470_to_677"])
def batched(request, ctx):
    """Root mean square errors of the batched eigensolver on 24 blocks, and of torch.linalg.eigh."""
    import torch

    n = [request.param[0] + request.param[1] * k for k in range(24)]
    blocks = [_dvr_block(m, k) for k, m in enumerate(n)]
    off, woff = np.cumsum([0] + [m * m for m in n]), np.cumsum([0] + n)
    a = torch.cat([b.reshape(-1) for b in blocks])
    w = torch.zeros(int(woff[-1]), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert _abi.load_library().dvr3d_b200_diag_batched(
        ctx._h, len(n), (C.c_int * len(n))(*n), (C.c_longlong * len(n))(*off[:-1].tolist()),
        (C.c_longlong * len(n))(*woff[:-1].tolist()), C.c_void_p(a.data_ptr()), C.c_void_p(w.data_ptr()), 1) == 0
    ours, theirs = [], []
    for b, m in enumerate(n):
        ours.append(_errors(blocks[b], a[off[b]:off[b + 1]].reshape(m, m).t().contiguous(), w[woff[b]:woff[b + 1]]))
        lam, z = torch.linalg.eigh(blocks[b])
        theirs.append(_errors(blocks[b], z, lam))
    return np.sqrt(np.mean(ours, 0)), np.sqrt(np.mean(theirs, 0))


def test_vectors_of_blocks(batched):
    """Both reduce a block by n reflectors and update it once a panel, so the errors are alike: no more
    than one and a half times torch's (0.9 and 1.1 measured, 2.1 and 2.4 with an update that rounds for
    every column of the panel)."""
    ours, theirs = batched
    assert ours[0] <= 1.5 * theirs[0]


def test_residuals_of_blocks(batched):
    """The back-transformation rounds a vector once a panel of 32 reflectors: residuals of 0.43 times
    torch's measured, 0.48 and 0.50 where it rounds once a reflector."""
    ours, theirs = batched
    assert ours[1] <= 0.46 * theirs[1]
