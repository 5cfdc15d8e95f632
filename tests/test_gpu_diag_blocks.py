"""dvr3d_b200_diag_batched against LAPACK: orders around the 16-row tiles, the 32-reflector panels
and the change of the column tile (536), and spectra that strain the Sturm counts and the inverse
iteration (decoupled, degenerate, graded, scaled far from one)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from dvr3d_b200 import _abi

pytestmark = pytest.mark.gpu


def _diag(ctx, blocks):
    import torch

    n = [b.shape[0] for b in blocks]
    off = np.concatenate([[0], np.cumsum(np.square(n))])
    woff = np.concatenate([[0], np.cumsum(n)])
    a = torch.tensor(np.concatenate([b.ravel(order="F") for b in blocks]), device="cuda")
    w = torch.zeros(int(woff[-1]), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    nb = len(n)
    rc = _abi.load_library().dvr3d_b200_diag_batched(
        ctx._h, nb, (C.c_int * nb)(*n), (C.c_longlong * nb)(*off[:-1].tolist()), (C.c_longlong * nb)(*woff[:-1].tolist()),
        C.c_void_p(a.data_ptr()), C.c_void_p(w.data_ptr()), 1)
    if rc != 0:
        return rc
    a, w = a.cpu().numpy(), w.cpu().numpy()
    return [(w[woff[b]:woff[b + 1]], a[off[b]:off[b + 1]].reshape(n[b], n[b], order="F")) for b in range(nb)]


def _check(ctx, blocks):
    got = _diag(ctx, blocks)
    assert not isinstance(got, int), got
    for a, (w, z) in zip(blocks, got):
        n = len(w)
        # backward error of a stable eigensolver: a modest multiple of n eps ||A||
        tol = 20 * np.finfo(float).eps * max(n, 8) * np.abs(a).sum(1).max()
        assert np.abs(w - np.linalg.eigvalsh(a)).max() <= tol, n
        assert np.abs(a @ z - z * w).max() <= tol, n
        assert np.abs(z.T @ z - np.eye(n)).max() <= 1e-9, n


def _random(n, seed):
    a = np.random.default_rng(seed).standard_normal((n, n))
    return 0.5 * (a + a.T)


@pytest.mark.parametrize("sizes", [[1, 2, 3, 4, 5], [15, 16, 17, 18, 31, 32, 33, 34, 35], [63, 64, 65, 66, 67, 130],
                                   [535, 536, 537], [1, 1023, 40], [1024], [40] * 200])
def test_orders(ctx, sizes):
    _check(ctx, [_random(n, 100 + i) for i, n in enumerate(sizes)])


def test_spectra(ctx):
    rng = np.random.default_rng(5)
    q, _ = np.linalg.qr(rng.standard_normal((60, 60)))
    graded = np.diag(10.0 ** np.linspace(-12, 3, 50)) + 1e-9 * _random(50, 3)
    _check(ctx, [np.eye(24), np.diag(np.arange(40.0)), np.diag(np.repeat([1.0, 2.0, 2.5], 11)),
                 (q * np.repeat([-1.0, 0.0, 4.0], 20)) @ q.T, graded, 1e120 * _random(37, 1), 1e-120 * _random(37, 2),
                 np.kron(np.eye(8), _random(6, 4))])


def test_zero_block_is_reported(ctx):
    """A block of zeros has no norm for dstein's growth test to refer to: non-convergence, as ever."""
    assert _diag(ctx, [np.zeros((9, 9))]) == -5  # DVR3D_ERR_NOCONV
