"""Eigenvalues of decoupled and graded blocks by dvr3d_b200_diag_batched: each decoupled part has its
eigenvalues to the accuracy of that part's own norm, however small it is beside the others, as the
quotient form of the Sturm counts gives them (LAPACK dstebz)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from dvr3d_b200 import _abi

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _eigenvalues(ctx, blocks):
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
        C.c_void_p(a.data_ptr()), C.c_void_p(w.data_ptr()), 0)
    assert rc == 0
    w = w.cpu().numpy()
    return [w[woff[b]:woff[b + 1]] for b in range(nb)]


def _random(n, seed):
    a = np.random.default_rng(seed).standard_normal((n, n))
    return 0.5 * (a + a.T)


def _joined(parts):
    n = sum(p.shape[0] for p in parts)
    a, q = np.zeros((n, n)), 0
    for p in parts:
        m = p.shape[0]
        a[q:q + m, q:q + m] = p
        q += m
    return a


@pytest.mark.parametrize("d", [[0.5, 1e-20, 3e-20], [1e-30, 2.0, 1e-30, -4e-25], [-1.0, 1e-60, 1e-45, 7.0],
                               [3e-20] * 9 + [1.0], list(10.0 ** -np.arange(60.0)),
                               list(-(10.0 ** -np.arange(0.0, 50.0, 0.5))), [1e120, 1e100, 1e98], [1e-160, 1e-175]])
def test_diagonal_blocks_to_relative_accuracy(ctx, d):
    """Counts of a diagonal matrix are exact, so an eigenvalue is known to its last bisection step
    (two units in the last place)."""
    d = np.array(d)
    got, = _eigenvalues(ctx, [np.diag(d)])
    ref = np.sort(d)
    assert (np.abs(got - ref) <= 4 * EPS * np.abs(ref)).all(), (got, ref)


@pytest.mark.parametrize("n1,n2,count", [(3, 2, 1), (7, 30, 2), (40, 40, 5), (100, 52, 3), (101, 60, 80), (17, 16, 200)])
@pytest.mark.parametrize("small", [1e-19, 1e-25, 1e-40])
def test_parts_far_below_the_norm(ctx, n1, n2, count, small):
    """Blocks of two decoupled parts, the second `small` times the size of the first. Its levels sit
    beside zero and are ordered with the first part's."""
    blocks, refs, tols = [], [], []
    for q in range(count):
        a, b = _random(n1, 10 + q), _random(n2, 1000 + q)
        blocks.append(_joined([a, small * b]))
        la, lb = np.linalg.eigvalsh(a), np.linalg.eigvalsh(b)
        refs.append((la, small * lb))
        # backward error of a stable eigensolver, each part by its own norm
        tols.append((20 * EPS * n1 * np.abs(a).sum(1).max(), 20 * EPS * n2 * small * np.abs(b).sum(1).max()))
    for got, (la, lb), (ta, tb) in zip(_eigenvalues(ctx, blocks), refs, tols):
        neg = int((la < 0).sum())
        assert np.abs(got[neg:neg + n2] - lb).max() <= tb
        assert np.abs(np.delete(got, np.s_[neg:neg + n2]) - la).max() <= ta


def test_blocks_of_equal_parts_beside_ordinary_ones(ctx):
    """Both forms of the counts in one batch."""
    a = [_random(33, 5), np.kron(np.eye(4), _random(8, 6)), np.eye(20) * 1e-25, _random(150, 7), np.zeros((5, 5))]
    for got, m in zip(_eigenvalues(ctx, a), a):
        ref = np.linalg.eigvalsh(m)
        assert np.abs(got - ref).max() <= 20 * EPS * len(ref) * max(np.abs(m).sum(1).max(), 1e-290)
