"""Amplitudes at the grid points of a block that keeps no 2D state: zero in the wavefunction file,
also after a larger job of the same context has used the buffers."""
from __future__ import annotations

import struct

import numpy as np
import pytest

import dvr3d_b200
from dvr3d_b200 import configs

pytestmark = pytest.mark.gpu


def _job(emax2: float):
    w = configs.jacobi_h3p_like(8, 9, 12, 45000.0, emax2, 10, title="empty blocks")
    w.deck = w.deck.replace("ZTHETA=.FALSE.", "ZTHETA=.TRUE.").replace("ZR2R1=.TRUE.", "ZR2R1=.FALSE.")
    w.deck = w.deck.replace("ZPMIN=.TRUE.", "ZPMIN=.TRUE., ZTRAN=.TRUE.")
    return w


def _amplitudes(path, nlev: int, shape):
    data, pos, rec = path.read_bytes(), 0, []
    while pos < len(data):
        n = struct.unpack_from("<i", data, pos)[0]
        rec.append(data[pos + 4:pos + 4 + n])
        pos += n + 8
    return np.array([np.frombuffer(r) for r in rec[-nlev:]]).reshape(nlev, *shape)


@pytest.mark.parametrize("first", [None, 40000.0], ids=["alone", "after_a_larger_job"])
def test_empty_blocks_have_zero_amplitudes(tmp_path, first):
    w = _job(20000.0)
    with dvr3d_b200.Context() as c:
        c.set_pes(w.pes)
        r = c.solve(dvr3d_b200.parse_deck(w.deck))
        empty = np.flatnonzero(r.iv2 == 0)
        assert empty.size and r.iv2.size == 9
        if first:
            c.run_deck(_job(first).deck, wave_path=str(tmp_path / "first"))
        c.run_deck(w.deck, wave_path=str(tmp_path / "f"))
    psi = _amplitudes(tmp_path / "f", r.eval.size, (9, 8, 12))  # psi(angle, r1, r2), Fortran order
    assert not psi[:, empty].any()
    kept = np.flatnonzero(r.iv2 > 0)
    assert psi[:, kept].any(axis=(0, 2, 3)).all()
