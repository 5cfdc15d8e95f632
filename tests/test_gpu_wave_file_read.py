"""What ROTLEV3B takes as a wavefunction file: a file, a pipe with the same bytes, and with an error that
names the path a directory, a missing file, a file cut short."""
from __future__ import annotations

import os
import threading

import numpy as np
import pytest
from test_gpu_rotlev3b import _first_step, _rot_deck

import dvr3d_b200

pytestmark = pytest.mark.gpu


def test_sources(ctx, tmp_path):
    w = _first_step(1, 1)
    ctx.set_pes(w.pes)
    path, deck = tmp_path / "fort.26", _rot_deck(30, 20, 1)
    ctx.run_deck(w.deck, wave_path=str(path))
    ref, _, _ = ctx.rotlev3b_pair(deck, str(path))
    data = path.read_bytes()

    pipe = tmp_path / "pipe"
    os.mkfifo(pipe)
    feed = threading.Thread(target=lambda: pipe.write_bytes(data))
    feed.start()
    got, _, _ = ctx.rotlev3b_pair(deck, str(pipe))
    feed.join()
    np.testing.assert_array_equal(got, ref)

    (tmp_path / "short").write_bytes(data[:len(data) // 2])
    for name, text in [("", "read"), ("absent", "open"), ("short", "")]:
        with pytest.raises(dvr3d_b200.DVR3DError) as e:
            ctx.rotlev3b_pair(deck, str(tmp_path / name) if name else str(tmp_path))
        assert e.value.code == -1 and text in str(e.value)  # DVR3D_ERR_ARG
