"""dvr3d_b200_run_deck_wave and the file at its path: a job that fails leaves the file that was
there as it was and makes none that was not; one that succeeds replaces all of it; a path that
cannot be written is refused."""
from __future__ import annotations

import pytest

import dvr3d_b200
from dvr3d_b200 import configs

pytestmark = pytest.mark.gpu


def _deck():
    w = configs.radau_water_like(8, 10, 30000.0, 6, title="wave file kept")
    w.deck = w.deck.replace("ZPMIN=.TRUE.", "ZPMIN=.TRUE., ZTRAN=.TRUE.")
    return w


@pytest.mark.parametrize("old", [None, b"", b"the run before" * 100000], ids=["none", "empty", "longer"])
def test_wave_file_replaced_only_by_a_job_that_succeeds(tmp_path, old):
    w = _deck()
    path = tmp_path / "fort.26"
    if old is not None:
        path.write_bytes(old)
    with dvr3d_b200.Context() as c:
        with pytest.raises(dvr3d_b200.DVR3DError):  # no surface set: the solve fails
            c.run_deck(w.deck, wave_path=str(path))
        assert (path.read_bytes() if path.exists() else None) == old
        c.set_pes(w.pes)
        text, _ = c.run_deck(w.deck, wave_path=str(path))
        other = tmp_path / "other.26"
        assert c.run_deck(w.deck, wave_path=str(other))[0] == text
        assert path.read_bytes() == other.read_bytes()
        assert len(path.read_bytes()) > 1000
        with pytest.raises(dvr3d_b200.DVR3DError):
            c.run_deck(w.deck, wave_path=str(tmp_path / "absent" / "fort.26"))
