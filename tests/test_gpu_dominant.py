"""The measurement counters of a default solve name what they cover: the reduction to a band as a
whole (five kernels), not one of its kernels."""
from __future__ import annotations

import pytest

import dvr3d_b200
from dvr3d_b200 import configs

pytestmark = pytest.mark.gpu


def test_counters_of_the_band_reduction(ctx):
    n = 513
    w = configs.radau_water_like(16, 24, 0.0, 20, zcut=False, max3d=n)
    ctx.set_pes(w.pes)
    x = ctx.solve(dvr3d_b200.parse_deck(w.deck), 0).extra
    assert x["dom_kernel"] == "band_reduction"
    assert x["dom_flops"] == pytest.approx(4.0 / 3.0 * n ** 3)
    panels = -(-n // 32)
    assert 4 * (panels - 1) < x["dom_launches"] <= 5 * panels + 1 and x["dom_ms"] > 0
