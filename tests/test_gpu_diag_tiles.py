"""dvr3d_b200_diag_batched on both sides of the changes that the largest order of a batch decides: the
reduction in shared memory up to order 152, one or two CTAs a block beyond it (two up to 74 blocks on
148 SMs), and 32 or 16 columns of vectors a CTA (32 up to order 527, where they fill shared memory)."""
from __future__ import annotations

import pytest
from test_gpu_diag_blocks import _check, _random

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[151, 152], [152, 153], [161] * 74, [161] * 75, [526, 527], [527, 528], [528]],
                         ids=lambda s: f"{len(s)}x{s[-1]}")
def test_orders(ctx, sizes):
    _check(ctx, [_random(n, 300 + i) for i, n in enumerate(sizes)])
