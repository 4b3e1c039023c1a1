"""The split-BF16 density's stages are refilled by bulk copies once its epilogue has
released them.  A copy that overtook the epilogue's loads would change a sum, so
repeated calls must give the same bits (one spin: every stage is reused at once)."""
import numpy as np
import pytest

import lcpgrid as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cell", ["si2", "mixed"])
def test_repeated_density_same_bits(cell):
    from test_gpu_parity import psd_dm
    from test_gpu_tc import _mixed_cell, _si2
    ctx = L.Context(0)
    u, orbs = (_si2 if cell == "si2" else _mixed_cell)(ctx)
    ctx.set_precision("bf16x3")
    dm = psd_dm(u, 71)
    rho = [np.zeros(u.NN)]
    L.Set_Density_Grid("off", u, orbs, dm, rho)
    first = rho[0].copy()
    for _ in range(100):
        L.Set_Density_Grid("off", u, orbs, dm, rho)
        assert np.array_equal(first, rho[0])
