"""The FP64 tensor-core kernels' tables leave a quarter of the device free.  Orbitals
first used while less was free take the pair kernels, and the tensor-core kernels
from the next call on after the memory came back."""
import numpy as np
import pytest

import lcpgrid as L

pytestmark = pytest.mark.gpu


def test_tables_are_made_once_there_is_room():
    torch = pytest.importorskip("torch")
    from test_gpu_parity import psd_dm
    from test_gpu_tc import _si2
    ctx = L.Context(0)
    u, orbs = _si2(ctx)
    dm, v = psd_dm(u, 61), np.random.default_rng(62).normal(size=u.NN)

    def call():
        rho, h = [np.zeros(u.NN)], [np.zeros(u.Total_Hsize)]
        l0 = ctx.launch_count
        L.Set_Density_Grid("off", u, orbs, dm, rho)
        L.Calc_MatrixElements_dVH_Vxc_off(u, orbs, [v], h)
        return rho[0], h[0], ctx.launch_count - l0

    free, total = torch.cuda.mem_get_info()
    held = torch.empty(max(free - total // 4, 1), dtype=torch.uint8, device="cuda")
    first = call()
    assert call()[2] == first[2] <= 4  # two orbital classes at most, for each of the two calls
    del held
    torch.cuda.empty_cache()
    call()
    again = call()
    assert again[2] == 7  # four kernels of the density, three of the elements
    for a, b in zip(first[:2], again[:2]):
        assert np.max(np.abs(a - b)) <= 1e-13 * np.max(np.abs(a))
