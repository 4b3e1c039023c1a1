"""Grid matrix elements in split-BF16 where the packing of the bricks' rows
changes: chunks of 16 orbitals (rows as the images hold them), 1 to 13 orbitals
end to end with images across blocks, groups and windows, 18 = 16 + 2; bricks of
one block and of many; against the FP64 path, to the split's bound (1e-6 of the
largest element, as the other split-BF16 tests).

And sphere lists with grid points exactly on the cutoff, where the FP32 bound of
the distance leaves the FP64 test to decide: identical to the host's."""
import numpy as np
import pytest

import lcpgrid as L
from test_gpu_setup import _same_lists
from test_gpu_tc import H_TOL

pytestmark = pytest.mark.gpu

BASES = {1: (1,), 2: (2,), 4: (1, 1), 9: (1, 1, 1), 13: (2, 2, 1), 16: (3, 1, 2), 18: (2, 2, 2)}
CELLS = {
    "one_orbital": ((1,), 7, 9.0, (15, 16, 18), 6.0),
    "sixteen": ((16,), 3, 8.0, (16, 16, 16), 6.0),
    "thirteen": ((13,), 5, 8.0, (17, 16, 18), 7.0),
    "mixed": ((18, 1, 4, 13, 2, 9), 6, 9.0, (18, 20, 19), 6.5),
    "one_image": ((4,), 1, 30.0, (24, 24, 24), 6.0),
}


@pytest.mark.parametrize("name", list(CELLS))
def test_packed_rows(name):
    from lcpgrid.workloads import synthetic_species
    orbitals, natom, side, ngrid, rc = CELLS[name]
    rng = np.random.default_rng(len(name))
    paos = [synthetic_species(30 + k, max_l=len(BASES[no]) - 1, num_basis=BASES[no], rc=rc) for k, no in enumerate(orbitals)]
    spe = [1 + a % len(paos) for a in range(natom)]
    pos = (np.arange(natom)[:, None] * np.array([[0.37, 0.61, 0.23]]) % 1.0) * side
    lat = np.diag([side, 1.05 * side, 0.95 * side])
    u = L.UCell(1, lat, natom, spe, pos, [rc] * natom, ngrid, [0, 0, 0], Total_NumOrbs=[orbitals[s - 1] for s in spe])
    ctx = L.Context(0)
    orbs = L.Set_Orbitals_Grid(paos, u, ctx=ctx)
    v = [rng.normal(size=u.NN)]
    h = {}
    for precision in ("fp64", "bf16x3"):
        ctx.set_precision(precision)
        h[precision] = [np.zeros(u.Total_Hsize)]
        L.Calc_MatrixElements_dVH_Vxc_off(u, orbs, v, h[precision])
    assert np.max(np.abs(h["bf16x3"][0] - h["fp64"][0])) <= H_TOL * np.max(np.abs(h["fp64"][0]))


@pytest.mark.parametrize("shift", [0.0, 1e-13, 1e4])
def test_sphere_lists_at_the_cutoff(shift):
    """Spacing 1/2 and cutoffs 3, 6.5 and 5 (3-4-5 points): many points at the very cutoff."""
    lat = np.eye(3) * 12.0
    pos = np.array([[0.0, 0.0, 0.0], [3.0, 4.0, 5.0], [6.5, 0.5, 2.0]]) + shift
    args = (1, lat, 3, [1, 1, 1], pos, [3.0, 6.5, 5.0], (24, 24, 24), [shift] * 3)
    _same_lists(L.UCell(*args, Total_NumOrbs=[1, 1, 1]), L.UCell(*args, Total_NumOrbs=[1, 1, 1], device=True, ctx=L.Context(0)))
