"""Orbital and gradient tables for every l (s to f, several radial functions
each), with grid points on the atom, on its axes and planes, inside the first
mesh point and at blocks' ends, against the oracle.  1e-12 of the largest
entry: both evaluate the same cubic of each interval, a few roundings apart."""
import numpy as np
import pytest

import lcpgrid as L
from oracle import lcp_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num_basis", [(1, 0, 0, 0), (2, 1, 1, 1), (0, 1, 0, 2), (1, 2)])
@pytest.mark.parametrize("r_lo", [1e-4, 0.9])
def test_tables_of_every_l(num_basis, r_lo):
    from lcpgrid.workloads import synthetic_species
    p = synthetic_species(5, max_l=len(num_basis) - 1, num_basis=num_basis, rc=5.0, nmesh=300, r_lo=r_lo, r_hi=4.5)
    no = sum((2 * l + 1) * n for l, n in enumerate(num_basis))
    lat = np.diag([9.0, 9.0, 9.0])
    lat[2, 0] = 1.5
    args = (lat, 2, [1, 1], np.array([[4.5, 4.5, 4.5], [1.03, 2.2, 3.1]]), [5.0, 5.0], (18, 18, 18), [0, 0, 0])
    u = L.UCell(1, *args, Total_NumOrbs=[no, no])
    uo = O.UCell(1, *args, total_numorbs=[no, no])
    op = [O.PAO(p.Spe_MaxL_Basis, p.Spe_Num_Basis, p.Spe_PAO_RV, p.Spe_PAO_RWF)]
    orbs = L.Set_dOrbitals_Grid([p], u, ctx=L.Context(0))
    ref = O.set_orbitals_grid(op, uo)
    dref = O.set_dorbitals_grid(op, uo)
    for a in range(2):
        for got, want in [(orbs.data(a), ref[a])] + [(orbs.data(a, k + 1), dref[k][a]) for k in range(3)]:
            assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
