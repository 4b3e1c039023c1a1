"""GGA-PBE with a caller's own gradient stencil: Diff_Coef is the caller's, and
weights that are not odd under inversion count as they are.  Tolerance of the
other GGA comparisons: 1e-11 of the largest magnitude."""
import numpy as np
import pytest

import lcpgrid as L
from oracle import lcp_oracle as O
from test_gpu_gga import NG, SKEW, close, smooth_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spin", ["off", "on"])
@pytest.mark.parametrize("pcc_on", [True, False])
def test_weights_with_an_even_part(spin, pcc_on):
    ns = 1 if spin == "off" else 2
    pcc, rho = smooth_fields(NG, ns, seed=11 + ns)
    gl = O.glatvecs_of(SKEW, NG)
    rng = np.random.default_rng(3)
    xf = L.XC_Func("GGA-PBE", spin, ns, NG, gl, ctx=L.Context(0))
    big = max(np.max(np.abs(c)) for c in xf.Diff_Coef)
    xf.Diff_Coef = [c + 0.1 * big * rng.uniform(-1, 1, 27) for c in xf.Diff_Coef]
    p = pcc if pcc_on else np.zeros_like(pcc)
    L.Set_XC_Grid(xf, p if pcc_on else None, rho)
    vref, dref, eref = O.set_xc_grid_gga(spin, NG, p, rho, [c.copy() for c in xf.Diff_Coef])
    for s in range(ns):
        close(xf.Vxc_Grid[s], vref[s])
        for a in range(3):
            close(xf.dDensity_Grid[s][a], dref[s][a])
            close(xf.dEXC_dGD[s][a], eref[s][a])
