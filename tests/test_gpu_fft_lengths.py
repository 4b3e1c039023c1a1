"""The FP64 Poisson solve at pencil lengths of every radix: 7 alone, repeated and
with other radices, 11 and 13 by the direct DFT, lengths of 1 and 2, fewer
pencils than a block takes and ragged last blocks; against the oracle.  1e-12 of
the largest value, as the other FP64 Poisson tests: a pencil's rounding grows
with the number of its stages, a few 2^-53 each."""
import numpy as np
import pytest

import lcpgrid as L
from helpers import FIX_LAT
from oracle import lcp_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng", [(7, 7, 7), (49, 14, 21), (35, 28, 42), (98, 63, 5), (1, 2, 7), (3, 343, 2),
                                (11, 26, 33), (105, 4, 126), (2, 1, 1)])
def test_poisson_lengths(ng):
    rec = 2 * np.pi * np.linalg.inv((FIX_LAT * 1.3).T)
    src = np.random.default_rng(sum(ng)).normal(size=int(np.prod(ng)))
    out = np.zeros(src.size)
    L.Solve_Poisson_xyz(ng, rec, src, out, ctx=L.Context(0))
    ref = O.solve_poisson_xyz(ng, rec, src)
    np.testing.assert_allclose(out, ref, rtol=0, atol=1e-12 * np.max(np.abs(ref)))
