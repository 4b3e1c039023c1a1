"""FP64 density and grid matrix elements on the tensor cores (56-bit fixed point
in base-256 digits) against the oracle, at the sizes where the tiling changes:
one short window of rows, several row tiles, bricks of 512 and more rows, ragged
bricks, orbital counts of 4 to 18, columns of D far apart in size, Inf/NaN.

Tolerance: both sides round like FP64 sums of at most a few thousand terms, so
they agree to a few hundred units of 2^-53 of the largest value: 1e-13."""
import numpy as np
import pytest

import lcpgrid as L

pytestmark = pytest.mark.gpu

TOL = 1e-13
BASES = {4: (1, 1, 0), 9: (1, 1, 1), 13: (2, 2, 1), 18: (2, 2, 2)}


def _cell(natom, side, ngrid, orbitals, rc):
    from lcpgrid.workloads import synthetic_species
    from oracle import lcp_oracle as O
    rng = np.random.default_rng(natom * 100 + ngrid[0])
    paos = []
    for k, (no, r) in enumerate(zip(orbitals, rc)):
        nb = BASES[no]
        max_l = 2 if nb[2] else 1
        paos.append(synthetic_species(70 + k, max_l=max_l, num_basis=nb[:max_l + 1], rc=r))
    spe = [1 + a % len(paos) for a in range(natom)]
    pos = (np.arange(natom)[:, None] * np.array([[0.37, 0.61, 0.23]]) % 1.0) * side + rng.uniform(0, 0.3, (natom, 3))
    lat = np.diag([side, 1.1 * side, 0.95 * side])
    lat[1, 0] = 0.1 * side
    cut = [rc[s - 1] for s in spe]
    no = [orbitals[s - 1] for s in spe]
    u = L.UCell(1, lat, natom, spe, pos, cut, ngrid, [0, 0, 0], Total_NumOrbs=no)
    uo = O.UCell(1, lat, natom, spe, pos, cut, ngrid, [0, 0, 0], total_numorbs=no)
    orbs = L.Set_Orbitals_Grid(paos, u, ctx=L.Context(0))
    return u, uo, orbs, [orbs.data(a) for a in range(natom)], rng


CELLS = {
    "one_window": (1, 14.0, (9, 10, 11), (4,), (6.0,)),
    "mixed": (5, 9.0, (18, 21, 20), (13, 18, 4), (7.0, 6.0, 8.0)),
    "over_512_rows": (4, 6.4, (12, 14, 13), (18,), (8.0,)),
}


@pytest.mark.parametrize("name", list(CELLS))
def test_f64_tensor_against_oracle(name):
    from oracle import lcp_oracle as O
    u, uo, orbs, phi, rng = _cell(*CELLS[name])
    dm = rng.normal(size=u.Total_Hsize)
    v = rng.normal(size=u.NN)
    # the second D: each pair's block scaled by its neighbour atom, 2^0 down to 2^-40
    wide = dm.copy()
    for p, j in enumerate(u.MPI_natn):
        n = int(u.Total_NumOrbs[u.MPI_atom[p] - 1]) * int(u.Total_NumOrbs[j - 1])
        wide[u.block_offset[p]:u.block_offset[p] + n] *= 2.0 ** (-10 * (j - 1))
    for d in (dm, wide):
        rho = [np.zeros(u.NN)]
        L.Set_Density_Grid("off", u, orbs, [d], rho)
        ref = O.set_density_grid("off", uo, phi, [d])[0]
        assert np.max(np.abs(rho[0] - ref)) <= TOL * np.max(np.abs(ref))
    h = [np.zeros(u.Total_Hsize)]
    L.Calc_MatrixElements_dVH_Vxc_off(u, orbs, [v], h)
    ref = O.calc_matrix_elements(uo, phi, [v], 1)[0]
    assert np.max(np.abs(h[0] - ref)) <= TOL * np.max(np.abs(ref))
    # extreme scales of V take the general exponent path (2^-900 and 2^500, exact in the reference's ratio)
    for s in (2.0 ** -900, 2.0 ** 500):
        L.Calc_MatrixElements_dVH_Vxc_off(u, orbs, [v * s], h)
        assert np.max(np.abs(h[0] / s - ref)) <= TOL * np.max(np.abs(ref))


def test_f64_tensor_non_finite():
    u, uo, orbs, phi, rng = _cell(*CELLS["mixed"])
    v = rng.normal(size=u.NN)
    v[int(u.GridListAtom[0][len(u.GridListAtom[0]) // 2])] = np.nan
    h = [np.zeros(u.Total_Hsize)]
    L.Calc_MatrixElements_dVH_Vxc_off(u, orbs, [v], h)
    onsite = next(p for p in range(u.Nloop) if u.MPI_atom[p] == 1 and u.MPI_natn[p] == 1 and u.MPI_ncn[p] == 0)
    n = int(u.Total_NumOrbs[0]) ** 2
    assert np.isnan(h[0][u.block_offset[onsite]:u.block_offset[onsite] + n]).any()
    dm = rng.normal(size=u.Total_Hsize)
    dm[u.block_offset[onsite]] = np.inf
    rho = [np.zeros(u.NN)]
    L.Set_Density_Grid("off", u, orbs, [dm], rho)
    inside = np.zeros(u.NN, bool)
    inside[u.GridListAtom[0]] = True
    assert not np.isfinite(rho[0][inside]).all()
    assert np.isfinite(rho[0][~inside]).all()


@pytest.mark.parametrize("name", list(CELLS))
def test_f64_tensor_force_against_oracle(name):
    """The force term on the same tilings, rows of every image.  1e-10 of the
    largest component, as the oracle's gradient tables agree to 1e-12."""
    from lcpgrid.workloads import synthetic_species
    from oracle import lcp_oracle as O
    natom, _, _, orbitals, rc = CELLS[name]
    u, uo, orbs, phi, rng = _cell(*CELLS[name])
    paos = [synthetic_species(70 + k, max_l=2 if BASES[no][2] else 1, num_basis=BASES[no][:3 if BASES[no][2] else 2], rc=r)
            for k, (no, r) in enumerate(zip(orbitals, rc))]
    dm = [rng.normal(size=u.Total_Hsize) for _ in range(2)]
    v = [rng.normal(size=u.NN) for _ in range(2)]
    dorbs = L.Set_dOrbitals_Grid(paos, u, ctx=L.Context(0))
    grad = [[dorbs.data(a, k + 1) for a in range(natom)] for k in range(3)]
    ref = O.calc_force3("on", uo, phi, grad, v, dm)
    f = L.Force3_spin(paos, dorbs, v, dm, u)
    assert np.max(np.abs(f - ref)) <= 1e-10 * np.max(np.abs(ref))
    for _ in range(10):  # every sum is taken in a fixed order
        assert np.array_equal(f, L.Force3_spin(paos, dorbs, v, dm, u))
    # a potential and a D that are not finite reach the atoms that have them, and no others
    bad = v[0].copy()
    outside = np.ones(u.NN, bool)
    outside[u.GridListAtom[0]] = False
    bad[outside] = np.nan
    ref = O.calc_force3("on", uo, phi, grad, [bad, v[1]], dm)
    f = L.Force3_spin(paos, dorbs, [bad, v[1]], dm, u)
    assert (np.isfinite(f) == np.isfinite(ref)).all()
    onsite = next(p for p in range(u.Nloop) if u.MPI_atom[p] == 1 and u.MPI_natn[p] == 1 and u.MPI_ncn[p] == 0)
    d = dm[0].copy()
    d[u.block_offset[onsite]] = np.inf
    f = L.Force3_spin(paos, dorbs, v, [d, dm[1]], u)
    assert not np.isfinite(f[0]).any() and np.isfinite(f[1:]).all()


def test_f64_tables_go_with_the_orbital_tables():
    """release_fp64 frees the FP64 kernels' tables too: the same bytes whether they were made or not."""
    held = []
    for made in (True, False):
        u, _, orbs, _, rng = _cell(*CELLS["mixed"])
        job = L.GridStepJob(u, orbs, "off", "LDA", None, None, np.zeros(u.NN))
        if made:
            job.set_dm([rng.normal(size=u.Total_Hsize)])
            job.step()
        orbs.ctx.set_precision("bf16x3")
        orbs.release_fp64()
        held.append(job.footprint())
    assert held[0] == held[1]
