"""FP64 density and matrix elements on the tensor cores where their fixed-point
grids could tell: potentials whose size at points that a pair does not hold is
out of proportion, many rows of like size and sign, columns of D far below the others'.

Tolerance, as for the other FP64 comparisons: both sides round like FP64 sums
of at most a few thousand terms, so they agree to a few hundred units of 2^-53
of the largest value of the compared part: 1e-13."""
import numpy as np
import pytest

import lcpgrid as L
from lcpgrid.pao import PAO
from lcpgrid.workloads import synthetic_species
from oracle import lcp_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-13


def _cell(lat, pos, spe, paos, ngrid, orbs_of=L.Set_Orbitals_Grid):
    """Product and oracle cells and the orbital tables (the oracle reads the product's values)."""
    cut = [paos[s - 1].Spe_Atom_Cut1 for s in spe]
    no = [paos[s - 1].Spe_Total_NumOrbs for s in spe]
    args = (1, np.asarray(lat, float), len(spe), spe, np.asarray(pos, float), cut, ngrid, [0, 0, 0])
    u = L.UCell(*args, Total_NumOrbs=no)
    orbs = orbs_of(paos, u, ctx=L.Context(0))
    return u, O.UCell(*args, total_numorbs=no), orbs, [orbs.data(a) for a in range(len(spe))]


def _sparse_cell():
    """Two overlapping atoms (13 and 4 orbitals) and a third apart, in a box with empty corners."""
    paos = [synthetic_species(81, rc=4.0), synthetic_species(82, max_l=1, num_basis=(1, 1), rc=4.5)]
    return _cell(np.diag([15.0, 15.5, 16.0]), [[4.0, 4.1, 4.2], [9.0, 4.5, 5.0], [10.5, 10.8, 11.0]], [1, 2, 1], paos,
                 (24, 25, 23))


def _counts(u):
    """Spheres (images included) that hold each grid point, and those of atom 1."""
    n = np.zeros(u.NN, int)
    for a in range(3):
        np.add.at(n, u.GridListAtom[a], 1)
    first = np.zeros(u.NN, int)
    np.add.at(first, u.GridListAtom[0], 1)
    return n, first


def _pair(u, atom, jatom):
    return [p for p in range(u.Nloop) if u.MPI_atom[p] == atom and u.MPI_natn[p] == jatom]


def _block(u, p):
    n = int(u.Total_NumOrbs[u.MPI_atom[p] - 1]) * int(u.Total_NumOrbs[u.MPI_natn[p] - 1])
    return slice(int(u.block_offset[p]), int(u.block_offset[p]) + n)


@pytest.mark.parametrize("value", [2.0 ** 6, 1e6, 1e12, 1e300, np.inf, np.nan])
@pytest.mark.parametrize("where", ["no_sphere", "first_sphere"])
def test_elements_do_not_see_v_outside_the_pair(where, value):
    """A pair's elements depend on V at the points that both its spheres hold, and on no other."""
    u, uo, orbs, phi = _sparse_cell()
    n, first = _counts(u)
    v = np.random.default_rng(7).normal(size=u.NN)
    at = np.flatnonzero(n == 0 if where == "no_sphere" else (n == 1) & (first == 1))
    if where == "first_sphere":
        at = at[::5]
    assert at.size > 100
    bad = v.copy()
    bad[at] = value
    h = [np.zeros(u.Total_Hsize)]
    L.Calc_MatrixElements_dVH_Vxc_off(u, orbs, [bad], h)
    with np.errstate(invalid="ignore"):
        ref = O.calc_matrix_elements(uo, phi, [bad], 1)[0]
    same = O.calc_matrix_elements(uo, phi, [v], 1)[0]
    own = _pair(u, 1, 1)[0]  # the self pair of the first atom comes first
    for p in range(u.Nloop):
        b = _block(u, p)
        if where == "first_sphere" and p == own:
            assert np.array_equal(np.isfinite(h[0][b]), np.isfinite(ref[b]))
            if np.isfinite(value):
                assert np.max(np.abs(h[0][b] - ref[b])) <= TOL * np.max(np.abs(ref[b]))
            continue
        assert np.max(np.abs(h[0][b] - same[b])) <= TOL * np.max(np.abs(same[b])) + 1e-300, (p, value)


def test_elements_of_one_infinite_point():
    """One infinite V inside two overlapping spheres: infinities of the oracle's signs, nothing elsewhere."""
    u, uo, orbs, phi = _sparse_cell()
    n, first = _counts(u)
    v = np.random.default_rng(8).normal(size=u.NN)
    v[np.flatnonzero((n == 2) & (first == 1))[3]] = -np.inf
    h = [np.zeros(u.Total_Hsize)]
    L.Calc_MatrixElements_dVH_Vxc_off(u, orbs, [v], h)
    with np.errstate(invalid="ignore"):
        ref = O.calc_matrix_elements(uo, phi, [v], 1)[0]
    ok = np.isfinite(ref)
    assert not ok.all() and np.array_equal(np.isfinite(h[0]), ok)
    assert np.array_equal(h[0][np.isinf(ref)], ref[np.isinf(ref)])
    assert np.max(np.abs(h[0][ok] - ref[ok])) <= TOL * np.max(np.abs(ref[ok]))


@pytest.mark.parametrize("shift", [6, 9, 40, 100, 140])
def test_density_of_an_atom_with_a_small_d(shift):
    """An atom whose D is 2^-shift of its neighbour's keeps its own accuracy where it is alone."""
    u, uo, orbs, phi = _sparse_cell()
    rng = np.random.default_rng(shift)
    dm = np.zeros(u.Total_Hsize)
    for p in range(u.Nloop):
        if u.MPI_atom[p] == u.MPI_natn[p]:
            dm[_block(u, p)] = rng.normal(size=dm[_block(u, p)].size) * (2.0 ** -shift if u.MPI_atom[p] == 2 else 1.0)
    rho = [np.zeros(u.NN)]
    L.Set_Density_Grid("off", u, orbs, [dm], rho)
    ref = O.set_density_grid("off", uo, phi, [dm])[0]
    n, _ = _counts(u)
    second = np.zeros(u.NN, bool)
    second[u.GridListAtom[1]] = True
    alone = second & (n == 1)
    for part in (alone, ~second):
        assert np.max(np.abs(rho[0] - ref)[part]) <= TOL * np.max(np.abs(ref[part]))


def _flat(nfun, values):
    """nfun s functions of constant value inside the cutoff."""
    rv = np.exp(np.linspace(np.log(1e-4), np.log(7.0), 400))
    return PAO(0, [nfun], rv, [[np.full(rv.size, float(x)) for x in values]], Spe_Atom_Cut1=6.0)


def _flat_cell(nfun, values, side=5.0, n=12):
    """At every point all orbitals of dozens of images count alike: 160 to 900 rows at a brick."""
    return _cell(np.diag([side] * 3), [[0.1, 0.2, 0.3], [2.0, 2.6, 1.1]], [1, 1], [_flat(nfun, values)], (n, n, n))


@pytest.mark.parametrize("nfun", [2, 8, 16, 32])
def test_density_of_many_like_rows(nfun):
    """Rows and D of one sign and nearly one size, up to the most rows that a brick
    takes: the sums over rows and columns are as large as they can be."""
    rng = np.random.default_rng(nfun)
    u, uo, orbs, phi = _flat_cell(nfun, np.ones(nfun))
    dm = np.ones(u.Total_Hsize)
    rho = [np.zeros(u.NN)]
    L.Set_Density_Grid("off", u, orbs, [dm], rho)
    ref = O.set_density_grid("off", uo, phi, [dm])[0]
    assert np.max(np.abs(rho[0] - ref) / ref) <= TOL
    v = 1.0 + 0.1 * rng.uniform(size=u.NN)
    h = [np.zeros(u.Total_Hsize)]
    L.Calc_MatrixElements_dVH_Vxc_off(u, orbs, [v], h)
    ref = O.calc_matrix_elements(uo, phi, [v], 1)[0]
    assert np.max(np.abs(h[0] - ref)) <= TOL * np.max(np.abs(ref))


def test_density_of_large_digits():
    """Up to 830 rows that count at one point, with phi's and D's two leading base-256
    digits large, odd and different from row to row: no sum of digit products may lose a unit."""
    rng = np.random.default_rng(5)
    phi0, d0 = 0.5 * (125 + 125 / 256) / 128, (63 + 120 / 256) / 128
    values = phi0 * 2 * np.sqrt(np.pi) * (1 + 2e-5 * rng.uniform(-1, 1, 32))
    u, uo, orbs, phi = _flat_cell(32, values, 4.4, 24)
    dm = d0 * (1 + 2e-5 * rng.uniform(-1, 1, u.Total_Hsize))
    l0 = orbs.ctx.launch_count
    rho = [np.zeros(u.NN)]
    L.Set_Density_Grid("off", u, orbs, [dm], rho)
    assert orbs.ctx.launch_count > l0 + 1  # the tensor-core kernels
    f = phi[0][:, 0]
    ref = np.zeros(u.NN)
    for p in range(u.Nloop):
        np.add.at(ref, uo.GridListAtom[u.MPI_atom[p] - 1][uo.MPI_GListTAtoms1[p]], f @ dm[_block(u, p)].reshape(32, 32) @ f)
    assert np.max(np.abs(rho[0] - ref) / ref) <= TOL


@pytest.mark.parametrize("value", [2.0 ** 6, 1e6, 1e12, 1e100])
def test_density_of_one_large_element_of_d(value):
    """An element of D between two atoms counts at the points that both hold, and
    takes no digits from the others."""
    u, uo, orbs, phi = _sparse_cell()
    dm = np.random.default_rng(11).normal(size=u.Total_Hsize)
    dm[_block(u, _pair(u, 1, 2)[0])][7:8] = value
    rho = [np.zeros(u.NN)]
    L.Set_Density_Grid("off", u, orbs, [dm], rho)
    ref = O.set_density_grid("off", uo, phi, [dm])[0]
    n, _ = _counts(u)
    for part in (n == 1, n > 1):
        assert np.max(np.abs(rho[0] - ref)[part]) <= TOL * np.max(np.abs(ref[part]))


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_density_of_a_d_that_is_not_finite(value):
    """An element of D between two atoms reaches the points that both hold, and no other."""
    u, uo, orbs, phi = _sparse_cell()
    dm = np.random.default_rng(9).normal(size=u.Total_Hsize)
    dm[_block(u, _pair(u, 1, 2)[0])][5:6] = value
    rho = [np.zeros(u.NN)]
    L.Set_Density_Grid("off", u, orbs, [dm], rho)
    with np.errstate(invalid="ignore"):
        ref = O.set_density_grid("off", uo, phi, [dm])[0]
    ok = np.isfinite(ref)
    assert not ok.all() and np.array_equal(np.isfinite(rho[0]), ok)
    assert np.max(np.abs(rho[0][ok] - ref[ok])) <= TOL * np.max(np.abs(ref[ok]))


def test_radial_functions_that_are_not_finite():
    """A radial function with a NaN marks the results of the points in that shell, as the oracle's are."""
    paos = [synthetic_species(81, rc=4.0), synthetic_species(82, max_l=1, num_basis=(1, 1), rc=4.5)]
    paos[1].Spe_PAO_RWF[1][0][int(np.searchsorted(paos[1].Spe_PAO_RV, 4.2))] = np.nan
    lat, pos = np.diag([15.0, 15.5, 16.0]), [[4.0, 4.1, 4.2], [9.0, 4.5, 5.0], [10.5, 10.8, 11.0]]
    u, uo, orbs, phi = _cell(lat, pos, [1, 2, 1], paos, (24, 25, 23), L.Set_dOrbitals_Grid)
    assert not all(np.isfinite(x).all() for x in phi)
    rng = np.random.default_rng(10)
    dm, v = rng.normal(size=u.Total_Hsize), rng.normal(size=u.NN)
    rho, h = [np.zeros(u.NN)], [np.zeros(u.Total_Hsize)]
    L.Set_Density_Grid("off", u, orbs, [dm], rho)
    L.Calc_MatrixElements_dVH_Vxc_off(u, orbs, [v], h)
    f = L.Force3_nospin(paos, orbs, [v], [dm], u)
    grad = [[orbs.data(a, k + 1) for a in range(3)] for k in range(3)]
    with np.errstate(invalid="ignore"):
        refs = [O.set_density_grid("off", uo, phi, [dm])[0], O.calc_matrix_elements(uo, phi, [v], 1)[0],
                O.calc_force3("off", uo, phi, grad, [v], [dm])]
    for got, ref, tol in zip((rho[0], h[0], f), refs, (TOL, TOL, 1e-10)):
        ok = np.isfinite(ref)
        assert not ok.all() and np.array_equal(np.isfinite(got), ok)
        assert np.max(np.abs(got[ok] - ref[ok]), initial=0.0) <= tol * np.max(np.abs(ref[ok]), initial=1.0)
