"""The grid-step work that users of lcpgrid have it do, as cases for timing.

An SCF program calls the library in a few ways, and each case is one of them
with everything the program does per call:

step      the device-resident grid step (GridStepJob): a new density matrix in,
          the step, energies and H out; one SCF iteration;
batch     the same step for many cells at once (Batch);
dropin    the reference's own call sequence of one SCF iteration with host
          arrays: density, Poisson, xc, potential, matrix elements;
potential the density-to-potential part alone with host arrays, and its
          energies (what a density-mixing loop and a post-processing run call);
newgeom   the first iteration on new atom positions: grid lists, orbital
          tables, job and one step (what every MD or relaxation move costs);
force     the grid force term with its gradient tables, once per move.

Cells: the Si cells of diamond structure at the grid spacing of the 64-atom 96^3
cell, MX2 monolayers with vacuum, and random mixed cells (1-3 species of 4, 9,
13 or 18 orbitals, cutoffs of 6-9 bohr) on the 150 Ry grids, whose sizes are odd
and ragged.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("lcpaodft.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

NSPIN = {"off": 1, "on": 2, "nc": 4}
_CTX = {}  # a program keeps one context per precision


def _context(prec):
    import lcpgrid as L
    if prec not in _CTX:
        _CTX[prec] = L.Context(0, prec)
    return _CTX[prec]


# ---------------------------------------------------------------- cases

def _step(name, cell, natom, prec, spin="off", xc="LDA", kind="step"):
    return {"name": name, "kind": kind, "cell": cell, "natom": natom, "prec": prec, "spin": spin, "xc": xc}


def listed():
    return [
        # one SCF iteration of a primitive cell: what a k-point or convergence study
        # runs thousands of, bound by latency and launches
        _step("si2_fp64", "si2", 2, "fp64"),
        _step("si2_bf16x3", "si2", 2, "bf16x3"),
        # the 64-atom supercell (a defect or phonon cell), drop-in and split-BF16 form
        _step("si64_fp64", "si", 64, "fp64"),
        _step("si64_bf16x3", "si", 64, "bf16x3"),
        # a magnetic or spin-polarised slab with vacuum, 13- and 18-orbital species
        _step("mx2_108_on_bf16x3", "mx2", 108, "bf16x3", "on", "LSDA"),
        # GGA on a mixed cell with a ragged grid, spin-polarised, drop-in precision
        _step("rand20_gga_on_fp64", "rand", 20, "fp64", "on", "GGA_PBE"),
        # non-collinear spin: four channels of D, V and H
        _step("si8_nc_bf16x3", "si", 8, "bf16x3", "nc", "LSDA"),
        # the reference's host-array call sites, unchanged
        _step("dropin_rand12_on", "rand", 12, "fp64", "on", "LSDA", kind="dropin"),
        # density to potential and energies on a large grid with odd factors
        {"name": "potential_gga_105x98x126", "kind": "potential", "n1": 105, "n2": 98, "n3": 126, "spin": "off",
         "xc": "GGA_PBE"},
        # an MD move: everything that depends on the positions, then one iteration
        _step("newgeom_si32_fp64", "randsi", 32, "fp64", kind="newgeom"),
        # forces of an MD move
        _step("force_randsi16", "randsi", 16, "fp64", kind="force"),
        # a screening run: many small mixed cells stepped together
        {"name": "batch16_bf16x3", "kind": "batch", "cells": 16, "nmax": 24, "pool": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# grid sizes are products of 2, 3, 5 and 7, as Calc_Ngrid chooses them
_SMOOTH = sorted({2 ** p * 3 ** q * 5 ** r * 7 ** t for p in range(8) for q in range(5) for r in range(3)
                  for t in range(3)})


def draw(rng):
    kind = rng.choice(["step", "step", "step", "dropin", "potential", "newgeom", "force", "batch"])
    if kind == "potential":
        spin = rng.choice(["off", "on"])
        n = [min(_SMOOTH, key=lambda m, x=_log_int(rng, 20, 110): abs(m - x)) for _ in range(3)]
        return {"kind": kind, "n1": n[0], "n2": n[1], "n3": n[2], "spin": spin,
                "xc": rng.choice(["GGA_PBE", "LDA" if spin == "off" else "LSDA"])}
    if kind == "batch":
        return {"kind": kind, "cells": rng.randint(2, 16), "nmax": _log_int(rng, 6, 24), "pool": rng.randint(1, 999)}
    if kind == "step":
        cell = rng.choice(["randsi", "rand", "rand", "mx2"])
        prec = rng.choice(["fp64", "bf16x3"])
        spin = rng.choice(["off", "on", "nc"])
        most = {"off": 24, "on": 12, "nc": 6}[spin] * (1 if prec == "fp64" else 2)
        natom = 3 * rng.choice([1, 4] if prec == "fp64" else [1, 4, 9]) if cell == "mx2" else _log_int(rng, 2, most)
    else:
        cell, prec = rng.choice(["randsi", "rand"]), "fp64"
        spin = rng.choice(["off", "on"])
        natom = _log_int(rng, 2, {"dropin": 20, "newgeom": 24, "force": 12}[kind])
    xc = rng.choice(["GGA_PBE", "LDA" if spin == "off" else "LSDA"])
    out = _step("", cell, natom, prec, spin, xc, kind=kind)
    del out["name"]
    return out


# ---------------------------------------------------------------- cells

def _cell(case, seed):
    """Host inputs of a case's cell.  The lattice and species are the case's; the
    seed shifts all atoms against the grid, so that every neighbour list stays
    the same length."""
    from lcpgrid import workloads as W
    kind, natom = case["cell"], case["natom"]
    rng = np.random.default_rng(1000003 * seed + natom)
    if kind == "si2":
        lat, pos = W.si2_primitive()
        paos = [W.synthetic_species(1234)]
        spe, ngrid = [1] * 2, (24, 24, 24)
    elif kind == "si":
        nrep = round((natom / 8) ** (1 / 3))
        lat, pos = W.si_supercell(nrep)
        paos = [W.synthetic_species(1234)]
        spe, ngrid = [1] * natom, (48 * nrep,) * 3
    elif kind == "mx2":
        nrep = round((natom / 3) ** 0.5)
        wl = W.mx2_monolayer(nrep=nrep, ngrid=(18 * nrep, 18 * nrep, 320))
        lat, pos, paos, spe, ngrid = wl["latvecs"], wl["gxyz"], wl["paos"], wl["atom2spe"], wl["ngrid"]
    elif kind == "randsi":
        lat, pos, _ = W.random_si_cell(natom, 77 + natom)
        paos = [W.synthetic_species(1234)]
        spe, ngrid = [1] * natom, W.calc_ngrid(150.0, lat)
    else:
        r = np.random.default_rng(4242 + natom)
        nspe = 1 + natom % 3
        paos = []
        for _ in range(nspe):
            rc = float(W.BATCH_CUTOFFS[r.integers(len(W.BATCH_CUTOFFS))])
            nb = W.BATCH_BASES[list(W.BATCH_BASES)[r.integers(len(W.BATCH_BASES))]]
            max_l = 2 if nb[2] else 1
            paos.append(W.synthetic_species(int(r.integers(1 << 30)), max_l=max_l, num_basis=nb[:max_l + 1], rc=rc))
        lat, pos, _ = W.random_si_cell(natom, 977 + natom)
        spe = [1 + i % nspe for i in range(natom)]
        ngrid = W.calc_ngrid(150.0, lat)
    pos = np.asarray(pos) + rng.uniform(0.0, 1.0, size=3)
    return {"lat": np.asarray(lat), "pos": pos, "paos": paos, "spe": spe, "ngrid": tuple(ngrid),
            "cut": [paos[s - 1].Spe_Atom_Cut1 for s in spe], "no": [paos[s - 1].Spe_Total_NumOrbs for s in spe]}


def _ucell(c, spin, ctx):
    import lcpgrid as L
    args = (NSPIN[spin], c["lat"], len(c["spe"]), c["spe"], c["pos"], c["cut"], c["ngrid"], [0.0, 0.0, 0.0])
    try:
        return L.UCell(*args, Total_NumOrbs=c["no"], device=True, ctx=ctx)
    except L.LCPError:  # cells so small that the device build refuses them
        return L.UCell(*args, Total_NumOrbs=c["no"], ctx=ctx)


def _gamma_matrices(no, seed, spin):
    """Gamma-point density matrices of the channels: PSD, two electrons per atom
    and spin, as the eigenvectors of a diagonalisation give them."""
    rng = np.random.default_rng(seed + 31)
    norb = int(sum(no))
    nocc = max(1, norb // 4)
    if spin == "nc":
        C = rng.normal(size=(2 * norb, nocc)) + 1j * rng.normal(size=(2 * norb, nocc))
        M = C @ C.conj().T
        M *= 4.0 * len(no) / np.trace(M).real
        return [M[:norb, :norb].real, M[norb:, norb:].real, M[:norb, norb:].real, M[:norb, norb:].imag]
    out = []
    for _ in range(NSPIN[spin]):
        C = rng.normal(size=(norb, nocc))
        M = C @ C.T
        out.append(M * (2.0 * len(no) / np.trace(M)))
    return out


def _pinned(n):
    t = torch.empty(int(n), dtype=torch.float64, pin_memory=True)
    t.zero_()
    return t.numpy()


def _pair_blocks(u, mats, no):
    """The matrices in the library's flat pair-block layout, in pinned memory."""
    off = np.concatenate([[0], np.cumsum(no)])
    out = [_pinned(u.Total_Hsize) for _ in mats]
    for p, (a, b) in enumerate(zip(u.MPI_atom, u.MPI_natn)):
        i0, i1, j0, j1 = off[a - 1], off[a], off[b - 1], off[b]
        o, n = u.block_offset[p], (i1 - i0) * (j1 - j0)
        for d, m in zip(out, mats):
            d[o:o + n] = m[i0:i1, j0:j1].ravel()
    return out


def _vna(c, seed):
    from lcpgrid import workloads as W
    return W.smooth_vna(c["ngrid"], c["lat"], seed + 17)


def _potential_inputs(case, seed):
    """Smooth positive densities (a few Gaussians per cell over a low
    background), a partial-core and an atomic density, on a skewed cell."""
    n = (case["n1"], case["n2"], case["n3"])
    rng = np.random.default_rng(seed + 5)
    lat = np.diag([0.21 * n[0], 0.21 * n[1], 0.21 * n[2]])
    lat[1, 0], lat[2, 1] = 0.05 * lat[1, 1], -0.04 * lat[2, 2]
    ax = [np.arange(m) / m for m in n]

    def bumps(count, amp, width, floor):
        rho = np.full(n, floor)
        for _ in range(count):
            x0 = rng.uniform(size=3)
            w = [width / lat[d, d] for d in range(3)]
            g = [np.exp(-0.5 * ((np.mod(ax[d] - x0[d] + 0.5, 1.0) - 0.5) / w[d]) ** 2) for d in range(3)]
            rho += amp * rng.uniform(0.5, 1.5) * g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :]
        return np.ascontiguousarray(rho.reshape(-1))
    den = [bumps(8, 0.2, 1.2, 1e-3) for _ in range(NSPIN[case["spin"]])]
    return {"lat": lat, "n": n, "den": den, "pcc": bumps(4, 0.1, 0.5, 1e-6), "aden": bumps(8, 0.15, 1.2, 5e-4)}


# ---------------------------------------------------------------- prepare and run

def prepare(case, seed):
    import lcpgrid as L
    kind = case["kind"]
    if kind == "potential":
        ctx = _context("fp64")
        s = _potential_inputs(case, seed)
        nn, nch = int(np.prod(s["n"])), NSPIN[case["spin"]]
        gl = s["lat"] / np.array(s["n"])[:, None]
        mix = L.Rhor_Mixing(s["n"], s["lat"], ctx=ctx)
        mix.GridVol = abs(np.linalg.det(s["lat"])) / nn
        s.update(case=case, ctx=ctx, mix=mix, xcf=L.XC_Func(case["xc"], case["spin"], nch, s["n"], gl, ctx=ctx),
                 dvh=np.zeros(nn), vpot=[np.zeros(nn) for _ in range(nch)])
        return s
    if kind == "batch":
        from lcpgrid import workloads as W
        ctx = _context("bf16x3")
        jobs, dms, hs = [], [], []
        for k, wl in enumerate(W.batch_pool(case["cells"], seed=4242 + case["pool"], nmin=2, nmax=case["nmax"])):
            c = {"lat": wl["latvecs"], "pos": wl["gxyz"], "paos": wl["paos"], "spe": wl["atom2spe"],
                 "ngrid": wl["ngrid"], "cut": wl["cut"], "no": wl["numorbs"]}
            u = _ucell(c, "off", ctx)
            orbs = L.Set_Orbitals_Grid(c["paos"], u, ctx=ctx)
            job = L.GridStepJob(u, orbs, "off", "LDA", None, None, _vna(c, seed + k))
            job.prepare()
            jobs.append(job)
            dms.append(_pair_blocks(u, _gamma_matrices(c["no"], seed + 100 * k, "off"), c["no"]))
            hs.append([_pinned(u.Total_Hsize)])
        return {"case": case, "batch": L.Batch(jobs), "jobs": jobs, "dm": dms, "h": hs}
    ctx = _context(case["prec"])
    spin = case["spin"]
    c = _cell(case, seed)
    u = _ucell(c, spin, ctx)
    s = {"case": case, "ctx": ctx, "c": c, "u": u, "vna": _vna(c, seed),
         "dm": _pair_blocks(u, _gamma_matrices(c["no"], seed, spin), c["no"])}
    if kind == "newgeom":  # the positions are new: the run makes everything that follows from them
        s["h"] = [_pinned(u.Total_Hsize) for _ in s["dm"]]
        del s["u"]
        return s
    s["orbs"] = L.Set_Orbitals_Grid(c["paos"], u, ctx=ctx)
    if kind == "step":
        s["job"] = L.GridStepJob(u, s["orbs"], spin, case["xc"], None, None, s["vna"])
        s["job"].prepare()
        s["e"] = _pinned(5)
        s["h"] = [_pinned(u.Total_Hsize) for _ in s["dm"]]
    elif kind == "dropin":
        nch = NSPIN[spin]
        s["mix"] = L.Rhor_Mixing(c["ngrid"], c["lat"], ctx=ctx)
        s["xcf"] = L.XC_Func(case["xc"], spin, nch, c["ngrid"], c["lat"] / np.array(c["ngrid"])[:, None], ctx=ctx)
        s["den"], s["vpot"] = ([np.zeros(u.NN) for _ in range(nch)] for _ in range(2))
        s["dvh"] = np.zeros(u.NN)
        s["h"] = [np.zeros(u.Total_Hsize) for _ in range(nch)]
        s["aden"] = np.full(u.NN, 0.5 * 4.0 * u.Natom / (u.NN * u.GridVol))
        s["pcc"] = np.zeros(u.NN)
    else:
        s["v"] = [s["vna"] * (1.0 + 0.1 * k) for k in range(NSPIN[spin])]
    return s


def run(s):
    import lcpgrid as L
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        s["job"].set_dm(s["dm"])
        s["job"].step()
        s["job"].energies_async(s["e"])
        return {"H": s["job"].hks(s["h"]), "energies": s["e"]}
    if kind == "batch":
        for job, dm in zip(s["jobs"], s["dm"]):
            job.set_dm(dm)
        s["batch"].step()
        e = s["batch"].energies()
        for job, h in zip(s["jobs"], s["h"]):
            job.hks(h)
        return {"H": s["h"], "energies": e}
    spin = case["spin"]
    if kind == "potential":
        L.Solve_Poisson(spin, s["mix"], s["den"], s["aden"], s["dvh"])
        L.Set_XC_Grid(s["xcf"], s["pcc"], s["den"])
        L.Set_Vpot_Grid(s["xcf"], s["dvh"], s["vpot"])
        eh1 = L.Calc_EH1(spin, s["mix"].GridVol, s["aden"], s["den"], s["dvh"], ctx=s["ctx"])
        exc = L.Calc_EXC1(spin, case["xc"], s["mix"], s["aden"], s["pcc"], s["den"])
        return {"dVH": s["dvh"], "V": s["vpot"], "EH1": np.array([eh1]), "EXC": exc[:NSPIN[spin]]}
    c = s["c"]
    if kind == "dropin":
        L.Set_Density_Grid(spin, s["u"], s["orbs"], s["dm"], s["den"])
        L.Solve_Poisson(spin, s["mix"], s["den"], s["aden"], s["dvh"])
        L.Set_XC_Grid(s["xcf"], s["pcc"], s["den"])
        L.Set_Vpot_Grid(s["xcf"], s["dvh"], s["vpot"])
        (L.Calc_MatrixElements_dVH_Vxc_on if spin == "on" else L.Calc_MatrixElements_dVH_Vxc_off)(
            s["u"], s["orbs"], s["vpot"], s["h"])
        return {"rho": s["den"], "V": s["vpot"], "H": s["h"]}
    if kind == "newgeom":
        u = _ucell(c, spin, s["ctx"])
        job = L.GridStepJob(u, L.Set_Orbitals_Grid(c["paos"], u, ctx=s["ctx"]), spin, case["xc"], None, None, s["vna"])
        job.set_dm(s["dm"])
        job.step()
        return {"energies": job.energies(), "H": job.hks(s["h"])}
    return (L.Force3_spin if spin == "on" else L.Force3_nospin)(c["paos"], s["orbs"], s["v"], s["dm"], s["u"])


# ---------------------------------------------------------------- work

def _geometry_work(case):
    """(grid points, folded-pair flops of one contraction, H entries, sphere
    points x orbitals) of a cell, from the spheres' and lenses' volumes."""
    c = _cell(case, 1)
    nn = float(np.prod(c["ngrid"]))
    dv = abs(np.linalg.det(c["lat"])) / nn
    rc, no = np.array(c["cut"]), np.array(c["no"], float)
    orbs_per_point = float((4 / 3 * math.pi * rc ** 3 * no).sum()) / (dv * nn)
    pairs = sum(4 / 3 * math.pi * (a + b) ** 3 / (dv * nn) * p * q for a, p in zip(rc, no) for b, q in zip(rc, no))
    return nn, nn * orbs_per_point ** 2, float(pairs), nn * orbs_per_point


def work(case):
    kind = case["kind"]
    if kind == "batch":
        from lcpgrid import workloads as W
        nb = nf = 0.0
        for wl in W.batch_pool(case["cells"], seed=4242 + case["pool"], nmin=2, nmax=case["nmax"]):
            nn = float(np.prod(wl["ngrid"]))
            vol = abs(np.linalg.det(wl["latvecs"]))
            opp = sum(4 / 3 * math.pi * r ** 3 * n for r, n in zip(wl["cut"], wl["numorbs"])) / vol
            nf += 2 * nn * opp ** 2
            nb += 8 * nn * opp + 8 * 6 * nn
        return {"bytes": nb, "flops": nf}
    nch = NSPIN[case["spin"]]
    if kind == "potential":
        nn = float(case["n1"] * case["n2"] * case["n3"])
        return {"bytes": 8 * nn * (2 * nch + 3), "flops": nn * (10 * math.log2(nn) + 150 * nch)}
    nn, pair, hsize, table = _geometry_work(case)
    if kind == "force":
        return {"bytes": 8 * (4 * table + nch * (hsize + nn)), "flops": nch * 2 * pair}
    once = table * (1 if kind != "newgeom" else 2)
    return {"bytes": float(8 * (once + 2 * nch * hsize + 3 * nch * nn)),
            "flops": nch * (2 * pair + 150 * nn) + 10 * nn * math.log2(nn)}


# ---------------------------------------------------------------- the same in plain torch, 64 bits

def _phi(pao, x, y, z):
    """Orbitals of a species at displacements: the reference's 4-point Hermite
    spline of each radial function times the real spherical harmonics."""
    dev = x.device
    rv = torch.as_tensor(pao.Spe_PAO_RV, device=dev)
    n = rv.numel()
    R = torch.sqrt(x * x + y * y + z * z)
    m = torch.searchsorted(rv, R.detach().contiguous()).clamp(2, n - 2)
    h1, h2, h3 = rv[m - 1] - rv[m - 2], rv[m] - rv[m - 1], rv[m + 1] - rv[m]
    y1, y2 = (R - rv[m - 1]) / h2, (R - rv[m]) / h2
    ux, uy, uz = x / R, y / R, z / R
    s3, s5, s15 = math.sqrt(3 / 4 / math.pi), 0.25 * math.sqrt(5 / math.pi), 0.5 * math.sqrt(15 / math.pi)
    ang = [[torch.full_like(R, 0.5 * math.sqrt(1 / math.pi))],
           [s3 * ux, s3 * uy, s3 * uz],
           [s5 * (3 * uz * uz - 1), 0.5 * s15 * (ux * ux - uy * uy), s15 * ux * uy, s15 * ux * uz, s15 * uy * uz]]
    out = []
    for l in range(pao.Spe_MaxL_Basis + 1):
        for p in range(pao.Spe_Num_Basis[l]):
            w = torch.as_tensor(pao.Spe_PAO_RWF[l][p], device=dev)
            f1, f2, f3, f4 = w[m - 2], w[m - 1], w[m], w[m + 1]
            g1 = (f3 - f2) * (h1 / h2 / (h1 + h2)) + (f2 - f1) * (h2 / h1 / (h1 + h2))
            g2 = (f4 - f3) * (h2 / h3 / (h2 + h3)) + (f3 - f2) * (h3 / h2 / (h2 + h3))
            f = y2 * y2 * (3 * f2 + h2 * g1 + (2 * f2 + h2 * g1) * y2) + \
                y1 * y1 * (3 * f3 - h2 * g2 - (2 * f3 - h2 * g2) * y1)
            out += [f * a for a in ang[l]]
    return torch.stack(out)


def _images(c, atom, pts, corners, grad=False):
    """(image cell, point indices, values [orbital, point], gradients) of an
    atom's images whose spheres reach points of the home cell."""
    lat, rc = c["lat"], c["cut"][atom]
    rec = np.linalg.inv(lat)                      # fractional = cartesian @ rec
    span = rc * np.linalg.norm(rec, axis=0)
    f = c["pos"][atom] @ rec
    lo, hi = np.floor(-span - f).astype(int), np.ceil(1 + span - f).astype(int)
    pao = c["paos"][c["spe"][atom] - 1]
    for i in range(lo[0], hi[0] + 1):
        for j in range(lo[1], hi[1] + 1):
            for k in range(lo[2], hi[2] + 1):
                at = torch.as_tensor(c["pos"][atom] + np.array([i, j, k]) @ lat, device=pts.device)
                d = pts - at
                sel = torch.nonzero((d * d).sum(1) <= rc * rc)[:, 0]
                if sel.numel():
                    d = d[sel]
                    if not grad:
                        yield (i, j, k), sel, _phi(pao, d[:, 0], d[:, 1], d[:, 2]), None
                    else:
                        one, zero = torch.ones_like(d[:, 0]), torch.zeros_like(d[:, 0])
                        g, v = [], None
                        for ax in range(3):
                            v, t = torch.func.jvp(lambda a, b, e: _phi(pao, a, b, e), (d[:, 0], d[:, 1], d[:, 2]),
                                                  tuple(one if ax == q else zero for q in range(3)))
                            g.append(t)
                        yield (i, j, k), sel, v, g


def _points(c):
    n = c["ngrid"]
    f = [torch.arange(m, device="cuda", dtype=torch.float64) / m for m in n]
    lat = torch.as_tensor(c["lat"], device="cuda")
    fr = torch.stack(torch.meshgrid(*f, indexing="ij"), -1).reshape(-1, 3)
    return fr @ lat


def _poisson(src, n, lat):
    a = torch.fft.fftn(src.reshape(n).to(torch.complex128))
    rec = torch.as_tensor(2 * math.pi * np.linalg.inv(lat.T), device=src.device)
    s = [torch.arange(m, device=src.device) for m in n]
    s = [torch.where(i < m // 2, i, i - m).double() for i, m in zip(s, n)]
    g = s[0][:, None, None, None] * rec[0] + s[1][None, :, None, None] * rec[1] + s[2][None, None, :, None] * rec[2]
    g2 = (g * g).sum(-1)
    g2[0, 0, 0] = 1.0
    a = a * (4 * math.pi / g2)
    a[0, 0, 0] = 0.0
    return torch.fft.ifftn(a).real.reshape(-1)


def _lsda(u, d):
    """Ceperley-Alder / Perdew-Zunger energy per electron and potentials."""
    t = u + d
    ok = t > 1e-15
    t = torch.where(ok, t, torch.ones_like(t))
    z = torch.where(ok, (u - d) / t, torch.zeros_like(t)).clamp(-1.0, 1.0)
    coe = 0.6203504908994
    rs = coe * t ** (-1 / 3)
    xp = -0.458165293632163 / rs
    dxp = -xp / rs
    big, sq, lr = rs >= 1.0, torch.sqrt(rs), torch.log(rs)

    def corr(g, b1, b2, a, b, cc, dd):
        den = 1.0 + b1 * sq + b2 * rs
        e = torch.where(big, -g / den, b + a * lr + rs * (cc * lr + dd))
        de = torch.where(big, g / den / den * (0.5 * b1 / sq + b2), a / rs + cc * lr + (cc + dd))
        return e, de
    ep, dep = corr(0.1423, 1.0529, 0.3334, 0.0311, -0.0480, 0.0020, -0.0116)
    ef, def_ = corr(0.0843, 1.3981, 0.2611, 0.01555, -0.0269, 0.0007, -0.0048)
    q = 1.25992104989487
    z0, z1 = (1 + z) ** (1 / 3), (1 - z) ** (1 / 3)
    fz = 1.92366105093154 * (z0 ** 4 + z1 ** 4 - 2.0)
    dfz = 2.56488140124205 * (z0 - z1)
    diff = q * xp + ef - xp - ep
    e = xp + ep + diff * fz
    de = dxp + dep + (q * dxp + def_ - dxp - dep) * fz
    v = e - rs / 3 * de
    zero = torch.zeros_like(t)
    return [torch.where(ok, a, zero) for a in (e, v + diff * (1 - z) * dfz, v + diff * (-1 - z) * dfz)]


def _exact_grids(c, spin, mats, vna, aden, pcc):
    """(Bloch-summed orbitals, rho, dVH, V, energies without <D, H>) in 64 bits."""
    pts = _points(c)
    nn = pts.shape[0]
    dv = abs(np.linalg.det(c["lat"])) / nn
    phi = torch.zeros(int(sum(c["no"])), nn, dtype=torch.float64, device="cuda")
    o = 0
    for a in range(len(c["spe"])):
        for _, sel, v, _ in _images(c, a, pts, None):
            phi[o:o + c["no"][a], sel] += v
        o += c["no"][a]
    rho = [(phi * (torch.as_tensor(np.ascontiguousarray(m), device="cuda") @ phi)).sum(0) for m in mats]
    src = (2 * rho[0] if spin == "off" else rho[0] + rho[1]) - 2 * aden
    dvh = _poisson(src, c["ngrid"], c["lat"])
    up, dn = rho[0] + pcc, rho[-1] + pcc
    e, vu, vd = _lsda(up, dn)
    v = [dvh + x + vna for x in (vu, vd)[:len(rho)]]
    eh1 = 0.5 * dv * float((src * dvh).sum())
    ea = _lsda(torch.zeros_like(up) + aden + pcc, torch.zeros_like(up) + aden + pcc)[0]
    exc = [dv * float(((r + pcc) * e - (aden + pcc) * ea).sum()) for r in rho]
    return pts, dv, phi, rho, dvh, v, eh1, exc


def _exact_h(c, pts, v, dv):
    """H in the flat pair-block layout: Gram matrices of the images that reach
    the home cell, summed along the pairs' lattice translations."""
    names, rows, where = [], [], {}
    for a in range(len(c["spe"])):
        for T, sel, val, _ in _images(c, a, pts, None):
            x = torch.zeros(c["no"][a], pts.shape[0], dtype=torch.float64, device="cuda")
            x[:, sel] = val
            where[(a, T)] = len(names)
            names.append((a, T))
            rows.append(x)
    off = np.concatenate([[0], np.cumsum([c["no"][a] for a, _ in names])])
    X = torch.cat(rows)
    del rows
    grams = [((X * w) @ X.T * dv).cpu().numpy() for w in v]
    out = [[] for _ in v]
    for a, b, R in _pair_list(c):
        blocks = [np.zeros((c["no"][a], c["no"][b])) for _ in v]
        for (a2, T), i in where.items():
            if a2 != a:
                continue
            j = where.get((b, tuple(int(p + q) for p, q in zip(T, R))))
            if j is not None:
                for blk, g in zip(blocks, grams):
                    blk += g[off[i]:off[i + 1], off[j]:off[j + 1]]
        for s, blk in zip(out, blocks):
            s.append(blk.ravel())
    return [np.concatenate(s) for s in out]


def _pair_list(c):
    """(atom, neighbour, cell) in the reference's order: the atom itself, then by
    neighbour and cell number (cell 0 first, then i, j, k ascending)."""
    lat, pos, rc = c["lat"], c["pos"], c["cut"]
    reach = int(math.ceil(2 * max(rc) * np.linalg.norm(np.linalg.inv(lat), axis=0).max())) + 1
    r = range(-reach, reach + 1)
    cells = [(0, 0, 0)] + [(i, j, k) for i in r for j in r for k in r if (i, j, k) != (0, 0, 0)]
    shift = np.array(cells) @ lat
    out = []
    for a in range(len(rc)):
        out.append((a, a, (0, 0, 0)))
        for b in range(len(rc)):
            d = np.linalg.norm(pos[a] - pos[b] - shift, axis=1)
            out += [(a, b, cells[q]) for q in np.nonzero(d <= rc[a] + rc[b])[0] if not (a == b and q == 0)]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch" or case["spin"] == "nc":
        return None
    if kind == "potential":
        s = _potential_inputs(case, seed)
        den, pcc, aden = ([torch.as_tensor(x, device="cuda") for x in s["den"]], torch.as_tensor(s["pcc"], device="cuda"),
                          torch.as_tensor(s["aden"], device="cuda"))
        src = (2 * den[0] if case["spin"] == "off" else den[0] + den[1]) - 2 * aden
        dvh = _poisson(src, s["n"], s["lat"])
        dv = abs(np.linalg.det(s["lat"])) / den[0].numel()
        eh1 = 0.5 * dv * float((src * dvh).sum())
        if case["xc"] == "GGA_PBE":
            return {"dVH": dvh, "V": [None] * len(den), "EH1": np.array([eh1]), "EXC": None}
        e, vu, vd = _lsda(den[0] + pcc, den[-1] + pcc)
        ea = _lsda(aden + pcc, aden + pcc)[0]
        return {"dVH": dvh, "V": [dvh + x for x in (vu, vd)[:len(den)]], "EH1": np.array([eh1]),
                "EXC": np.array([dv * float(((r + pcc) * e - (aden + pcc) * ea).sum()) for r in den])}
    c = _cell(case, seed)
    spin = case["spin"]
    mats = _gamma_matrices(c["no"], seed, spin)
    vna = torch.as_tensor(_vna(c, seed), device="cuda")
    if kind == "force":
        pts = _points(c)
        dv = abs(np.linalg.det(c["lat"])) / pts.shape[0]
        off = np.concatenate([[0], np.cumsum(c["no"])])
        phi = torch.zeros(int(off[-1]), pts.shape[0], dtype=torch.float64, device="cuda")
        dphi = [torch.zeros_like(phi) for _ in range(3)]
        for a in range(len(c["spe"])):
            for _, sel, v, g in _images(c, a, pts, None, grad=True):
                phi[off[a]:off[a + 1], sel] += v
                for ax in range(3):
                    dphi[ax][off[a]:off[a + 1], sel] += g[ax]
        F = np.zeros((len(c["spe"]), 3))
        for k, m in enumerate(mats):
            w = (4.0 if spin == "off" else 2.0) * dv * (1.0 + 0.1 * k) * vna
            # the gradients are those with respect to the atom
            y = (torch.as_tensor(np.ascontiguousarray(m), device="cuda") @ phi) * -w
            for ax in range(3):
                per = (dphi[ax] * y).sum(1).cpu().numpy()
                F[:, ax] += np.add.reduceat(per, off[:-1])
        return F
    if case["xc"] == "GGA_PBE":
        return None
    aden = 0.5 * 4.0 * len(c["spe"]) / abs(np.linalg.det(c["lat"])) if kind == "dropin" else 0.0
    pts, dv, _, rho, dvh, v, eh1, exc = _exact_grids(c, spin, mats, 0.0 if kind == "dropin" else vna, aden, 0.0)
    cols = float(sum(n * 4 / 3 * math.pi * (r + 0.62 * abs(np.linalg.det(c["lat"])) ** (1 / 3)) ** 3
                     for n, r in zip(c["no"], c["cut"]))) / abs(np.linalg.det(c["lat"]))
    h = [None] * len(v)
    if 2 * len(v) * pts.shape[0] * cols * cols < 6e12 and pts.shape[0] * cols * 8 < 4e10:
        h = _exact_h(c, pts, v, dv)
    if kind == "dropin":
        return {"rho": rho, "V": v, "H": h}
    dh = dv * sum(float((r * w).sum()) for r, w in zip(rho, v))
    e1 = exc[0] + exc[-1]
    energies = np.array([eh1, exc[0], exc[-1] if spin == "on" else exc[0], dh, (2.0 if spin == "off" else 1.0) * dh + eh1 + e1])
    return {"H": h, "energies": energies}
