"""Timed workloads of the H|psi> library, driven through its Python operator API.

Silicon-like diamond cells (the 2-atom fcc cell and supercells of the 8-atom
conventional cell), with the atoms displaced as in a snapshot of a molecular
dynamics run, at plane-wave cutoffs of 12 to 20 Ha.  A case names the cell, the
k-point, the call, its precision and the number of bands; the seed sets the
displacements, the Kleinman-Bylander strengths and the bands.  FP64 is the
operator API's default precision and the one of band-structure post-processing;
the mixed precisions are what a solver's inner loop uses on the same cells.
"""
from __future__ import annotations

import math

import numpy as np
import torch

A_CONV = 10.26  # conventional cubic lattice constant, bohr
DQ, Q_MAX = 0.01, 30.0
DEV = "cuda"
C128 = torch.complex128
F64 = torch.float64


def listed():
    return [
        # the reference's own call: one band of the primitive cell, one k-point of a band path
        dict(name="one_band_fcc2_fp64", op="apply", prec="fp64", cell="fcc", reps="1,1,1", ecut=15.0, lmax=1,
             kinds=1, k="0.25,0.25,0.25", nb=1),
        # an inner-loop block of the primitive cell in single precision
        dict(name="block_fcc2_fp32", op="apply", prec="fp32", cell="fcc", reps="1,1,1", ecut=15.0, lmax=1,
             kinds=1, k="0.1,-0.2,0.3", nb=32),
        # an ordinary block of the conventional cell at the default precision
        dict(name="block_sc8_fp64", op="apply", prec="fp64", cell="sc", reps="1,1,1", ecut=17.5, lmax=1,
             kinds=1, k="0.0,0.0,0.0", nb=48),
        # a compound slab: non-cubic grid, two species with s, p and d projectors, an odd number of bands
        dict(name="ragged_sc16_fp64", op="apply", prec="fp64", cell="sc", reps="1,1,2", ecut=14.3, lmax=2,
             kinds=2, k="0.13,-0.21,0.37", nb=37),
        # the benchmark's supercell block, at the default precision and on the tensor cores
        dict(name="block_sc64_fp64", op="apply", prec="fp64", cell="sc", reps="2,2,2", ecut=20.0, lmax=2,
             kinds=1, k="0.0,0.0,0.0", nb=128),
        dict(name="block_sc64_tc", op="apply", prec="tc", cell="sc", reps="2,2,2", ecut=20.0, lmax=2,
             kinds=1, k="0.0,0.0,0.0", nb=128),
        # band velocities along a path: dH/dk of a block in all three directions
        dict(name="grad_sc8_fp64", op="grad", prec="fp64", cell="sc", reps="1,1,1", ecut=17.5, lmax=1,
             kinds=1, k="0.05,0.0,0.0", nb=48),
        # k.p input of a supercell: the full band-pair velocity matrix
        dict(name="velocity_sc64_tc", op="velocity", prec="tc", cell="sc", reps="2,2,2", ecut=20.0, lmax=2,
             kinds=1, k="0.0,0.0,0.0", nb=256),
        # Rayleigh quotients beside H|psi> on a mid-sized cell
        dict(name="energies_sc32_tc", op="energies", prec="tc", cell="sc", reps="1,2,2", ecut=16.0, lmax=2,
             kinds=1, k="0.2,0.1,0.0", nb=64),
        # the charge density of one k-point of a compound cell
        dict(name="density_sc16_fp64", op="density", prec="fp64", cell="sc", reps="1,1,2", ecut=17.5, lmax=1,
             kinds=2, k="0.125,0.125,0.25", nb=40),
        # a Monkhorst-Pack mesh of the primitive cell in one plan
        dict(name="mesh_fcc2_fp32", op="batch", prec="fp32", cell="fcc", reps="1,1,1", ecut=15.0, lmax=1,
             kinds=1, k="0.0,0.0,0.0", nb=16, mesh=4),
        # one step of a loop over k-points: bind the G-sphere, then apply H to its bands
        dict(name="bind_sc8_fp64", op="bind", prec="fp64", cell="sc", reps="1,1,1", ecut=17.5, lmax=1,
             kinds=1, k="0.125,0.375,0.125", nb=16),
    ]


CELLS = [("fcc", "1,1,1"), ("sc", "1,1,1"), ("sc", "1,1,2"), ("sc", "1,2,2"), ("sc", "2,2,2")]


def draw(rng):
    op = rng.choice(["apply"] * 5 + ["grad", "velocity", "energies", "density", "batch", "bind"])
    prec = rng.choice(["fp64", "fp64", "fp64", "fp32", "tc", "tc", "tc_bf16"])
    if op == "density" and prec.startswith("tc"):
        prec = "fp32"
    if op == "batch":
        prec = rng.choice(["fp64", "fp32", "fp32", "tc"])
    cell, reps = rng.choice(CELLS[:2] if op == "batch" else CELLS)
    case = dict(op=op, prec=prec, cell=cell, reps=reps, ecut=round(rng.uniform(12.0, 20.0), 2),
                lmax=rng.choice([1, 2]), kinds=rng.choice([1, 2]),
                k=",".join("%.3f" % rng.uniform(-0.5, 0.5) for _ in range(3)),
                nb=int(round(2 ** rng.uniform(0.0, 7.0))))
    if op == "batch":
        case["mesh"] = rng.choice([2, 3])
    top = 0.95 * cost(listed()[4])  # block_sc64_fp64
    while case["nb"] > 1 and cost(case) > top:
        case["nb"] = max(1, case["nb"] * 2 // 3)
    return case


def cost(case):
    """Rough cost of a pass in FP64 operations: the projector sums, and the grid transforms."""
    c = counts(case)
    sums = 16.0 * c["P"] * c["npw"] * case["nb"] * {"grad": 5, "velocity": 6}.get(case["op"], 1)
    fft = 20.0 * c["N"] * math.log2(c["N"]) * case["nb"]
    every = case.get("mesh", 1) ** 3
    return every * (sums + fft) * (1.0 if case["prec"] == "fp64" else 0.03)


# ---- geometry ---------------------------------------------------------------

def smooth(n):
    """The smallest even-radix FFT length >= n (factors 2, 3 and 5)."""
    while True:
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


def geometry(case):
    """Lattice rows (bohr), ideal fractional positions, species of each atom, FFT grid."""
    if case["cell"] == "fcc":
        lat = 0.5 * A_CONV * np.array([[0.0, 1.0, 1.0], [1.0, 0.0, 1.0], [1.0, 1.0, 0.0]])
        tau = np.array([[0.0, 0.0, 0.0], [0.25, 0.25, 0.25]])
        kind = np.array([0, 1])
    else:
        reps = [int(x) for x in case["reps"].split(",")]
        fcc = np.array([[0, 0, 0], [0, 0.5, 0.5], [0.5, 0, 0.5], [0.5, 0.5, 0]])
        cells = [(i, j, k) for i in range(reps[0]) for j in range(reps[1]) for k in range(reps[2])]
        tau = np.concatenate([(np.concatenate([fcc, fcc + 0.25]) + np.array(c)) / np.array(reps) for c in cells])
        kind = np.tile(np.repeat([0, 1], 4), len(cells))
        lat = A_CONV * np.diag([float(r) for r in reps])
    kmax = math.sqrt(2.0 * case["ecut"])
    # 3.4 times the sphere's radius along each axis: holds the sphere, and most of V|psi>
    grid = [smooth(int(math.ceil(3.4 * np.linalg.norm(a) * kmax / (2 * math.pi))) + 1) for a in lat]
    return lat, tau, np.minimum(kind, case["kinds"] - 1).astype(np.int32), grid


def sphere(lat, k_frac, ecut):
    """G-vectors with |k+G|^2/2 < ecut in order of kinetic energy: (g, K, kinetic), numpy."""
    B = 2.0 * np.pi * np.linalg.inv(lat).T
    r = [np.arange(-m, m + 1) for m in
         (int(math.ceil(np.linalg.norm(a) * math.sqrt(2.0 * ecut) / (2 * math.pi))) + 1 for a in lat)]
    g = np.stack(np.meshgrid(*r, indexing="ij"), axis=-1).reshape(-1, 3)
    K = (g + np.asarray(k_frac)) @ B
    kin = 0.5 * np.einsum("ij,ij->i", K, K)
    keep = kin < ecut
    g, K, kin = g[keep], K[keep], kin[keep]
    order = np.lexsort((g[:, 2], g[:, 1], g[:, 0], kin))
    return g[order].astype(np.int32), np.ascontiguousarray(K[order]), np.ascontiguousarray(kin[order])


def kpoints(case):
    k = [float(x) for x in case["k"].split(",")]
    m = case.get("mesh", 0)
    if not m:
        return [tuple(k)]
    v = [(2 * i - m - 1) / (2.0 * m) for i in range(1, m + 1)]
    return [(a, b, c) for a in v for b in v for c in v]


_counts = {}


def counts(case):
    key = (case["cell"], case["reps"], case["ecut"], case["lmax"], case["k"])
    if key not in _counts:
        lat, tau, _, n = geometry(case)
        k = kpoints(case)[0]
        npw = sphere(lat, k, case["ecut"])[0].shape[0]
        _counts[key] = dict(P=len(tau) * 2 * (case["lmax"] + 1) ** 2, npw=npw, N=n[0] * n[1] * n[2])
    return _counts[key]


def radial(l, rc, q):
    """Projector q^l exp(-q^2 rc^2 / 4) and its derivative."""
    e = np.exp(-q * q * rc * rc / 4.0)
    db = (l * q ** max(l - 1, 0) if l else 0.0) * e - 0.5 * rc * rc * q ** (l + 1) * e
    return q ** l * e, db


def tables(case, seed):
    """Per species: l, lambda, beta(q) and dbeta/dq of two projectors per l, D_l diagonalised per l."""
    q = np.arange(int(math.ceil(Q_MAX / DQ)) + 4) * DQ
    got = []
    for kind in range(case["kinds"]):
        rng = np.random.default_rng(1000 * kind + seed % 100003)
        ls, lam, bq, dbq = [], [], [], []
        for l in range(case["lmax"] + 1):
            D = rng.uniform(-2.0, 2.0, size=(2, 2))
            w, U = np.linalg.eigh(0.5 * (D + D.T))
            raw = [radial(l, rc, q) for rc in ((1.0, 1.4), (1.1, 1.5))[kind]]
            for i in range(2):
                ls.append(l)
                lam.append(w[i])
                bq.append(U[0, i] * raw[0][0] + U[1, i] * raw[1][0])
                dbq.append(U[0, i] * raw[0][1] + U[1, i] * raw[1][1])
        got.append((np.array(ls, dtype=np.int32), np.array(lam), np.array(bq), np.array(dbq)))
    return got


def physics(case, seed):
    """What both the library and the plain evaluation start from: displaced atoms, V_loc, tables, bands."""
    lat, tau, kind, n = geometry(case)
    rng = np.random.default_rng(seed)
    tau = tau + rng.normal(scale=0.08, size=tau.shape) @ np.linalg.inv(lat)
    omega = float(abs(np.linalg.det(lat)))
    B = torch.tensor(2.0 * np.pi * np.linalg.inv(lat).T, device=DEV)
    f = [torch.fft.fftfreq(m, 1.0 / m, device=DEV, dtype=F64) for m in n]
    G = torch.stack(torch.meshgrid(*f, indexing="ij"), -1) @ B
    t = torch.tensor(tau, device=DEV)
    e = [torch.exp(-2j * math.pi * torch.outer(t[:, d], f[d])) for d in range(3)]
    S = torch.einsum("ai,aj,ak->ijk", *e)
    form = -3.0 * math.pi ** 1.5 * 1.2 ** 3 * torch.exp(-(G * G).sum(-1) * 1.2 ** 2 / 4.0)
    v = (torch.fft.ifftn(form * S / omega) * (n[0] * n[1] * n[2])).real.contiguous()
    ks = []
    for i, k in enumerate(kpoints(case)):
        g, K, kin = sphere(lat, k, case["ecut"])
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed * 1009 + i)
        x = torch.randn(case["nb"], kin.shape[0], 2, generator=gen, device=DEV, dtype=F64)
        x = torch.view_as_complex(x) / (1.0 + 2.0 * torch.tensor(kin, device=DEV)) ** 2
        for _ in range(2):  # orthonormal bands
            L = torch.linalg.cholesky(x.conj() @ x.T)
            x = torch.linalg.solve_triangular(L.conj(), x, upper=False)
        ks.append((k, g, K, kin, x.contiguous()))
    return dict(lat=lat, tau=tau, kind=kind, n=n, omega=omega, v=v, tables=tables(case, seed), ks=ks)


# ---- the library ------------------------------------------------------------

def prepare(case, seed):
    from effmass_gb300.batch import Batch
    from effmass_gb300.hamiltonian import Hamiltonian
    from effmass_gb300.system import KPoint, Species, System

    p = physics(case, seed)
    sp = [Species(z=6 + i, proj_l=l, lam=lam, dq=DQ, q_max=Q_MAX, beta_q=b, dbeta_q=db)
          for i, (l, lam, b, db) in enumerate(p["tables"])]
    system = System(name=case["cell"], lattice=p["lat"], omega=p["omega"], n1=p["n"][0], n2=p["n"][1], n3=p["n"][2],
                    v_loc=p["v"].cpu().numpy().reshape(-1), species=sp, atom_species=p["kind"],
                    atom_z=6 + p["kind"], atom_tau=p["tau"], ecut=case["ecut"])
    H = Hamiltonian(system, precision=case["prec"])
    ks = [KPoint(npw=len(kin), k_frac=np.array(k), g_idx=g, kvec=K, kinetic=kin) for k, g, K, kin, _ in p["ks"]]
    op, nb, psi = case["op"], case["nb"], p["ks"][0][4]
    s = dict(op=op, nb=nb, H=H, kpoint=ks[0], psi=psi)
    if op != "bind":
        for i, kp in enumerate(ks):
            H.set_kpoint(i, kp)
    if op in ("apply", "energies", "bind"):
        s["out"] = torch.zeros_like(psi)
    if op == "apply":
        s["call"] = H.at_k(0)
    elif op == "grad":
        s["out"] = torch.zeros((3,) + tuple(psi.shape), dtype=C128, device=DEV)
        s["call"] = H.gradient().at_k(0)
    elif op == "velocity":
        s["out"] = torch.zeros((3, nb, nb), dtype=C128, device=DEV)
    elif op == "density":
        s["occ"] = torch.linspace(2.0, 0.5, nb, dtype=F64, device=DEV)
        s["out"] = torch.zeros(tuple(p["n"]), dtype=F64, device=DEV)
    elif op == "batch":
        # the mixed precisions with the built-in tiles: tuned ones may sum in another order in another process
        s["plan"] = Batch([(H, i, nb) for i in range(len(ks))], precision=case["prec"], tune=case["prec"] == "fp64")
        s["psi"] = torch.cat([x[4].reshape(-1) for x in p["ks"]])
        s["out"] = torch.zeros_like(s["psi"])
    return s


def run(s):
    from effmass_gb300.hamiltonian import GradHPsi

    op, H, nb, psi, out = s["op"], s["H"], s["nb"], s["psi"], s["out"]
    if op != "velocity":
        out.zero_()  # outputs accumulate: the caller clears them
    if op == "apply":
        s["call"](nb, psi, out)
    elif op == "bind":
        H.at_k(0, s["kpoint"])(nb, psi, out)
    elif op == "energies":
        return out, H.apply_energies(0, nb, psi, out)
    elif op == "grad":
        s["call"](psi, GradHPsi(out[0], out[1], out[2]), n_bands=nb)
    elif op == "velocity":
        H.velocity_matrix(0, nb, psi, out=out)
    elif op == "density":
        H.density(0, nb, psi, s["occ"], rho=out)
    else:
        s["plan"].apply(psi, out, device=True)
    return out


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    c = counts(case)
    nb, op, every = case["nb"], case["op"], case.get("mesh", 1) ** 3
    block = 16.0 * c["npw"] * nb
    N, P, npw = c["N"], c["P"], c["npw"]
    transform = 5.0 * N * math.log2(N) * nb
    sums = 8.0 * P * npw * nb  # one complex projection or expansion
    geometry_bytes = 8.0 * N + 40.0 * npw  # V_loc; K, g and kinetic energies
    if op == "density":
        return dict(bytes=block + 8.0 * N + 12.0 * npw, flops=transform + 3.0 * N * nb)
    if op == "grad":
        return dict(bytes=4.0 * block + 40.0 * npw, flops=10.0 * sums)
    if op == "velocity":
        return dict(bytes=block + 48.0 * nb * nb + 40.0 * npw, flops=4.0 * sums + 24.0 * (npw + 2 * P) * nb * nb)
    return dict(bytes=every * (2.0 * block + geometry_bytes), flops=every * (2.0 * transform + 2.0 * sums + 3.0 * N * nb))


# ---- the same in plain torch, 64 bits ---------------------------------------

def interpolate(t, q):
    """Cubic Lagrange interpolation of the table rows t[i][q_j = j dq], the stencil one node left of q."""
    x = q / DQ
    i0 = torch.clamp(torch.floor(x).long() - 1, min=0)
    p = x - i0
    u, v, w = 1.0 - p, 2.0 - p, 3.0 - p
    return (t[:, i0] * (u * v * w / 6.0) + t[:, i0 + 1] * (p * v * w / 2.0) - t[:, i0 + 2] * (p * u * w / 2.0)
            + t[:, i0 + 3] * (p * u * v / 6.0))


def harmonics(l, K):
    """Real solid harmonics |K|^l Y_lm [2l+1][npw] and their gradients [3][2l+1][npw]."""
    x, y, z = K.T
    o, one = torch.zeros_like(x), torch.ones_like(x)
    if l == 0:
        R, D = [one], [[o], [o], [o]]
        c = [math.sqrt(1 / (4 * math.pi))]
    elif l == 1:
        R, D = [y, z, x], [[o, o, one], [one, o, o], [o, one, o]]
        c = [math.sqrt(3 / (4 * math.pi))] * 3
    else:
        R = [x * y, y * z, 2 * z * z - x * x - y * y, x * z, x * x - y * y]
        D = [[y, o, -2 * x, z, 2 * x], [x, z, -2 * y, o, -2 * y], [o, y, 4 * z, x, o]]
        a = math.sqrt(15 / (4 * math.pi))
        c = [a, a, math.sqrt(5 / (16 * math.pi)), a, a / 2]
    c = torch.tensor(c, dtype=F64, device=DEV)[:, None]
    return torch.stack(R) * c, torch.stack([torch.stack(d) * c for d in D])


def projectors(p, k, g, K, derivatives):
    """Projector rows [P][npw], lambda [P] and the rows' K-derivatives."""
    Kt = torch.tensor(K, device=DEV)
    q = torch.sqrt((Kt * Kt).sum(1))
    safe = torch.where(q > 1e-12, q, torch.ones_like(q))
    phase = (torch.tensor(g, device=DEV).to(F64) + torch.tensor(k, dtype=F64, device=DEV)) @ torch.tensor(p["tau"], device=DEV).T
    S = torch.exp(-2j * math.pi * phase).T / math.sqrt(p["omega"])
    per_kind = []
    for ls, lam, bq, dbq in p["tables"]:
        b = interpolate(torch.tensor(bq, device=DEV), q)
        db = interpolate(torch.tensor(dbq, device=DEV), q)
        rows, drows, strength = [], [[], [], []], []
        for i, l in enumerate(ls):
            R, D = harmonics(int(l), Kt)
            f0 = torch.where(q > 1e-12, b[i] / safe ** int(l), (db[i] if l == 1 else b[i] if l == 0 else 0 * b[i]))
            rows.append(f0 * R)
            strength += [lam[i]] * R.shape[0]
            if derivatives:
                f1 = torch.where(q > 1e-12, (db[i] - int(l) * b[i] / safe) / safe ** int(l), 0 * q)
                for a in range(3):
                    drows[a].append(f1 * Kt[:, a] / safe * R + f0 * D[a])
        per_kind.append((torch.cat(rows), [torch.cat(d) for d in drows] if derivatives else [], strength))
    pr = torch.cat([per_kind[kd][0] * S[a] for a, kd in enumerate(p["kind"])])
    lam = torch.tensor(sum((per_kind[kd][2] for kd in p["kind"]), []), device=DEV)
    d = [torch.cat([per_kind[kd][1][x] * S[a] for a, kd in enumerate(p["kind"])]) for x in range(3)] if derivatives else []
    return pr, lam, d


def local(p, g, kin, psi):
    """(kinetic + V_loc) psi through full grids, sixteen bands at a time."""
    n = p["n"]
    gi = torch.tensor(g, device=DEV).long()
    at = ((gi[:, 0] % n[0]) * n[1] + gi[:, 1] % n[1]) * n[2] + gi[:, 2] % n[2]
    out = torch.tensor(kin, device=DEV) * psi
    for b in range(0, psi.shape[0], 16):
        x = psi[b:b + 16]
        grid = torch.zeros((x.shape[0], n[0] * n[1] * n[2]), dtype=C128, device=DEV)
        grid[:, at] = x
        r = torch.fft.ifftn(grid.reshape(-1, *n), dim=(1, 2, 3)) * p["v"]
        out[b:b + 16] += torch.fft.fftn(r, dim=(1, 2, 3)).reshape(x.shape[0], -1)[:, at]
    return out


def exact(case, seed):
    p = physics(case, seed)
    op = case["op"]
    if op == "density":
        k, g, K, kin, psi = p["ks"][0]
        n = p["n"]
        gi = torch.tensor(g, device=DEV).long()
        rho = torch.zeros(tuple(n), dtype=F64, device=DEV)
        for b, occ in enumerate(torch.linspace(2.0, 0.5, case["nb"], dtype=F64, device=DEV)):
            grid = torch.zeros(tuple(n), dtype=C128, device=DEV)
            grid[gi[:, 0] % n[0], gi[:, 1] % n[1], gi[:, 2] % n[2]] = psi[b]
            r = torch.fft.ifftn(grid) * (n[0] * n[1] * n[2])
            rho += occ * (r.real ** 2 + r.imag ** 2)
        return rho
    found = []
    for k, g, K, kin, psi in p["ks"]:
        pr, lam, d = projectors(p, k, g, K, op in ("grad", "velocity"))
        c = psi @ pr.conj().T  # <p|psi_b>, [nb][P]
        Kt = torch.tensor(K, device=DEV)
        if op == "velocity":
            m = []
            for a in range(3):
                x = (c.conj() * lam) @ (psi @ d[a].conj().T).T  # sum_p lambda <psi_m|p><d_a p|psi_n>
                m.append((psi.conj() * Kt[:, a]) @ psi.T + x + x.conj().T)
            return torch.stack(m)
        if op == "grad":
            return torch.stack([Kt[:, a] * psi + ((psi @ d[a].conj().T) * lam) @ pr + (c * lam) @ d[a] for a in range(3)])
        h = local(p, g, kin, psi) + (c * lam) @ pr
        if op == "energies":
            return h, (psi.conj() * h).sum(1).real.contiguous()
        found.append(h.reshape(-1))
    return torch.cat(found) if op == "batch" else h
