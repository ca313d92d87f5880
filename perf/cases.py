"""The work that the speed of this framework is measured on.

Each case is a piece of a plane-wave DFT run as a user's program makes it
through the public entry points: a few electronic steps from given
coefficients (FP64 or mixed precision, with or without forces and stress), a
batch of independent cells, k points off Gamma, molecular dynamics, and the
reference's class methods on the caller's own host arrays.  Every pass starts
from the coefficients in the caller's pinned memory and ends with the new ones
there, as a program does that keeps or saves them.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  contexts, inputs and buffers a program has in hand
    run(state)           one pass, returning energies, forces and coefficients
    work(case)           bytes and operations a pass cannot do without
    tolerance(case)      how far two correct implementations may lie apart
    exact(case, seed)    the same outputs in 64 bits, in plain torch

Cells are diamond-lattice supercells of the Si-like species (a0 = 10.26 bohr,
the configurations' lattice constant) with every atom displaced, boxes of
water-like molecules, and random cubic cells; coefficients are Gaussian random
with the reference's exp(-|G|^2/4) envelope of a fresh wavefunction, then
orthonormalised.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "qbox-public_b200"))

A0 = 10.26          # bohr, diamond lattice constant
AMU = 1822.89       # electron masses
DT = 20.0           # a.u., MD time step
KT = 9.5e-4         # Ha, 300 K

# norm-conserving species on a 0.01-bohr mesh to 10 bohr: -Z erf(r/rc)/r plus
# a Gaussian, one s and one p projector r^l exp(-(r/w)^2)
SPECIES = {
    "Si": dict(zval=4, mass=28.0855, rc=0.5, amp=1.2, width=0.9, w=1.0, d=(2.0, -1.0)),
    "O": dict(zval=6, mass=15.9994, rc=0.4, amp=0.0, width=1.0, w=0.7, d=(3.0, -1.5)),
    "H": dict(zval=1, mass=1.00794, rc=0.3, amp=0.0, width=1.0, w=None, d=()),
}
KPOINTS = {2: (((0.25, 0.25, 0.25), 0.5), ((-0.25, 0.25, 0.25), 0.5)),
           1: (((0.0, 0.25, 0.5), 1.0),)}


def _step(name, reps, ecut_ry, bands, xc, precision, steps, **more):
    c = dict(kind="step", cell="si", nx=reps[0], ny=reps[1], nz=reps[2], ecut_ry=ecut_ry,
             bands=bands, xc=xc, precision=precision, steps=steps, forces=False, stress=False,
             tune=False)
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest run: an 8-atom cell, 20 steps, where launches and the
        # n x n algebra of 16 bands are all there is
        _step("si8_lda_fp64", (1, 1, 1), 20.0, 16, "LDA", "fp64", 20),
        # the precision configuration: 64 atoms, PBE, in both precisions
        _step("si64_pbe_mixed", (2, 2, 2), 30.0, 128, "PBE", "mixed", 10),
        _step("si64_pbe_fp64", (2, 2, 2), 30.0, 128, "PBE", "fp64", 10),
        # an elongated supercell (a surface or interface slab) with an odd
        # band count: a grid of three different lengths
        _step("si48_slab_mixed", (3, 2, 1), 27.0, 97, "PBE", "mixed", 6),
        # a middle-sized cubic cell whose grid length is none of the others'
        _step("si216_pbe_mixed", (3, 3, 3), 24.0, 432, "PBE", "mixed", 4),
        # the large cell, tuned as a long run would be, and its FP64 form
        _step("si512_pbe_mixed", (4, 4, 4), 25.0, 1024, "PBE", "mixed", 8, tune=True),
        _step("si512_pbe_fp64", (4, 4, 4), 25.0, 1024, "PBE", "fp64", 2),
        # the differentiation configuration: 32 water molecules at 70 Ry,
        # one step and one with the adjoint forces and the stress tensor
        _step("water32_forces_stress", (0, 0, 0), 70.0, 128, "PBE", "mixed", 2, cell="water",
              molecules=32, length=18.6, forces=True, stress=True),
        # the batching configuration: uneven cells stepped together
        dict(name="batch12_lda_mixed", kind="batch", systems=12, xc="LDA", precision="mixed",
             steps=5, tune=False),
        # k points off Gamma: complex wavefunctions on two bases
        dict(name="si64_2k_fp64", kind="kpoints", cell="si", nx=2, ny=2, nz=2, ecut_ry=30.0,
             bands=128, xc="PBE", precision="fp64", steps=4, nkp=2, tune=False),
        # molecular dynamics: forces every ionic step, the wavefunction
        # extrapolation and two electronic steps each
        dict(name="si64_md_mixed", kind="md", cell="si", nx=2, ny=2, nz=2, ecut_ry=25.0,
             bands=128, xc="PBE", precision="mixed", steps=2, ionic=3, tune=False),
        # the reference's class methods one by one on the caller's host
        # arrays (a Qbox build linked with this library)
        dict(name="si64_class_calls_fp64", kind="classes", cell="si", nx=2, ny=2, nz=2,
             ecut_ry=25.0, bands=128, xc="LDA", precision="fp64", tune=False),
    ]


def draw(rng):
    """A case of the ranges above: any kind, supercells of 1 to 4 by 1 to 4 by
    1 to 4 lattice cells, cutoffs of 20 to 35 Ry, odd band counts too."""
    kind = rng.choice(("step", "step", "step", "step", "batch", "kpoints", "md", "classes"))
    precision = rng.choice(("mixed", "mixed", "fp64"))
    xc = rng.choice(("LDA", "PBE"))
    if kind == "batch":
        return dict(kind="batch", systems=rng.randint(3, 14), xc=xc, precision=precision,
                    steps=rng.randint(2, 6), tune=False)
    most = {"step": 512 if precision == "mixed" else 256, "kpoints": 64, "md": 128,
            "classes": 96}[kind]
    while True:
        r = [max(1, min(4, int(round(math.exp(rng.uniform(-0.3, math.log(4.4))))))) for _ in range(3)]
        atoms = 8 * r[0] * r[1] * r[2]
        if atoms <= most:
            break
    ecut = round(rng.uniform(20.0, 35.0 if atoms <= 128 else 26.0), 1)
    bands = max(8, 2 * atoms + rng.randint(-atoms // 4, atoms // 8))
    steps = rng.randint(2, 10 if atoms <= 64 else 3)
    if kind == "step":
        if rng.random() < 0.2:
            mol = rng.randint(4, 32)
            return _step("", (0, 0, 0), round(rng.uniform(40.0, 70.0), 1), 4 * mol, xc, precision,
                         2, cell="water", molecules=mol, forces=True, stress=rng.random() < 0.5,
                         length=round(4.65 * math.ceil(mol ** (1.0 / 3.0) - 1e-9)
                                      + rng.uniform(0.0, 0.5), 2))
        return _step("", r, ecut, bands, xc, precision, steps, forces=rng.random() < 0.3)
    c = dict(kind=kind, cell="si", nx=r[0], ny=r[1], nz=r[2], ecut_ry=ecut, bands=bands, xc=xc,
             precision=precision, tune=False)
    if kind == "kpoints":
        c.update(precision="fp64", steps=min(steps, 4), nkp=rng.choice((1, 2)))
    elif kind == "md":
        c.update(steps=rng.randint(1, 2), ionic=rng.randint(2, 3))
    return c


# ------------------------------------------------------------------ systems
def _diamond(nx, ny, nz, rng):
    f = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0], [.25, .25, .25],
                  [.25, .75, .75], [.75, .25, .75], [.75, .75, .25]])
    cells = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"),
                     -1).reshape(-1, 1, 3)
    pos = ((cells + f[None]) * A0).reshape(-1, 3)
    return np.diag([nx * A0, ny * A0, nz * A0]).astype(float), \
        pos + rng.uniform(-0.05, 0.05, pos.shape)


def _sites(length, count, spacing, jitter, rng):
    """count points at least spacing - 2 sqrt(3) jitter apart in a cubic cell."""
    n = max(int(length / spacing), math.ceil(count ** (1.0 / 3.0) - 1e-9))
    g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    g = g[rng.permutation(len(g))[:count]]
    return (g + 0.5) * (length / n) + rng.uniform(-jitter, jitter, (count, 3))


def _water(case, rng):
    length, n = case["length"], case["molecules"]
    oxy = _sites(length, n, 4.65, 0.05, rng)
    ang = math.radians(104.5) / 2
    local = 1.81 * np.array([[math.sin(ang), 0, math.cos(ang)], [-math.sin(ang), 0, math.cos(ang)]])
    hyd = []
    for o in oxy:
        q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
        hyd.append(o + local @ q.T)
    return np.eye(3) * length, [oxy, np.concatenate(hyd)]


def _systems(case, seed):
    """[(cell, species names, positions per species, ecut in Ha, bands)]"""
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        out = []
        # the cells of a batch are of the case, the positions of the seed
        sizes = np.random.default_rng(case["systems"])
        for _ in range(case["systems"]):
            length = sizes.uniform(10.0, 20.0)
            ecut = sizes.uniform(20.0, 30.0) / 2
            n = min(int(sizes.integers(8, 65)), int(length / 3.9) ** 3)
            out.append((np.eye(3) * length, ["Si"], [_sites(length, n, 3.9, 0.11, rng)], ecut, 2 * n))
        return out
    if case["cell"] == "water":
        cell, tau = _water(case, rng)
        return [(cell, ["O", "H"], tau, case["ecut_ry"] / 2, case["bands"])]
    cell, tau = _diamond(case["nx"], case["ny"], case["nz"], rng)
    return [(cell, ["Si"], [tau], case["ecut_ry"] / 2, case["bands"])]


def _miller(cell, ecut, k=None):
    """Sorted (h,k,l) of the basis: the half sphere |G|^2 < 2 ecut at Gamma,
    the whole sphere |k+G|^2 < 2 ecut at a k point."""
    b = 2 * math.pi * np.linalg.inv(cell).T
    m = [int(1.5 + math.sqrt(2 * ecut) / (2 * math.pi) * np.linalg.norm(cell[i])) for i in range(3)]
    h, q, l = [x.ravel() for x in np.meshgrid(*[np.arange(-x, x + 1) for x in m], indexing="ij")]
    g = np.stack([h, q, l], 1) + (0.0 if k is None else np.asarray(k))
    keep = ((g @ b) ** 2).sum(1) < 2 * ecut
    if k is None:
        keep &= (h > 0) | ((h == 0) & (q > 0)) | ((h == 0) & (q == 0) & (l >= 0))
    return np.stack([h, q, l], 1)[keep].astype(np.int32)


def _random_coeffs(cell, hkl, bands, seed, k=None):
    """(bands, ng) complex Gaussian with the envelope exp(-|k+G|^2/4)."""
    b = torch.from_numpy(2 * math.pi * np.linalg.inv(cell).T).cuda()
    h = torch.from_numpy(hkl.astype(float)).cuda()
    if k is not None:
        h = h + torch.tensor(k, dtype=torch.float64, device="cuda")
    env = torch.exp(-0.25 * ((h @ b) ** 2).sum(1))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    c = torch.randn(bands, len(hkl), 2, dtype=torch.float64, device="cuda", generator=gen)
    c = torch.view_as_complex(c) * env
    if k is None:
        g0 = int(np.flatnonzero((hkl == 0).all(1))[0])
        c[:, g0] = c[:, g0].real.to(c.dtype)
    return c


def _velocities(tau, names, seed):
    rng = np.random.default_rng(seed + 17)
    return np.concatenate([rng.standard_normal(t.shape) * math.sqrt(KT / (SPECIES[s]["mass"] * AMU))
                           for s, t in zip(names, tau)])


def _local_mesh(sp):
    r = torch.arange(1001, dtype=torch.float64) * 0.01
    v = torch.empty_like(r)
    v[1:] = -sp["zval"] * torch.erf(r[1:] / sp["rc"]) / r[1:]
    v[0] = -2.0 * sp["zval"] / (sp["rc"] * math.sqrt(math.pi))
    return r.numpy(), (v + sp["amp"] * torch.exp(-(r / sp["width"]) ** 2)).numpy()


def _projectors(sp):
    if sp["w"] is None:
        return []
    r = np.arange(1001) * 0.01
    g = np.exp(-(r / sp["w"]) ** 2)
    return [(0, g), (1, r * g)]


# --------------------------------------------------------- prepare and run
def _pinned(shape, like=None):
    t = torch.empty(shape, dtype=torch.complex128, pin_memory=True)
    if like is not None:
        t.copy_(like)
    return t


def _context(case, system, seed):
    from qbx import capi
    cell, names, tau, ecut, bands = system
    ctx = capi.Context(0, capi.MIXED if case["precision"] == "mixed" else capi.FP64)
    ctx.set_cell(cell, ecut, bands, case["xc"])
    hkl = _miller(cell, ecut)
    if not np.array_equal(ctx.miller(), hkl):
        ctx.set_coeff_order(hkl)
    for s in names:
        sp = SPECIES[s]
        ctx.add_species(sp["zval"], 0.01, _local_mesh(sp)[1], _projectors(sp), list(sp["d"]))
    ctx.set_atoms([len(t) for t in tau], np.concatenate(tau))
    c = _pinned((bands, ctx.ngw), _random_coeffs(cell, hkl, bands, seed))
    ctx.set_coeffs(c.numpy())
    ctx.gram()
    _read(ctx, c)
    return ctx, c


def _read(ctx, out):
    ctx.get_coeffs_async(torch.view_as_real(out).reshape(-1).numpy())
    ctx.synchronize()


def prepare(case, seed):
    systems = _systems(case, seed)
    made = [_context(case, s, 1000 * seed % (1 << 40) + i) for i, s in enumerate(systems)]
    st = dict(case=case, ctxs=[m[0] for m in made], start=[m[1] for m in made])
    ctx = st["ctxs"][0]
    st["out"] = [_pinned(c.shape) for c in st["start"]]
    if case["kind"] == "kpoints":
        kpts = KPOINTS[case["nkp"]]
        ctx.set_kpoints([k for k, _ in kpts], [w for _, w in kpts])
        cell, _, _, ecut, bands = systems[0]
        st["start"], st["out"] = [], []
        for ik, (k, _) in enumerate(kpts):
            c = _random_coeffs(cell, _miller(cell, ecut, k), bands, 1000 * seed % (1 << 40) + 50 + ik, k)
            st["start"].append(_pinned(c.shape, c))
            st["out"].append(_pinned(c.shape))
            ctx.set_kpoint_coeffs(ik, st["start"][ik].numpy())
        ctx.gram()
        for ik in range(len(kpts)):
            _read_k(ctx, ik, st["start"][ik])
    if case["kind"] == "classes":
        cell, names, tau, ecut, bands = systems[0]
        other = _random_coeffs(cell, _miller(cell, ecut), bands, 1000 * seed % (1 << 40) + 90)
        near = st["start"][0].cuda() + 0.01 * other
        st["near"] = _pinned(near.shape, near)
        st["v"] = _potential(ctx.grid, seed)
        st["rho"] = np.zeros(ctx.grid[0] * ctx.grid[1] * ctx.grid[2])
        st["dc"] = np.zeros((bands, ctx.ngw), np.complex128)
    if case["kind"] == "md":
        cell, names, tau, ecut, bands = systems[0]
        st["tau"] = np.concatenate(tau)
        st["vel"] = _velocities(tau, names, seed)
        st["masses"] = [SPECIES[s]["mass"] for s in names]
    if case["kind"] != "classes":
        for c in st["ctxs"]:
            if case["tune"]:
                c.autotune()
            c.set_step_graph(True)
    return st


def _read_k(ctx, ik, out):
    import ctypes
    ctx._ok(ctx.lib.qbx_get_kpoint_coeffs(ctx.h, ik, ctypes.cast(
        out.data_ptr(), ctypes.POINTER(ctypes.c_double))), "get_kpoint_coeffs")


def _potential(grid, seed):
    """A smooth negative potential on the grid (x fastest), as a caller has."""
    rng = np.random.default_rng(seed + 5)
    x = [np.cos(2 * math.pi * np.arange(n) / n + rng.uniform(0, 6.28)) for n in grid]
    return np.ascontiguousarray(-0.8 + 0.3 * x[2][:, None, None] * x[1][None, :, None]
                                + 0.4 * x[0][None, None, :] * x[1][None, :, None]).reshape(-1)


_NAMES = ("ekin", "eps", "enl", "ehart", "ecoul", "exc", "esr", "eself", "etotal",
          "eigenvalue_sum", "total_charge")


def _energies(e):
    return [e[n] for n in _NAMES]


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    ctx = st["ctxs"][0]
    if kind == "step":
        ctx.set_coeffs(st["start"][0].numpy())
        rows, out = [], {}
        for i in range(case["steps"]):
            last = i == case["steps"] - 1
            e = ctx.scf_step(forces=case["forces"] and last, stress=case["stress"] and last)
            rows.append(_energies(e))
        _read(ctx, st["out"][0])
        if case["forces"]:
            out["forces"] = e["fion"]
        if case["stress"]:
            out["stress"] = e["sigma"]
        out.update(energies=np.array(rows), c=st["out"][0])
        return out
    if kind == "batch":
        from qbx import capi
        for c, start in zip(st["ctxs"], st["start"]):
            c.set_coeffs(start.numpy())
        rows = [[_energies(e) for e in capi.scf_step_batch(st["ctxs"])]
                for _ in range(case["steps"])]
        for c, out in zip(st["ctxs"], st["out"]):
            _read(c, out)
        return {"energies": np.array(rows), "c": list(st["out"])}
    if kind == "kpoints":
        for ik, c in enumerate(st["start"]):
            ctx.set_kpoint_coeffs(ik, c.numpy())
        rows = [_energies(ctx.scf_step()) for _ in range(case["steps"])]
        for ik, out in enumerate(st["out"]):
            _read_k(ctx, ik, out)
        return {"energies": np.array(rows), "c": list(st["out"])}
    if kind == "md":
        ctx.move_atoms(st["tau"])
        ctx.set_coeffs(st["start"][0].numpy())
        r = ctx.md_run(case["ionic"], case["steps"], DT, st["masses"], st["vel"])
        _read(ctx, st["out"][0])
        return {"ionic": r["ionic"], "scf": np.array([_energies(e) for e in r["scf"]]),
                "positions": r["positions"], "velocities": r["velocities"], "c": st["out"][0]}
    # class calls: density, V psi, the nonlocal energy with its H psi and
    # forces, and the orthonormalisation of a neighbouring wavefunction
    ctx.set_coeffs(st["start"][0].numpy())
    st["rho"].fill(0.0)
    st["dc"].fill(0.0)
    ctx.compute_density(1.0, st["rho"])
    ctx.rs_mul_add(st["v"], st["dc"])
    nl = ctx.nonlocal_energy(st["dc"], forces=True)
    ctx.set_coeffs(st["near"].numpy())
    ctx.ortho_align(st["start"][0].numpy())
    _read(ctx, st["out"][0])
    return {"rho": st["rho"], "hc": st["dc"], "enl": nl["enl"], "fion": nl["fion"],
            "c": st["out"][0]}


# ------------------------------------------------------------------- work
def _fft_sizes(cell, ecut):
    """The density grid: twice the +-h range of the 4 ecut sphere, plus two,
    each rounded up to an even 2^a 3^{0..2} 5^{0,1} 7^{0,1} 11^{0,1}."""
    def good(n):
        for p in (11, 7, 5, 3, 3):
            n = n // p if n % p == 0 else n
        return n & (n - 1) == 0
    out = []
    for i in range(3):
        n = 2 * int(1.5 + math.sqrt(8 * ecut) / (2 * math.pi) * np.linalg.norm(cell[i]))
        while not good(n):
            n += 2
        n += 2
        while not good(n):
            n += 2
        out.append(n)
    return out


def _one_step_work(cell, names, counts, ecut, bands, k=None, products=True):
    n0, n1, n2 = _fft_sizes(cell, ecut)
    vol = abs(np.linalg.det(cell))
    ng = vol * (2 * ecut) ** 1.5 / (6 * math.pi ** 2) * (1.0 if k else 0.5)
    kmax = math.sqrt(2 * ecut)
    rods = np.linalg.norm(np.cross(cell[0], cell[1])) * kmax ** 2 / (4 * math.pi)
    cols = 2 * kmax * np.linalg.norm(cell[0]) / (2 * math.pi)
    lanes = bands if k else (bands + 1) / 2
    line = lambda n: 5.0 * n * math.log2(n)  # noqa: E731
    fft = lanes * (rods * line(n2) + cols * n2 * line(n1) + n1 * n2 * line(n0))
    nproj = sum(4 * c for s, c in zip(names, counts) if SPECIES[s]["w"])
    mul = 8.0 if k else 4.0           # complex x complex rows; real rows of +-G twice
    gemm = mul * ng * bands * (2.0 * nproj + 5.0 * bands)
    wf = 16.0 * ng * bands
    grid = 8.0 * n0 * n1 * n2
    flops = 2 * fft + 12 * line(n0) * n1 * n2 * 3 + (gemm + 20.0 * bands ** 3 if products else 0)
    # C, C_last and dC_last read, C and dC_last written, rho and v on the grid
    return dict(bytes=5 * wf + 4 * grid + 16.0 * ng * nproj, flops=flops, wf=wf, nproj=nproj,
                ng=ng, fft=fft, grid=grid, mul=mul)


def work(case):
    total = dict(bytes=0.0, flops=0.0)
    for cell, names, tau, ecut, bands in _systems(case, 1):
        counts = [len(t) for t in tau]
        kpts = KPOINTS[case["nkp"]] if case["kind"] == "kpoints" else (None,)
        for k in kpts:
            w = _one_step_work(cell, names, counts, ecut, bands, k)
            if case["kind"] == "classes":
                total["bytes"] += 7 * w["wf"] + 3 * w["grid"]
                total["flops"] += 3 * w["fft"] + w["mul"] * w["ng"] * bands * (
                    5.0 * w["nproj"] + 3.0 * bands)
                continue
            steps = case["steps"]
            total["bytes"] += steps * w["bytes"] + 2 * w["wf"]
            total["flops"] += steps * w["flops"]
            deriv = w["mul"] * w["ng"] * bands * w["nproj"]
            if case.get("forces"):
                total["flops"] += 3 * deriv
            if case.get("stress"):
                total["flops"] += 6 * deriv
            if case["kind"] == "md":
                # per ionic step: density and forces, the alignment and the
                # orthonormalisation; once more at the end
                n = case["ionic"]
                total["flops"] += (n - 1) * steps * w["flops"] + (n + 1) * (
                    w["fft"] + 4 * deriv + 4 * w["mul"] * w["ng"] * bands * bands)
                total["bytes"] += (n - 1) * steps * w["bytes"] + (n + 1) * 3 * w["wf"]
    return total


def tolerance(case):
    """Mixed precision: FP32 transforms and split products over a few steps
    leave the coefficients 2e-6 to 7e-6 from 64 bits (energies 1e-6 at most).
    FP64: 1e-14 after the steps here; sums in another order pass through the
    same Cholesky factors and polar iterations, which amplify rounding by the
    condition of a fresh wavefunction's overlap."""
    return {"rel": 3e-5, "max": 1.2e-3} if case["precision"] == "mixed" else \
        {"rel": 1e-12, "max": 4e-11}


# ------------------------------------------------- the same in 64 bits, plain torch
_RCPS = 1.5         # Gaussian pseudocharge radius
_FPI = 4 * math.pi
_VOIGT = ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2))


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _cubic(x, y, left_slope):
    """Second derivatives of a cubic spline: zero slope (or natural) on the
    left, natural on the right."""
    n, h = len(x), x[1] - x[0]
    d = np.full(n, 4.0)
    e = np.ones(n)
    f = np.ones(n)
    r = np.zeros(n)
    r[1:-1] = 6.0 * (y[2:] - 2 * y[1:-1] + y[:-2]) / h ** 2
    d[-1], f[-1] = 1.0, 0.0
    if left_slope:
        d[0], e[0], r[0] = 2.0, 1.0, 6.0 * (y[1] - y[0]) / h ** 2
    else:
        d[0], e[0] = 1.0, 0.0
    for i in range(1, n):
        m = f[i] / d[i - 1]
        d[i] -= m * e[i - 1]
        r[i] -= m * r[i - 1]
    r[-1] /= d[-1]
    for i in range(n - 2, -1, -1):
        r[i] = (r[i] - e[i] * r[i + 1]) / d[i]
    return r


class _Table:
    """A radial function of |G| on a uniform mesh, by its cubic spline."""

    def __init__(self, g, y, left_slope):
        self.h, self.n = float(g[1] - g[0]), len(g)
        self.y, self.y2 = _t(y), _t(_cubic(g, y, left_slope))

    def __call__(self, g):
        i = torch.clamp((g.detach() / self.h).floor().long(), 0, self.n - 2)
        b = g / self.h - i
        a = 1 - b
        return a * self.y[i] + b * self.y[i + 1] + self.h ** 2 / 6 * (
            (a ** 3 - a) * self.y2[i] + (b ** 3 - b) * self.y2[i + 1])


class _SpeciesTables:
    """V_loc(G) plus the pseudocharge's potential, and V_l(G), from the radial
    mesh by sine and cosine sums on 4096 points."""

    def __init__(self, sp):
        self.z, self.d = float(sp["zval"]), sp["d"]
        n, dr = 4096, 0.01
        r = np.arange(n) * dr
        mesh, vin = _local_mesh(sp)
        v = np.empty(n)
        v[:len(vin)] = vin
        v[len(vin):] = -self.z / r[len(vin):]
        v[0] += self.z / _RCPS * 2 / math.sqrt(math.pi)
        v[1:] += self.z / r[1:] * torch.erf(torch.from_numpy(r[1:] / _RCPS)).numpy()
        v *= _FPI * r * dr
        g = np.arange(n) * math.pi / (n * dr)
        y = self._sine(v)
        y[0] = self._ends(v * r)
        y[1:] /= g[1:]
        self.loc = _Table(g, y, True)
        self.proj = []
        for l, p in _projectors(sp):
            u = np.zeros(n)
            u[:len(p)] = _FPI * dr * p
            if l == 0:
                y = self._sine(u * r)
                y[0] = self._ends(u * r * r)
                y[1:] /= g[1:]
                self.proj.append(_Table(g, y, True))
            else:
                y = np.zeros(n)
                w = np.zeros(n + 1)
                w[:n] = u * r
                even = np.concatenate([w, w[1:n][::-1]])
                cos = np.fft.fft(even).real[:n] / 2
                y[1:] = self._sine(u)[1:] / g[1:] ** 2 - cos[1:] / g[1:]
                self.proj.append(_Table(g, y, False))

    @staticmethod
    def _sine(y):
        n = len(y)
        z = np.concatenate([[0.0], y[1:], [0.0], -y[1:][::-1]])
        return -0.5 * np.fft.fft(z).imag[:n]

    @staticmethod
    def _ends(t):
        c = (17.0 / 48, 59.0 / 48, 43.0 / 48, 49.0 / 48)
        return sum(c[i] * (t[i] + t[-1 - i]) for i in range(4)) + t[4:-4].sum()


def _exc(xc, rho, grad2):
    """Sum of rho times the exchange-correlation energy per electron."""
    if xc == "LDA":
        r = rho.clamp_min(1e-300)
        rs = 0.6203504908994001 / r ** (1.0 / 3.0)
        A, B, b1, b2, G = 0.0311, -0.048, 1.0529, 0.3334, -0.1423
        D = G / (1 + b1 + b2) - B
        C = -A - D - G * ((b1 / 2 + b2) / (1 + b1 + b2) ** 2)
        lo = rs < 1
        rl = torch.where(lo, rs, torch.ones_like(rs))
        ec = torch.where(lo, A * rl.log() + B + C * rl * rl.log() + D * rl,
                         G / (1 + b1 * rs.sqrt() + b2 * rs))
        return (rho * torch.where(rho > 0, 0.75 * -0.610887057711 / rs + ec,
                                  torch.zeros_like(rho))).sum()
    on = rho >= 1e-18
    r = torch.where(on, rho, torch.ones_like(rho))
    fk = 3.09366772628014 * r ** (1.0 / 3.0)
    ul = 0.2195149727645171 / 0.804
    s2 = grad2 / (2 * fk * r) ** 2
    ex = -0.7385587663820224 * r ** (1.0 / 3.0) * (1.804 - 0.804 / (1 + ul * s2))
    rs = 1.91915829267751 / fk
    t2 = grad2 / (4 * 1.27323954473516 * fk * r * r)
    x = rs.sqrt()
    q1 = 2 * 0.0310907 * x * (7.5957 + x * (3.5876 + x * (1.6382 + x * 0.49294)))
    ec = -2 * 0.0310907 * (1 + 0.2137 * rs) * torch.log1p(1 / q1)
    gamma, delt = 0.03109069086965489, 0.06672455060314922 / 0.03109069086965489
    b = delt / torch.expm1(-ec / gamma)
    h = gamma * torch.log1p(delt * (1 + b * t2) * t2 / (1 + b * t2 + b * b * t2 * t2))
    return (rho * torch.where(on, ex + ec + h, torch.zeros_like(rho))).sum()


class _Basis:
    def __init__(self, cell, hkl, shape, k=None):
        self.real = k is None
        self.hkl = _t(hkl.astype(float)) + (0 if k is None else _t(np.array(k, float)))
        n0, n1, n2 = shape
        h = _t(hkl.astype(np.int64))
        self.ip = ((h[:, 2] % n2) * n1 + h[:, 1] % n1) * n0 + h[:, 0] % n0
        self.im = ((-h[:, 2] % n2) * n1 + -h[:, 1] % n1) * n0 + -h[:, 0] % n0
        self.shape, self.N = (n2, n1, n0), n0 * n1 * n2
        on = np.flatnonzero((hkl[:, 0] == 0) & (hkl[:, 1] == 0))
        # G = 0 at Gamma; the lowest l of the rod (0, 0) at a k point
        self.first = int(np.flatnonzero((hkl == 0).all(1))[0]) if k is None else \
            int(on[np.argmin(hkl[on, 2])])
        self.at(_t(np.asarray(cell, float)))

    def at(self, cell):
        b = 2 * math.pi * torch.linalg.inv(cell).T
        self.gx = self.hkl @ b
        self.g2 = (self.gx ** 2).sum(1)
        self.g = torch.sqrt(torch.where(self.g2 > 0, self.g2, torch.ones_like(self.g2)))
        self.on = self.g2 > 0
        self.g = torch.where(self.on, self.g, torch.zeros_like(self.g))
        return self

    def back(self, c):
        """Real function(s) of c (..., ng) at Gamma, as the complex grid."""
        z = torch.zeros(c.shape[:-1] + (self.N,), dtype=torch.complex128, device="cuda")
        z = z.index_copy(-1, self.ip, c)
        if self.real:
            z = z.index_copy(-1, self.im, c.conj())
        return torch.fft.ifftn(z.reshape(c.shape[:-1] + self.shape), dim=(-3, -2, -1),
                               norm="forward").reshape(z.shape)

    def back2(self, c1, c2):
        """c1 + i c2 of two real functions."""
        z = torch.zeros(c1.shape[:-1] + (self.N,), dtype=torch.complex128, device="cuda")
        z[..., self.ip] = c1 + 1j * c2
        z[..., self.im] = c1.conj() + 1j * c2.conj()
        return torch.fft.ifftn(z.reshape(c1.shape[:-1] + self.shape), dim=(-3, -2, -1),
                               norm="forward").reshape(z.shape)

    def grid_fft(self, f):
        return torch.fft.fftn(f.reshape(f.shape[:-1] + self.shape), dim=(-3, -2, -1),
                              norm="forward").reshape(f.shape)

    def dot(self, x, y):
        if not self.real:
            return x.conj() @ y.T
        n, m = x.shape[0], y.shape[0]
        s = 2 * (torch.view_as_real(x).reshape(n, -1) @ torch.view_as_real(y).reshape(m, -1).T)
        return s - torch.outer(x[:, self.first].real, y[:, self.first].real)

    def mix(self, x, m):
        """sum_n x[n] m[n, j] for each j"""
        if not self.real:
            return m.T @ x
        y = m.T.contiguous() @ torch.view_as_real(x).reshape(x.shape[0], -1)
        return torch.view_as_complex(y.reshape(m.shape[1], -1, 2))


def _solve_l(L, b):
    return torch.linalg.solve_triangular(L, b, upper=False)


def _polar(x):
    eye = torch.eye(len(x), dtype=x.dtype, device="cuda")
    for _ in range(20):
        q = eye - x.mH @ x
        nq = float(torch.linalg.norm(q))
        x = x @ (eye + 0.5 * q @ (eye + 0.75 * q)) if nq < 1 else \
            0.5 * (x + torch.linalg.inv(x.mH))
        if nq <= 1e-6:
            break
    return x


class _Exact:
    """One system: bases, species tables, potentials and the operations of
    the electronic step on one SlaterDet per k point (or the one at Gamma)."""

    def __init__(self, system, xc, kpts=None):
        self.cell, self.names, tau, self.ecut, self.nst = system
        self.xc = xc
        self.cell = np.asarray(self.cell, float)
        shape = _fft_sizes(self.cell, self.ecut)
        self.vb = _Basis(self.cell, _miller(self.cell, 4 * self.ecut), shape)
        self.N = self.vb.N
        self.kw = [1.0] if kpts is None else [w for _, w in kpts]
        self.wbs = [_Basis(self.cell, _miller(self.cell, self.ecut, k), shape, k)
                    for k in ([None] if kpts is None else [k for k, _ in kpts])]
        self.tables = [_SpeciesTables(SPECIES[s]) for s in self.names]
        self.omega = abs(np.linalg.det(self.cell))
        self.c_last, self.dc_last = [None] * len(self.wbs), [None] * len(self.wbs)
        self.extrapolate = False
        self.move([np.asarray(t, float) for t in tau])

    # energies of the ions' positions; frac and strain carry derivatives
    def move(self, tau):
        self.tau = tau
        self.frac = [_t(t @ np.linalg.inv(self.cell)) for t in tau]
        self.vion, self.rhops = self._ions(self.vb, self.frac, self.omega)
        self.anl = [self._projector_block(wb, self.frac) for wb in self.wbs]
        self.dfac = torch.cat([torch.cat([_t(np.full(len(f) * m, d)) for d, m in zip(t.d, (1, 3))])
                               for t, f in zip(self.tables, self.frac) if t.proj] or [_t(np.zeros(0))])
        with torch.no_grad():
            self.esr = float(self._esr(self.frac, _t(self.cell)))
        self.eself = sum(t.z ** 2 / (math.sqrt(2 * math.pi) * _RCPS) * len(f)
                         for t, f in zip(self.tables, self.frac))

    def _ions(self, vb, frac, omega):
        vion = rhops = 0
        for t, f in zip(self.tables, frac):
            s = torch.exp(-2j * math.pi * (vb.hkl @ f.T)).sum(1)
            vion = vion + s * (t.loc(vb.g) / omega)
            rhops = rhops - s * (t.z * torch.exp(-0.25 * _RCPS ** 2 * vb.g2) / omega)
        return vion, rhops

    def _projector_block(self, wb, frac):
        rows = []
        for t, f in zip(self.tables, frac):
            if not t.proj:
                continue
            e = torch.exp(-2j * math.pi * (f @ wb.hkl.T))
            inv = torch.where(wb.on, 1 / torch.where(wb.on, wb.g, torch.ones_like(wb.g)),
                              torch.zeros_like(wb.g))
            rows.append(math.sqrt(1 / _FPI) * t.proj[0](wb.g) * e)
            for j in range(3):
                rows.append(-1j * (math.sqrt(3 / _FPI) * wb.gx[:, j] * inv * t.proj[1](wb.g)) * e)
        return torch.cat(rows) if rows else None

    def _esr(self, frac, cell):
        """Repulsion of the Gaussian pseudocharges over neighbouring images."""
        pos = torch.cat([f @ cell for f in frac])
        z = torch.cat([_t(np.full(len(f), t.z)) for t, f in zip(self.tables, frac)])
        rc = math.sqrt(2.0) * _RCPS
        d = [2 * math.pi / np.linalg.norm(2 * math.pi * np.linalg.inv(self.cell).T[i]) for i in range(3)]
        nc = [int(8.0 * rc / x) for x in d]
        df = torch.cat(frac)
        df = df[:, None, :] - df[None, :, :]
        shift = torch.round(df.detach())
        x0 = pos[:, None, :] - pos[None, :, :] - shift @ cell
        e = 0.0
        for i0 in range(-nc[0], nc[0] + 1):
            for i1 in range(-nc[1], nc[1] + 1):
                for i2 in range(-nc[2], nc[2] + 1):
                    x = x0 + _t(np.array([i0, i1, i2], float)) @ cell
                    r2 = (x ** 2).sum(-1)
                    on = r2 > 1e-12
                    r = torch.sqrt(torch.where(on, r2, torch.ones_like(r2)))
                    e = e + 0.5 * torch.where(on, z[:, None] * z[None, :] * torch.erfc(r / rc) / r,
                                              torch.zeros_like(r)).sum()
        return e

    # the SlaterDet's operations
    def gram(self, cs):
        out = []
        for wb, c in zip(self.wbs, cs):
            c = self._clean(wb, c)
            L = torch.linalg.cholesky(wb.dot(c, c))
            out.append(wb.mix(c, torch.linalg.inv(L).mH))
        return out

    def _clean(self, wb, c):
        if wb.real:
            c = c.clone()
            c[:, wb.first] = c[:, wb.first].real.to(c.dtype)
        return c

    def ortho_align(self, wb, c, ref):
        c = self._clean(wb, c)
        L = torch.linalg.cholesky(wb.dot(c, c))
        x = _polar(_solve_l(L, wb.dot(c, ref)))
        return wb.mix(c, torch.linalg.solve_triangular(L.mH, x, upper=True))

    def density(self, cs):
        rho = torch.zeros(self.N, dtype=torch.float64, device="cuda")
        for wb, w, c in zip(self.wbs, self.kw, cs):
            for i in range(0, self.nst, 32):
                if wb.real:
                    d = c[i:i + 32]
                    if len(d) % 2:
                        d = torch.cat([d, torch.zeros_like(d[:1])])
                    f = wb.back2(d[0::2], d[1::2])
                else:
                    f = wb.back(c[i:i + 32])
                rho += w * 2.0 / self.omega * (f.real ** 2 + f.imag ** 2).sum(0)
        return rho

    def potentials(self, rho):
        vb, om = self.vb, self.omega
        self.rho = rho
        self.charge = float(rho.sum()) * om / self.N
        r = rho.clone().requires_grad_(True)
        exc = self._exc_of(r, vb) * om / self.N
        vxc, = torch.autograd.grad(exc, r)
        self.exc = float(exc.detach())
        self.rhog = vb.grid_fft(rho.to(torch.complex128))[vb.ip]      # electrons per volume
        self.eps = float(self._eps(self.rhog, self.vion, om))
        rt = self.rhog + self.rhops
        self.ehart = float(self._ehart(rt, vb, om))
        g2i = torch.where(vb.on, 1 / torch.where(vb.on, vb.g2, torch.ones_like(vb.g2)),
                          torch.zeros_like(vb.g2))
        self.v = vxc * self.N / om + vb.back(self.vion + _FPI * rt * g2i).real

    def _exc_of(self, rho, vb):
        if self.xc == "LDA":
            return _exc("LDA", rho, None)
        g = vb.grid_fft(rho.to(torch.complex128))[vb.ip]
        grad2 = 0
        for j in range(3):
            grad2 = grad2 + vb.back(1j * vb.gx[:, j] * g).real ** 2
        return _exc("PBE", rho, grad2)

    def _eps(self, rhog, vion, om):
        t = (rhog.conj() * vion).real
        return om * (2 * t.sum() - t[self.vb.first])

    @staticmethod
    def _ehart(rt, vb, om):
        g2 = torch.where(vb.on, vb.g2, torch.ones_like(vb.g2))
        return om * _FPI * torch.where(vb.on, (rt.real ** 2 + rt.imag ** 2) / g2,
                                       torch.zeros_like(g2)).sum()

    def _ekin(self, wb, c):
        p = (c.real ** 2 + c.imag ** 2).sum(0)
        return ((2.0 if wb.real else 1.0) * p * wb.g2).sum()

    def _enl(self, wb, a, c, om):
        f = wb.dot(a, c)
        return 2.0 / om * (self.dfac[:, None] * (f.real ** 2 + f.imag ** 2 if f.is_complex()
                                                 else f * f)).sum()

    def local_h(self, wb, c, v, kinetic=True):
        h = 0.5 * wb.g2 * c if kinetic else torch.zeros_like(c)
        for i in range(0, self.nst, 32):
            if not wb.real:
                h[i:i + 32] += wb.grid_fft(wb.back(c[i:i + 32]) * v)[:, wb.ip]
                continue
            d = c[i:i + 32]
            n = len(d)
            if n % 2:
                d = torch.cat([d, torch.zeros_like(d[:1])])
            z = wb.grid_fft(wb.back2(d[0::2], d[1::2]) * v)
            p, m = z[:, wb.ip], z[:, wb.im].conj()
            out = torch.empty_like(d)
            out[0::2], out[1::2] = 0.5 * (p + m), -0.5j * (p - m)
            h[i:i + n] += out[:n]
        return h

    def nonlocal_h(self, wb, a, c):
        f = wb.dot(a, c)
        return wb.mix(a, self.dfac[:, None] / self.omega * f)

    def energies(self, cs, eig=0.0):
        self.ekin = sum(w * float(self._ekin(wb, c)) for wb, w, c in zip(self.wbs, self.kw, cs))
        self.enl = sum(w * float(self._enl(wb, a, c, self.omega)) for wb, w, a, c in
                       zip(self.wbs, self.kw, self.anl, cs) if a is not None)
        ecoul = self.ehart + self.esr - self.eself
        self.etotal = self.ekin + self.eps + self.enl + ecoul + self.exc
        return [self.ekin, self.eps, self.enl, self.ehart, ecoul, self.exc, self.esr, self.eself,
                self.etotal, eig, self.charge]

    def step(self, cs):
        """(the row of energies, the new coefficients)"""
        self.potentials(self.density(cs))
        new, eig = [], 0.0
        for i, (wb, w, a, c) in enumerate(zip(self.wbs, self.kw, self.anl, cs)):
            hc = self.local_h(wb, c, self.v)
            if a is not None:
                hc += self.nonlocal_h(wb, a, c)
            d = (c.conj() * hc).real
            eig += w * float(2 * d.sum() - d[:, wb.first].sum() if wb.real else d.sum())
            hc = hc - wb.mix(c, wb.dot(c, hc))
            p = c.real ** 2 + c.imag ** 2
            ek = 0.5 * (p * wb.g2).sum(1) / (p.sum(1) - 0.5 * p[:, wb.first])
            dc = -0.5 / torch.maximum(0.5 * wb.g2[None], ek[:, None]) * hc
            if self.extrapolate:
                df = dc - self.dc_last[i]
                av, bv = ((x.real * df.real + x.imag * df.imag) for x in (dc, df))
                av, bv = ((2 * float(x.sum()) - float(x[:, wb.first].sum())) if wb.real
                          else float(x.sum()) for x in (av, bv))
                th = -av / bv if bv else 0.0
                th = min(2.0, 0.0 if th < -1.0 else th)
                x = c + th * (c - self.c_last[i]) + dc + th * df
            else:
                x = c + dc
            self.c_last[i], self.dc_last[i] = c, dc
            new.append(self.ortho_align(wb, x, c))
        self.extrapolate = True
        return self.energies(cs, eig), new

    # derivatives of the energy at fixed coefficients (Gamma)
    def _energy_at(self, c, rho_n, frac, strain):
        """Energy at moved ions and a strained cell; rho_n = rho times volume."""
        cell = _t(self.cell) @ (torch.eye(3, dtype=torch.float64, device="cuda") + strain)
        om = torch.linalg.det(cell).abs()
        wb, vb = self.wbs[0], self.vb
        wb.at(cell)
        vb.at(cell)
        vion, rhops = self._ions(vb, frac, om)
        rho = rho_n / om
        rhog = vb.grid_fft(rho.to(torch.complex128))[vb.ip]
        a = self._projector_block(wb, frac)
        e = self._ekin(wb, c) + self._eps(rhog, vion, om) + self._ehart(rhog + rhops, vb, om) \
            + self._exc_of(rho, vb) * om / self.N + self._esr(frac, cell)
        return e + (self._enl(wb, a, c, om) if a is not None else 0.0)

    def forces_stress(self, c, stress=True):
        frac = [f.clone().requires_grad_(True) for f in self.frac]
        strain = torch.zeros(3, 3, dtype=torch.float64, device="cuda", requires_grad=True)
        e = self._energy_at(c, self.rho * self.omega, frac, strain)
        d = torch.autograd.grad(e, frac + [strain])
        self.wbs[0].at(_t(self.cell))
        self.vb.at(_t(self.cell))
        to = _t(np.linalg.inv(self.cell)).T
        f = torch.cat([-g @ to for g in d[:-1]])
        s = -d[-1] / self.omega
        return f.cpu().numpy(), np.array([float(s[i, j] + s[j, i]) / 2 for i, j in _VOIGT])

    def forces(self, c):
        self.potentials(self.density([c]))
        self.energies([c])
        return self.forces_stress(c)[0]


def _exact_md(ex, case, cs, names, tau, vel):
    wb = ex.wbs[0]
    counts = [len(t) for t in tau]
    mass = np.concatenate([np.full((n, 1), SPECIES[s]["mass"] * AMU) for s, n in zip(names, counts)])
    r0, v0, rm, c = np.concatenate(tau), vel.copy(), None, cs[0]
    cv = torch.zeros_like(c)
    ionic, scf = [], []
    speeds = lambda f: (r0 - rm) / DT + DT / (2 * mass) * f  # noqa: E731
    for it in range(case["ionic"]):
        f = ex.forces(c)
        v0 = speeds(f) if it else v0
        ek = float((0.5 * mass * v0 ** 2).sum())
        ionic.append([ex.etotal, ek, ex.etotal + ek])
        rm, r0 = r0, r0 + v0 * DT + DT * DT / (2 * mass) * f
        ex.move(np.split(r0, np.cumsum(counts)[:-1]))
        if it == 0:
            c, cv = ex.gram([c + DT * cv])[0], c
        else:
            cv = wb.mix(cv, _polar(wb.dot(cv, c)))
            x, cv = ex._clean(wb, 2 * c - cv), c
            L = torch.linalg.cholesky(wb.dot(x, x))
            u = _polar(L.mH.contiguous())
            c = wb.mix(x, torch.linalg.solve_triangular(L.mH, u, upper=True))
        ex.extrapolate = False
        for _ in range(case["steps"]):
            e, (c,) = ex.step([c])
            scf.append(e)
    c = ex.gram([c])[0]
    v0 = speeds(ex.forces(c))
    return {"ionic": np.array(ionic), "scf": np.array(scf), "positions": r0, "velocities": v0,
            "c": c.cpu()}


def exact(case, seed):
    torch.set_grad_enabled(True)
    systems = _systems(case, seed)
    kind, base = case["kind"], 1000 * seed % (1 << 40)
    cols, outs = [], []
    for i, s in enumerate(systems):
        cell, names, tau, ecut, bands = s
        if kind == "kpoints":
            kpts = KPOINTS[case["nkp"]]
            ex = _Exact(s, case["xc"], kpts)
            cs = [_random_coeffs(cell, _miller(cell, ecut, k), bands, base + 50 + ik, k)
                  for ik, (k, _) in enumerate(kpts)]
        else:
            ex = _Exact(s, case["xc"])
            cs = [_random_coeffs(cell, _miller(cell, ecut), bands, base + i)]
        cs = ex.gram(cs)
        if kind == "md":
            return _exact_md(ex, case, cs, names, tau, _velocities(tau, names, seed))
        if kind == "classes":
            return _exact_classes(ex, case, cs[0], seed, base)
        rows = []
        for k in range(case["steps"]):
            before = cs
            e, cs = ex.step(cs)
            rows.append(e)
        cols.append(rows)
        outs += [c.cpu() for c in cs]
    if kind == "batch":
        return {"energies": np.array(cols).transpose(1, 0, 2), "c": outs}
    if kind == "kpoints":
        return {"energies": np.array(cols[0]), "c": outs}
    out = {"energies": np.array(cols[0]), "c": outs[0]}
    if case["forces"] or case["stress"]:
        f, sig = ex.forces_stress(before[0])
        if case["forces"]:
            out["forces"] = f
        if case["stress"]:
            out["stress"] = sig
    return out


def _exact_classes(ex, case, c, seed, base):
    wb = ex.wbs[0]
    n2, n1, n0 = wb.shape
    near = c + 0.01 * _random_coeffs(ex.cell, _miller(ex.cell, ex.ecut), ex.nst, base + 90)
    v = _t(_potential((n0, n1, n2), seed))
    hc = ex.local_h(wb, c, v, kinetic=False) + ex.nonlocal_h(wb, ex.anl[0], c)
    frac = [f.clone().requires_grad_(True) for f in ex.frac]
    e = ex._enl(wb, ex._projector_block(wb, frac), c, ex.omega)
    d = torch.autograd.grad(e, frac)
    to = _t(np.linalg.inv(ex.cell)).T
    return {"rho": ex.density([c]).cpu().numpy(), "hc": hc.cpu(), "enl": float(e.detach()),
            "fion": torch.cat([-g @ to for g in d]).cpu().numpy(),
            "c": ex.ortho_align(wb, near, c).cpu()}
