"""The work a user of this framework has it do, as cases that can be timed and compared.

A case is one call (or the two or three calls of one task) through the public entry points:
``Context.fit_batch`` (what ``ChargeCalculator.fit_charges``, the command line and the batched
workload run), ``Context.batch_submit`` (what the server runs), ``Context.qeq`` (``--charge qeq``) and
``Context.filter`` + ``Context.potential`` (what ``compute_stats`` and ``--output`` run).  Sizes are those of
the synthetic workloads of ``pyrepeat_gb300.synth`` and of the benchmark: water, the MOF-like and the
triclinic cell, the batched distribution (20-300 atoms, 12-30 Bohr, 40-96 points per axis at
0.2-0.3 Bohr) and its large requests (800-1500 atoms, 160^3).

Inputs are made here from a seed: atoms by rejection at a minimum separation, neutral charges, and
an ESP equal to the Ewald potential of those charges in the convention of the fit (a Fourier sum
of Gaussian charges of width 0.45 Bohr, indistinguishable from point charges outside the vdW radii)
plus noise of 1e-4 Hartree.  ``exact`` restates every path in plain torch in 64 bits.
"""
import math

import numpy as np
import torch

from pyrepeat_gb300 import _lib, qeq as qeq_params
from pyrepeat_gb300.constants import z_to_symbol
from pyrepeat_gb300.fit import Context
from pyrepeat_gb300.synth import Cube

CUTOFF = 20.0
SIGMA = 0.45
ELEMENTS = (1, 6, 7, 8, 16, 30)
SHARES = (0.4, 0.3, 0.1, 0.15, 0.03, 0.02)
# RESP towards 0 on every element: what keeps densely packed cells well conditioned
RESP_ALL = {"H": (0.1, 0.0), "C": (0.1, 0.0), "N": (0.1, 0.0), "O": (0.1, 0.0), "S": (0.1, 0.0), "Zn": (0.1, 0.0)}
RESP_HEAVY = {"C": (0.1, 0.0), "N": (0.1, 0.0), "O": (0.1, 0.0), "S": (0.1, 0.0)}


def listed():
    return [
        # one molecular cube from the command line: 9 atoms, the grid in ordinary host memory (latency)
        dict(name="water", kind="fit", model="water", cubes=1, atoms=9, grid=72, kmax=7, grids="host", call="batch",
             precision="mixed"),
        # one micro-batch of a served stream: eight small requests, grids in page-locked host memory
        dict(name="served8", kind="fit", model="batch", cubes=8, atoms=0, grid=0, mix=5, kmax=7, grids="pinned",
             call="submit", precision="mixed"),
        # the batched workload: many independent cubes of uneven sizes, grids resident on the device
        dict(name="batch64", kind="fit", model="batch", cubes=64, atoms=0, grid=0, mix=11, kmax=7, grids="device",
             call="batch", precision="mixed"),
        # a served stream's large request: about a thousand atoms at 160^3
        dict(name="large", kind="fit", model="large", cubes=1, atoms=1064, grid=160, kmax=7, grids="device",
             call="batch", precision="mixed"),
        # a densely packed MOF-like cell at a larger k-cutoff: few kept points, the any-KMAX kernels
        dict(name="mof_k12", kind="fit", model="mof", cubes=1, atoms=424, grid=128, kmax=12, grids="device",
             call="batch", precision="mixed"),
        # the largest cell: triclinic, ragged grid, symmetry groups and RESP
        dict(name="tric", kind="fit", model="tric", cubes=1, atoms=2000, grid=200, kmax=7, grids="device",
             call="batch", precision="mixed"),
        # a mixed fit whose condition limit sends it to the FP64 refit (as every ill-conditioned cell does)
        dict(name="escalated", kind="fit", model="tric", cubes=1, atoms=900, grid=150, kmax=7, grids="device",
             call="batch", precision="mixed", kappa_limit=1e-3),
        # --fp64: two cubes of the batched distribution in plain FP64
        dict(name="fp64", kind="fit", model="batch", cubes=2, atoms=0, grid=0, mix=3, kmax=7, grids="device",
             call="batch", precision="fp64"),
        # --fit-type 0: the non-periodic 1/r basis of one molecule in a box
        dict(name="nonperiodic", kind="fit", model="box", cubes=1, atoms=77, grid=90, kmax=0, grids="host",
             call="batch", precision="mixed"),
        # --charge qeq of a large cell, and of an ordinary one
        dict(name="qeq2000", kind="qeq", atoms=2000, kmax=7),
        dict(name="qeq150", kind="qeq", atoms=150, kmax=7),
        # compute_stats / --output: the filter and the fitted potential at every kept point
        dict(name="stats", kind="stats", model="batch", atoms=270, grid=93, mix=7, kmax=7),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("single", "single", "served", "batch", "large", "mof", "tric", "escalated", "fp64", "box",
                       "qeq", "stats"))
    grids = rng.choice(("host", "pinned", "device"))
    mix = rng.randrange(1, 1 << 20)
    fit = dict(kind="fit", atoms=0, grid=0, mix=mix, kmax=7, grids=grids, call="batch", precision="mixed")
    if kind == "single":
        if rng.random() < 0.3:
            return dict(fit, model="water", cubes=1, atoms=9, grid=rng.randrange(24, 97))
        return dict(fit, model="batch", cubes=1)
    if kind == "served":
        return dict(fit, model="batch", cubes=log_int(1, 32), call="submit")
    if kind == "batch":
        return dict(fit, model="batch", cubes=log_int(9, 64))
    if kind == "large":
        return dict(fit, model="large", cubes=1, atoms=rng.randrange(800, 1065), grid=rng.randrange(128, 161))
    if kind == "mof":
        return dict(fit, model="mof", cubes=1, atoms=rng.randrange(53, 425), grid=rng.randrange(64, 129),
                    kmax=rng.randrange(8, 13))
    if kind == "tric":
        return dict(fit, model="tric", cubes=1, atoms=rng.randrange(100, 2000), grid=rng.randrange(60, 200))
    if kind == "escalated":
        return dict(fit, model="tric", cubes=1, atoms=rng.randrange(60, 900), grid=rng.randrange(60, 150),
                    kappa_limit=1e-3)
    if kind == "fp64":
        return dict(fit, model="batch", cubes=1, precision="fp64")
    if kind == "box":
        return dict(fit, model="box", cubes=1, atoms=log_int(3, 150), grid=rng.randrange(40, 97), kmax=0)
    if kind == "qeq":
        return dict(kind="qeq", atoms=log_int(20, 2000), kmax=rng.choice((0, 7, 7)))
    return dict(kind="stats", model="batch", atoms=rng.randrange(20, 301), grid=rng.randrange(40, 97), mix=mix, kmax=7)


# ----------------------------------------------------------------------------- sizes and inputs

def _cell(a, b, c, al=90.0, be=90.0, ga=90.0):
    al, be, ga = (math.radians(x) for x in (al, be, ga))
    cx = c * math.cos(be)
    cy = c * (math.cos(al) - math.cos(be) * math.cos(ga)) / math.sin(ga)
    cell = np.array([[a, 0.0, 0.0], [b * math.cos(ga), b * math.sin(ga), 0.0],
                     [cx, cy, math.sqrt(max(c * c - cx * cx - cy * cy, 0.0))]])
    cell[np.abs(cell) < 1e-14] = 0.0
    return cell


def _sizes(case):
    """[(atoms, cell rows, points per axis, minimum separation)] of the case's cubes."""
    m = case["model"]
    if m == "batch":
        out = []
        rng = np.random.default_rng(case["mix"])
        for _ in range(case.get("cubes", 1)):
            n = case["atoms"] or int(rng.integers(20, 301))
            L = rng.uniform(12.0, 30.0, size=3) if rng.random() < 0.5 else np.full(3, rng.uniform(12.0, 30.0))
            if np.prod(L) < 90.0 * n:  # at most one atom per 90 Bohr^3: the vdW spheres leave ESP points
                L = L * (90.0 * n / np.prod(L)) ** (1 / 3)
            ng = np.clip(np.round(L / rng.uniform(0.2, 0.3)).astype(int), 40, 96)
            if case["grid"]:
                ng = np.maximum(case["grid"] - np.array([0, 3, 8]), 24)
            out.append((n, _cell(*L), ng, 2.0))
        return out
    n, g = case["atoms"], case["grid"]
    if m == "water":
        return [(9, _cell(18.0, 18.0, 18.0), np.array([g, g, g]), 2.0)]
    if m == "large":
        L = max(28.0, (90.0 * n) ** (1 / 3))
        return [(n, _cell(L, L, L), np.array([g, g, g]), 2.0)]
    if m == "mof":  # the density of 424 atoms in 25.8 Bohr
        L = 25.8 * (n / 424.0) ** (1 / 3)
        return [(n, _cell(L, L, L), np.array([g, g, g]), 2.2)]
    if m == "tric":  # the density of 2000 atoms in 40 x 42 x 45 Bohr, 85/95/100 degrees
        s = (n / 2000.0) ** (1 / 3)
        return [(n, _cell(40.0 * s, 42.0 * s, 45.0 * s, 85.0, 95.0, 100.0),
                 np.array([g, int(round(1.05 * g)), int(round(1.125 * g))]), 2.0)]
    L = 12.0 + 2.0 * (90.0 * n) ** (1 / 3) / 2.0  # a box around a molecule
    return [(n, _cell(L, L, L), np.array([g, g, g]), 2.0)]


def _place(rng, cell, n, sep):
    pos = np.empty((n, 3))
    frac = np.empty((n, 3))
    m = 0
    while m < n:
        for f in rng.random((64, 3)):
            if m == n:
                break
            if m:
                d = frac[:m] - f
                d -= np.round(d)
                d = d @ cell
                if np.min(np.einsum("ij,ij->i", d, d)) < sep * sep:
                    continue
            frac[m] = f
            pos[m] = f @ cell
            m += 1
    return pos


def _water(rng, cell):
    half = math.radians(104.5) / 2
    pos, Z, q = [], [], []
    for o in _place(rng, cell, 3, 5.0):
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        v = rng.normal(size=3)
        v -= u * np.dot(u, v)
        v /= np.linalg.norm(v)
        qo = rng.normal(-0.8, 0.05)
        for z, qq, p in ((8, qo, o), (1, -qo / 2, o + 1.81 * (math.cos(half) * u + math.sin(half) * v)),
                         (1, -qo / 2, o + 1.81 * (math.cos(half) * u - math.sin(half) * v))):
            pos.append(p)
            Z.append(z)
            q.append(qq)
    frac = np.array(pos) @ np.linalg.inv(cell)
    return (frac - np.floor(frac)) @ cell, np.array(Z), np.array(q)


def _groups(rng, n, count):
    perm, out, at = rng.permutation(n), [], 0
    for _ in range(count):
        k = int(rng.integers(2, 7))
        if at + k > n:
            break
        out.append(sorted(int(x) for x in perm[at:at + k]))
        at += k
    return out


def _reciprocal(cell):
    return 2.0 * math.pi * np.linalg.inv(cell).T


def _k_share(n1, n2, n3, kmax):
    """The share of +-k that the fit's k-set keeps: k1 >= 0, 0 < |n|^2 < KMAX^2, no factor 2."""
    inside = (n1 * n1 + n2 * n2 + n3 * n3) < kmax * kmax
    return inside * torch.where(n1 == 0, 1.0, 0.5)


def _fourier(pos, q, cell, ng, weight, dtype):
    """sum_k weight(k) S(k) e^{i k.g} on every grid point (nx, ny, nz), S = sum_a q_a e^{-i k.r_a}."""
    dev = "cuda"
    frac = torch.from_numpy(pos @ np.linalg.inv(cell)).to(dev)
    cdt = torch.complex128 if dtype == torch.float64 else torch.complex64
    n = [torch.fft.fftfreq(int(g), 1.0 / int(g), device=dev, dtype=torch.float64).round() for g in ng]
    e = [torch.polar(torch.ones((), dtype=torch.float64, device=dev), -2.0 * math.pi * frac[:, d:d + 1] * n[d]).to(cdt)
         for d in range(3)]
    e[0] = e[0] * torch.from_numpy(q).to(dev)[:, None].to(cdt)
    rec = torch.from_numpy(_reciprocal(cell)).to(dev)
    out = torch.empty(tuple(int(g) for g in ng), dtype=cdt, device=dev)
    step = max(1, int(2e8) // max(1, len(q) * int(ng[2])))
    for j in range(0, int(ng[1]), step):
        yz = (e[1][:, j:j + step, None] * e[2][:, None, :]).reshape(len(q), -1)
        out[:, j:j + step] = (e[0].T @ yz).reshape(int(ng[0]), -1, int(ng[2]))
    n1, n2, n3 = n[0][:, None, None], n[1][None, :, None], n[2][None, None, :]
    k2 = sum((n1 * rec[0, d] + n2 * rec[1, d] + n3 * rec[2, d]) ** 2 for d in range(3))
    k2[0, 0, 0] = 1.0
    w = weight(k2, n1, n2, n3)
    w[0, 0, 0] = 0.0
    return torch.fft.ifftn(out * w.to(cdt)).real * float(np.prod(ng))


def _esp(pos, q, cell, ng, kmax):
    """The planted charges' potential on the grid, flat order i + j nx + k nx ny."""
    vol = abs(float(np.linalg.det(cell)))
    if kmax == 0:
        ax = torch.from_numpy(cell / np.asarray(ng)[:, None]).cuda()
        f = torch.arange(int(np.prod(ng)), device="cuda")
        V = torch.empty(len(f), dtype=torch.float64, device="cuda")
        p, qq = torch.from_numpy(pos).cuda(), torch.from_numpy(q).cuda()
        for s in range(0, len(f), 1 << 17):
            g = _points(f[s:s + (1 << 17)], ng, ax)
            V[s:s + (1 << 17)] = (1.0 / torch.cdist(g, p, compute_mode="donot_use_mm_for_euclid_dist").clamp_min(0.3)) @ qq
        return V
    beta = CUTOFF * CUTOFF / (4.0 * math.pi * math.pi)

    def weight(k2, n1, n2, n3):
        gauss = torch.exp(-0.5 * SIGMA * SIGMA * k2) - torch.exp(-beta * k2) * (1.0 - _k_share(n1, n2, n3, kmax))
        return 4.0 * math.pi / vol * gauss / k2
    V = _fourier(pos, q, cell, ng, weight, torch.float32)
    return V.permute(2, 1, 0).reshape(-1).double()


def _cubes(case, seed):
    """The case's cubes, their grid values on the device (V_dev)."""
    out = []
    for i, (n, cell, ng, sep) in enumerate(_sizes(case)):
        # the statistics come back per kept point: their geometry is the case's, so that their shape is too
        rng = np.random.default_rng([case["mix"] if case["kind"] == "stats" else int(seed), i])
        m = case["model"]
        groups, resp = None, None
        if m == "water":
            pos, Z, q = _water(rng, cell)
        else:
            pos = _place(rng, cell, n, sep)
            Z = rng.choice(np.array(ELEMENTS), size=n, p=SHARES)
            if m == "mof":  # Zn : O : C : H = 4 : 13 : 24 : 12
                Z = rng.choice(np.array([30, 8, 6, 1]), size=n, p=np.array([4, 13, 24, 12]) / 53)
            if case["kind"] == "stats":
                rng = np.random.default_rng([int(seed), i])
            q = rng.normal(0.0, 0.5, size=n)
            if m in ("mof", "tric"):
                resp = RESP_ALL
            if m == "tric":
                groups = _groups(rng, n, max(1, int(0.075 * n)))
            if m in ("batch", "large"):
                if i % 2 == 0:
                    groups = _groups(rng, n, max(1, n // 20))
                else:
                    resp = RESP_HEAVY
            for g in groups or []:
                q[g] = q[g].mean()
            q -= q.mean()
            if m == "box":  # the molecule in the middle of its box
                pos = 6.0 + pos * (1.0 - 12.0 / cell[0, 0])
        V = _esp(pos, q, cell, ng, case["kmax"])
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int(rng.integers(0, 2 ** 62)))
        V += 1e-4 * torch.randn(V.shape, dtype=torch.float64, device="cuda", generator=gen)
        out.append(Cube(Z, pos, np.asarray(ng), cell / np.asarray(ng)[:, None], None, charges_true=q,
                        symm_groups=groups, resp=resp, kmax=case["kmax"], cutoff=CUTOFF, V_dev=V))
    return out


def _qeq_cell(n, seed):
    """A jittered 5 Bohr lattice of H, C, O and Zn: the benchmark's QEq cell."""
    rng = np.random.default_rng(int(seed))
    side = int(np.ceil((1.2 * n) ** (1.0 / 3.0)))
    site = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    site = site[rng.choice(len(site), size=n, replace=False)]
    pos = (site + 0.5 + rng.uniform(-0.15, 0.15, size=(n, 3))) * 5.0
    Z = rng.choice([1, 6, 8, 30], size=n)
    ng = np.array([10 * side] * 3)
    return pos, Z, ng, np.eye(3) * 0.5


# ----------------------------------------------------------------------------- the calls

_CTX = {}


def _ctx(limit=None):
    """The library context that a program keeps; one of its own for a condition limit of its own."""
    if limit not in _CTX:
        _CTX[limit] = Context(0)
        if limit is not None:
            _CTX[limit].set_kappa_limit(limit)
    return _CTX[limit]


def prepare(case, seed):
    ctx = _ctx(case.get("kappa_limit"))
    if case["kind"] == "qeq":
        pos, Z, ng, axis = _qeq_cell(case["atoms"], seed)
        chi, jself, _, _ = qeq_params.charge_parameters(Z)
        return dict(ctx=ctx, case=case, pos=pos, chi=chi, jself=jself, ng=ng, axis=axis)
    cubes = _cubes(case, seed)
    if case["kind"] == "fit" and case["grids"] != "device":
        for c in cubes:
            V = c.V_dev.cpu()
            c.V = (V.pin_memory() if case["grids"] == "pinned" else V).numpy()
            c.V_dev = None
    return dict(ctx=ctx, case=case, cubes=cubes)


def run(state):
    ctx, case = state["ctx"], state["case"]
    if case["kind"] == "qeq":
        q, _, _ = ctx.qeq(state["ng"], state["axis"], state["pos"], state["chi"], state["jself"], 0.0, CUTOFF,
                          case["kmax"])
        return {"charges": q}
    cubes = state["cubes"]
    if case["kind"] == "stats":
        c = cubes[0]
        kept, Vc, _, _ = ctx.filter(c.n_grid, c.axis_vector, c.atom_pos, c.atom_index, c.V_dev)
        ew = ctx.ewald(c.n_grid, c.axis_vector, c.cutoff, c.kmax)
        V = ctx.potential(ew, c.atom_pos, c.charges_true, kept)
        ew.close()
        return {"kept": kept, "Vc": Vc, "V_coul": V}
    prec = _lib.PREC_FP64 if case["precision"] == "fp64" else _lib.PREC_MIXED
    V_dev = [c.V_dev for c in cubes] if case["grids"] == "device" else None
    if case["call"] == "submit":
        q, M, _ = ctx.batch_submit(cubes, prec, V_dev=V_dev).result()
    else:
        q, M, _ = ctx.fit_batch(cubes, prec, V_dev=V_dev)
    return {"charges": q[:8], "more": np.concatenate(q[8:]) if len(q) > 8 else None, "kept": M}


def _radius(z):
    # vdW radii in Bohr of the elements used here, the filter's table
    return {1: 2.72687, 6: 3.63867, 7: 3.45820, 8: 3.30702, 16: 3.81252, 30: 2.61066}[int(z)]


def work(case):
    """Bytes: the grid values, atoms and parameters in, the charges (or the potential) out.  Operations per kept
    point and atom: ~40 for each image within the cutoff, 4 KMAX for the separable reciprocal sum, and the
    atoms' share of one triangle of the Gram; the bordered system's (2/3) n^3 once per cube."""
    if case["kind"] == "qeq":
        n, K = case["atoms"], 754 if case["kmax"] else 0
        images = 1.0 if case["kmax"] == 0 else 1.1
        return {"bytes": 8.0 * 6 * n, "flops": n * n / 2.0 * (60 * images + 4 * K) + 2.0 / 3.0 * n ** 3}
    total_b = total_f = 0.0
    for n, cell, ng, _ in _sizes(case):
        vol, pts = abs(float(np.linalg.det(cell))), float(np.prod(ng))
        r = np.mean([_radius(z) for z in ELEMENTS[:4]])
        full = n * 4.0 / 3.0 * math.pi * r ** 3 / vol
        kept = pts * math.exp(-1.79 * (full / 1.52) ** 1.33)
        images = 4.0 / 3.0 * math.pi * CUTOFF ** 3 / vol if case["kmax"] else 1.0
        total_b += 8.0 * pts + 40.0 * n
        if case["kind"] == "stats":
            total_b += 20.0 * kept
            total_f += kept * n * 40 * images
        else:
            total_f += kept * n * (40 * images + 4 * case["kmax"] + (n + 1)) + 2.0 / 3.0 * n ** 3
    return {"bytes": total_b, "flops": total_f}


# ----------------------------------------------------------------------------- the same in 64 bits

def _points(f, ng, ax):
    nx, ny = int(ng[0]), int(ng[1])
    i, j, k = (f % nx).double(), ((f // nx) % ny).double(), (f // (nx * ny)).double()
    return i[:, None] * ax[0] + j[:, None] * ax[1] + k[:, None] * ax[2]


def _kept(c):
    """Flat indices of the grid points outside every vdW sphere (any of the 27 images)."""
    ng = [int(v) for v in c.n_grid]
    ax = torch.from_numpy(c.axis_vector).cuda()
    box = ax * torch.tensor(ng, dtype=torch.float64, device="cuda")[:, None]
    keep = torch.ones(ng[0] * ng[1] * ng[2], dtype=torch.bool, device="cuda")
    inv = np.linalg.inv(c.axis_vector)
    for p, z in zip(c.atom_pos, c.atom_index):
        r = _radius(z)
        at = p @ inv
        reach = r * np.linalg.norm(inv, axis=0) + 1.0
        lo, hi = np.floor(at - reach).astype(int), np.ceil(at + reach).astype(int)
        idx = [torch.arange(lo[d], hi[d] + 1, device="cuda") for d in range(3)]
        w = [torch.div(idx[d], ng[d], rounding_mode="floor") for d in range(3)]
        ok = [(x >= -1) & (x <= 1) for x in w]
        idx, w = [x[o] for x, o in zip(idx, ok)], [x[o] for x, o in zip(w, ok)]
        n = [x - y * g for x, y, g in zip(idx, w, ng)]
        d2 = None
        for d in range(3):
            g = (n[0].double() * ax[0, d])[:, None, None] + (n[1].double() * ax[1, d])[None, :, None]
            g = g + (n[2].double() * ax[2, d])[None, None, :]
            s = (-w[0].double() * box[0, d])[:, None, None] + (-w[1].double() * box[1, d])[None, :, None]
            s = s + (-w[2].double() * box[2, d])[None, None, :]
            t = g - (float(p[d]) + s)
            d2 = t * t if d2 is None else d2 + t * t
        f = n[0][:, None, None] + ng[0] * (n[1][None, :, None] + ng[1] * n[2][None, None, :])
        keep[f[d2 <= r * r]] = False
    return torch.nonzero(keep)[:, 0]


def _shifts(cell):
    nm = [int(math.floor(CUTOFF / float(np.linalg.norm(cell[d])))) + 1 for d in range(3)]
    return [i * cell[0] + j * cell[1] + k * cell[2] for i in range(-nm[0], nm[0] + 1)
            for j in range(-nm[1], nm[1] + 1) for k in range(-nm[2], nm[2] + 1)]


def _real(g, p, cell):
    """sum over images within the cutoff of erfc(sqrt(alpha) r)/r, every point by every atom."""
    out = torch.zeros((len(g), len(p)), dtype=torch.float64, device="cuda")
    lo, hi = g.min(0).values, g.max(0).values
    for s in _shifts(cell):
        ps = p + torch.from_numpy(s).cuda()
        near = ((torch.maximum(lo - ps, ps - hi).clamp_min(0.0) ** 2).sum(1) <= CUTOFF ** 2 * 1.0001).nonzero()[:, 0]
        if not len(near):
            continue
        r = torch.cdist(g, ps[near], compute_mode="donot_use_mm_for_euclid_dist")
        r = torch.where((r <= CUTOFF) & (r > 1e-10), r, torch.inf)
        out[:, near] += torch.erfc(math.pi / CUTOFF * r) / r
    return out


def _k_set(cell, kmax):
    n = torch.cartesian_prod(torch.arange(0, kmax), torch.arange(1 - kmax, kmax), torch.arange(1 - kmax, kmax)).cuda()
    n2 = (n * n).sum(1)
    n = n[(n2 > 0) & (n2 < kmax * kmax)]
    k = n.double() @ torch.from_numpy(_reciprocal(cell)).cuda()
    k2 = (k * k).sum(1)
    beta = CUTOFF * CUTOFF / (4.0 * math.pi * math.pi)
    return k, 4.0 * math.pi / abs(float(np.linalg.det(cell))) * torch.exp(-beta * k2) / k2


def _charges(c):
    ng, N = [int(v) for v in c.n_grid], c.n_atoms
    cell = c.axis_vector * np.asarray(ng)[:, None]
    ax, p = torch.from_numpy(c.axis_vector).cuda(), torch.from_numpy(c.atom_pos).cuda()
    f = _kept(c)
    V = c.V_dev[f]
    V = V - V.mean()
    if c.kmax:
        k, w = _k_set(cell, c.kmax)
        ph = p @ k.T
        B = torch.cat([w * torch.cos(ph), w * torch.sin(ph)], 1)
    G, r = torch.zeros((N, N), dtype=torch.float64, device="cuda"), torch.zeros(N, dtype=torch.float64, device="cuda")
    s, shift = torch.zeros(N, dtype=torch.float64, device="cuda"), None
    step = max(1024, min(1 << 16, int(1e8) // max(N, 1500)))
    for m in range(0, len(f), step):
        g = _points(f[m:m + step], ng, ax)
        if c.kmax:
            ph = g @ k.T
            phi = torch.cat([torch.cos(ph), torch.sin(ph)], 1) @ B.T
            phi += _real(g, p, cell)
        else:
            phi = 1.0 / torch.cdist(g, p, compute_mode="donot_use_mm_for_euclid_dist")
        shift = phi.mean(0) if shift is None else shift  # any shift: the covariance does not depend on it
        phi -= shift
        G += phi.T @ phi
        r += phi.T @ V[m:m + step]
        s += phi.sum(0)
    A = (G - s[:, None] * s / len(f)).cpu().numpy()
    b = (r - s * V.sum() / len(f)).cpu().numpy()
    base = np.arange(N)
    for grp in c.symm_groups or []:
        base[grp[1:]] = grp[0]
    ind = np.flatnonzero(base == np.arange(N))
    T = np.zeros((N, len(ind)))
    T[np.arange(N), np.searchsorted(ind, base)] = 1.0
    A, b, n = T.T @ A @ T, T.T @ b, len(ind)
    for t, a in enumerate(ind):
        st = (c.resp or {}).get(z_to_symbol(int(c.atom_index[a])))
        if st:
            A[t, t] += st[0]
            b[t] += st[0] * st[1]
    K = np.zeros((n + 1, n + 1))
    K[:n, :n] = A
    K[:n, n] = K[n, :n] = T.sum(0)
    return T @ np.linalg.solve(K, np.append(b, 0.0))[:n]


def exact(case, seed):
    if case["kind"] == "qeq":
        pos, Z, ng, axis = _qeq_cell(case["atoms"], seed)
        chi, jself, _, _ = qeq_params.charge_parameters(Z)
        cell, p = axis * ng[:, None], torch.from_numpy(pos).cuda()
        n = len(p)
        if case["kmax"]:
            J = torch.zeros((n, n), dtype=torch.float64, device="cuda")
            for s in _shifts(cell):
                d = p[:, None, :] - p[None, :, :] + torch.from_numpy(s).cuda()
                rr = (d * d).sum(2).sqrt()
                rr[rr <= 1e-10] = torch.inf
                J += torch.erfc(math.pi / CUTOFF * rr) / rr
            k, w = _k_set(cell, case["kmax"])
            ph = p @ k.T
            c, s = torch.cos(ph), torch.sin(ph)
            J += (w * c) @ c.T + (w * s) @ s.T
        else:
            J = torch.cdist(p, p, compute_mode="donot_use_mm_for_euclid_dist")
            J = 1.0 / torch.where(J > 1e-10, J, torch.inf)
        K = np.zeros((n + 1, n + 1))
        K[:n, :n] = J.cpu().numpy()
        K[np.arange(n), np.arange(n)] = jself
        K[:n, n] = K[n, :n] = 1.0
        return {"charges": np.linalg.solve(K, np.append(-chi, 0.0))[:n]}
    cubes = _cubes(case, seed)
    if case["kind"] == "stats":
        c = cubes[0]
        cell = c.axis_vector * np.asarray(c.n_grid)[:, None]
        f = _kept(c)
        Vc = c.V_dev[f]
        vol, beta = abs(float(np.linalg.det(cell))), CUTOFF * CUTOFF / (4.0 * math.pi * math.pi)
        V = _fourier(c.atom_pos, c.charges_true, cell, c.n_grid, lambda k2, a, b, d: 4.0 * math.pi / vol
                     * torch.exp(-beta * k2) / k2 * _k_share(a, b, d, c.kmax), torch.float64)
        V = V.permute(2, 1, 0).reshape(-1)[f].contiguous()
        ax, p = torch.from_numpy(c.axis_vector).cuda(), torch.from_numpy(c.atom_pos).cuda()
        q = torch.from_numpy(c.charges_true).cuda()
        for m in range(0, len(f), 1 << 15):
            V[m:m + (1 << 15)] += _real(_points(f[m:m + (1 << 15)], c.n_grid, ax), p, cell) @ q
        return {"kept": None, "Vc": Vc - Vc.mean(), "V_coul": V}
    return {"charges": [_charges(c) for c in cubes[:8]], "more": None, "kept": None}
