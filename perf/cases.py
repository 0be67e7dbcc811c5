"""Performance cases: what a user of the pressure solver has it do, through its public entry points.

A CFD program builds a mesh's hierarchy once, then hands over a matrix and a source every time step
(``pcg_gamg_solve``), solves many resident cases together (``Batch``), or drives single pieces of the
solve itself (a smoothing call). The systems are pressure equations on hex boxes: 7-point LDU
matrices in OpenFOAM's face order, graded toward the walls, with a face coefficient that varies from
cell to cell as 1/A does, optionally across a 1000:1 density step.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import brae_b200.native as b2g

# Cells a drawn case may have: that of the largest listed one.
_MAX_CELLS = 160 ** 3


# ---- the systems ---------------------------------------------------------------------------------

def _spacing(n: int, length: float, grading: float, dev) -> torch.Tensor:
    """Cell sizes along an axis, geometric toward both ends (``grading``: middle over wall cell)."""
    if grading == 1.0 or n < 4:
        return torch.full((n,), length / n, dtype=torch.float64, device=dev)
    i = torch.arange(n, dtype=torch.float64, device=dev)
    d = torch.minimum(i, n - 1 - i)
    h = (grading ** (1.0 / (n // 2 - 1))) ** d
    return h * (length / h.sum())


def _box(case: dict, seed: int, dev: str = "cuda") -> dict:
    """Addressing, face areas and the folded matrix of one box, on the device.

    Beside the LDU arrays: ``cx, cy, cz``, the coefficients of the +x, +y, +z faces as [nz, ny, nx]
    arrays (zero where there is no face, or the periodic face's in z), and ``diag3``, ``source3``."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    lx, ly, lz = case.get("lx", 2.0), 1.0, case.get("lz", 1.0)
    periodic = case.get("periodic", False)
    g = torch.Generator(device=dev)
    g.manual_seed(seed * 1000003 + nx * 7919 + ny * 101 + nz)
    dx = _spacing(nx, lx, 1.0, dev)[None, None, :]
    dy = _spacing(ny, ly, case.get("grading", 1.0), dev)[None, :, None]
    dz = _spacing(nz, lz, 1.0, dev)[:, None, None]
    one = torch.ones(nz, ny, nx, dtype=torch.float64, device=dev)
    ax, ay, az = (dy * dz) * one, (dx * dz) * one, (dx * dy) * one
    # 1/A varies by +-20 % from cell to cell; a face takes its two cells' mean
    rau = 0.8 + 0.4 * torch.rand(nz, ny, nx, dtype=torch.float64, device=dev, generator=g)
    if case.get("two_phase", False):
        z = (torch.arange(nz, dtype=torch.float64, device=dev)[:, None, None] + 0.5) * (lz / nz)
        rau = rau / (1.0 + 999.0 * 0.5 * (1.0 - torch.tanh((z - 0.5 * lz) / (3.0 * lz / nz))))

    def face(axis, area, d):
        nxt = torch.roll(rau, -1, axis)
        dist = 0.5 * (d + torch.roll(d, -1, axis)) if d.shape[axis] > 1 else d
        return -0.5 * (rau + nxt) * area / dist

    cx, cy, cz = face(2, ax, dx), face(1, ay, dy), face(0, az, dz)
    cx[:, :, -1] = 0.0
    cy[:, -1, :] = 0.0
    if not periodic:
        cz[-1] = 0.0
    diag = -(cx + torch.roll(cx, 1, 2) + cy + torch.roll(cy, 1, 1) + cz + torch.roll(cz, 1, 0))
    # fixed pressure at the outlet x = lx
    diag[:, :, -1] += rau[:, :, -1] * (ax / (0.5 * dx))[:, :, -1]

    # internal faces per cell: +x, +y, +z, cells ascending (upper-triangular order)
    c = torch.arange(nx * ny * nz, dtype=torch.int32, device=dev).view(nz, ny, nx)
    have = torch.ones(nz, ny, nx, 3, dtype=torch.bool, device=dev)
    have[:, :, -1, 0] = False
    have[:, -1, :, 1] = False
    have[-1, :, :, 2] = False
    nb = torch.stack([c + 1, c + nx, c + nx * ny], dim=3)
    lower = c[..., None].expand(nz, ny, nx, 3)[have].contiguous()
    upper = nb[have].contiguous()
    coef = torch.stack([cx, cy, cz], dim=3)[have].contiguous()
    mag = torch.stack([ax, ay, az], dim=3)[have].contiguous()
    kind = torch.arange(3, device=dev).expand(nz, ny, nx, 3)[have]
    sf = torch.zeros(mag.shape[0], 3, dtype=torch.float64, device=dev)
    sf.scatter_(1, kind[:, None], mag[:, None])
    # the source: the divergence of random face fluxes
    phi = 2.0 * torch.rand(coef.shape[0], dtype=torch.float64, device=dev, generator=g) - 1.0
    flux = torch.zeros(nz, ny, nx, 3, dtype=torch.float64, device=dev)
    flux[have] = phi
    src = (flux.sum(3) - torch.roll(flux[..., 0], 1, 2) - torch.roll(flux[..., 1], 1, 1)
           - torch.roll(flux[..., 2], 1, 0))
    out = dict(lower=lower, upper=upper, Sf=sf, magSf=mag, diag=diag.reshape(-1).clone(), coef=coef,
               source=src.reshape(-1).clone(), n=nx * ny * nz, cx=cx, cy=cy, cz=cz, diag3=diag,
               source3=src, generator=g)
    if periodic:
        low, high = c[0].reshape(-1), c[-1].reshape(-1)
        pc = -cz[-1].reshape(-1)  # Amul subtracts the pair coefficient times the value across
        out["pair_own"] = torch.cat([low, high])
        out["pair_nbr"] = torch.cat([high, low])
        out["pair_coef"] = torch.cat([pc, pc]).contiguous()
    return out


def _mesh(s: dict) -> b2g.Mesh:
    return b2g.Mesh(s["lower"], s["upper"], s["Sf"], s["magSf"], s["n"], 10, True)


def _controls(case: dict) -> b2g.Controls:
    return b2g.controls_default(tolerance=case.get("tol", 1e-6), relTol=case.get("relTol", 0.0),
                                precision=case.get("precision", "fp64"),
                                smoother=case.get("smoother", "GaussSeidel"))


def _batch_boxes(case: dict) -> list[dict]:
    """A batch's boxes: cell counts log-uniform in [lo, hi], aspects 1..8, grading 1..20; the same
    meshes for every seed."""
    r = np.random.default_rng(case["sizes_seed"])
    out = []
    for _ in range(case["count"]):
        n = math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"])))
        ax, az, gr = r.uniform(1.0, 8.0), r.uniform(1.0, 8.0), r.uniform(1.0, 20.0)
        base = (n / (ax * az)) ** (1.0 / 3.0)
        out.append(dict(nx=max(2, round(base * ax)), ny=max(4, round(base)), nz=max(2, round(base * az)),
                        lx=ax, lz=az, grading=gr))
    return out


# ---- the cases -----------------------------------------------------------------------------------

def listed() -> list[dict]:
    return [
        # a small case of a served stream, solved alone in the parity form: launches and the chain of
        # dependent sweep steps are its time
        dict(name="small_fp64", kind="solve", nx=46, ny=23, nz=23, grading=20.0),
        # the same stream's fast form: FP32 V-cycle, the smoother colour by colour
        dict(name="small_multicolour", kind="solve", nx=61, ny=29, nz=30, grading=20.0,
             precision="fp32_precond_multicolour"),
        # the classic uniform cube, one pressure corrector solved to the absolute tolerance
        dict(name="cube_64_fp64", kind="solve", nx=64, ny=64, nz=64, lx=1.0),
        # an ordinary channel mesh of a million cells, FP64
        dict(name="channel_1m_fp64", kind="solve", nx=160, ny=80, nz=80, grading=20.0),
        # a large channel, one corrector of a time step: a relative tolerance, as transient runs set it
        dict(name="channel_4m_fp64", kind="solve", nx=160, ny=160, nz=160, grading=20.0, relTol=0.05),
        # free-surface flow, a 1000:1 density step, the fast form on a large mesh
        dict(name="two_phase_4m_multicolour", kind="solve", nx=160, ny=160, nz=160, grading=20.0,
             two_phase=True, precision="fp32_precond_multicolour"),
        # the same flow with the FP32 V-cycle in the exact sweep order, odd sizes
        dict(name="two_phase_800k_fp32", kind="solve", nx=101, ny=87, nz=93, grading=20.0, two_phase=True,
             precision="fp32_precond"),
        # symGaussSeidel, the other smoother that fvSolution files name
        dict(name="channel_150k_sym", kind="solve", nx=61, ny=47, nz=53, grading=10.0,
             smoother="symGaussSeidel"),
        # a parameter study: many uneven cases resident, solved together
        dict(name="batch_24_fp32", kind="batch", count=24, lo=4096, hi=262144, sizes_seed=1,
             precision="fp32_precond"),
        # a spanwise-periodic channel: the standalone GAMG solver with a cyclic pair
        dict(name="periodic_300k", kind="coupled", nx=81, ny=64, nz=59, grading=20.0, periodic=True),
        # one smoothing call of a program that drives its own multigrid
        dict(name="smooth_2m", kind="smooth", nx=128, ny=128, nz=128, grading=20.0, sweeps=2),
        # the hierarchy of a new mesh, once per mesh change
        dict(name="mesh_260k", kind="mesh", nx=80, ny=57, nz=57, grading=20.0),
    ]


def _log_int(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_box(rng, lo, hi) -> dict:
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    ax, az = rng.uniform(0.8, 2.5), rng.uniform(0.8, 1.6)
    base = (n / (ax * az)) ** (1.0 / 3.0)
    return dict(nx=max(4, round(base * ax)), ny=max(4, round(base)), nz=max(4, round(base * az)),
                grading=rng.choice([1.0, 5.0, 20.0]), lx=ax)


def draw(rng) -> dict:
    kind = rng.choice(["solve"] * 6 + ["batch", "coupled", "smooth", "mesh"])
    if kind == "solve":
        precision = rng.choice(["fp64", "fp64", "fp32_precond_multicolour", "fp32_precond"])
        smoother = rng.choice(["GaussSeidel"] * 4 + ["symGaussSeidel"])
        # a relative tolerance (about one iteration) on the largest meshes, the absolute one below
        hi = _MAX_CELLS * 0.9
        c = dict(kind=kind, precision=precision, smoother=smoother,
                 **_draw_box(rng, 8000, hi if smoother == "GaussSeidel" else 120000))
        big = c["nx"] * c["ny"] * c["nz"] > 8e5
        c["relTol"] = 0.05 if precision != "fp32_precond_multicolour" and big else rng.choice([0.0, 0.0, 0.05])
        c["two_phase"] = rng.random() < 0.3
        return c
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 24), lo=4096, hi=rng.choice([65536, 131072, 262144]),
                    sizes_seed=rng.randint(2, 10 ** 6),
                    precision=rng.choice(["fp64", "fp32_precond", "fp32_precond_multicolour"]))
    if kind == "coupled":
        return dict(kind=kind, periodic=True, **_draw_box(rng, 8000, 300000))
    if kind == "smooth":
        return dict(kind=kind, sweeps=rng.randint(1, 4), **_draw_box(rng, 8000, 2.1e6))
    return dict(kind=kind, **_draw_box(rng, 8000, 262144))


def prepare(case: dict, seed: int):
    if case["kind"] == "batch":
        st = {"controls": _controls(case), "matrices": [], "sources": [], "psis": []}
        # a batch's meshes are built with the part rule it prefers
        b2g.set_part_cells(128)
        try:
            for k, box in enumerate(_batch_boxes(case)):
                s = _box(box, seed * 257 + k)
                st["matrices"].append(b2g.Matrix(_mesh(s), s["diag"], s["coef"]))
                st["sources"].append(s["source"])
                st["psis"].append(torch.zeros_like(s["source"]))
        finally:
            b2g.set_part_cells(48)
        st["batch"] = b2g.Batch(st["matrices"])
        return dict(kind="batch", **st)
    s = _box(case, seed)
    keep = {k: s[k] for k in ("lower", "upper", "Sf", "magSf", "diag", "coef", "source", "n")}
    st = dict(kind=case["kind"], controls=_controls(case), **keep)
    if case["kind"] == "mesh":
        # points moved a little: the face areas vary by 2 % and the pairing meets no ties
        w = 0.98 + 0.04 * torch.rand(s["magSf"].shape[0], dtype=torch.float64, device="cuda", generator=s["generator"])
        st["Sf"] = s["Sf"] * w[:, None]
        st["magSf"] = s["magSf"] * w
        st["n_faces"] = int(w.shape[0])
        return st
    st["mesh"] = _mesh(s)
    st["psi"] = torch.zeros_like(s["source"])
    if case["kind"] == "coupled":
        st["mesh"].set_pair(s["pair_own"].cpu().numpy(), s["pair_nbr"].cpu().numpy())
        st["pair_coef"] = s["pair_coef"]
    if case["kind"] == "smooth":
        st["matrix"] = b2g.Matrix(st["mesh"], s["diag"], s["coef"])
        st["psi0"] = torch.rand(s["n"], dtype=torch.float64, device="cuda", generator=s["generator"])
        st["sweeps"] = case["sweeps"]
    return st


def _end_to_end(arrays: list, size: int) -> np.ndarray:
    out = np.full(size, -1, np.int32)
    at = 0
    for a in arrays:
        out[at:at + a.shape[0]] = a
        at += a.shape[0]
    return out


def run(st):
    kind = st["kind"]
    if kind == "batch":
        for x in st["psis"]:
            x.zero_()
        st["batch"].solve(st["sources"], st["psis"], st["controls"])
        return st["psis"]
    if kind == "mesh":
        mesh = _mesh(st)
        steps = [mesh.step(i) for i in range(mesh.n_levels)]
        # every level's maps and addressing end to end; the levels' sizes depend on the areas, so the
        # arrays are as long as they can get
        return [_end_to_end([s[k] for s in steps], size)
                for k, size in (("restrict", 3 * st["n"]), ("face_restrict", 3 * st["n_faces"]),
                                ("lower", 3 * st["n_faces"]), ("upper", 3 * st["n_faces"]))]
    if kind == "smooth":
        st["psi"].copy_(st["psi0"])
        st["matrix"].smooth(0, st["psi"], st["source"], st["sweeps"])
        return st["psi"]
    st["psi"].zero_()
    if kind == "coupled":
        b2g.gamg_solve_coupled(st["mesh"], st["diag"], st["coef"], st["pair_coef"], st["source"], st["psi"],
                               st["controls"])
    else:
        b2g.pcg_gamg_solve(st["mesh"], st["diag"], st["coef"], st["source"], st["psi"], st["controls"])
    return st["psi"]


# ---- what a pass cannot do without ----------------------------------------------------------------

def _work_box(case: dict) -> dict:
    n = case["nx"] * case["ny"] * case["nz"]
    f = 3 * n
    if case["kind"] == "mesh":
        # addressing, face areas in; the maps and the coarse addressing of every level out
        return {"bytes": 40.0 * f + 2.0 * (4.0 * n + 12.0 * f), "flops": 10.0 * f}
    if case["kind"] == "smooth":
        # the matrix, source and psi once, psi out; every sweep's operations
        return {"bytes": 8.0 * (4 * n + f) + 8.0 * f, "flops": case["sweeps"] * (4.0 * f + n)}
    # a solve reads matrix and source once and writes psi; its iterations' operations: per V-cycle
    # about 3 sweeps and 2 products on each level (twice the finest level's in all), and 2 V-cycles and
    # one product an iteration
    tol = case.get("relTol", 0.0)
    iters = 1 if tol > 0 else 7
    return {"bytes": 8.0 * (3 * n + f) + 8.0 * f, "flops": iters * (2 * 2 * 5 + 1) * (4.0 * f + n)}


def work(case: dict) -> dict:
    if case["kind"] != "batch":
        return _work_box(case)
    out = {"bytes": 0.0, "flops": 0.0}
    for b in _batch_boxes(case):
        w = _work_box(dict(kind="solve", **b))
        out = {k: out[k] + w[k] for k in out}
    return out


def tolerance(case: dict):
    if case["kind"] == "mesh":
        return "exact"
    if case["kind"] == "smooth":
        return {"rel": 1e-14}
    if case["kind"] == "coupled" or case.get("precision", "fp64") == "fp64":
        # sums of up to 4 M terms in another order, through a few iterations: 7e-15 measured with the
        # sums in serial order on 24 k to 262 k cells
        return {"rel": 1e-12}
    # the FP32 V-cycle's rounding moves the path of the iteration, and the result is as far from the
    # system's solution as the solver's tolerance leaves open: 5e-6 to 3.3e-4 measured
    return {"rel": 5e-4}


# ---- the results in plain 64-bit torch ------------------------------------------------------------

def _apply(s: dict, x: torch.Tensor) -> torch.Tensor:
    y = s["diag3"] * x
    for axis, c in ((2, s["cx"]), (1, s["cy"]), (0, s["cz"])):
        y = y + c * torch.roll(x, -1, axis) + torch.roll(c * x, 1, axis)
    return y


def _solve_exact(s: dict) -> torch.Tensor:
    """Conjugate gradients with the diagonal as preconditioner, to rounding."""
    x = torch.zeros_like(s["source3"])
    r = s["source3"].clone()
    z = r / s["diag3"]
    p = z.clone()
    rz = (r * z).sum()
    stop = 1e-13 * s["source3"].abs().sum()
    for it in range(20000):
        q = _apply(s, p)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        if it % 50 == 49 and r.abs().sum() < stop:
            break
        z = r / s["diag3"]
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x.reshape(-1)


def _smooth_exact(s: dict, psi0: torch.Tensor, sweeps: int) -> torch.Tensor:
    """Gauss-Seidel in ascending cell order, one plane i + j + k = d after another."""
    nz, ny, nx = s["diag3"].shape
    dev = psi0.device
    k, j, i = torch.meshgrid(torch.arange(nz, device=dev), torch.arange(ny, device=dev),
                             torch.arange(nx, device=dev), indexing="ij")
    plane = (i + j + k).reshape(-1)
    order = torch.argsort(plane, stable=True)
    bounds = torch.cumsum(torch.bincount(plane), 0).tolist()
    n = nx * ny * nz
    x = torch.zeros(n + 1, dtype=torch.float64, device=dev)  # the last entry stands for no neighbour
    x[:n] = psi0
    idx = torch.arange(n, device=dev).view(nz, ny, nx)
    cols, vals = [], []
    for axis, c, st in ((0, s["cz"], nx * ny), (1, s["cy"], nx), (2, s["cx"], 1)):
        pos = {0: k, 1: j, 2: i}[axis]
        m = (nz, ny, nx)[axis]
        cols += [torch.where(pos > 0, idx - st, n).reshape(-1), torch.where(pos + 1 < m, idx + st, n).reshape(-1)]
        vals += [torch.roll(c, 1, axis).reshape(-1), c.reshape(-1)]
    cols = torch.stack(cols, 1)[order]
    vals = torch.stack(vals, 1)[order]
    b, d = s["source"][order], s["diag"][order]
    for _ in range(sweeps):
        a = 0
        for e in bounds:
            x[order[a:e]] = (b[a:e] - (vals[a:e] * x[cols[a:e]]).sum(1)) / d[a:e]
            a = e
    return x[:n]


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "mesh":
        return None
    if kind == "batch":
        return [_solve_exact(_box(b, seed * 257 + k)) for k, b in enumerate(_batch_boxes(case))]
    if kind != "smooth" and case.get("relTol", 0.0) > 0:
        return None  # stopped after an iteration or two: not the system's solution
    s = _box(case, seed)
    if kind == "smooth":
        psi0 = torch.rand(s["n"], dtype=torch.float64, device="cuda", generator=s["generator"])
        return _smooth_exact(s, psi0, case["sweeps"])
    return _solve_exact(s)
