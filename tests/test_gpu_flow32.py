"""The FP32 data-flow smoothing launch (flow_kernels.cuh) against the sequential sweeps, one rounded operation at a
time: its 8-byte mailboxes, its quotient's exponent range, and operands outside it.

gaussSeidelSweeps (src/OpenFOAM/matrices/smooth_solver_cpp.cu:87-166) restated in FP32: a row's terms are rounded
products subtracted in the row's order, lower neighbours then upper ones, then one division.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from brae_b200 import cases  # noqa: E402


@pytest.fixture(scope="module")
def b2g():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import brae_b200.native as n
    return n


def dev(a, dtype=torch.float32):
    return torch.as_tensor(np.ascontiguousarray(a)).to(device="cuda", dtype=dtype)


def _rows(lower, upper, coef, n):
    rows = [[] for _ in range(n)]
    for f in range(len(lower)):
        rows[upper[f]].append((int(lower[f]), coef[f]))
    for f in range(len(lower)):
        rows[lower[f]].append((int(upper[f]), coef[f]))
    return rows


def _sweeps(rows, diag, psi, b, n_sweeps, symmetric):
    x = psi.astype(np.float32).copy()
    n = len(rows)
    with np.errstate(all="ignore"):
        for _ in range(n_sweeps):
            for order in ((range(n), range(n - 1, -1, -1)) if symmetric else (range(n),)):
                for c in order:
                    acc = b[c]
                    for o, v in rows[c]:
                        acc = np.float32(acc - np.float32(v * x[o]))
                    x[c] = np.float32(acc / diag[c])
    return x


def _same(got, want):
    return np.array_equal(got, want, equal_nan=True) and np.array_equal(
        np.signbit(got[~np.isnan(want)]), np.signbit(want[~np.isnan(want)]))


@pytest.mark.parametrize("symmetric", [False, True])
def test_sweeps_bitexact(b2g, symmetric):
    c = cases.box_case(19, 13, 11, (2.0, 1.0, 1.0), 5.0)
    mesh = b2g.Mesh(c.lower, c.upper, c.Sf, c.magSf, c.n_cells, 10, True)
    A = b2g.Matrix(mesh, c.diag, c.coef)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(9)
    for lv in (0, 1, 3):
        lo, up = (c.lower, c.upper) if lv == 0 else (mesh.step(lv - 1)["lower"], mesh.step(lv - 1)["upper"])
        d, u = (a.astype(np.float32) for a in A.level(lv))
        n = d.shape[0]
        rows = _rows(lo, up, u, n)
        x0, b = (rng.uniform(-1.0, 1.0, n).astype(np.float32) for _ in range(2))
        for sweeps in (1, 3):
            want = _sweeps(rows, d, x0, b, sweeps, symmetric)
            for ranks, weight in ((0, 1), (1, 1), (2, 4), (7, 1), (sms, 4)):
                if ranks > n:
                    continue
                x = dev(x0)
                A.smooth_flow32(lv, x, dev(b), sweeps, ranks, weight, symmetric)
                assert _same(x.cpu().numpy(), want), (lv, sweeps, ranks)


# the quick quotient takes operands of exponents within 60 of 1: diagonals and sources at the bounds and past them,
# subnormal, zero, infinite and NaN ones
@pytest.mark.parametrize("exponent", [0, 58, 61, 100, -58, -61, -100])
def test_quotient_edges(b2g, exponent):
    c = cases.box_case(11, 9, 8, (2.0, 1.0, 1.0), 5.0)
    # (the magnitudes of diagonal and coefficients about 1 before scaling)
    s = 2.0 ** exponent / np.abs(c.diag).max()
    mesh = b2g.Mesh(c.lower, c.upper, c.Sf, c.magSf, c.n_cells, 10, True)
    A = b2g.Matrix(mesh, c.diag * s, c.coef * s)
    d, u = (c.diag * s).astype(np.float32), (c.coef * s).astype(np.float32)
    rows = _rows(c.lower, c.upper, u, c.n_cells)
    rng = np.random.default_rng(10)
    x0 = np.zeros(c.n_cells, np.float32)
    for special in (None, np.inf, np.nan):
        b = (rng.uniform(-1.0, 1.0, c.n_cells) * 2.0 ** rng.uniform(-140, 120, c.n_cells)).astype(np.float32)
        near = rng.random(c.n_cells) < 0.5
        b[near] = (rng.uniform(0.5, 2.0, near.sum()) * 2.0 ** rng.choice([-61, -60, -59, 59, 60, 61], near.sum())).astype(np.float32)
        b[::5] = np.where(rng.random(b[::5].size) < 0.5, np.float32(0.0), np.float32(-0.0))
        if special is not None:
            b[c.n_cells // 2] = special
        want = _sweeps(rows, d, x0, b, 2, False)
        for ranks in (0, 1, 8):
            x = dev(x0)
            A.smooth_flow32(0, x, dev(b), 2, ranks, 4 if ranks > 1 else 1)
            assert _same(x.cpu().numpy(), want), (special, ranks)
