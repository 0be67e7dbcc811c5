"""The data-flow smoothing launch (flow_kernels.cuh) and the V-cycle's fused transfers on small levels
(scaleProlongCluster, restrictChain in ldu_kernels.cuh) against the oracle.

The smoothing launch must give the oracle's sequential sweeps (gaussSeidelSweeps,
src/OpenFOAM/matrices/smooth_solver_cpp.cu:87-166) bit for bit, for any number of CTAs and any step
weight, forward and symmetric, and with operands that leave the quick quotient's exponent range.
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


def dev(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to(device="cuda", dtype=dtype)


def _build(b2g, c, scale=1.0):
    mesh = b2g.Mesh(c.lower, c.upper, c.Sf, c.magSf, c.n_cells, 10, True)
    return mesh, b2g.Matrix(mesh, dev(c.diag * scale), dev(c.coef * scale))


def _level_system(mesh, A, c, lv):
    if lv == 0:
        lo, up = c.lower, c.upper
    else:
        st = mesh.step(lv - 1)
        lo, up = st["lower"], st["upper"]
    d, u = A.level(lv)
    return lo, up, d, u


# a slab one cell thick, odd sizes, a level of many chunks a step; levels down to a dozen cells with rows
# past the register entries
BOXES = [(37, 3, 1, 1.0), (23, 20, 21, 20.0), (48, 44, 45, 1.0)]


@pytest.mark.parametrize("nx,ny,nz,grading", BOXES)
@pytest.mark.parametrize("symmetric", [False, True])
def test_sweeps_bitexact(b2g, oracle, nx, ny, nz, grading, symmetric):
    c = cases.box_case(nx, ny, nz, (2.0, 1.0, 1.0), grading)
    mesh, A = _build(b2g, c)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(3)
    ran = 0
    for lv in range(mesh.n_levels + 1):
        lo, up, d, u = _level_system(mesh, A, c, lv)
        n = d.shape[0]
        x0, b = rng.uniform(-1.0, 1.0, n), rng.uniform(-1.0, 1.0, n)
        for sweeps in (1, 2, 5):
            want = oracle.smooth(lo, up, d, u, x0, b, sweeps, "symGaussSeidel" if symmetric else "GaussSeidel")
            for ranks, weight in ((1, 1), (2, 4), (7, 1), (sms, 4)):
                if ranks > n:
                    continue
                x = dev(x0)
                try:
                    A.smooth_flow(lv, x, dev(b), sweeps, ranks, weight, symmetric=symmetric)
                except b2g.GamgError as e:
                    # the live values of so many cells do not fit one or two CTAs
                    assert e.status == "ARGUMENT" and n / ranks > 10000
                    continue
                assert np.array_equal(x.cpu().numpy(), want), (lv, sweeps, ranks)
                ran += 1
    assert ran > 20


# the quotient's quick form holds for exponents within its bounds only: diagonals and sources past them on
# both sides, subnormal, zero, infinite and NaN operands take the division itself
@pytest.mark.parametrize("scale", [1.0, 1e-160, 1e-300, 1e155, 1e300])
def test_quotient_edges(b2g, oracle, scale):
    c = cases.box_case(19, 17, 13, (2.0, 1.0, 1.0), 5.0)
    mesh, A = _build(b2g, c, scale)
    lo, up, d, u = _level_system(mesh, A, c, 0)
    n = d.shape[0]
    rng = np.random.default_rng(4)
    # magnitudes over the whole range, one row in three of them zero or negative zero
    b = rng.uniform(-1.0, 1.0, n) * 10.0 ** rng.uniform(-320, 300, n)
    b[::3] = np.where(rng.random(b[::3].size) < 0.5, 0.0, -0.0)
    x0 = np.zeros(n)
    with np.errstate(all="ignore"):
        for special in (None, np.inf, np.nan):
            bs = b.copy()
            if special is not None:
                bs[n // 2] = special
            want = oracle.smooth(lo, up, d, u, x0, bs, 2)
            for ranks in (1, 8):
                x = dev(x0)
                A.smooth_flow(0, x, dev(bs), 2, ranks, 4 if ranks > 1 else 1)
                got = x.cpu().numpy()
                assert np.array_equal(got, want, equal_nan=True), (special, ranks)
                finite = np.isfinite(want)
                assert np.array_equal(np.signbit(got[finite]), np.signbit(want[finite]))


# CTA counts and limits that make waits run out at different places of a launch: at the first hand-over, with the
# ring full of chunks under way, on levels of few and of many chunks a CTA
@pytest.mark.parametrize("ranks,limit", [(2, 1 << 10), (7, 1 << 12), (16, 1 << 14), (0, 1 << 12)])
@pytest.mark.parametrize("symmetric", [False, True])
def test_wait_gives_up(b2g, oracle, ranks, limit, symmetric):
    # no rank hands its values over: every rank's wait runs out after a short limit, the launch ends and the
    # call reports a device time-out; the next call on the same matrix is the oracle's
    c = cases.box_case(40, 40, 40, (2.0, 1.0, 1.0), 20.0)
    ranks = ranks or torch.cuda.get_device_properties(0).multi_processor_count
    mesh, A = _build(b2g, c)
    rng = np.random.default_rng(5)
    for lv in (0, 2):
        lo, up, d, u = _level_system(mesh, A, c, lv)
        x0, b = rng.uniform(-1.0, 1.0, d.shape[0]), rng.uniform(-1.0, 1.0, d.shape[0])
        want = oracle.smooth(lo, up, d, u, x0, b, 3, "symGaussSeidel" if symmetric else "GaussSeidel")
        for sweeps in (1, 3):
            status = "OK"
            try:
                A.smooth_flow(lv, dev(x0), dev(b), sweeps, ranks, 4, stall_limit=limit, symmetric=symmetric)
            except b2g.GamgError as e:
                status = e.status
            assert status in ("DEVICE_TIMEOUT", "ARGUMENT"), (lv, sweeps)
            assert status == "DEVICE_TIMEOUT" or d.shape[0] / ranks > 10000  # (ARGUMENT: too many cells for so few)
        x = dev(x0)
        A.smooth_flow(lv, x, dev(b), 3, max(ranks, 7), 4, symmetric=symmetric)
        assert np.array_equal(x.cpu().numpy(), want)


def test_smoothing_calls_on_streams_and_threads(b2g, oracle):
    # two matrices of one mesh share its schedules, not the hand-over words: their smoothing calls, from two
    # threads on streams of their own, give the oracle's sweeps each
    import threading

    c = cases.box_case(40, 38, 36, (2.0, 1.0, 1.0), 20.0)
    mesh = b2g.Mesh(c.lower, c.upper, c.Sf, c.magSf, c.n_cells, 10, True)
    mats = [b2g.Matrix(mesh, dev(c.diag * s), dev(c.coef * s)) for s in (1.0, 3.0)]
    rng = np.random.default_rng(6)
    x0, b = rng.uniform(-1.0, 1.0, c.n_cells), rng.uniform(-1.0, 1.0, c.n_cells)
    for A in mats:  # the schedule is tuned on the first call of a mesh
        A.smooth(0, dev(x0), dev(b), 2)
    got = [[], []]
    torch.cuda.synchronize()

    def work(k):
        for _ in range(10):
            x = dev(x0)
            torch.cuda.current_stream().synchronize()
            mats[k].smooth(0, x, dev(b), 2)
            got[k].append(x.cpu().numpy())

    th = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for k, s in enumerate((1.0, 3.0)):
        want = oracle.smooth(c.lower, c.upper, c.diag * s, c.coef * s, x0, b, 2)
        assert len(got[k]) == 10
        for x in got[k]:
            assert np.array_equal(x, want)


# finest sizes that put a coarse level at, just under and just over a block's, a cluster's and the chain's
# share (1,024 cells a CTA and pass, 32,768 the cluster, 4,096 the chain): a whole tree-order solve against
# the oracle's serial one. Tolerance: sums of n terms in another order differ by at most n eps relative to the
# sum of magnitudes, through 2 dots and a scaling per level and iteration: 1e-10 for these n < 7e4.
@pytest.mark.parametrize("nx,ny,nz", [(32, 32, 2), (41, 25, 2), (32, 16, 16), (33, 25, 10), (64, 32, 32), (64, 33, 32)])
def test_solve_at_transfer_edges(b2g, oracle, nx, ny, nz):
    c = cases.box_case(nx, ny, nz, (2.0, 1.0, 1.0), 3.0)
    mesh, A = _build(b2g, c)
    agg = oracle.agglomerate(c.lower, c.upper, c.Sf, c.magSf, c.n_cells, 10, True)
    want = oracle.pcg_gamg_solve(agg, c.diag, c.coef, c.source, np.zeros(c.n_cells), 1e-8, 0.0)
    x = dev(np.zeros(c.n_cells))
    perf, _, _ = A.solve(dev(c.source), x, b2g.controls_default(tolerance=1e-8))
    assert perf.nIterations == want["perf"][2]
    assert np.abs(x.cpu().numpy() - want["psi"]).max() <= 1e-10 * np.abs(want["psi"]).max()
    # the order of the sums is fixed: every further solve gives the same bits
    for _ in range(4):
        again = dev(np.zeros(c.n_cells))
        A.solve(dev(c.source), again, b2g.controls_default(tolerance=1e-8))
        assert torch.equal(again, x)


_FULL_DEVICE = """
import sys
sys.path.insert(0, {repo!r})
import numpy as np
import torch
import brae_b200.native as b
from brae_b200 import cases

c = cases.box_case(180, 110, 100, (2.0, 1.0, 1.0), 5.0)
mesh = b.Mesh(c.lower, c.upper, c.Sf, c.magSf, c.n_cells, 10, True)
A = b.Matrix(mesh, c.diag, c.coef)
batch_mesh = b.Mesh(c.lower, c.upper, c.Sf, c.magSf, c.n_cells, 10, True)
batch = b.Batch([b.Matrix(batch_mesh, c.diag, c.coef)])
forms = [(p, s) for p in ("fp64", "fp32_precond", "fp32_precond_multicolour") for s in ("GaussSeidel", "symGaussSeidel")]


def solve_all():
    out = {{}}
    for p, s in forms:
        ctl = b.controls_default(tolerance=1e-12, relTol=0.0, precision=p, smoother=s, maxIter=2)
        psi = np.zeros(c.n_cells)
        A.solve(c.source, psi, ctl)
        out[p, s] = psi
        if s == "GaussSeidel":
            psi = np.zeros(c.n_cells)
            batch.solve([c.source], [psi], ctl)
            out[p, "batch"] = psi
    return out


# everything but the smoothing calls' schedules is there once these have run
b.set_sweep_pipeline(False)
want = solve_all()
torch.cuda.synchronize()
free, _ = torch.cuda.mem_get_info()
hold = torch.empty(free - (160 << 20), dtype=torch.uint8, device="cuda")
b.set_sweep_pipeline(True)
got = solve_all()
assert all(np.array_equal(want[k], got[k]) for k in want), [k for k in want if not np.array_equal(want[k], got[k])]
print("SAME", mesh.pipe_shape(0, 2, 8)["ranks"])
"""


def test_no_memory_takes_the_other_forms():
    # a device that has no room for the finest levels' schedules (2 M cells: 0.7 GB and more each): every form
    # solves as it does without them, bit for bit. In a process of its own, whose memory pool holds nothing else.
    import os
    import subprocess
    import sys
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _FULL_DEVICE.format(repo=repo)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "SAME" in r.stdout, (r.stdout[-500:], r.stderr[-1500:])


def test_long_chain_of_steps(b2g):
    # a line of cells is one chain of steps: the last CTA waits for nearly all of them without taking that for a
    # stall; the result is the sweep-by-sweep one
    n = 200_000
    c = cases.box_case(n, 1, 1)
    mesh, A = _build(b2g, c)
    rng = np.random.default_rng(8)
    x0, b = dev(rng.uniform(-1.0, 1.0, n)), dev(rng.uniform(-1.0, 1.0, n))
    x, want = x0.clone(), x0.clone()
    A.smooth_flow(0, x, b, 1, torch.cuda.get_device_properties(0).multi_processor_count, 4)
    A.smooth(0, want, b, 1)  # one sweep: no data flow
    assert torch.equal(x, want)


_SCHEDULES_GO = """
import sys
sys.path.insert(0, {repo!r})
import numpy as np
import torch
import brae_b200.native as b
from brae_b200 import cases

c = cases.box_case(180, 110, 100, (2.0, 1.0, 1.0), 5.0)
new_mesh = lambda: b.Mesh(c.lower, c.upper, c.Sf, c.magSf, c.n_cells, 10, True)
ctl = b.controls_default(tolerance=1e-12, relTol=0.0, maxIter=2)


def solve(A):
    psi = np.zeros(c.n_cells)
    A.solve(c.source, psi, ctl)
    return psi


mesh = new_mesh()
A = b.Matrix(mesh, c.diag, c.coef)
batch_mesh = new_mesh()
batch = b.Batch([b.Matrix(batch_mesh, c.diag, c.coef)])


def solve_batch():
    psi = np.zeros(c.n_cells)
    batch.solve([c.source], [psi], ctl)
    return psi


want, want_batch = solve(A), solve_batch()
assert mesh.schedule_bytes > 100 * c.n_cells
before = mesh.pipe_shape(0, 2, 8)
assert before["ranks"] > 0 and not before["grid"], before
# leave a few GB (and the room rule's eighth is gone): the next matrices, without pipelined launches, take it all
free, _ = torch.cuda.mem_get_info()
hold = torch.empty(free - (2 << 30), dtype=torch.uint8, device="cuda")
more = new_mesh()
b.set_sweep_pipeline(False)
kept = []
try:
    for k in range(200):
        kept.append(b.Matrix(more, c.diag, c.coef))
        solve(kept[-1])
except b.GamgError as e:
    assert e.status == "NO_MEMORY", e
else:
    raise AssertionError("the device was never full")
b.set_sweep_pipeline(True)
after = mesh.pipe_shape(0, 2, 8)
assert after["ms_sweep_by_sweep"] == 0.0, after   # the mesh's schedules went before the call failed
assert mesh.schedule_bytes == 0 and batch_mesh.schedule_bytes == 0
assert np.array_equal(solve(A), want)
assert np.array_equal(solve_batch(), want_batch)
print("SAME", len(kept))
"""


def test_schedules_go_when_memory_is_short():
    # matrices are made until none fits: the schedules of idle meshes are dropped before a call fails, and what
    # had been captured or tabulated with them (a solve's graph, a batch's tables) is remade without, bit for bit
    import os
    import subprocess
    import sys
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _SCHEDULES_GO.format(repo=repo)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "SAME" in r.stdout, (r.stdout[-500:], r.stderr[-1500:])
