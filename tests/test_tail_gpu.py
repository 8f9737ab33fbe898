"""The fused V-cycle tail (csrc/cycle_tail.cu) against the oracle's V-cycle and, bit for
bit, against the cycle with every pass in its own launch: entry at level 0 (few rows; odd
and even sizes, an odd address), with and without the entry level's restriction and
prolongation in the launch, several sweeps, FP64 and FP32."""
import ctypes as C

import numpy as np
import pytest

from linalglib_b200 import _lib as L
from linalglib_b200 import problems as P

pytestmark = pytest.mark.gpu

CASES = [  # with the entry level and whether R and P are in the launch
    ("2d 11", lambda: P.poisson2d(11), 0, 1),  # odd: in the launch for no FP64 iterate
    ("2d 12", lambda: P.poisson2d(12), 0, 1),
    ("2d 40", lambda: P.poisson2d(40), 0, 0),
    ("2d 61", lambda: P.poisson2d(61), 1, 1),
    ("2d 100x83", lambda: P.poisson2d(100, 83), 1, 0),
    ("3d 13", lambda: P.poisson3d(13), 1, 1),  # long rows
    ("3d 24", lambda: P.poisson3d(24), 2, 1),
    ("27pt 12", lambda: P.diffusion27(12), 1, 1),
]


def _tail_info(H, opts):
    entry, transfers = C.c_int(), C.c_int()
    L.call("lab_hierarchy_tail_info", H.h, C.byref(opts), C.byref(entry), C.byref(transfers))
    return entry.value, transfers.value


@pytest.mark.parametrize("n1, n2", [(1, 1), (2, 1), (1, 0), (3, 2)])
@pytest.mark.parametrize("name, make, entry, transfers", CASES, ids=[c[0] for c in CASES])
def test_tail_matches_oracle_cycle(gpu, oracle, name, make, entry, transfers, n1, n2):
    import torch
    A = make()
    m = A[0].size - 1
    H = gpu.Hierarchy(gpu.CsrMatrix.from_arrays(*A), kind=L.AMG_SA)
    r = np.random.default_rng(m).uniform(-1, 1, m)
    zo = oracle.amg_setup(A, kind=0).vcycle(r, n1=n1, n2=n2, omega=2.0 / 3.0, coarse=1)
    # sums of at most ~200 products on each of a few dozen passes: 2^-53 and 2^-24 times
    # a few hundred, in the norm of the result
    for precision, tol in ((L.PREC_FP64, 1e-12), (L.PREC_FP32, 4e-5)):
        opts = gpu.amg_options(n1=n1, n2=n2, omega=2.0 / 3.0, precision=precision)
        M = gpu.Preconditioner.amg(H, opts)
        L.call("lab_hierarchy_set_tail", H.h, 0)
        assert _tail_info(H, opts) == (-1, 0)
        passes = M.apply(gpu.vec(r)).cpu().numpy()
        L.call("lab_hierarchy_set_tail", H.h, 1)
        assert _tail_info(H, opts) == (entry, transfers)
        for shift in (0, 1):  # z at a 16-byte boundary and 8 bytes off it
            z = torch.full((m + 3,), 7.0, dtype=torch.float64, device="cuda")
            M.apply(gpu.vec(r), z[shift:shift + m])
            z = z.cpu().numpy()
            assert np.max(np.abs(z[shift:shift + m] - zo)) <= tol * np.max(np.abs(zo))
            assert np.array_equal(z[shift:shift + m].view(np.int64), passes.view(np.int64))
            assert np.all(z[:shift] == 7.0) and np.all(z[shift + m:] == 7.0)


def _lone(A, rows):
    """A with the rows and columns of the given unknowns cut down to their diagonal: they
    have no strong neighbour, so no aggregate, and their rows of P are empty."""
    rp, ci, v = A[:3]
    r = np.repeat(np.arange(rp.size - 1), np.diff(rp))
    keep = ~(np.isin(r, rows) | np.isin(ci, rows)) | (r == ci)
    cnt = np.bincount(r[keep], minlength=rp.size - 1)
    return np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32), ci[keep], v[keep]


@pytest.mark.parametrize("lanes", [0, 2, 8, 32])
@pytest.mark.parametrize("make", [lambda: P.poisson2d(14), lambda: P.poisson2d(16),
                                  lambda: P.poisson3d(13)], ids=["2d 14", "2d 16", "3d 13"])
def test_tail_empty_rows(gpu, oracle, make, lanes):
    """Empty rows of P, in the middle and at the end (its entries not a multiple of four,
    so that the row starts inside a group of four), with P and R summed by several
    lanes a row: a row without entries reads none."""
    A = make()
    m = A[0].size - 1
    A = _lone(A, [m // 2, m - 2, m - 1])
    H = gpu.Hierarchy(gpu.CsrMatrix.from_arrays(*A), kind=L.AMG_SA)
    rp = H.P(0).to_numpy()[0]
    assert rp[m - 2] == rp[m] and rp[m // 2] == rp[m // 2 + 1]
    r = np.random.default_rng(m).uniform(-1, 1, m)
    zo = oracle.amg_setup(A, kind=0).vcycle(r, n1=1, n2=1, omega=2.0 / 3.0, coarse=1)
    if lanes:
        for l in range(H.levels):
            for M in (H.P(l), H.R(l)):
                M.set_algorithm(L.SPMV_VECTOR, lanes)
    for precision, tol in ((L.PREC_FP64, 1e-12), (L.PREC_FP32, 4e-5)):
        opts = gpu.amg_options(omega=2.0 / 3.0, precision=precision)
        M = gpu.Preconditioner.amg(H, opts)
        assert _tail_info(H, opts)[0] == (1 if m > 1000 else 0)
        z = M.apply(gpu.vec(r)).cpu().numpy()
        assert np.max(np.abs(z - zo)) <= tol * np.max(np.abs(zo))
        L.call("lab_hierarchy_set_tail", H.h, 0)
        passes = M.apply(gpu.vec(r)).cpu().numpy()
        L.call("lab_hierarchy_set_tail", H.h, 1)
        assert np.array_equal(z.view(np.int64), passes.view(np.int64))


@pytest.mark.parametrize("n, launches", [(14, 3), (16, 3), (18, 5), (20, 5), (26, 5)])
def test_tail_dense_coarse_rows(gpu, oracle, n, launches):
    """Coarsest levels of 50 and 64 rows are solved in the tail's one launch (after the
    first pass over level 0 and before its last), of 82, 98 and 170 rows on the whole GPU."""
    A = P.poisson2d(n)
    H = gpu.Hierarchy(gpu.CsrMatrix.from_arrays(*A), kind=L.AMG_SA, max_level=1)
    M = gpu.Preconditioner.amg(H, gpu.amg_options(omega=2.0 / 3.0))
    r = np.random.default_rng(n).uniform(-1, 1, n * n)
    rd = gpu.vec(r)
    n0 = gpu.launch_count()
    z = M.apply(rd)
    assert gpu.launch_count() - n0 == launches
    zo = oracle.amg_setup(A, kind=0, max_level=1).vcycle(r, n1=1, n2=1, omega=2.0 / 3.0, coarse=1)
    # the two inverses round differently, by the coarsest operator's condition number (< 1e4)
    assert np.max(np.abs(z.cpu().numpy() - zo)) <= 1e-11 * np.max(np.abs(zo))


def test_first_cycle_of_a_process_can_be_captured(gpu):
    """A preconditioner's first application may run inside the caller's stream capture:
    what the cycle needs is allocated when the preconditioner is built.  (In a process
    of its own, where nothing has run before.)"""
    import os
    import subprocess
    import sys
    code = """
import numpy as np, torch
from linalglib_b200 import core, _lib as L, problems as P
A = P.poisson2d(61)
r = core.vec(np.random.default_rng(0).uniform(-1, 1, 61 * 61))
for precision in (L.PREC_FP64, L.PREC_FP32):
    M = core.Preconditioner.amg(core.Hierarchy(core.CsrMatrix.from_arrays(*A)),
                                core.amg_options(omega=2.0 / 3.0, precision=precision))
    z = torch.zeros_like(r)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        M.apply(r, z)
    g.replay()
    assert torch.equal(z, M.apply(r)) and float(z.abs().max()) > 0.0
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]


def _timeouts(gpu):
    n = C.c_int64()
    L.call("lab_wait_timeouts", C.byref(n), gpu.stream_handle())
    return n.value


def test_tail_wait_that_runs_out(gpu):
    """The tail's wait for its operators is bounded.  Held back (a barrier that waits for
    an arrival that never comes), the cycle's result is NaN, the wait is counted, every
    solve returns LAB_TIMEOUT, and the next solves run as if nothing had been.  (In a process
    of its own: the device's count stays 0 in this one.)"""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    p = subprocess.run([sys.executable, "-c", "import sys; sys.path.insert(0, 'tests'); "
                        "import test_tail_gpu as t; t._wait_that_runs_out()"],
                       cwd=os.path.dirname(here), capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]


def _wait_that_runs_out():
    from linalglib_b200 import core as gpu
    for make in (lambda: P.poisson2d(61), lambda: P.poisson2d(100, 83)):  # with R and P, without
        for precision in (L.PREC_FP64, L.PREC_FP32):
            _solves_with_a_held_wait(gpu, make, precision)


def _solves_with_a_held_wait(gpu, make, precision):
    A = make()
    m = A[0].size - 1
    dA = gpu.CsrMatrix.from_arrays(*A)
    H = gpu.Hierarchy(dA, kind=L.AMG_SA)
    opts = gpu.amg_options(omega=2.0 / 3.0, precision=precision)
    b = gpu.vec(np.random.default_rng(m).uniform(-1, 1, m))
    M = gpu.Preconditioner.amg(H, opts)
    want, info = gpu.pcg(dA, b, M=M)
    L.call("lab_hierarchy_wait_control", H.h, 256, 1)
    M = gpu.Preconditioner.amg(H, opts)
    n0 = _timeouts(gpu)
    assert np.isnan(M.apply(b).cpu().numpy()).all() and _timeouts(gpu) == n0 + 1
    offsets = np.array([0, m], dtype=np.int64)
    for solve in (lambda: gpu.pcg(dA, b, M=M), lambda: gpu.gmres(dA, b, M=M),
                  lambda: gpu.adjoint_solve(dA, b, M), lambda: H.solve(b, options=opts),
                  lambda: gpu.batched_pcg(dA, offsets, b, M)):
        with pytest.raises(L.LabError) as e:
            solve()
        assert e.value.status == L.LAB_TIMEOUT
    L.call("lab_hierarchy_wait_control", H.h, 0, 0)
    M = gpu.Preconditioner.amg(H, opts)
    n0 = _timeouts(gpu)
    x, again = gpu.pcg(dA, b, M=M)
    assert again.iterations == info.iterations and bool((x == want).all()) and _timeouts(gpu) == n0


@pytest.mark.parametrize("alg, lanes", [(L.SPMV_ROWSEQ, 0), (L.SPMV_VECTOR, 4),
                                        (L.SPMV_VECTOR_STREAM, 8), (L.SPMV_VECTOR_HALO, 4),
                                        (L.SPMV_VECTOR_HALO, 32)])
def test_tail_keeps_the_order_of_the_schedules(gpu, alg, lanes):
    """The tail sums a row in the order of its operator's schedule, also where that is
    the streamed or the halo form of several lanes a row."""
    A = P.poisson2d(61)
    H = gpu.Hierarchy(gpu.CsrMatrix.from_arrays(*A), kind=L.AMG_SA)
    for l in range(1, H.levels):
        for M in (H.A(l), H.P(l), H.R(l)):
            M.set_algorithm(alg, lanes)
    r = gpu.vec(np.random.default_rng(61).uniform(-1, 1, 61 * 61))
    for precision in (L.PREC_FP64, L.PREC_FP32):
        opts = gpu.amg_options(n1=2, n2=2, omega=2.0 / 3.0, precision=precision)
        M = gpu.Preconditioner.amg(H, opts)
        assert _tail_info(H, opts)[0] == 1
        z = M.apply(r)
        L.call("lab_hierarchy_set_tail", H.h, 0)
        passes = M.apply(r)
        L.call("lab_hierarchy_set_tail", H.h, 1)
        assert bool((z == passes).all())
