"""Block PCG over interleaved columns (csrc/cycle_blk.cu) at odd and even column counts,
one and two blocks, short and long rows, a zero column and a nonzero guess, against the
oracle's PCG column by column."""
import numpy as np
import pytest

from linalglib_b200 import _lib as L
from linalglib_b200 import problems as P

pytestmark = pytest.mark.gpu

OPS = {"2d 31x40": lambda: P.poisson2d(31, 40), "3d 12": lambda: P.poisson3d(12),
       "27pt 9": lambda: P.diffusion27(9)}


@pytest.mark.parametrize("n1, n2", [(1, 1), (2, 2)])
@pytest.mark.parametrize("ncols", [1, 2, 5, 32, 65])
@pytest.mark.parametrize("op", list(OPS))
def test_block_pcg(gpu, oracle, op, ncols, n1, n2):
    A = OPS[op]()
    m = A[0].size - 1
    rng = np.random.default_rng(ncols)
    B = np.stack([P.csr_matvec(*A, rng.uniform(-1, 1, m)) for _ in range(ncols)])
    X0 = np.zeros((ncols, m))
    if ncols > 2:
        B[1] = 0.0
        X0[2] = rng.uniform(-1, 1, m)
    dA = gpu.CsrMatrix.from_arrays(*A)
    M = gpu.Preconditioner.amg(gpu.Hierarchy(dA, kind=L.AMG_SA),
                               gpu.amg_options(n1=n1, n2=n2, omega=2.0 / 3.0))
    X, iters, conv, info = gpu.multi_rhs_pcg(
        dA, gpu.vec(B).reshape(ncols, m), M, X=gpu.vec(X0).reshape(ncols, m),
        control=gpu.iter_control(rel_tol=1e-9, abs_tol=0.0))
    assert info.converged == 1 and np.all(conv == 1)
    X = X.cpu().numpy()
    H = oracle.amg_setup(A, kind=0)
    for k in range(min(ncols, 6)):
        if k == 1 and ncols > 2:
            assert iters[k] == 0 and np.all(X[k] == 0.0)
            continue
        xo, it, _ = H.pcg(B[k], x0=X0[k], n1=n1, n2=n2, omega=2.0 / 3.0, coarse=1, rel_tol=1e-9)
        assert abs(int(iters[k]) - it) <= 1
        # both stop at a relative residual of 1e-9; condition numbers are below 1e4
        assert np.max(np.abs(X[k] - xo)) <= 1e-5 * np.max(np.abs(xo))
    for k in range(ncols):
        r = B[k] - P.csr_matvec(*A, X[k])
        assert np.max(np.abs(r)) <= 2e-9 * max(np.max(np.abs(B[k] - P.csr_matvec(*A, X0[k]))), 1e-30)


@pytest.mark.parametrize("ncols", [1, 2, 5, 33, 64])
@pytest.mark.parametrize("n, nc", [(16, 64), (26, 170), (48, 545), (52, 647)])
def test_block_dense_coarse_level(gpu, oracle, n, nc, ncols):
    """A coarsest level solved by its dense inverse, on both sides of the number of rows
    (four per SM) from which a CTA takes four of them, the last ones a remainder."""
    A = P.poisson2d(n)
    rng = np.random.default_rng(n + ncols)
    B = np.stack([P.csr_matvec(*A, rng.uniform(-1, 1, n * n)) for _ in range(ncols)])
    dA = gpu.CsrMatrix.from_arrays(*A)
    H = gpu.Hierarchy(dA, kind=L.AMG_SA, max_level=1)
    assert H.A(1).m == nc
    M = gpu.Preconditioner.amg(H, gpu.amg_options(omega=2.0 / 3.0))
    X, iters, conv, info = gpu.multi_rhs_pcg(dA, gpu.vec(B).reshape(ncols, n * n), M,
                                             control=gpu.iter_control(rel_tol=1e-9, abs_tol=0.0))
    assert info.converged == 1 and np.all(conv == 1)
    X = X.cpu().numpy()
    Ho = oracle.amg_setup(A, kind=0, max_level=1)
    for k in range(min(ncols, 3)):
        xo, it, _ = Ho.pcg(B[k], omega=2.0 / 3.0, coarse=1, rel_tol=1e-9)
        assert abs(int(iters[k]) - it) <= 1
        assert np.max(np.abs(X[k] - xo)) <= 1e-5 * np.max(np.abs(xo))
    for k in range(ncols):
        assert np.max(np.abs(B[k] - P.csr_matvec(*A, X[k]))) <= 2e-9 * np.max(np.abs(B[k]))


@pytest.mark.parametrize("op", list(OPS))
def test_one_column_takes_the_single_cycle(gpu, op):
    """One right-hand side takes the single-vector cycle (whose last levels are one launch:
    fewer launches than the block cycle of two columns makes in as many iterations)."""
    A = OPS[op]()
    m = A[0].size - 1
    dA = gpu.CsrMatrix.from_arrays(*A)
    M = gpu.Preconditioner.amg(gpu.Hierarchy(dA, kind=L.AMG_SA), gpu.amg_options(omega=2.0 / 3.0))
    b = gpu.vec(np.random.default_rng(m).uniform(-1, 1, m))
    ctl = gpu.iter_control(rel_tol=1e-9, abs_tol=0.0)
    launches, out = [], []
    for k in (1, 2):
        n0 = gpu.launch_count()
        X, it, _, _ = gpu.multi_rhs_pcg(dA, b.expand(k, m).contiguous(), M, control=ctl)
        launches.append((gpu.launch_count() - n0) / (int(it[0]) + 1))
        out.append(X[0].cpu().numpy())
    assert launches[0] < launches[1]
    assert np.max(np.abs(out[0] - out[1])) <= 1e-5 * np.max(np.abs(out[0]))


@pytest.mark.parametrize("ncols", [64, 33])
def test_block_width_by_memory(gpu, ncols):
    """A block that does not fit the memory it may take is solved in narrower ones; two
    columns that do not fit are an error that leaves X as it was.  Scratch of more than
    64 MB is given back after the solve."""
    A = P.poisson3d(40)
    m = A[0].size - 1
    rng = np.random.default_rng(ncols)
    dA = gpu.CsrMatrix.from_arrays(*A)
    H = gpu.Hierarchy(dA, kind=L.AMG_SA)
    M = gpu.Preconditioner.amg(H, gpu.amg_options(omega=2.0 / 3.0))
    B = gpu.vec(np.stack([P.csr_matvec(*A, rng.uniform(-1, 1, m)) for _ in range(ncols)]))
    B = B.reshape(ncols, m)
    ctl = gpu.iter_control(rel_tol=1e-9, abs_tol=0.0)
    want, it0, conv, _ = gpu.multi_rhs_pcg(dA, B, M, control=ctl)
    assert np.all(conv == 1)
    want = want.cpu().numpy()
    column = 8 * (7 * m + sum(4 * H.A(l).m for l in range(1, H.levels + 1)))
    for width in (16, 3, 2):
        L.call("lab_hierarchy_block_memory", H.h, column * (width + width % 2))
        X, it, conv, info = gpu.multi_rhs_pcg(dA, B, M, control=ctl)
        assert info.converged == 1 and np.all(conv == 1) and np.max(np.abs(it - it0)) <= 1
        X = X.cpu().numpy()
        assert np.max(np.abs(X - want)) <= 1e-5 * np.max(np.abs(want))
    L.call("lab_hierarchy_block_memory", H.h, 2 * column - 1)
    X = B.clone()
    with pytest.raises(L.LabError) as e:
        gpu.multi_rhs_pcg(dA, B, M, X=X, control=ctl)
    assert e.value.status == L.LAB_OOM and bool((X == B).all())
    L.call("lab_hierarchy_block_memory", H.h, 0)


def test_block_scratch_is_given_back(gpu):
    """The level scratch of a wide block does not stay allocated: after the solve the
    pool holds no more than before it, but for a bounded rest."""
    import ctypes as C
    import torch
    rt = C.CDLL("libcudart.so.12")
    pool = C.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0

    def used():
        torch.cuda.synchronize()
        v = C.c_uint64()
        assert rt.cudaMemPoolGetAttribute(pool, 7, C.byref(v)) == 0  # UsedMemCurrent
        return v.value

    A = P.poisson3d(64)
    m = A[0].size - 1
    dA = gpu.CsrMatrix.from_arrays(*A)
    H = gpu.Hierarchy(dA, kind=L.AMG_SA)
    M = gpu.Preconditioner.amg(H, gpu.amg_options(omega=2.0 / 3.0))
    B = torch.rand((64, m), dtype=torch.float64, device="cuda")
    gpu.multi_rhs_pcg(dA, B[:1], M)
    before = used()
    gpu.multi_rhs_pcg(dA, B, M)
    rows = sum(H.A(l).m for l in range(H.levels + 1))
    assert used() - before <= max(256 * rows, 64 << 20)
