"""Level-scheduled triangular path on the GPU: lab_csrtrsv, lab_csrilu0 /
lab_csric0 and the ILU(0) / IC(0) / Gauss-Seidel / SOR / SSOR preconditioners are
bit-identical to the oracle (which is pinned bit-exact to the reference's
host_csrtrsv.cpp, host_csrilu0.cpp, host_csric0.cpp and preconditioner.cpp), and
PCG with them behaves as the reference's cg_solver does."""
import numpy as np
import pytest

from linalglib_b200 import problems as P

pytestmark = pytest.mark.gpu

CASES = {
    "poisson2d_20": lambda: P.poisson2d(20),
    "laplacian3d_8": lambda: P.graph_laplacian3d(8, seed=1),
    "diffusion27_6": lambda: P.diffusion27(6, seed=2),
    "poisson3d_24": lambda: P.poisson3d(24),
}


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float64).view(np.int64)


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("unit", [True, False])
def test_trsv_bit_exact(gpu, oracle, name, lower, unit):
    A = CASES[name]()
    b = np.random.default_rng(3).uniform(-1, 1, A[0].size - 1)
    x = gpu.CsrMatrix.from_arrays(*A[:3]).trsv(gpu.vec(b), lower=lower, unit_diag=unit)
    assert np.array_equal(_bits(x.cpu().numpy()), _bits(oracle.trsv(A, b, lower, unit)))


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("kind", ["ilu0", "ic0"])
def test_factor_bit_exact(gpu, oracle, name, kind):
    A = CASES[name]()
    dA = gpu.CsrMatrix.from_arrays(*A[:3])
    sz, nz = dA.factor(kind)
    vo, so, no = getattr(oracle, "csr" + kind)(A)
    big = np.iinfo(np.int32).max
    assert (sz, nz) == (-1 if so == big else so, -1 if no == big else no)
    assert np.array_equal(_bits(dA.to_numpy()[2]), _bits(vo))


def test_factor_zero_pivots(gpu, oracle):
    # numeric zero on row 3's diagonal, structural zero (no diagonal) in row 5:
    # the level-parallel and sequential paths must both report the smallest column
    rp, ci, v = P.poisson2d(4)
    v = v.copy()
    for j in range(rp[3], rp[4]):
        if ci[j] == 3:
            v[j] = 0.0
    keep = np.ones(v.size, dtype=bool)
    for j in range(rp[5], rp[6]):
        if ci[j] == 5:
            keep[j] = False
    rows = np.repeat(np.arange(rp.size - 1), np.diff(rp))[keep]
    A = (np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=rp.size - 1))]).astype(np.int32),
         ci[keep].copy(), v[keep].copy())
    for kind in ("ilu0", "ic0"):
        dA = gpu.CsrMatrix.from_arrays(*A)
        sz, nz = dA.factor(kind)
        vo, so, no = getattr(oracle, "csr" + kind)(A)
        big = np.iinfo(np.int32).max
        assert (sz, nz) == (-1 if so == big else so, -1 if no == big else no), kind
        assert np.array_equal(_bits(dA.to_numpy()[2]), _bits(vo)), kind


def _precond(gpu, kind, dA, omega=1.3):
    return [gpu.Preconditioner.ilu0, gpu.Preconditioner.ic0, gpu.Preconditioner.gauss_seidel,
            lambda X: gpu.Preconditioner.sor(X, omega),
            lambda X: gpu.Preconditioner.ssor(X, omega)][kind](dA)


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("kind", [0, 1, 2, 3, 4])
def test_precond_apply_bit_exact(gpu, oracle, name, kind):
    A = CASES[name]()
    dA = gpu.CsrMatrix.from_arrays(*A[:3])
    M = _precond(gpu, kind, dA)
    r = np.random.default_rng(4).uniform(-1, 1, A[0].size - 1)
    z = M.apply(gpu.vec(r)).cpu().numpy()
    assert np.array_equal(_bits(z), _bits(oracle.precond_apply(kind, A, r, omega=1.3)))
    # the preconditioner works on a copy: A itself is unchanged
    assert np.array_equal(_bits(dA.to_numpy()[2]), _bits(A[2]))


@pytest.mark.parametrize("kind,omega,expected", [(0, 1.0, 24), (4, 1.3, 32), (4, 1.0, 26)])
def test_ilu_ssor_pcg_matches_reference(gpu, reference, kind, omega, expected):
    A = P.poisson2d(24)
    b, xt = P.rhs_from_solution(*A[:3], seed=0)
    dA = gpu.CsrMatrix.from_arrays(*A[:3])
    x, info = gpu.pcg(dA, gpu.vec(b), M=_precond(gpu, kind, dA, omega),
                      control=gpu.iter_control(rel_tol=1e-8, abs_tol=0.0, max_iter=1000))
    xr, itr = reference.precond_cg(kind, A, b, omega=omega, rel_tol=1e-8, abs_tol=1e-300)
    assert itr == expected  # the reference's count on this problem
    assert info.converged == 1
    assert abs(info.iterations - itr) <= 1, (info.iterations, itr)
    assert np.max(np.abs(x.cpu().numpy() - xr)) <= 1e-7 * np.max(np.abs(xr))
    assert np.max(np.abs(x.cpu().numpy() - xt)) <= 1e-6


@pytest.mark.parametrize("kind", [1, 2, 3])
def test_nonsymmetric_precond_pcg_like_reference(gpu, reference, kind):
    # The reference's IC(0) factor overwrites only the lower triangle and its
    # upper solve reads the unfactored upper part (host_csric0.cpp:70-115,
    # preconditioner.cpp:512-525); Gauss-Seidel and SOR are one-sided.  None is
    # symmetric, so the reference's CG stagnates with them: the device path must
    # do the same (not converged, the same iterate after 50 iterations).
    A = P.poisson2d(24)
    b, _ = P.rhs_from_solution(*A[:3], seed=0)
    dA = gpu.CsrMatrix.from_arrays(*A[:3])
    M = _precond(gpu, kind, dA)
    x, info = gpu.pcg(dA, gpu.vec(b), M=M,
                      control=gpu.iter_control(rel_tol=1e-8, abs_tol=0.0, max_iter=50))
    xr, itr = reference.precond_cg(kind, A, b, omega=1.3, rel_tol=1e-8, abs_tol=1e-300,
                                   max_iter=50)
    assert itr == 51 and info.converged == 0
    assert np.max(np.abs(x.cpu().numpy() - xr)) <= 1e-6 * np.max(np.abs(xr))


@pytest.mark.parametrize("name", ["poisson3d_24", "diffusion27_6"])
def test_nonsymmetric_preconds_under_gmres(gpu, name):
    # Gauss-Seidel and SOR are one-sided: they work under GMRES (the reference's
    # IC(0), whose upper solve reads the unfactored upper part, does not converge
    # under GMRES either: its application is checked bit for bit above)
    A = CASES[name]()
    b, xt = P.rhs_from_solution(*A[:3], seed=1)
    dA = gpu.CsrMatrix.from_arrays(*A[:3])
    for M in (gpu.Preconditioner.gauss_seidel(dA), gpu.Preconditioner.sor(dA, 1.2)):
        x, info = gpu.gmres(dA, gpu.vec(b), M=M, restart=30,
                            control=gpu.iter_control(rel_tol=1e-10, abs_tol=0.0, max_iter=2000))
        assert info.converged == 1
        assert np.max(np.abs(x.cpu().numpy() - xt)) <= 1e-6 * np.max(np.abs(xt))


def test_trsv_in_place_and_ssor_arg_check(gpu, oracle):
    A = P.poisson3d(12)
    b = np.random.default_rng(7).uniform(-1, 1, A[0].size - 1)
    dA = gpu.CsrMatrix.from_arrays(*A[:3])
    for lower in (True, False):
        xb = gpu.vec(b)
        dA.trsv(xb, lower=lower, unit_diag=False, x=xb)  # b and x the same array
        assert np.array_equal(_bits(xb.cpu().numpy()), _bits(oracle.trsv(A, b, lower, False)))
    from linalglib_b200 import _lib as L
    for bad in (0.0, 2.0, -1.0):
        with pytest.raises(L.LabError):
            gpu.Preconditioner.ssor(dA, bad)


def _random_nonsym(n, per_row, seed):
    """Random nonsymmetric pattern (sorted rows, stored diagonal, a few empty
    off-diagonal rows) with diagonally dominant values."""
    rng = np.random.default_rng(seed)
    rp, ci, v = [0], [], []
    for i in range(n):
        k = 0 if i % 17 == 5 else rng.integers(1, per_row + 1)
        cols = set(rng.choice(n, size=min(k, n), replace=False).tolist()) - {i}
        cols = sorted(cols | {i})
        vals = rng.uniform(-1, 1, len(cols))
        vals[cols.index(i)] = len(cols) + 1.0
        ci += cols
        v += vals.tolist()
        rp.append(len(ci))
    return (np.array(rp, np.int32), np.array(ci, np.int32), np.array(v, np.float64))


@pytest.mark.parametrize("n,per_row,seed", [(1, 1, 0), (2, 2, 1), (300, 6, 2), (2000, 12, 3)])
def test_nonsymmetric_patterns_bit_exact(gpu, oracle, n, per_row, seed):
    # the level analysis reads the dependents of a row through the pattern's
    # transpose: nonsymmetric patterns exercise it
    A = _random_nonsym(n, per_row, seed)
    b = np.random.default_rng(seed + 10).uniform(-1, 1, n)
    dA = gpu.CsrMatrix.from_arrays(*A)
    for lower in (True, False):
        for unit in (True, False):
            x = dA.trsv(gpu.vec(b), lower=lower, unit_diag=unit)
            assert np.array_equal(_bits(x.cpu().numpy()), _bits(oracle.trsv(A, b, lower, unit)))
    for kind in (0, 1, 2, 3, 4):
        z = _precond(gpu, kind, dA).apply(gpu.vec(b)).cpu().numpy()
        assert np.array_equal(_bits(z), _bits(oracle.precond_apply(kind, A, b, omega=1.3))), kind


@pytest.mark.parametrize("lower", [True, False])
def test_trsv_bounded_wait_reports_timeout(gpu, oracle, lower):
    """The solves poll for their dependencies with a bounded wait.  A held row
    (its value never written) makes every row that depends on it run out of its
    wait: the launch must return and the call report LAB_TIMEOUT, and the same
    matrix must solve bit-exactly again once the hold is lifted."""
    import ctypes as C
    from linalglib_b200 import _lib as L
    A = P.poisson3d(24)
    m = A[0].size - 1
    b = np.random.default_rng(4).uniform(-1, 1, m)
    dA = gpu.CsrMatrix.from_arrays(*A[:3])
    held = 0 if lower else m - 1  # the first row solved; every other row depends on it
    L.call("lab_csrtrsv_wait_control", dA.h, 1 << 12, held, gpu.stream_handle())
    bx, x = gpu.vec(b), gpu.vec(np.zeros(m))
    st = L.lib().lab_csrtrsv(dA.h, int(lower), 0, gpu.ptr(bx), gpu.ptr(x), gpu.stream_handle())
    assert st == L.LAB_TIMEOUT, L.lib().lab_last_error().decode()
    assert "wait" in L.lib().lab_last_error().decode()
    L.call("lab_csrtrsv_wait_control", dA.h, 0, -1, gpu.stream_handle())
    x = dA.trsv(gpu.vec(b), lower=lower)
    assert np.array_equal(_bits(x.cpu().numpy()), _bits(oracle.trsv(A, b, lower, False)))


MEMBER_CASES = {
    "poisson2d_20": lambda: P.poisson2d(20),
    "diffusion27_6": lambda: P.diffusion27(6, seed=2),
    "nonsym_18": lambda: _nonsym(18),
}


def _nonsym(n):
    rp, ci, v = P.poisson2d(n)
    v = v.copy()
    rows = np.repeat(np.arange(rp.size - 1), np.diff(rp))
    v[ci == rows + 1] *= 0.37
    v[ci == rows - n] *= 1.9
    return rp, ci, v


@pytest.mark.parametrize("name", list(MEMBER_CASES))
def test_triangle_copies_match_reference(gpu, reference, name):
    """copy_lower_triangular_from / copy_upper_triangular_from
    (csr_matrix.cpp:170-225): same pattern, same values."""
    from helpers import csr_diff, csr_equal
    A = MEMBER_CASES[name]()
    dA = gpu.CsrMatrix.from_arrays(*A)
    for upper in (False, True):
        g = dA.triangle(upper=upper).to_numpy()
        r = reference.triangle(A, upper=upper)
        assert csr_equal(g, r), csr_diff(g, r)


@pytest.mark.parametrize("name", list(MEMBER_CASES))
def test_diagonal_scalings_match_reference(gpu, reference, name):
    """scale_diagonal_by and scale_by_inverse_diagonal (host_scale.cpp:34-69)."""
    A = MEMBER_CASES[name]()
    dA = gpu.CsrMatrix.from_arrays(*A)
    dA.scale_diagonal(-2.75)
    assert np.array_equal(_bits(dA.to_numpy()[2]), _bits(reference.scale_diagonal(A, -2.75)))
    dB = gpu.CsrMatrix.from_arrays(*A)
    dB.scale_by_inverse_diagonal()
    assert np.array_equal(_bits(dB.to_numpy()[2]), _bits(reference.scale_by_inverse_diagonal(A)))
    # the scaled matrix's cached diagonal is rebuilt (the next Jacobi sees new values)
    assert np.array_equal(dB.diagonal().cpu().numpy(),
                          [dB.to_numpy()[2][j] for j in
                           [next(k for k in range(A[0][i], A[0][i + 1]) if A[1][k] == i)
                            for i in range(A[0].size - 1)]])


def _band(n, k, seed, shuffle):
    """Rows with up to k columns on each side of the diagonal, among the 40 nearest;
    shuffle: the columns of a row in any order."""
    rng = np.random.default_rng(seed)
    rp, ci, v = [0], [], []
    for i in range(n):
        lo, hi = np.arange(max(0, i - 40), i), np.arange(i + 1, min(n, i + 41))
        cols = np.concatenate([rng.choice(lo, min(k, lo.size), replace=False), [i],
                               rng.choice(hi, min(k, hi.size), replace=False)]).astype(int)
        cols = rng.permutation(cols) if shuffle else np.sort(cols)
        vals = np.where(cols == i, 4.0 * k, rng.uniform(-1, 1, cols.size))
        ci += cols.tolist()
        v += vals.tolist()
        rp.append(len(ci))
    return np.array(rp, np.int32), np.array(ci, np.int32), np.array(v, np.float64)


@pytest.mark.parametrize("shuffle", [False, True])
@pytest.mark.parametrize("n,k", [(31, 3), (32, 3), (33, 4), (257, 7), (257, 8), (4100, 3),
                                 (1000, 16)])
def test_trsv_row_lengths_bit_exact(gpu, oracle, n, k, shuffle):
    """Rows of at most, of more and of many times the entries a lane holds (4 or 8,
    the diagonal among them), chunks of 32 rows with a remainder, rows in any column
    order, and b solved in place."""
    from linalglib_b200 import _lib as L
    A = _band(n, k, n + k, shuffle)
    b = np.random.default_rng(n).uniform(-1, 1, n)
    dA = gpu.CsrMatrix.from_arrays(*A)
    for lower in (True, False):
        for unit in (True, False):
            want = _bits(oracle.trsv(A, b, lower, unit))
            x = dA.trsv(gpu.vec(b), lower=lower, unit_diag=unit)
            assert np.array_equal(_bits(x.cpu().numpy()), want)
            y = gpu.vec(b)
            L.call("lab_csrtrsv", dA.h, int(lower), int(unit), gpu.ptr(y), gpu.ptr(y),
                   gpu.stream_handle())
            assert np.array_equal(_bits(y.cpu().numpy()), want)


def _two_levels(n):
    """Half the rows depend on one of the other half: two levels of n / 2 rows."""
    h = n // 2
    rng = np.random.default_rng(n)
    lo, hi = rng.permutation(h), h + rng.permutation(h)
    rp = np.arange(0, 2 * n + 1, 2)
    ci = np.empty((n, 2), np.int64)
    ci[:h] = np.stack([np.arange(h), hi], 1)
    ci[h:] = np.stack([lo, np.arange(h, n)], 1)
    v = np.where(ci == np.arange(n)[:, None], 3.0, rng.uniform(-1, 1, (n, 2)))
    return rp.astype(np.int32), ci.reshape(-1).astype(np.int32), v.reshape(-1)


def _ctas(gpu, dA, lower):
    import ctypes as C
    from linalglib_b200 import _lib as L
    n, c = C.c_int64(), C.c_int()
    L.call("lab_csrtrsv_info", dA.h, int(lower), C.byref(n), C.byref(c), gpu.stream_handle())
    return c.value


@pytest.mark.parametrize("make, ctas", [
    (lambda: P.poisson2d(40), 1),
    (lambda: P.poisson2d(130), 2),       # levels of 65 rows
    (lambda: P.poisson3d(20), 4),        # 138
    (lambda: P.poisson3d(30), 8),        # 307
    (lambda: P.poisson3d(41), 16),       # 570
    (lambda: P.poisson2d(700), 0),       # more than 16 CTAs' shared memory holds: the grid
    (lambda: _two_levels(9000), 0),      # wide and shallow: the grid
], ids=["c1", "c2", "c4", "c8", "c16", "large", "wide"])
def test_trsv_cluster_sizes_bit_exact(gpu, oracle, make, ctas):
    A = make()[:3]
    b = np.random.default_rng(5).uniform(-1, 1, A[0].size - 1)
    dA = gpu.CsrMatrix.from_arrays(*A)
    for lower in (True, False):
        want = _bits(oracle.trsv(A, b, lower, False))
        assert _ctas(gpu, dA, lower) == ctas
        for _ in range(2):
            x = dA.trsv(gpu.vec(b), lower=lower, unit_diag=False)
            assert np.array_equal(_bits(x.cpu().numpy()), want)


def test_trsv_bounded_wait_on_grid(gpu, oracle):
    """The bounded wait of the form that solves on the whole grid (a wide triangle)."""
    from linalglib_b200 import _lib as L
    A = _two_levels(9000)
    b = np.random.default_rng(6).uniform(-1, 1, 9000)
    dA = gpu.CsrMatrix.from_arrays(*A)
    L.call("lab_csrtrsv_wait_control", dA.h, 1 << 12, 0, gpu.stream_handle())
    bx, x = gpu.vec(b), gpu.vec(np.zeros(9000))
    st = L.lib().lab_csrtrsv(dA.h, 1, 0, gpu.ptr(bx), gpu.ptr(x), gpu.stream_handle())
    assert st == L.LAB_TIMEOUT, L.lib().lab_last_error().decode()
    L.call("lab_csrtrsv_wait_control", dA.h, 0, -1, gpu.stream_handle())
    x = dA.trsv(gpu.vec(b), lower=True)
    assert np.array_equal(_bits(x.cpu().numpy()), _bits(oracle.trsv(A, b, True, False)))


@pytest.mark.parametrize("lower", [True, False])
@pytest.mark.parametrize("make, held", [
    (lambda: P.poisson3d(24), 5000),        # a row in the middle, 4 CTAs
    (lambda: P.poisson2d(40), 800),         # one CTA
    (lambda: _two_levels(9000), 4400),      # the grid
], ids=["cluster", "one", "grid"])
def test_trsv_rows_that_time_out_are_nan(gpu, oracle, make, held, lower):
    """A solve that gives up leaves NaN in every row it did not solve (the held row's
    dependents at least), and the solution in the others; an earlier solve's values
    stay nowhere."""
    from linalglib_b200 import _lib as L
    A = make()[:3]
    m = A[0].size - 1
    b = np.random.default_rng(7).uniform(-1, 1, m)
    want = oracle.trsv(A, b, lower, False)
    dA = gpu.CsrMatrix.from_arrays(*A)
    row = held if lower else m - 1 - held
    L.call("lab_csrtrsv_wait_control", dA.h, 1 << 12, row, gpu.stream_handle())
    bx, x = gpu.vec(b), gpu.vec(np.full(m, 3.0))
    st = L.lib().lab_csrtrsv(dA.h, int(lower), 0, gpu.ptr(bx), gpu.ptr(x), gpu.stream_handle())
    assert st == L.LAB_TIMEOUT
    x = x.cpu().numpy()
    solved = ~np.isnan(x)
    assert np.array_equal(_bits(x[solved]), _bits(want[solved]))
    need = np.zeros(m, bool)  # the held row and the rows that depend on it
    need[row] = True
    for i in (range(row, m) if lower else range(row, -1, -1)):
        c = A[1][A[0][i]:A[0][i + 1]]
        need[i] |= bool(need[c[c < i] if lower else c[c > i]].any())
    assert not solved[need].any()


def _levels(widths):
    """Lower triangle whose level k has widths[k] rows, each with one entry in level
    k - 1 and the diagonal."""
    rng = np.random.default_rng(len(widths))
    rp, ci, v, base, below = [np.zeros(1, np.int64)], [], [], 0, None
    for w in widths:
        i = np.arange(base, base + w)
        if below is None:
            ci.append(i)
        else:
            ci.append(np.stack([below[0] + rng.integers(0, below[1], w), i], 1).reshape(-1))
        v.append(np.where(ci[-1] >= base, 2.0, rng.uniform(-1, 1, ci[-1].size)))
        rp.append(rp[-1][-1] + (ci[-1].size // w) * np.arange(1, w + 1))
        below, base = (base, w), base + w
    return tuple(np.concatenate(a).astype(t) for a, t in zip((rp, ci, v),
                                                             (np.int32, np.int32, np.float64)))


@pytest.mark.parametrize("widths, launches", [
    ([20000] + [64] * 30, 1),          # one wide level and enough others: the cluster
    ([20000] + [64] * 10, 2),          # too few others to make up for it: the grid
    ([10000] * 40 + [64] * 80, 2),     # many wide levels, a mean of 3376 rows: the grid
    ([4096] * 12, 1), ([4097] * 12, 2),
], ids=["head", "short", "heads", "4096", "4097"])
def test_trsv_form_by_level_widths(gpu, oracle, widths, launches):
    """The form is chosen by the widths of the levels and not by their mean; the cluster
    is one launch, the grid two."""
    A = _levels(widths)
    b = np.random.default_rng(8).uniform(-1, 1, A[0].size - 1)
    dA = gpu.CsrMatrix.from_arrays(*A)
    x = dA.trsv(gpu.vec(b), lower=True)
    assert np.array_equal(_bits(x.cpu().numpy()), _bits(oracle.trsv(A, b, True, False)))
    bx = gpu.vec(b)
    n0 = gpu.launch_count()
    dA.trsv(bx, lower=True)
    assert gpu.launch_count() - n0 == launches and (_ctas(gpu, dA, True) > 0) == (launches == 1)
