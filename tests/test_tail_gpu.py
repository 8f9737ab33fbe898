"""The fused V-cycle tail (csrc/cycle_tail.cu) against the oracle's V-cycle: entry at
level 0 (few rows; odd and even sizes, an odd address), with and without the entry
level's restriction and prolongation in the launch, several sweeps, FP64 and FP32."""
import numpy as np
import pytest

from linalglib_b200 import _lib as L
from linalglib_b200 import problems as P

pytestmark = pytest.mark.gpu

CASES = [
    ("2d 11", lambda: P.poisson2d(11)),           # entry 0, odd number of rows
    ("2d 12", lambda: P.poisson2d(12)),           # entry 0
    ("2d 61", lambda: P.poisson2d(61)),           # entry 1 with R and P
    ("2d 100x83", lambda: P.poisson2d(100, 83)),  # entry 1 without R and P
    ("3d 13", lambda: P.poisson3d(13)),           # long rows
    ("27pt 12", lambda: P.diffusion27(12)),
]


@pytest.mark.parametrize("n1, n2", [(1, 1), (2, 1), (1, 0), (3, 2)])
@pytest.mark.parametrize("name, make", CASES, ids=[c[0] for c in CASES])
def test_tail_matches_oracle_cycle(gpu, oracle, name, make, n1, n2):
    import torch
    A = make()
    m = A[0].size - 1
    H = gpu.Hierarchy(gpu.CsrMatrix.from_arrays(*A), kind=L.AMG_SA)
    r = np.random.default_rng(m).uniform(-1, 1, m)
    zo = oracle.amg_setup(A, kind=0).vcycle(r, n1=n1, n2=n2, omega=2.0 / 3.0, coarse=1)
    # sums of at most ~200 products on each of a few dozen passes: 2^-53 and 2^-24 times
    # a few hundred, in the norm of the result
    for precision, tol in ((L.PREC_FP64, 1e-12), (L.PREC_FP32, 4e-5)):
        M = gpu.Preconditioner.amg(H, gpu.amg_options(n1=n1, n2=n2, omega=2.0 / 3.0,
                                                      precision=precision))
        for shift in (0, 1):  # z at a 16-byte boundary and 8 bytes off it
            z = torch.full((m + 3,), 7.0, dtype=torch.float64, device="cuda")
            M.apply(gpu.vec(r), z[shift:shift + m])
            z = z.cpu().numpy()
            assert np.max(np.abs(z[shift:shift + m] - zo)) <= tol * np.max(np.abs(zo))
            assert np.all(z[:shift] == 7.0) and np.all(z[shift + m:] == 7.0)
