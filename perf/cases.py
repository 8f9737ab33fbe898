"""The work a user has the library do, as cases that can be timed.

Every case goes through the package's public entry points (``linalglib_b200.core``)
the way a program that links the library does: a sparse operator is on the device,
a hierarchy is set up from it, a preconditioner is kept, systems are solved.

Paths
    spmv      y = A x with an analysed matrix: the pass everything else is made of
    setup     from a matrix that is on the device to a preconditioner: the AMG level loop
              (strength, aggregation, P, R = P^T, R A P), the build, and
              one application z = M r, as a program with a Krylov loop of its own has it
              at every new matrix (time steps, Newton)
    solve     preconditioned CG with a kept AMG preconditioner (one matrix, many
              right-hand sides one after another), in FP64 or with a V-cycle of FP32
              or FP32 + BF16 values
    systems   a batch of independent systems of different sizes in one call
    rhs       one matrix, a block of right-hand sides in one call
    ilu0      CG with a kept ILU(0) factorisation (two triangular solves an iteration)
    adjoint   the backward direction: lambda = A^-T g and dL/dA on A's pattern

Operators
    poisson2d, poisson3d   5- and 7-point Laplacians, times one coefficient
    diffusion27            27-point operator, lognormal link conductances, strong in z
    graph3d                weighted 7-point graph Laplacian plus a shift
"""
import math
import random

import torch

from linalglib_b200 import _lib as L
from linalglib_b200 import core

KIND = {"sa": L.AMG_SA, "ua": L.AMG_UA}
PRECISION = {"fp64": L.PREC_FP64, "fp32": L.PREC_FP32, "bf16": L.PREC_FP32_BF16}


def listed():
    return [
        # the FP64 SpMV of the headline system
        {"name": "spmv_3d_128", "path": "spmv", "op": "poisson3d", "n": 128},
        # and of a 27-point operator with a ragged grid
        {"name": "spmv_27pt_101", "path": "spmv", "op": "diffusion27", "n": 101},
        # setup of the headline system
        {"name": "setup_sa_3d_128", "path": "setup", "kind": "sa", "op": "poisson3d", "n": 128},
        # setup of a variable-coefficient 27-point system
        {"name": "setup_sa_27pt_64", "path": "setup", "kind": "sa", "op": "diffusion27", "n": 64},
        # a small 2D setup: launches and host round trips
        {"name": "setup_sa_2d_61", "path": "setup", "kind": "sa", "op": "poisson2d", "n": 61},
        # the solve of the headline system, and a small and a mixed-precision one
        {"name": "solve_3d_128", "path": "solve", "op": "poisson3d", "n": 128, "precision": "fp64"},
        {"name": "solve_2d_64", "path": "solve", "op": "poisson2d", "n": 64, "precision": "fp64"},
        {"name": "solve_27pt_96_fp32", "path": "solve", "op": "diffusion27", "n": 96,
         "precision": "fp32"},
        # many uneven systems, many right-hand sides
        {"name": "systems_256", "path": "systems", "op": "poisson2d", "n": 256, "count": 256},
        {"name": "rhs_32_3d_64", "path": "rhs", "op": "poisson3d", "n": 64, "count": 32},
        # triangular solves
        {"name": "ilu0_3d_64", "path": "ilu0", "op": "poisson3d", "n": 64},
        # the backward direction on a graph Laplacian
        {"name": "adjoint_graph_80", "path": "adjoint", "op": "graph3d", "n": 80},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["spmv", "setup", "setup", "solve", "solve", "systems", "rhs", "ilu0",
                       "adjoint"])
    if path == "systems":
        return {"path": path, "op": "poisson2d", "n": _log(rng, 40, 256),
                "count": _log(rng, 4, 200)}
    if path == "rhs":
        op = rng.choice(["poisson3d", "graph3d", "poisson2d"])
        n = _log(rng, 40, 400) if op == "poisson2d" else _log(rng, 12, 64)
        return {"path": path, "op": op, "n": n, "count": rng.randint(2, 32)}
    if path == "ilu0":
        op = rng.choice(["poisson3d", "poisson2d"])
        n = _log(rng, 24, 120) if op == "poisson2d" else _log(rng, 10, 64)
        return {"path": path, "op": op, "n": n}
    op = rng.choice(["poisson2d", "poisson3d", "diffusion27", "graph3d"])
    n = {"poisson2d": lambda: _log(rng, 32, 900), "poisson3d": lambda: _log(rng, 16, 120),
         "diffusion27": lambda: _log(rng, 12, 72), "graph3d": lambda: _log(rng, 16, 100)}[op]()
    if path == "spmv":
        n = max(n, 24)
        return {"path": path, "op": op, "n": n}
    if path == "setup":
        return {"path": path, "kind": rng.choice(["sa", "sa", "sa", "ua"]), "op": op, "n": n}
    if path == "adjoint":
        return {"path": path, "op": op, "n": n}
    return {"path": path, "op": op, "n": n, "precision": rng.choice(["fp64", "fp64", "fp32",
                                                                      "bf16"])}


# ------------------------------------------------------------------ operators
def _stencil(shape, offsets, weights):
    """CSR on the device of a Dirichlet stencil, columns ascending in each row.
    offsets in ascending order of their linear index; weights broadcast to shape."""
    nd = len(shape)
    m = math.prod(shape)
    stride = [math.prod(shape[d + 1:]) for d in range(nd)]
    at = torch.arange(m, device="cuda")
    idx = [(at // stride[d]) % shape[d] for d in range(nd)]
    valid = torch.empty((m, len(offsets)), dtype=torch.bool, device="cuda")
    val = torch.empty((m, len(offsets)), dtype=torch.float64, device="cuda")
    for k, (o, w) in enumerate(zip(offsets, weights)):
        ok = torch.ones(m, dtype=torch.bool, device="cuda")
        for d in range(nd):
            if o[d]:
                ok &= (idx[d] + o[d] >= 0) & (idx[d] + o[d] < shape[d])
        valid[:, k] = ok
        val[:, k] = w.reshape(-1) if isinstance(w, torch.Tensor) else w
    lin = torch.tensor([sum(a * b for a, b in zip(o, stride)) for o in offsets], device="cuda")
    rp = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(valid.sum(1), 0, out=rp[1:])
    col = (at[:, None] + lin[None, :])[valid]
    return rp.to(torch.int32), col.to(torch.int32), val[valid]


def _operator(op, n, g):
    """(row_ptr, col_ind, val) on the device; g is the case's generator."""
    if op == "poisson2d":
        s = float(torch.empty((), device="cuda").uniform_(0.5, 2.0, generator=g))
        offs = [(-1, 0), (0, -1), (0, 0), (0, 1), (1, 0)]
        return _stencil((n, n), offs, [4.0 * s if o == (0, 0) else -s for o in offs])
    offs7 = [(-1, 0, 0), (0, -1, 0), (0, 0, -1), (0, 0, 0), (0, 0, 1), (0, 1, 0), (1, 0, 0)]
    if op == "poisson3d":
        s = float(torch.empty((), device="cuda").uniform_(0.5, 2.0, generator=g))
        return _stencil((n, n, n), offs7, [6.0 * s if o == (0, 0, 0) else -s for o in offs7])

    def links(d, sigma, scale):
        """conductance of the link from grid point q - 1 to q - 1 + d, q in the padded grid"""
        c = torch.empty((n + 2,) * 3, dtype=torch.float64, device="cuda")
        return c.normal_(0.0, sigma, generator=g).exp_().mul_(scale)

    def cut(c, d):
        return c[1 - d[0]:n + 1 - d[0], 1 - d[1]:n + 1 - d[1], 1 - d[2]:n + 1 - d[2]]

    weights = {}
    if op == "graph3d":
        diag = torch.full((n, n, n), 1e-3, dtype=torch.float64, device="cuda")
        for d in ((0, 0, 1), (0, 1, 0), (1, 0, 0)):
            c = links(d, 1.0, 1.0)
            for a in range(3):  # no link leaves the grid
                if d[a]:
                    c.select(a, 0).zero_()
                    c.select(a, n).zero_()
            weights[d] = -cut(c, (0, 0, 0))
            weights[tuple(-x for x in d)] = -cut(c, d)
            diag += cut(c, (0, 0, 0)) + cut(c, d)
        weights[(0, 0, 0)] = diag
        return _stencil((n, n, n), offs7, [weights[o] for o in offs7])
    offs = [(z, y, x) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)]
    diag = torch.zeros((n, n, n), dtype=torch.float64, device="cuda")
    for d in offs:
        if d > (0, 0, 0):
            r2 = sum(x * x for x in d)
            c = links(d, 1.5, (d[2] ** 2 + d[1] ** 2 + 100.0 * d[0] ** 2) / float(r2) ** 2)
            weights[d] = -cut(c, (0, 0, 0))
            weights[tuple(-x for x in d)] = -cut(c, d)
            diag += cut(c, (0, 0, 0)) + cut(c, d)
    weights[(0, 0, 0)] = diag
    return _stencil((n, n, n), offs, [weights[o] for o in offs])


def _rows(rp):
    return torch.repeat_interleave(torch.arange(rp.numel() - 1, device="cuda"), rp.diff().long())


def _apply(A, x):
    """A x in plain torch, 64 bits."""
    rp, ci, v = A
    return torch.zeros(rp.numel() - 1, dtype=torch.float64, device="cuda").index_add_(
        0, _rows(rp), v * x[ci.long()])


def _uniform(m, g):
    return torch.empty(m, dtype=torch.float64, device="cuda").uniform_(-1.0, 1.0, generator=g)


def _sides(case):
    """The batch's grid sides: evenly from an eighth of the largest to the largest, shuffled."""
    lo, count = max(8, case["n"] // 8), case["count"]
    sides = [lo + (case["n"] - lo) * k // (count - 1) for k in range(count)]
    random.Random(count).shuffle(sides)
    return sides


def _inputs(case, seed):
    """(operators, true solutions) of the case."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["path"] == "systems":
        ops = [_operator(case["op"], n, g) for n in _sides(case)]
        return ops, [_uniform(A[0].numel() - 1, g) for A in ops]
    A = _operator(case["op"], case["n"], g)
    m = A[0].numel() - 1
    return [A], [_uniform(m, g) for _ in range(case.get("count", 1))]


# ------------------------------------------------------------------ cases
def _omega(case):
    return 1.0 if case["op"] == "poisson3d" else 2.0 / 3.0


def prepare(case, seed):
    path = case["path"]
    ops, xs = _inputs(case, seed)
    A = ops[0]
    s = {"case": case, "control": core.iter_control(rel_tol=1e-8, abs_tol=0.0)}
    if path == "systems":
        s["A"], s["offsets"] = core.block_diag([core.CsrMatrix.from_arrays(*a) for a in ops])
        s["b"] = torch.cat([_apply(a, x) for a, x in zip(ops, xs)])
    else:
        s["A"] = core.CsrMatrix.from_arrays(*A)
    if path == "spmv":
        s["A"].analyse()
        s["x"], s["y"] = xs[0], torch.zeros_like(xs[0])
    elif path in ("setup", "solve", "ilu0"):
        s["b"] = _apply(A, xs[0])
    elif path == "rhs":
        s["b"] = torch.stack([_apply(A, x) for x in xs])
    elif path == "adjoint":
        s["g"], s["x"] = _apply(A, xs[0]), xs[0].flip(0).contiguous()
    if path == "ilu0":
        s["M"] = core.Preconditioner.ilu0(s["A"])
    elif path not in ("spmv", "setup"):
        s["M"] = core.Preconditioner.amg(
            core.Hierarchy(s["A"], kind=KIND["sa"]),
            core.amg_options(omega=_omega(case),
                             precision=PRECISION[case.get("precision", "fp64")]))
    return s


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "spmv":
        return state["A"].spmv(state["x"], state["y"])
    if path == "setup":
        H = core.Hierarchy(state["A"], kind=KIND[case["kind"]])
        return core.Preconditioner.amg(H, core.amg_options(omega=_omega(case))).apply(state["b"])
    if path == "systems":
        return core.batched_pcg(state["A"], state["offsets"], state["b"], state["M"],
                                control=state["control"])[0]
    if path == "rhs":
        return core.multi_rhs_pcg(state["A"], state["b"], state["M"],
                                  control=state["control"])[0]
    if path == "adjoint":
        lam, _ = core.adjoint_solve(state["A"], state["g"], state["M"], control=state["control"])
        return lam, core.adjoint_grad_A(state["A"], lam, state["x"])
    return core.pcg(state["A"], state["b"], M=state["M"], control=state["control"])[0]


def exact(case, seed):
    path = case["path"]
    if path == "setup":
        return None  # what the aggregates (whole numbers, greedy in row order) lead to
    ops, xs = _inputs(case, seed)
    if path == "spmv":
        return _apply(ops[0], xs[0])
    if path == "systems":
        return torch.cat(xs)
    if path == "rhs":
        return torch.stack(xs)
    if path == "adjoint":
        rp, ci, _ = ops[0]
        return xs[0], -xs[0][_rows(rp)] * xs[0].flip(0)[ci.long()]
    return xs[0]


# ------------------------------------------------------------------ sizes
#: nonzeros of all levels over those of the first, and CG iterations to 1e-8 with an
#: SA V-cycle (ILU(0)'s grow with the side), as these operators show them
COMPLEXITY = {"poisson2d": 1.5, "poisson3d": 2.7, "diffusion27": 1.3, "graph3d": 2.5}
ITERATIONS = {"poisson2d": 15, "poisson3d": 24, "diffusion27": 40, "graph3d": 35}


def _size(op, n):
    """(rows, nonzeros)"""
    if op == "poisson2d":
        return n * n, 5 * n * n - 4 * n
    if op == "diffusion27":
        return n ** 3, (3 * n - 2) ** 3
    return n ** 3, 7 * n ** 3 - 6 * n * n


def work(case):
    """Operators are read as 8-byte values and 4-byte columns.  A solve reads them once
    for A p and twice (down and up) on every level of the V-cycle in each iteration, and
    ten vectors; a setup reads A and P and writes every coarser level."""
    path = case["path"]
    m, z = _size(case["op"], case["n"])
    if path == "systems":
        lo = max(8, case["n"] // 8)
        side2 = (case["n"] ** 3 - lo ** 3) / (3.0 * max(1, case["n"] - lo))
        m, z = int(case["count"] * side2), int(5 * case["count"] * side2)
    mat = 12.0 * z + 4.0 * (m + 1)
    if path == "spmv":
        return {"bytes": mat + 16.0 * m, "flops": 2.0 * z}
    more = COMPLEXITY[case["op"]]
    if path == "setup":
        return {"bytes": mat * more, "flops": 8.0 * z}
    if path == "ilu0":
        its = 0.8 * case["n"] + 6
        return {"bytes": its * (2.0 * mat + 80.0 * m), "flops": its * 4.0 * z}
    its = ITERATIONS[case["op"]]
    half = {"fp64": 1.0, "fp32": 2.0 / 3.0, "bf16": 2.0 / 3.0}[case.get("precision", "fp64")]
    count = case["count"] if path == "rhs" else 1
    blocks = -(-count // 8) if path == "rhs" else 1
    reads = its * mat * (1.0 + 2.0 * more * half)
    return {"bytes": blocks * reads + count * its * 80.0 * m * (1.0 + half),
            "flops": count * its * 2.0 * z * (1.0 + 2.0 * more)}


def tolerance(case):
    """One SpMV row sums at most 27 products in 64 bits; a V-cycle sums a few thousand of
    them on the way to each value.  A solve stops at a relative residual of 1e-8, an
    iteration more or less on the way."""
    path = case["path"]
    if path == "setup":
        return {"rel": 1e-11, "max": 1e-9}
    if path == "spmv":
        return {"rel": 1e-14, "max": 1e-12}
    return {"rel": 2e-6, "max": 4e-5}
