"""PCG on device scalars: iterates, iteration counts and stops against the same recurrence in
numpy, with the preconditioner whose solves queue an iteration ahead of the host's read
(JACOBI) and with one that does not (NONE)."""
import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg
from gpu_helpers import box

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


def _cg(A, M, b, flexible, steps):
    """x after `steps` iterations, and r.r of each"""
    x, r, p, Ap, rz, alpha, rr = np.zeros_like(b), b.copy(), 0, 0 * b, 1.0, 0.0, []
    for k in range(steps):
        z = M * r
        new = r @ z
        beta = 0.0 if k == 0 else (-alpha * (z @ Ap) / rz if flexible else new / rz)
        rz = new
        p = z + beta * p
        Ap = A(p)
        alpha = rz / (p @ Ap)
        x = x + alpha * p
        r = r - alpha * Ap
        rr.append(r @ r)
    return x, rr


@pytest.mark.parametrize("solver", ["PCG", "FPCG"])
@pytest.mark.parametrize("precon", ["JACOBI", "NONE"])
@pytest.mark.parametrize("N,dims", [(2, (3, 2, 2)), (5, (4, 3, 5))])
def test_iterates_match_numpy(solver, precon, N, dims):
    e = lpg.Elliptic(box(**{"POLYNOMIAL DEGREE": N, "BOX NX": dims[0], "BOX NY": dims[1], "BOX NZ": dims[2],
                            "LINEAR SOLVER": solver, "PRECONDITIONER": precon}))
    n = e.Nglobal
    q, Aq = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")

    def A(v):
        q.copy_(torch.tensor(v))
        e.Operator(q, Aq)
        return Aq.cpu().numpy()

    M = e.get("invDiag") if precon == "JACOBI" else np.ones(n)
    b = np.random.default_rng(2).uniform(-1, 1, n)
    for steps in (1, 2, 5):
        ref, rr = _cg(A, M, b, solver == "FPCG", steps)
        x, r = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.tensor(b, device="cuda")
        before = e.info("operator_applications")
        assert e.Solve(x, r, tol=1e-14, maxit=steps) == steps
        assert e.info("operator_applications") - before == steps + 1   # one for the residual
        assert np.max(np.abs(x.cpu().numpy() - ref)) < 1e-12 * np.max(np.abs(ref))
        assert abs(float(r @ r) - rr[-1]) < 1e-10 * rr[0]
        # the same number of iterations when it is the tolerance that ends them
        if steps < 5:
            continue
        tol = np.sqrt(0.5 * (rr[2] + rr[3]) / (b @ b))
        want = next(k for k, v in enumerate(rr) if v <= max(tol * tol * (b @ b), tol * tol)) + 1
        x.zero_()
        r.copy_(torch.tensor(b))
        before = e.info("operator_applications")
        assert e.Solve(x, r, tol=tol, maxit=50) == want
        assert e.info("operator_applications") - before == want + 1
        ref, _ = _cg(A, M, b, solver == "FPCG", want)
        assert np.max(np.abs(x.cpu().numpy() - ref)) < 1e-12 * np.max(np.abs(ref))
