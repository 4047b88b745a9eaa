"""How solves end early: right-hand sides that are not finite, operators that are not positive
(p.Ap <= 0 in the first or a later iteration) and residuals that overflow, with the
preconditioner whose solves queue an iteration ahead of the host's read (JACOBI) and with one
that does not (NONE). Iterates against the same recurrence in numpy; the next solve of the
object is that of a fresh one."""
import ctypes

import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg
from gpu_helpers import box

pytestmark = pytest.mark.gpu
BREAKDOWN = -7


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


class Problem:
    def __init__(self, solver, precon, **over):
        self.s = box(**{"POLYNOMIAL DEGREE": 3, "BOX NX": 3, "BOX NY": 2, "BOX NZ": 3, "LINEAR SOLVER": solver,
                        "PRECONDITIONER": precon, **over})
        self.e = lpg.Elliptic(self.s)
        n = self.n = self.e.Nglobal
        q, Aq = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2))
        self.A = np.zeros((n, n))
        for k in range(n):
            q.zero_()
            q[k] = 1.0
            self.e.Operator(q, Aq)
            self.A[:, k] = Aq.cpu().numpy()
        self.M = self.e.get("invDiag") if precon == "JACOBI" else np.ones(n)
        self.flexible = solver == "FPCG"

    def solve(self, b, tol=1e-10, maxit=400, e=None):
        e = e or self.e
        x, r = torch.zeros(self.n, dtype=torch.float64, device="cuda"), torch.tensor(b, device="cuda")
        it, ops = ctypes.c_int(-1), e.info("operator_applications")
        st = lpg.lib().lpg_elliptic_solve(e.h, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(r.data_ptr()), tol, maxit,
                                          ctypes.byref(it))
        return st, it.value, x.cpu().numpy(), r.cpu().numpy(), e.info("operator_applications") - ops

    def cg(self, b):
        """(x, r, p.Ap) after each iteration's start: the recurrence up to p.Ap <= 0 or r.r not finite"""
        x, r, p, Ap, rz, alpha = np.zeros_like(b), b.copy(), 0, 0 * b, 1.0, 0.0
        for k in range(400):
            z = self.M * r
            new = r @ z
            beta = 0.0 if k == 0 else (-alpha * (z @ Ap) / rz if self.flexible else new / rz)
            rz = new
            p = z + beta * p
            Ap = self.A @ p
            if not p @ Ap > 0:
                return k, x, r
            alpha = rz / (p @ Ap)
            x = x + alpha * p
            r = r - alpha * Ap
            with np.errstate(over="ignore"):
                if not np.isfinite(r @ r):
                    return k + 1, x, r
        raise AssertionError("no early end")

    def next_solve_is_a_fresh_one(self):
        b = np.random.default_rng(11).uniform(-1, 1, self.n)
        b = self.A @ b if self.s["LAMBDA"] >= 0 else b
        got, ref = self.solve(b, maxit=5), self.solve(b, maxit=5, e=lpg.Elliptic(self.s))
        assert got[0] == ref[0] and got[1] == ref[1] and got[4] == ref[4]
        assert np.max(np.abs(got[2] - ref[2])) <= 1e-12 * np.max(np.abs(ref[2]))


SOLVERS = [(s, p) for s in ("PCG", "FPCG") for p in ("JACOBI", "NONE")]


@pytest.mark.parametrize("solver,precon", SOLVERS)
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_right_hand_side_not_finite(solver, precon, bad):
    p = Problem(solver, precon)
    b = np.random.default_rng(1).uniform(-1, 1, p.n)
    b[p.n // 2] = bad
    st, it, x, r, ops = p.solve(b)
    assert st == BREAKDOWN and it == 0 and ops == 1
    assert np.array_equal(x, np.zeros(p.n))
    p.next_solve_is_a_fresh_one()


@pytest.mark.parametrize("solver,precon", SOLVERS)
@pytest.mark.parametrize("lam", [-1e4, "some"])
def test_operator_not_positive(solver, precon, lam):
    """lambda far below 0: p.Ap < 0 at once; below the fourth eigenvalue of the pencil: later"""
    if lam == "some":
        K = Problem(solver, precon, LAMBDA=0.0)
        mass = Problem(solver, precon, LAMBDA=1.0).A - K.A
        w = np.sqrt(np.diag(mass))
        ev = np.linalg.eigvalsh(K.A / w[:, None] / w[None, :])
        lam = -float(0.5 * (ev[3] + ev[4]))
    p = Problem(solver, precon, LAMBDA=lam)
    if precon == "JACOBI":
        p.M = p.e.get("invDiag")
    b = np.random.default_rng(2).uniform(-1, 1, p.n)
    want, xr, rr = p.cg(b)
    st, it, x, r, ops = p.solve(b, tol=1e-14)
    assert st == BREAKDOWN and it == want
    assert ops == want + 2   # the residual's and the one whose p.Ap was not positive
    top = max(np.max(np.abs(xr)), np.max(np.abs(p.M * b)))
    assert np.max(np.abs(x - xr)) <= 1e-9 * top
    assert np.max(np.abs(r - rr)) <= 1e-9 * max(np.max(np.abs(rr)), np.max(np.abs(b)))
    p.next_solve_is_a_fresh_one()


@pytest.mark.parametrize("solver", ["PCG", "FPCG"])
def test_residual_overflows(solver):
    """Steepest descent's worst start, of the smallest and the largest eigenvalue of the scaled
    operator in the ratio of their roots: the first step grows r.r, here past the largest FP64
    number, and the solve ends after one iteration."""
    p = Problem(solver, "JACOBI", LAMBDA=0.0, **{"BOX DIMX": 2e6, "BOX DIMY": 2e6, "BOX DIMZ": 2e6})
    d = np.sqrt(np.diag(p.A))
    ev, V = np.linalg.eigh(0.5 * (p.A + p.A.T) / d[:, None] / d[None, :])
    b = d * (V[:, 0] + np.sqrt(ev[0] / ev[-1]) * V[:, -1])
    r = b - (b @ (b / d**2)) / ((b / d**2) @ p.A @ (b / d**2)) * (p.A @ (b / d**2))
    growth = (r @ r) / (b @ b)
    assert growth > 1.5
    b *= np.sqrt(1.7e308 / growth * 1.4 / (b @ b))
    assert np.isfinite(b @ b)
    want, xr, _ = p.cg(b)
    assert want == 1
    st, it, x, r, ops = p.solve(b)
    assert st == BREAKDOWN and it == 1 and ops == 2
    assert np.max(np.abs(x - xr)) <= 1e-12 * np.max(np.abs(xr))
    p.next_solve_is_a_fresh_one()
