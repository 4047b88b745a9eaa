"""The derivative matrix that the operators use: mirrored exactly, rows that add up to exactly 0
(N >= 4; below, the plain formula's own), entries right to the rounding of the nodes."""
from fractions import Fraction

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


def _plain(N):
    """D at the GLL nodes in extended precision"""
    LD = np.longdouble
    P = np.polynomial.legendre.Legendre.basis(N)
    x = np.concatenate([[-1.0], np.sort(P.deriv().roots().real) if N > 1 else [], [1.0]]).astype(LD)
    c = P.convert(kind=np.polynomial.Polynomial)
    d1, d2 = c.deriv().coef.astype(LD), c.deriv(2).coef.astype(LD)
    val = lambda a, v: sum(a[k] * v ** k for k in range(len(a)))
    for _ in range(4):
        if N > 1:
            x[1:-1] -= val(d1, x[1:-1]) / val(d2, x[1:-1])
    x = (x - x[::-1]) / 2
    w = [np.prod([x[j] - x[k] for k in range(N + 1) if k != j]) for j in range(N + 1)]
    D = np.array([[w[i] / w[j] / (x[i] - x[j]) if i != j else LD(0) for j in range(N + 1)] for i in range(N + 1)])
    return D - np.diag(D.sum(1))


@pytest.mark.parametrize("N", range(1, 9))
def test_derivative_matrix(N):
    D = lpg.Elliptic(box(**{"POLYNOMIAL DEGREE": N})).get("D").reshape(N + 1, N + 1)
    assert np.array_equal(D, -D[::-1, ::-1])
    sums = [sum(Fraction(float(v)) for v in row) for row in D]
    assert max(abs(s) for s in sums) <= (0 if N > 3 else Fraction(1, 2 ** 52))
    # a node's rounding, 2^-54, moves an entry by at most its distance to the nearest node's
    # inverse, 2 / N^2 at least, for each of the N factors: N^3 2^-55 of the row's largest
    ref = _plain(N)
    top = np.abs(ref).max(axis=1, keepdims=True)
    assert np.all(np.abs(D - ref) <= (N ** 3 * 2.0 ** -55 + 2.0 ** -52) * top)
