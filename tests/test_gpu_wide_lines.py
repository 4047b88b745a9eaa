"""The FP64 operator on lines that one entry outweighs, with metric factors over 15 decades and
derivative matrices with zeros: error per dof relative to the magnitudes summed.

Bound, u = 2^-53, mag = |D|^T (|G| |D| |q|): an FP64 chain has 2 Nq + 16 roundings (see
test_gpu_ax_entry_forms.py). An integer line errs by at most Nq 2^-57 R M (R, M the largest of
the row and of the line). It is used where the entries but the largest sum to at least
2^-(T + 1) M and the off-diagonal entries of a row are at least rho R; then the magnitudes
summed for any output are at least rho 2^-(T + 1) R M (the largest entry's own output; rho R M
for the others), so the error is at most Nq 2^(T - 3) / rho roundings of them, once in each of
the two contractions."""
import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg
from test_gpu_ax_entry_forms import _apply

pytestmark = pytest.mark.gpu
LD, U = np.longdouble, 2.0 ** -53
T = {1: 0, 2: 8, 3: 6, 4: 5, 5: 4, 6: 3, 7: 3, 8: 3}   # N = 1: every entry is part of both outputs


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


def _gll_derivative(N):
    x = np.polynomial.legendre.Legendre.basis(N).deriv().roots().real if N > 1 else np.zeros(0)
    x = np.concatenate([[-1.0], np.sort(x), [1.0]])
    x = 0.5 * (x - x[::-1])
    w = np.array([np.prod([x[j] - x[k] for k in range(N + 1) if k != j]) for j in range(N + 1)])
    D = np.array([[w[i] / w[j] / (x[i] - x[j]) if i != j else 0.0 for j in range(N + 1)] for i in range(N + 1)])
    D -= np.diag(D.sum(1))
    return 0.5 * (D - D[::-1, ::-1])


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("field", ["decades", "spike"])
@pytest.mark.parametrize("matrix", ["gll", "central"])
def test_error_relative_to_terms(N, field, matrix):
    rng = np.random.default_rng(N)
    Nq = N + 1
    E = 1101 if N == 7 else 37   # N = 7: also the kernel for larger problems
    if matrix == "gll":
        D = _gll_derivative(N)
        rows = np.abs(np.concatenate([D, D.T]))
        off = np.where(np.concatenate([np.eye(Nq)] * 2) > 0, np.inf, rows).min(1)
        chain = Nq * 2.0 ** (T[N] - 3) / (off / rows.max(1)).min()
    else:   # central differences: an output has two terms
        D = np.diag(np.ones(N), 1) - np.diag(np.ones(N), -1)
        chain = 0.0
    G = rng.uniform(-1, 1, (E, 6, Nq, Nq, Nq)) * 10.0 ** rng.uniform(-12, 3, (E, 1, Nq, Nq, Nq))
    shape = (E, Nq, Nq, Nq)
    q = rng.uniform(-1, 1, shape) * 10.0 ** rng.uniform(-12, 3 if field == "decades" else -6, shape)
    if field == "spike":
        for e in range(E):
            q[(e, *rng.integers(0, Nq, 3))] = rng.uniform(0.5, 1)
    dev = lambda x: torch.tensor(x, device="cuda").reshape(-1)
    n = E * Nq ** 3
    out = torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
    lpg.ax_hex("f64", N, E, dev(np.arange(n, dtype=np.int32)), dev(G), 6 * Nq ** 3, dev(np.zeros(n)), Nq ** 3, dev(D), 0.0,
               dev(q), out, n)
    torch.cuda.synchronize()
    zero = np.zeros(E, LD)
    ref = _apply(G.astype(LD), 0 * q, D.astype(LD), zero, q.astype(LD)).reshape(-1)
    mag = _apply(np.abs(G).astype(LD), 0 * q, np.abs(D).astype(LD), zero, np.abs(q).astype(LD)).reshape(-1)
    err = np.abs(out.cpu().numpy().astype(LD) - ref)
    assert np.all(err <= (2 * chain + 2 * Nq + 16) * U * mag)
