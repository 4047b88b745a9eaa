"""The FP64 operator's block fixed-point contractions against extended precision.

The bound is derived per node from the arithmetic, with u = 2^-53:
  * one contraction of a line: a representation and rounding error of at most Nq 2^-57 times
    (largest |D| of the row) times (largest entry of the line), and the conversion to FP64, u;
  * G . grad q: three products and two sums, 3 u of the magnitudes summed;
  * the three transposed parts and the mass term: two shifts by less than one unit, u for the
    conversion, 2 u for the mass term; the assembly of at most 8 copies, 8 u.
"""
import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg
from gpu_helpers import box

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
LD = np.longdouble


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


class Problem:
    def __init__(self, N, dims, **over):
        s = box(**{"POLYNOMIAL DEGREE": N, "BOX NX": dims[0], "BOX NY": dims[1], "BOX NZ": dims[2], **over})
        self.e = e = lpg.Elliptic(s)
        self.E, self.Nq = int(np.prod(dims)), N + 1
        shape = (self.E, self.Nq, self.Nq, self.Nq)
        self.g2l, self.shape = e.get("GlobalToLocal"), shape
        self.G = e.get("geo").reshape(self.E, 7, *shape[1:])
        self.D = e.get("D").reshape(self.Nq, self.Nq)
        # N = 3, 7 are contracted through the mirror symmetry of D and D^T: rows N - t are rows
        # t reversed and negated, which the stored D satisfies to its last bits only
        self.A, self.T = self.D.copy(), self.D.T.copy()
        if self.Nq in (4, 8):
            for M in (self.A, self.T):
                M[self.Nq // 2:] = -M[self.Nq // 2 - 1::-1, ::-1]
        lam = e.get("lambdaE") if s.get("LAMBDA FIELD") else np.full(self.E, float(s["LAMBDA"]))
        self.lam = lam[:, None, None, None]

    def local(self, q):
        return np.where(self.g2l < 0, 0.0, q[np.maximum(self.g2l, 0)]).reshape(self.shape)

    def gather(self, f):
        out = np.zeros(self.e.Nglobal + 1, dtype=f.dtype)
        np.add.at(out, np.where(self.g2l < 0, self.e.Nglobal, self.g2l), f.reshape(-1))
        return out[:-1]

    def along(self, M, f, d):
        """sum_m M[a][m] f[.. m ..] along r (d = 0), s (1), t (2)."""
        return np.moveaxis(np.einsum("am,...m->...a", M, np.moveaxis(f, 3 - d, -1)), -1, 3 - d)

    def both(self, q):
        """(operator, error bound) of q in extended precision."""
        G, A, T, u, Nq = (self.G.astype(LD), self.A.astype(LD), self.T.astype(LD), self.local(q).astype(LD),
                         self.Nq)
        sym = [[0, 1, 2], [1, 3, 4], [2, 4, 5]]

        def line(M, f, d):
            """|error| of one fixed-point contraction"""
            top = np.max(np.abs(f), axis=3 - d, keepdims=True)
            rows = np.max(np.abs(M), axis=1).reshape([-1 if 2 - d == k else 1 for k in range(3)])
            return Nq * 2.0 ** -57 * top * rows

        du = [self.along(A, u, d) for d in range(3)]
        err = [U * np.abs(du[d]) + line(A, u, d) for d in range(3)]
        out, bound = G[:, 6] * self.lam * u, 2 * U * np.abs(G[:, 6] * self.lam * u)
        for a in range(3):
            row = [G[:, sym[a][b]] for b in range(3)]
            v = sum(row[b] * du[b] for b in range(3))
            ev = sum(np.abs(row[b]) * (err[b] + 3 * U * np.abs(du[b])) for b in range(3))
            out = out + self.along(T, v, a)
            bound = bound + self.along(np.abs(T), ev, a) + line(T, np.abs(v) + ev, a)
        bound = bound + 3 * U * np.abs(out)
        return self.gather(out), self.gather(bound) + 8 * U * self.gather(np.abs(out))

    def apply(self, q):
        qd = torch.tensor(q, device="cuda")
        Aq = torch.full_like(qd, np.nan)
        self.e.Operator(qd, Aq)
        torch.cuda.synchronize()
        return Aq.cpu().numpy()


def _check(p, q):
    ref, bound = p.both(q)
    got = p.apply(q)
    assert np.all(np.isfinite(got))
    assert np.all(np.abs(got.astype(LD) - ref) <= bound)


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("dims,over", [((1, 1, 1), {"BOX BOUNDARY FLAG": 2}), ((3, 2, 3), {"LAMBDA": 0.0}),
                                       ((5, 3, 2), {"LAMBDA FIELD": "LOGNORMAL", "LAMBDA SEED": 4})])
def test_operator_within_derived_bound(N, dims, over):
    """Every degree; one element, an odd count that leaves the last CTA partly empty, Dirichlet
    boxes (lines of zeros), each mass-term variant."""
    p = Problem(N, dims, **over)
    rng = np.random.default_rng(5 + N)
    n = p.e.Nglobal
    _check(p, rng.uniform(-1, 1, n))
    # 15 decades in one vector: the lines' exponents differ, entries drop below a line's unit
    _check(p, rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-12, 3, n))
    _check(p, np.where(rng.uniform(size=n) < 0.7, 0.0, rng.uniform(-1, 1, n)))
    _check(p, np.ones(n))


@pytest.mark.parametrize("N", [2, 3, 7])
@pytest.mark.parametrize("exp", [-1000, -880, -500, 500, 880, 900])
def test_operator_scales_with_its_input(N, exp):
    """Powers of two scale the result exactly as long as nothing leaves the normal range: the
    FP64 lines (outside 2^-895..2^897) and the integer ones agree to rounding."""
    p = Problem(N, (2, 3, 2), **{"LAMBDA": 0.5})
    q = np.random.default_rng(3).uniform(-1, 1, p.e.Nglobal)
    ref, bound = p.both(q)
    got = p.apply(np.ldexp(q, exp))
    fp64 = 4 * p.Nq   # roundings of two plain FP64 dot products
    scale = np.ldexp(LD(1), exp)
    mag = bound / U
    assert np.all(np.abs(got.astype(LD) / scale - ref) <= fp64 * U * mag)


@pytest.mark.parametrize("N", [1, 3, 5, 7, 8])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e300])
def test_operator_keeps_non_finite_entries_where_they_belong(N, value):
    p = Problem(N, (3, 2, 2), **{"BOX BOUNDARY FLAG": 2})
    q = np.random.default_rng(9).uniform(-1, 1, p.e.Nglobal)
    at = p.e.Nglobal // 2
    q[at] = value
    with np.errstate(all="ignore"):
        u = p.local(q)
        sym = [[0, 1, 2], [1, 3, 4], [2, 4, 5]]
        du = [p.along(p.D, u, d) for d in range(3)]
        out = p.G[:, 6] * p.lam * u
        for a in range(3):
            out = out + p.along(p.D.T, sum(p.G[:, sym[a][b]] * du[b] for b in range(3)), a)
        ref = p.gather(out)
    got = p.apply(q)
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    fine = np.isfinite(ref)
    assert np.allclose(got[fine], ref[fine], rtol=1e-12, atol=1e-12 * np.max(np.abs(ref[fine])))
