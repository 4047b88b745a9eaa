"""The FP64 IPDG operator at every degree against extended precision, formed from the object's
own metric factors: grad d / |grad d| is the normal of a face of direction d, |grad d|^2 =
G_dd / wJ, sJ / J = |grad d|, and WsJ = wJ |grad d| / w with the GLL weight w = 2 / (N (N + 1))
of the face.

Bound per node: mag is the sum of the magnitudes with every contraction at the largest entry of
its line and row. Two contractions of Nq terms (FP64 lines; integer lines err less), the
metric product, the face's jump, flux, penalty (two roots and their quotient, from factors
that are themselves rounded differences: 20) and sums: 2 Nq + 48 roundings of mag."""
import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg
from gpu_helpers import box

pytestmark = pytest.mark.gpu
LD, U = np.longdouble, 2.0 ** -53
SYM = [[0, 1, 2], [1, 3, 4], [2, 4, 5]]
DIMS = (5, 3, 3)   # odd: the last CTA is partly empty
BC = {"dirichlet": 1, "neumann": 2, "periodic": -1}


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


class Problem:
    def __init__(self, N, bc, **over):
        nx, ny, nz = DIMS
        s = box(**{"POLYNOMIAL DEGREE": N, "BOX NX": nx, "BOX NY": ny, "BOX NZ": nz, "BOX BOUNDARY FLAG": BC[bc],
                   "DISCRETIZATION": "IPDG", "MESH JITTER": 0.0 if bc == "periodic" else 0.1, **over})
        self.e, self.bc, self.N, Nq = lpg.Elliptic(s), bc, N, N + 1
        E = nx * ny * nz
        self.shape = (nz, ny, nx, Nq, Nq, Nq)
        geo = self.e.get("geo").reshape(nz, ny, nx, 7, Nq, Nq, Nq)
        self.G, self.wJ = [geo[:, :, :, c] for c in range(6)], geo[:, :, :, 6]
        self.D = self.e.get("D").reshape(Nq, Nq)
        lamE = self.e.get("lambdaE") if s.get("LAMBDA FIELD") else np.full(E, float(s["LAMBDA"]))
        self.lam = lamE.reshape(nz, ny, nx, 1, 1, 1)

    def operator(self, q, mag=False, dtype=LD):
        """A q, or the magnitudes summed"""
        f = (lambda v: np.abs(v)) if mag else (lambda v: v)
        D, G = f(self.D.astype(dtype)), [f(g.astype(dtype)) for g in self.G]
        wJ, u, N = self.wJ.astype(dtype), f(q.astype(dtype).reshape(self.shape)), self.N
        minus = 1 if mag else -1

        def line(M, v, d):
            v = np.moveaxis(v, 5 - d, -1)
            if mag:
                v = np.broadcast_to(v.max(axis=-1, keepdims=True), v.shape)
                M = np.broadcast_to(M.max(axis=1, keepdims=True), M.shape)
            return np.moveaxis(np.einsum("am,...m->...a", M, v), -1, 5 - d)

        du = [line(D, u, d) for d in range(3)]
        rows = [sum(G[SYM[a][b]] * du[b] for b in range(3)) for a in range(3)]
        val = self.lam.astype(dtype) * wJ * u
        invw = dtype(N * (N + 1)) / 2
        tau = dtype(2 * (N + 1) * (N + 3))
        jump = [np.zeros_like(u) for _ in range(3)]
        for d in range(3):
            axis, cells = 5 - d, 2 - d
            n = np.sqrt(np.abs(G[SYM[d][d]]) / wJ)   # |grad d|
            for hi in (0, 1):
                s, mine, theirs, roll = (1, N, 0, -1) if hi else (-1, 0, N, 1)
                own = lambda v: np.take(v, mine, axis=axis)
                oth = lambda v: np.roll(np.take(v, theirs, axis=axis), roll, axis=cells)
                edge = np.zeros(own(u).shape, dtype=bool)
                if self.bc != "periodic":
                    np.moveaxis(edge, cells, 0)[-1 if hi else 0] = True
                qM, qP = own(u), oth(u)
                fM, fP = s * own(rows[d]) * invw, s * oth(rows[d]) * invw
                if mag:
                    fM, fP = np.abs(fM), np.abs(fP)
                h = np.where(edge, own(n), np.maximum(own(n), oth(n)))
                if self.bc == "dirichlet":
                    qP, fP = np.where(edge, minus * qM, qP), np.where(edge, fM, fP)
                elif self.bc == "neumann":
                    qP, fP = np.where(edge, qM, qP), np.where(edge, minus * fM, fP)
                dq = qP + minus * qM
                pen = own(wJ * n) * invw * tau * h / 2
                if mag:
                    np.moveaxis(jump[d], axis, 0)[mine] += invw / 2 * dq
                    np.moveaxis(val, axis, 0)[mine] += (fM + fP) / 2 + pen * dq
                else:
                    np.moveaxis(jump[d], axis, 0)[mine] += s * invw / 2 * dq
                    np.moveaxis(val, axis, 0)[mine] += -(fM + fP) / 2 - pen * dq
        for a in range(3):
            val = val + line(D.T, rows[a] + sum(G[SYM[a][b]] * jump[b] for b in range(3)), a)
        return val.reshape(-1)

    def apply(self, q):
        qd = torch.tensor(q, device="cuda")
        Aq = torch.full_like(qd, np.nan)
        self.e.Operator(qd, Aq)
        torch.cuda.synchronize()
        same = qd.clone()
        self.e.Operator(same, same)   # the result may take the input's place
        torch.cuda.synchronize()
        assert torch.equal(same, Aq) or not torch.isfinite(Aq).all()
        return Aq.cpu().numpy()


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("bc", sorted(BC))
@pytest.mark.parametrize("over", [{"LAMBDA": 0.0}, {"LAMBDA": 1.0}, {"LAMBDA FIELD": "LOGNORMAL", "LAMBDA SEED": 4}])
def test_operator_within_derived_bound(N, bc, over):
    p = Problem(N, bc, **over)
    rng = np.random.default_rng(N)
    uniform = rng.uniform(-1, 1, p.e.Nglobal)
    for q in (uniform, uniform * 10.0 ** rng.uniform(-12, 3, uniform.size), np.ldexp(uniform, -960), np.ldexp(uniform, 900)):
        err = np.abs(p.apply(q).astype(LD) - p.operator(q))
        assert np.all(err <= (2 * (N + 1) + 48) * U * p.operator(q, mag=True))


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_non_finite_entries_stay_where_they_belong(N, value):
    """A node that is not finite reaches its element's lines and the face nodes across: entries
    that are finite in plain FP64 are finite and right, and none else."""
    p = Problem(N, "dirichlet")
    q = np.random.default_rng(9).uniform(-1, 1, p.e.Nglobal)
    q[p.e.Nglobal // 2] = value
    with np.errstate(all="ignore"):
        ref = p.operator(q, dtype=np.float64)
    got = p.apply(q)
    fine = np.isfinite(ref)
    assert 0 < fine.sum() < fine.size
    assert np.array_equal(np.isfinite(got), fine)
    assert np.allclose(got[fine], ref[fine], rtol=1e-11, atol=1e-11 * np.max(np.abs(ref[fine])))
