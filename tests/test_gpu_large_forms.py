"""The FP64 operator's one-thread-a-line form, which serves every problem but small ones, at each
degree and mass term: boxes about twice the size where it takes over, with an odd number of
elements (the last CTA is partly empty where a CTA holds several). The reference is formed for
blocks of 3 x 3 x 3 elements, at two corners, at the last element and inside, and compared at the
dofs all of whose elements are in a block.

Bound per dof, u = 2^-53: an integer line errs by Nq 2^-57 (largest of the row) (largest of the
line) and u of its result; a line left to FP64 by Nq u of the magnitudes summed; G . grad q by
3 u of the magnitudes summed, the sum of the three parts and the mass term by 5 u, and the
assembly of at most 8 copies by 8 u."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg
from gpu_helpers import box

pytestmark = pytest.mark.gpu
LD, U = np.longdouble, 2.0 ** -53
SYM = [[0, 1, 2], [1, 3, 4], [2, 4, 5]]
DIMS = {1: (35, 33, 33), 2: (27, 25, 25), 3: (21, 21, 21), 4: (19, 17, 19), 5: (17, 17, 15), 6: (15, 15, 15),
        7: (13, 13, 15), 8: (13, 13, 11)}
LAMBDAS = {"zero": {"LAMBDA": 0.0}, "one": {"LAMBDA": 1.0}, "const": {"LAMBDA": 2.5},
           "field": {"LAMBDA FIELD": "LOGNORMAL", "LAMBDA SEED": 4}}


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


def _along(M, f, d):
    return np.moveaxis(np.einsum("am,...m->...a", M, np.moveaxis(f, 3 - d, -1)), -1, 3 - d)


class Blocks:
    def __init__(self, N, lam):
        dims = DIMS[N]
        s = box(**{"POLYNOMIAL DEGREE": N, "BOX NX": dims[0], "BOX NY": dims[1], "BOX NZ": dims[2], **LAMBDAS[lam]})
        self.e = e = lpg.Elliptic(s)
        E, Nq = int(np.prod(dims)), N + 1
        assert E % 2 == 1
        at = {(0, 0, 0), tuple(d - 3 for d in dims), tuple(d // 2 for d in dims), (dims[0] - 3, 0, dims[2] // 3),
              (1, dims[1] // 2, dims[2] - 3)}
        S = sorted({(i + a) + dims[0] * ((j + b) + dims[1] * (k + c)) for i, j, k in at for a in range(3) for b in range(3)
                    for c in range(3)})
        assert 0 in S and E - 1 in S
        g2l = e.get("GlobalToLocal")
        self.g2l = g2l.reshape(E, -1)[S].reshape(-1)
        self.Ng, self.Nq, self.shape = e.Nglobal, Nq, (len(S), Nq, Nq, Nq)
        count = lambda v: np.bincount(v[v >= 0], minlength=self.Ng)
        mine = count(self.g2l)
        self.whole = np.flatnonzero((mine > 0) & (mine == count(g2l)))
        geo = e.get("geo").reshape(E, 7, *self.shape[1:])[S]
        self.G, self.wJ = geo[:, :6], geo[:, 6]
        self.D = e.get("D").reshape(Nq, Nq)
        lamE = e.get("lambdaE") if lam == "field" else np.full(E, float(s["LAMBDA"]))
        self.lam = lamE[S][:, None, None, None]

    def local(self, q):
        return np.where(self.g2l < 0, 0.0, q[np.maximum(self.g2l, 0)]).reshape(self.shape)

    def gather(self, f):
        out = np.zeros(self.Ng + 1, dtype=f.dtype)
        np.add.at(out, np.where(self.g2l < 0, self.Ng, self.g2l), f.reshape(-1))
        return out[:-1][self.whole]

    def both(self, q):
        G, D, u = self.G.astype(LD), self.D.astype(LD), self.local(q).astype(LD)

        def line(M, f, d):
            top = np.max(np.abs(f), axis=3 - d, keepdims=True)
            sure = np.sum(np.abs(f), axis=3 - d, keepdims=True) >= 2.3 * top   # none outweighs the rest: integers
            rows = np.max(np.abs(M), axis=1).reshape([-1 if 2 - d == k else 1 for k in range(3)])
            return self.Nq * (2.0 ** -57 * top * rows + np.where(sure, 0, U * _along(np.abs(M), np.abs(f), d)))

        du = [_along(D, u, d) for d in range(3)]
        err = [U * np.abs(du[d]) + line(D, u, d) for d in range(3)]
        mass = self.wJ * self.lam * u
        out, bound = mass, 2 * U * np.abs(mass)
        for a in range(3):
            row = [G[:, SYM[a][b]] for b in range(3)]
            v = sum(row[b] * du[b] for b in range(3))
            ev = sum(np.abs(row[b]) * (err[b] + 3 * U * np.abs(du[b])) for b in range(3))
            part = _along(D.T, v, a)
            out = out + part
            bound = bound + _along(np.abs(D.T), ev, a) + line(D.T, np.abs(v) + ev, a) + U * np.abs(part)
        return self.gather(out), self.gather(bound + 3 * U * np.abs(out)) + 8 * U * self.gather(np.abs(out))

    def apply(self, q):
        qd = torch.tensor(q, device="cuda")
        Aq = torch.full_like(qd, np.nan)
        self.e.Operator(qd, Aq)
        torch.cuda.synchronize()
        return Aq.cpu().numpy()[self.whole]


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("lam", sorted(LAMBDAS))
def test_operator_within_derived_bound(N, lam):
    p = Blocks(N, lam)
    rng = np.random.default_rng(7 + N)
    uniform = rng.uniform(-1, 1, p.Ng)
    for q in (uniform, uniform * 10.0 ** rng.uniform(-12, 3, p.Ng)):
        ref, bound = p.both(q)
        got = p.apply(q)
        assert np.all(np.isfinite(got))
        assert np.all(np.abs(got.astype(LD) - ref) <= bound)


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("exp", [-960, 940])
def test_lines_outside_the_integers_range(N, exp):
    """A vector scaled by a power of two gives the scaled result; its lines (below 2^-895, above
    2^897) are FP64 lines."""
    p = Blocks(N, "const")
    q = np.random.default_rng(N).uniform(-1, 1, p.Ng)
    ref, _ = p.both(q)
    # FP64 lines: Nq roundings in each contraction, and 16 of the metric product, the sum and the assembly
    A, u = np.abs(p.D).astype(LD), np.abs(p.local(q)).astype(LD)
    du = [_along(A, u, d) for d in range(3)]
    G = np.abs(p.G).astype(LD)
    mag = p.gather(p.wJ * p.lam * u + sum(_along(A.T, sum(G[:, SYM[a][b]] * du[b] for b in range(3)), a) for a in range(3)))
    got = p.apply(np.ldexp(q, exp)).astype(LD) / np.ldexp(LD(1), exp)
    assert np.all(np.abs(got - ref) <= (2 * p.Nq + 16) * U * mag)


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_non_finite_entries_stay_where_they_belong(N, value):
    p = Blocks(N, "one")
    q = np.random.default_rng(9).uniform(-1, 1, p.Ng)
    inside = p.g2l[p.g2l >= 0]
    q[[inside[0], inside[len(inside) // 2], inside[-1]]] = value
    with np.errstate(all="ignore"):
        u = p.local(q)
        du = [_along(p.D, u, d) for d in range(3)]
        ref = p.gather(p.wJ * p.lam * u + sum(
            _along(p.D.T, sum(p.G[:, SYM[a][b]] * du[b] for b in range(3)), a) for a in range(3)))
    got = p.apply(q)
    fine = np.isfinite(ref)
    assert 0 < fine.sum() < fine.size
    assert np.array_equal(np.isfinite(got), fine)
    assert np.allclose(got[fine], ref[fine], rtol=1e-12, atol=1e-12 * np.max(np.abs(ref[fine])))


RUN = """
import sys
import numpy as np
import torch
import libparanumal_gb300 as lpg
from gpu_helpers import box
N, out = int(sys.argv[1]), sys.argv[2]
n = {7: (13, 13, 15), 5: (17, 17, 15), 3: (21, 21, 21)}[N]
e = lpg.Elliptic(box(**{"POLYNOMIAL DEGREE": N, "BOX NX": n[0], "BOX NY": n[1], "BOX NZ": n[2], "LAMBDA": 0.5,
                        "PRECONDITIONER": "MULTIGRID"}))
r = torch.tensor(np.random.default_rng(N).uniform(-1, 1, e.Nglobal), device="cuda")
z = torch.zeros_like(r)
e.precon(r, z)
torch.cuda.synchronize()
np.save(out, z.cpu().numpy())
"""


@pytest.mark.parametrize("N", [3, 5, 7])
def test_subtracting_smoother_matches_the_one_with_a_vector_for_the_product(N, tmp_path):
    """u -= A d assembled into u against A d formed apart (LPG_CHEB = unfused): the same V-cycle
    but for the order of additions. Each level's sweep adds a few rounding errors of the
    residual, which the cycle's operator (norm near 1 on it) carries on: 10^-11 leaves two
    digits above the 10^-13 of a product of FP64 operators."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    z = []
    for mode in ("", "unfused"):
        f = str(tmp_path / ("z%s.npy" % mode))
        env = dict(os.environ, PYTHONPATH=root + os.pathsep + os.path.join(root, "tests"))
        env.pop("LPG_CHEB", None)
        if mode:
            env["LPG_CHEB"] = mode
        subprocess.run([sys.executable, "-c", RUN, str(N), f], check=True, env=env, cwd=root, timeout=300)
        z.append(np.load(f))
    assert np.max(np.abs(z[0] - z[1])) <= 1e-11 * np.max(np.abs(z[1]))
