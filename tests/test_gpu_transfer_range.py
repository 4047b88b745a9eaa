"""FP64 transfers on lines whose entries differ by many orders of magnitude.

Nodes that both levels share (the ends, and the midpoints where both degrees are even) take
the other level's value as it is: a prolongation onto zero gives it bit for bit.

Bound per entry, relative to the magnitudes summed, u = 2^-53: a contraction of n terms has an
error of n u (an FP64 chain), or n 2^-57 of (largest entry of the line) x (largest of the row),
which is at most kappa times the sum of the products' magnitudes, kappa being the largest ratio
of two entries in a row or column of P off the shared nodes, and 2 u for the conversion and the
addition of a shared node. So 3 (n (1 + kappa / 16) + 2) u for the three, and 10 u for the
weight, the assembly of 8 copies and the addition to the old value."""
import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg
from gpu_helpers import box
from test_gpu_kernel_exports import dev
from test_gpu_transfer_lines import PAIRS, _tensor3

pytestmark = pytest.mark.gpu
LD, U = np.longdouble, 2.0 ** -53


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


def _problem(Nf, Nc):
    base = box(**{"BOX NX": 3, "BOX NY": 3, "BOX NZ": 3})
    return [lpg.Elliptic(dict(base, **{"POLYNOMIAL DEGREE": N})) for N in (Nf, Nc)]


def _interp(ef, ec, Nf, Nc):
    """P[i][m] = l_m(x_i) with the factors that vanish or are 1 exactly so"""
    def nodes(N):
        x = np.polynomial.legendre.Legendre.basis(N).deriv().roots().real if N > 1 else np.zeros(0)
        x = np.concatenate([[-1.0], np.sort(x), [1.0]])
        return 0.5 * (x - x[::-1])
    xf, xc = nodes(Nf), nodes(Nc)
    P = np.ones((Nf + 1, Nc + 1))
    for m in range(Nc + 1):
        for k in range(Nc + 1):
            if k != m:
                P[:, m] *= (xf - xc[k]) / (xc[m] - xc[k])
    shared = {0: 0, Nf: Nc}
    if Nf % 2 == 0 and Nc % 2 == 0:
        shared[Nf // 2] = Nc // 2
    for i, m in shared.items():
        assert np.array_equal(P[i], np.eye(Nc + 1)[m])
    inner = np.abs(P[[i for i in range(Nf + 1) if i not in shared]])
    kappa = max((inner.max(1) / inner.min(1)).max(), (inner.max(0) / inner.min(0)).max())
    return P, shared, kappa


@pytest.mark.parametrize("Nf,Nc", PAIRS)
@pytest.mark.parametrize("seed", [0, 1])
def test_wide_lines(Nf, Nc, seed):
    ef, ec = _problem(Nf, Nc)
    P, shared, kappa = _interp(ef, ec, Nf, Nc)
    E, nf, nc = ef.info("nelements"), Nf + 1, Nc + 1
    g2lf, g2lc, owner, wf = ef.get("GlobalToLocal"), ec.get("GlobalToLocal"), ef.get("ownerLocal"), ef.get("weightG")
    rng = np.random.default_rng(seed)
    wide = lambda n: rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-12, 3, n)
    rF, xC = wide(ef.Nglobal), wide(ec.Nglobal)
    L = lpg.lib()
    a = [dev(v) for v in (g2lf, g2lc, owner, wf, rF, P, xC)]
    d_rC = torch.full((ec.Nglobal,), np.nan, device="cuda", dtype=torch.float64)
    d_xF = torch.zeros(ef.Nglobal, device="cuda", dtype=torch.float64)
    lpg.check(L.lpg_pmg_restrict_f64(Nf, Nc, E, a[0].data_ptr(), a[3].data_ptr(), a[4].data_ptr(), a[5].data_ptr(),
                                     a[1].data_ptr(), d_rC.data_ptr(), ec.Nglobal, None))
    lpg.check(L.lpg_pmg_prolong_add_f64(Nf, Nc, E, a[1].data_ptr(), a[6].data_ptr(), a[5].data_ptr(), a[0].data_ptr(),
                                        a[2].data_ptr(), d_xF.data_ptr(), None))
    torch.cuda.synchronize()
    gotF, gotC = d_xF.cpu().numpy(), d_rC.cpu().numpy()

    vC = np.where(g2lc >= 0, xC[np.maximum(g2lc, 0)], 0.0).reshape(E, nc, nc, nc)
    n = owner % nf ** 3
    i, j, k = n % nf, (n // nf) % nf, n // nf ** 2
    at = np.array([shared.get(v, -1) for v in range(nf)])
    both = (at[i] >= 0) & (at[j] >= 0) & (at[k] >= 0)
    assert both.sum() >= 8
    assert np.array_equal(gotF[both], vC[owner // nf ** 3, at[k], at[j], at[i]][both])

    def up(M, x):
        return _tensor3(M.astype(LD), x.astype(LD), E).reshape(-1)[owner]

    def down(M, x):
        y = _tensor3(M.T.astype(LD), x.astype(LD), E).reshape(-1)
        r = np.zeros(ec.Nglobal, dtype=LD)
        np.add.at(r, g2lc[g2lc >= 0], y[g2lc >= 0])
        return r

    uF = np.where(g2lf >= 0, (wf.astype(LD) * rF)[np.maximum(g2lf, 0)], 0).reshape(E, nf, nf, nf)
    for got, op, x, terms in ((gotF, up, vC, nc), (gotC, down, uF, nf)):
        err, mag = np.abs(got.astype(LD) - op(P, x)), op(np.abs(P), np.abs(x))
        assert np.all(err <= (3 * (terms * (1 + kappa / 16) + 2) + 10) * U * mag)
