"""The transfers of fixed degree pairs over every pair, with element counts that leave the last
block partly empty, lines with an infinite or NaN entry and an interpolation of another scale.

Bound per entry: three contractions of at most n = Nf + 1 terms, each with n roundings of the
magnitudes summed (FP64 lines: n 2^-57 of the line's largest magnitude times the row's, less
than one rounding of it), carried on by the others' absolute sums, at most S each; the
assembly of at most 8 copies, the weight and the addition to the old value: 10 more. So
(3 (n + 1) + 10) roundings of S^3 times the largest input, 8 copies of it in a restriction."""
import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg
from gpu_helpers import box
from test_gpu_kernel_exports import dev, interp

pytestmark = pytest.mark.gpu
LD = np.longdouble
PAIRS = [(7, 3), (3, 1), (8, 6), (7, 5), (6, 4), (5, 3), (4, 2), (3, 2), (2, 1)]


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


def _tensor3(P, u, E):
    with np.errstate(invalid="ignore"):
        for axis in (1, 2, 3):   # k, then j, then i
            u = np.moveaxis(np.einsum("am,...m->...a", P, np.moveaxis(u, axis, -1)), -1, axis)
    return u.reshape(E, -1)


@pytest.mark.parametrize("Nf,Nc", PAIRS)
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("form", ["plain", "nonfinite", "scaled"])
def test_transfer_lines(Nf, Nc, prec, form):
    base = box(**{"BOX NX": 3, "BOX NY": 3, "BOX NZ": 3, "LAMBDA": 1.0})
    ef = lpg.Elliptic(dict(base, **{"POLYNOMIAL DEGREE": Nf}))
    ec = lpg.Elliptic(dict(base, **{"POLYNOMIAL DEGREE": Nc}))
    E = ef.info("nelements")
    g2lf, g2lc = ef.get("GlobalToLocal"), ec.get("GlobalToLocal")
    dt, vec, u = ((torch.float64, np.float64, 2.0 ** -53) if prec == "f64" else (torch.float32, np.float32, 2.0 ** -24))
    scale = 2.0 ** (-80 if prec == "f64" else -20) if form == "scaled" else 1.0
    P = (scale * interp(Nf, Nc)).astype(vec)
    rng = np.random.default_rng(100 * Nf + Nc)
    wf, owner = ef.get("weightG").astype(vec), ef.get("ownerLocal")
    rF = (rng.uniform(-1, 1, ef.Nglobal) * 10.0 ** rng.integers(-9, 1, ef.Nglobal)).astype(vec)
    xC = rng.uniform(-1, 1, ec.Nglobal).astype(vec)
    xF0 = (scale ** 3 * rng.uniform(-1, 1, ef.Nglobal)).astype(vec)
    if form == "nonfinite":
        rF[[0, ef.Nglobal // 2]] = np.inf, np.nan
        xC[[0, ec.Nglobal // 2]] = np.nan, -np.inf
    with np.errstate(invalid="ignore"):
        nf, nc = Nf + 1, Nc + 1
        uF = np.where(g2lf >= 0, (wf.astype(LD) * rF)[np.maximum(g2lf, 0)], 0).reshape(E, nf, nf, nf)
        uC = _tensor3(P.T.astype(LD), uF, E).reshape(-1)
        refC = np.zeros(ec.Nglobal, dtype=LD)
        np.add.at(refC, g2lc[g2lc >= 0], uC[g2lc >= 0])
        vC = np.where(g2lc >= 0, xC.astype(LD)[np.maximum(g2lc, 0)], 0).reshape(E, nc, nc, nc)
        refF = xF0 + _tensor3(P.astype(LD), vC, E).reshape(-1)[owner]
    L = lpg.lib()
    a = [dev(g2lf), dev(g2lc), dev(owner), dev(wf, dt), dev(rF, dt), dev(P, dt)]
    d_rC = torch.full((ec.Nglobal,), np.nan, device="cuda", dtype=dt)
    d_xC, d_xF = dev(xC, dt), dev(xF0, dt)
    lpg.check(getattr(L, "lpg_pmg_restrict_" + prec)(Nf, Nc, E, a[0].data_ptr(), a[3].data_ptr(), a[4].data_ptr(),
                                                     a[5].data_ptr(), a[1].data_ptr(), d_rC.data_ptr(), ec.Nglobal, None))
    lpg.check(getattr(L, "lpg_pmg_prolong_add_" + prec)(Nf, Nc, E, a[1].data_ptr(), d_xC.data_ptr(), a[5].data_ptr(),
                                                        a[0].data_ptr(), a[2].data_ptr(), d_xF.data_ptr(), None))
    torch.cuda.synchronize()
    top = lambda v: float(np.max(np.abs(v[np.isfinite(v)])))
    for got, ref, M, n, size in ((d_rC, refC, P.T, nf, 8 * top(wf * rF)), (d_xF, refF, P, nc, top(xC))):
        got = got.cpu().numpy().astype(LD)
        S = float(np.max(np.sum(np.abs(M), axis=1)))
        ok = np.isfinite(ref)
        assert np.array_equal(np.isfinite(got), ok)
        assert np.all(np.abs(got[ok] - ref[ok]) <= (3 * (n + 1) + 10) * u * (S ** 3 * size + top(xF0) * (n == nc)))
