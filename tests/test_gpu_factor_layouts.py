"""The operator on factor layouts whose last element ends before a full stride: wJ stored in
front of the six factors, and padded factors with the mass factors elsewhere. Bound: that of
test_gpu_ax_entry_forms.py (2 Nq + 8 roundings and the copies of the assembly)."""
import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg
from test_gpu_ax_entry_forms import _apply

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("prec", ["f64", "f32", "bf16g"])
@pytest.mark.parametrize("layout", ["wJ_first", "padded"])
@pytest.mark.parametrize("lam", [0.0, 0.7])
def test_layouts(N, prec, layout, lam):
    rng = np.random.default_rng(N)
    Nq, E = N + 1, 37
    Np = Nq ** 3
    vec = np.float64 if prec == "f64" else np.float32
    tvec = torch.float64 if prec == "f64" else torch.float32
    tgeo = torch.bfloat16 if prec == "bf16g" else tvec
    D = rng.uniform(-2, 2, (Nq, Nq)).astype(vec)
    if N in (3, 7):
        D = (0.5 * (D - D[::-1, ::-1])).astype(vec)
    geo = torch.tensor(rng.uniform(-1, 1, (E, 7, Np))).to(tgeo)   # wJ, then the factors
    q = rng.uniform(-1, 1, E * Np).astype(vec)
    dev = lambda x, t: torch.tensor(x, device="cuda").to(t).reshape(-1)
    if layout == "wJ_first":
        buf = geo.to("cuda").reshape(-1).clone()
        dW, dG, gs, ws = buf, buf[Np:], 7 * Np, 7 * Np
    else:   # strides of 6 Np + 8, the last element without its padding
        buf = torch.zeros((E - 1) * (6 * Np + 8) + 6 * Np, dtype=tgeo, device="cuda")
        for e in range(E):
            buf[e * (6 * Np + 8):e * (6 * Np + 8) + 6 * Np] = geo[e, 1:].reshape(-1).to("cuda")
        dG, gs, dW, ws = buf, 6 * Np + 8, geo[:, 0].contiguous().to("cuda").reshape(-1), Np
    out = torch.full((E * Np,), float("nan"), dtype=tvec, device="cuda")
    lpg.ax_hex(prec, N, E, dev(np.arange(E * Np), torch.int32), dG, gs, dW, ws, dev(D, tvec), lam, dev(q, tvec), out,
               E * Np)
    torch.cuda.synchronize()
    LD = np.longdouble
    g = geo.double().numpy().astype(LD).reshape(E, 7, Nq, Nq, Nq)
    u, lams = q.astype(LD).reshape(E, Nq, Nq, Nq), np.full(E, vec(lam)).astype(LD)
    ref = _apply(g[:, 1:], g[:, 0], D.astype(LD), lams, u)
    mag = _apply(np.abs(g[:, 1:]), np.abs(g[:, 0]), np.abs(D).astype(LD), lams, np.abs(u), top=prec == "f64")
    err = np.abs(out.cpu().numpy().astype(LD) - ref.reshape(-1))
    roundoff = 2.0 ** -53 if prec == "f64" else 2.0 ** -24
    assert np.all(err <= (2 * Nq + 8 + 1) * roundoff * mag.reshape(-1))
