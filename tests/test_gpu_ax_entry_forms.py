"""The assembled operator through the C entry points with a caller's own arrays, over the
forms they accept: every degree, element lists, the reference's and the packed factor layout,
arrays that start off a 16-byte boundary, a D without mirror symmetry, a lambda field.

Bound per dof: the longest chain of roundings of one term is the Nq products and sums of each
of the two contractions, five operations of the metric product, three of the sum and the mass
term and eight of the assembly: 2 Nq + 16 roundings of the magnitudes summed. The FP64 kernels'
integer lines err by at most Nq 2^-57 of the largest magnitudes of a line and a row, which
replace the plain magnitudes there; BF16 factors are exact inputs."""
import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


def _line(M, f, d, top):
    """sum_m M[a][m] f[.. m ..] along r (0), s (1), t (2); top: with the line's and the row's
    largest magnitudes in place of every term's"""
    g = np.moveaxis(f, 3 - d, -1)
    if top:
        g = np.broadcast_to(g.max(axis=-1, keepdims=True), g.shape)
        M = np.broadcast_to(M.max(axis=1, keepdims=True), M.shape)
    return np.moveaxis(np.einsum("am,...m->...a", M, g), -1, 3 - d)


def _apply(G, wJ, D, lam, u, top=False):
    sym = [[0, 1, 2], [1, 3, 4], [2, 4, 5]]
    du = [_line(D, u, d, top) for d in range(3)]
    out = lam[:, None, None, None] * wJ * u
    for a in range(3):
        out = out + _line(D.T, sum(G[:, sym[a][b]] * du[b] for b in range(3)), a, top)
    return out


def _off(x, dtype, offset):
    """device copy of x that starts `offset` entries behind an aligned address"""
    buf = torch.zeros(x.size + 16, dtype=dtype, device="cuda")
    v = buf[offset:offset + x.size]
    v.copy_(torch.tensor(x.reshape(-1)))
    return v


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("prec", ["f64", "f32", "bf16g"])
@pytest.mark.parametrize("form", ["packed", "reference", "list_offset", "field_zero"])
def test_entry_point_forms(N, prec, form):
    rng = np.random.default_rng(100 * N + len(form))
    Nq, E = N + 1, 37
    Np = Nq ** 3
    vec = np.float64 if prec == "f64" else np.float32
    tvec = torch.float64 if prec == "f64" else torch.float32
    tgeo = torch.bfloat16 if prec == "bf16g" else tvec
    D = rng.uniform(-2, 2, (Nq, Nq)).astype(vec)
    if N in (3, 7):   # these degrees contract through the mirror symmetry
        D = (0.5 * (D - D[::-1, ::-1])).astype(vec)
    geo = torch.tensor(rng.uniform(-1, 1, (E, 7, Nq, Nq, Nq))).to(tgeo).double().numpy()
    Ng = 5 * Np
    g2l = rng.integers(-1, Ng, E * Np).astype(np.int32)
    q = rng.uniform(-1, 1, Ng).astype(vec)
    lamE = rng.uniform(0, 2, E).astype(vec)
    lam, field, elems, offset = 0.7, None, np.arange(E), 0
    if form == "field_zero":
        lam = 0.0
        field = lamE if N % 2 else None
    if form == "list_offset":
        elems, offset = rng.permutation(E)[:21], 3
    t = lambda x, dt, o=offset: _off(x, dt, o)
    dD, dq, dg2l = t(D, tvec), t(q, tvec), t(g2l, torch.int32)
    if form == "reference":
        dG, dW, gs, ws = t(geo[:, :6].copy(), tgeo), t(geo[:, 6].copy(), tgeo), 6 * Np, Np
    else:
        dG = t(geo, tgeo)
        dW, gs, ws = dG[6 * Np:], 7 * Np, 7 * Np
    dl = t(field, tvec) if field is not None else None
    lst = torch.tensor(elems.astype(np.int32), device="cuda") if form == "list_offset" else None
    out = _off(np.full(Ng, np.nan), tvec, offset)
    lpg.ax_hex(prec, N, len(elems), dg2l, dG, gs, dW, ws, dD, lam, dq, out, Ng, lambdaE=dl, element_list=lst)
    torch.cuda.synchronize()

    LD = np.longdouble
    lams = (field if field is not None else np.full(E, lam)).astype(LD)[elems]
    idx = g2l.reshape(E, Np)[elems]
    u = np.where(idx < 0, 0, q[np.maximum(idx, 0)]).astype(LD).reshape(-1, Nq, Nq, Nq)
    G, W, Dl = geo[elems][:, :6].astype(LD), geo[elems][:, 6].astype(LD), D.astype(LD)

    def gather(f):
        r = np.zeros(Ng + 1, dtype=LD)
        np.add.at(r, np.where(idx < 0, Ng, idx).reshape(-1), f.reshape(-1))
        return r[:-1]

    ref = gather(_apply(G, W, Dl, lams, u))
    mag = gather(_apply(np.abs(G), np.abs(W), np.abs(Dl), np.abs(lams), np.abs(u), top=prec == "f64"))
    roundoff = 2.0 ** -53 if prec == "f64" else 2.0 ** -24
    copies = np.bincount(idx[idx >= 0], minlength=Ng).max()   # the assembly of random indices
    err = np.abs(out.cpu().numpy().astype(LD) - ref)
    assert np.all(err <= (2 * Nq + 8 + copies) * roundoff * mag)


@pytest.mark.parametrize("N", [2, 3, 6, 7])
@pytest.mark.parametrize("scale", [2.0 ** -90, 2.0 ** 90])
def test_scaled_derivative(N, scale):
    """A D outside the integers' range of rows is served by FP64 lines: same bound."""
    rng = np.random.default_rng(N)
    Nq, E = N + 1, 5
    Np = Nq ** 3
    D = rng.uniform(-2, 2, (Nq, Nq)) * scale
    if N in (3, 7):
        D = 0.5 * (D - D[::-1, ::-1])
    geo, q = rng.uniform(-1, 1, (E, 7, Nq, Nq, Nq)), rng.uniform(-1, 1, E * Np)
    dev = lambda x: torch.tensor(x, device="cuda").reshape(-1)
    dG, out = dev(geo), torch.empty(E * Np, dtype=torch.float64, device="cuda")
    lpg.ax_hex("f64", N, E, dev(np.arange(E * Np, dtype=np.int32)), dG, 7 * Np, dG[6 * Np:], 7 * Np, dev(D), 0.0,
               dev(q), out, E * Np)
    torch.cuda.synchronize()
    LD = np.longdouble
    G, W, u = geo[:, :6].astype(LD), geo[:, 6].astype(LD), q.astype(LD).reshape(-1, Nq, Nq, Nq)
    ref = _apply(G, W, D.astype(LD), np.zeros(E, LD), u)
    mag = _apply(np.abs(G), W, np.abs(D).astype(LD), np.zeros(E, LD), np.abs(u), top=True)
    err = np.abs(out.cpu().numpy().astype(LD) - ref.reshape(-1))
    assert np.all(err <= (2 * Nq + 8 + 1) * 2.0 ** -53 * mag.reshape(-1))


@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("prec", ["f32", "bf16g"])
@pytest.mark.parametrize("form", ["one", "list", "nomass", "nomass_list"])
def test_fp32_line_kernel(N, prec, form):
    """One element, a partly empty last block, aligned element lists, no mass term."""
    rng = np.random.default_rng(10 * N + len(form))
    Nq, E = N + 1, 1 if form == "one" else 75
    Np = Nq ** 3
    tgeo = torch.bfloat16 if prec == "bf16g" else torch.float32
    D = rng.uniform(-2, 2, (Nq, Nq)).astype(np.float32)
    geo = torch.tensor(rng.uniform(-1, 1, (E, 7, Nq, Nq, Nq))).to(tgeo).double().numpy()
    g2l = rng.integers(-1, 5 * Np, E * Np).astype(np.int32)
    q = rng.uniform(-1, 1, 5 * Np).astype(np.float32)
    lam = 0.0 if "nomass" in form else 0.7
    elems = rng.permutation(E)[:41] if "list" in form else np.arange(E)
    dG = _off(geo, tgeo, 0)
    out = torch.empty(5 * Np, dtype=torch.float32, device="cuda")
    lst = torch.tensor(elems.astype(np.int32), device="cuda") if "list" in form else None
    lpg.ax_hex(prec, N, len(elems), _off(g2l, torch.int32, 0), dG, 7 * Np, dG[6 * Np:], 7 * Np,
               _off(D, torch.float32, 0), lam, _off(q, torch.float32, 0), out, 5 * Np, element_list=lst)
    torch.cuda.synchronize()
    LD = np.longdouble
    lams = np.full(len(elems), lam, dtype=np.float32).astype(LD)
    idx = g2l.reshape(E, Np)[elems]
    u = np.where(idx < 0, 0, q[np.maximum(idx, 0)]).astype(LD).reshape(-1, Nq, Nq, Nq)
    G, W, Dl = geo[elems][:, :6].astype(LD), geo[elems][:, 6].astype(LD), D.astype(LD)

    def gather(f):
        r = np.zeros(5 * Np + 1, dtype=LD)
        np.add.at(r, np.where(idx < 0, 5 * Np, idx).reshape(-1), f.reshape(-1))
        return r[:-1]

    ref = gather(_apply(G, W, Dl, lams, u))
    mag = gather(_apply(np.abs(G), np.abs(W), np.abs(Dl), lams, np.abs(u)))
    copies = np.bincount(idx[idx >= 0], minlength=5 * Np).max()
    assert np.all(np.abs(out.cpu().numpy().astype(LD) - ref) <= (2 * Nq + 8 + copies) * 2.0 ** -24 * mag)
