"""What a user of this framework has it do, as measurable cases.

The cases go through the public entry points (libparanumal_gb300.Elliptic): the assembled
screened-Poisson operator in each precision (device and host arrays), the interior-penalty
operator, one preconditioner application and whole solves, on jittered hexahedral boxes
over the polynomial degrees the library supports. `exact` restates the operators in plain
torch FP64 from the mesh definition alone.
"""
import math

import numpy as np
import torch

import libparanumal_gb300 as lpg

# ---------------------------------------------------------------- the cases
_DEFAULTS = {"kind": "op", "prec": "f64", "N": 7, "nx": 8, "ny": 8, "nz": 8, "bc": 1, "lam": "one"}


def _case(name=None, **over):
    c = dict(_DEFAULTS)
    c.update(over)
    if name is not None:
        c["name"] = name
    return c


def _box(n):
    return {"nx": n, "ny": n, "nz": n}


def listed():
    return [
        # the throughput workload of the benchmark: FP64 assembled operator, 64^3, N = 7
        _case("op_f64_n7_64", **_box(64)),
        # a small FP64 operator: a coarse or strongly partitioned problem, launch latency counts
        _case("op_f64_n7_small", nx=5, ny=4, nz=3, lam="zero"),
        # FP64 operator at a degree without mirror-pair kernel, odd sizes, lambda per element
        _case("op_f64_n5_odd", N=5, nx=31, ny=23, nz=29, lam="field"),
        # the FP64-accurate double-FP32 operator: outer operator of the mixed-precision solves
        _case("op_df64_n7_40", prec="df64", lam="zero", **_box(40)),
        # FP32 operator of the preconditioner's fine level
        _case("op_f32_n7_48", prec="f32", **_box(48)),
        # FP32 operator at an even degree and odd sizes: intermediate p-multigrid level
        _case("op_f32_n4_odd", prec="f32", N=4, nx=47, ny=51, nz=45, lam="field"),
        # FP64 operator on page-locked host arrays: a caller that keeps its vectors on the host
        _case("host_f64_n7_40", kind="host", **_box(40)),
        # interior-penalty operator in FP64
        _case("ipdg_f64_n7_24", kind="ipdg", lam="zero", **_box(24)),
        # interior-penalty operator in double-FP32, odd degree and sizes
        _case("ipdg_df64_n5_odd", kind="ipdg", prec="df64", N=5, nx=21, ny=27, nz=25),
        # one p-multigrid V-cycle over the algebraic coarse levels, the default precision
        _case("vcycle_f64_n7_20", kind="vcycle", lam="zero", **_box(20)),
        # a small solve: flexible CG with Jacobi, 8^3, N = 5
        _case("solve_jacobi_f64_n5_8", kind="solve", precon="JACOBI", N=5, lam="zero", **_box(8)),
        # a time step's solve: flexible CG, FP32 p-multigrid, double-FP32 outer operator
        _case("solve_pmg_mixed_n7_32", kind="solve", precon="MULTIGRID", prec="mixed", **_box(32)),
    ]


def _sizes(rng, nodes, N):
    """Three element counts, uneven, whose box has about `nodes` local nodes."""
    e = max(8.0, nodes / (N + 1) ** 3)
    side = e ** (1.0 / 3.0)
    a, b = (math.exp(rng.uniform(-0.35, 0.35)) for _ in range(2))
    n = [side * a, side * b, side / (a * b)]
    return {k: max(2, int(round(v))) for k, v in zip(("nx", "ny", "nz"), n)}


def draw(rng):
    kind = rng.choice(["op", "op", "op", "op", "host", "ipdg", "ipdg", "vcycle", "solve"])
    N = rng.choice([1, 2, 3, 4, 5, 6, 7, 7, 7, 8])
    lam = rng.choice(["zero", "one", "field", "const"])
    if kind == "op":
        prec = rng.choice(["f64", "f64", "df64", "f32", "f32", "bf16g"])
        nodes = math.exp(rng.uniform(math.log(1e4), math.log(4e7)))
        return _case(kind=kind, prec=prec, N=N, lam=lam, bc=rng.choice([1, 1, 1, 2, -1]), **_sizes(rng, nodes, N))
    if kind == "host":
        prec = rng.choice(["f64", "f64", "f32"])
        nodes = math.exp(rng.uniform(math.log(1e5), math.log(2e7)))
        return _case(kind=kind, prec=prec, N=N, lam=lam, **_sizes(rng, nodes, N))
    if kind == "ipdg":
        prec = rng.choice(["f64", "df64", "f32"])
        nodes = math.exp(rng.uniform(math.log(1e4), math.log(8e6)))
        return _case(kind=kind, prec=prec, N=N, lam=lam, bc=rng.choice([1, 1, -1]), **_sizes(rng, nodes, N))
    N = rng.choice([3, 4, 5, 6, 7, 7])
    if kind == "vcycle":
        nodes = math.exp(rng.uniform(math.log(3e4), math.log(4e6)))
        return _case(kind=kind, N=N, lam=lam, **_sizes(rng, nodes, N))
    precon, prec, most = rng.choice([("JACOBI", "f64", 1e6), ("MULTIGRID", "f64", 1e6), ("MULTIGRID", "mixed", 4e6)])
    nodes = math.exp(rng.uniform(math.log(3e4), math.log(most)))
    return _case(kind=kind, precon=precon, prec=prec, N=N, lam=lam, **_sizes(rng, nodes, N))


# ---------------------------------------------------------------- preparing and running
_LAMBDA = {"zero": 0.0, "one": 1.0, "const": 2.5, "field": 1.0}


def _settings(c, seed):
    s = {"BOX NX": c["nx"], "BOX NY": c["ny"], "BOX NZ": c["nz"], "BOX DIMX": 2, "BOX DIMY": 2, "BOX DIMZ": 2,
         "BOX BOUNDARY FLAG": c["bc"], "POLYNOMIAL DEGREE": c["N"], "LAMBDA": _LAMBDA[c["lam"]],
         "MESH JITTER": 0.1, "MESH JITTER SEED": seed, "LINEAR SOLVER": "FPCG", "PRECONDITIONER": "NONE"}
    if c["lam"] == "field":
        s["LAMBDA FIELD"] = "LOGNORMAL"
        s["LAMBDA SEED"] = seed
    if c["kind"] == "ipdg":
        s["DISCRETIZATION"] = "IPDG"
    if c["kind"] in ("vcycle", "solve"):
        s["PRECONDITIONER"] = c.get("precon", "MULTIGRID")
        if c["N"] == 7:
            s["MULTIGRID DEGREES"] = "7,3,1"
        if c["prec"] == "mixed":
            s["PRECONDITIONER PRECISION"] = "FP32"
            s["OPERATOR PRECISION"] = "DF64"
    return s


def _uniform(n, seed, dtype=torch.float64):
    """n values of U[-1, 1)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.rand(n, generator=g, dtype=torch.float64, device="cuda").mul_(2).sub_(1).to(dtype)


def _waves(seed):
    """A smooth field on [-1, 1]^3 with zero boundary values: eight sine products."""
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    return [(r.uniform(-1, 1), r.randint(1, 5), r.randint(1, 5), r.randint(1, 5)) for _ in range(8)]


def _smooth(c, seed, m):
    u = torch.zeros_like(m.x)
    for a, kx, ky, kz in _waves(seed):
        h = math.pi / 2
        u += a * torch.sin(kx * h * (m.x + 1)) * torch.sin(ky * h * (m.y + 1)) * torch.sin(kz * h * (m.z + 1))
    return u


def prepare(case, seed):
    c = dict(case)
    e = lpg.Elliptic(_settings(c, seed))
    n = e.Nglobal
    st = {"case": c, "e": e}
    if c["kind"] == "host":
        dt = torch.float64 if c["prec"] == "f64" else torch.float32
        st["q"] = _uniform(n, seed, dt).cpu().pin_memory()
        st["Aq"] = torch.empty(n, dtype=dt, pin_memory=True)
    elif c["kind"] == "solve":
        # right-hand side of a time step: the mass product of a smooth field
        m = _Mesh(c, seed)
        u = m.to_dofs(_smooth(c, seed, m))
        st["b"], st["r"], st["x"] = torch.empty_like(u), torch.empty_like(u), torch.empty_like(u)
        e.mass(u, st["b"])
        torch.cuda.synchronize()
    else:
        dt = torch.float32 if c["prec"] in ("f32", "bf16g") else torch.float64
        st["q"] = _uniform(n, seed, dt)
        st["Aq"] = torch.empty(n, dtype=dt, device="cuda")
    return st


def run(st):
    c, e = st["case"], st["e"]
    if c["kind"] == "solve":
        st["r"].copy_(st["b"])
        st["x"].zero_()
        e.Solve(st["x"], st["r"], tol=1e-8, maxit=2000)
        return {"x": st["x"]}
    q, Aq = st["q"], st["Aq"]
    if c["kind"] == "host":
        e.OperatorHost(q, Aq, "FP64" if c["prec"] == "f64" else "FP32")
    elif c["kind"] == "vcycle":
        e.precon(q, Aq)
    elif c["prec"] == "f64":
        e.Operator(q, Aq)
    elif c["prec"] == "df64":
        e.OperatorDF64(q, Aq)
    else:
        e.OperatorF32(q, Aq, bf16geo=(c["prec"] == "bf16g"))
    return {"Aq": Aq}


# ---------------------------------------------------------------- work
def _dofs(c, N):
    n = 1
    for d in ("nx", "ny", "nz"):
        n *= c[d] * N + (-1 if c["bc"] == 1 else 0 if c["bc"] == -1 else 1)
    return n


def _op_work(c, N, prec):
    """Bytes and operations of one operator application at degree N."""
    E, Nq = c["nx"] * c["ny"] * c["nz"], N + 1
    nl, size = E * Nq ** 3, {"f64": 8, "df64": 8, "f32": 4, "bf16g": 2}[prec]
    vec = 8 if size == 8 else 4
    if c["kind"] == "ipdg":
        return nl * (10 * size + 2 * vec) + E * 6 * Nq * Nq * (5 * size + 4), (12 * Nq + 33) * nl
    factors = 6 if c["lam"] == "zero" else 7
    return nl * (factors * size + 4) + 2 * vec * _dofs(c, N), (12 * Nq + 18) * nl


def _schedule(N):
    if N == 7:
        return [7, 3]
    deg, n = [N], N   # each level at most half the nodes of the one above
    while n > 1:
        half = (n + 1) ** 3 / 2
        while (n + 1) ** 3 > half and n > 1:
            n -= 1
        deg.append(n)
    return [d for d in deg if d > 1]


def _vcycle_work(c, prec):
    """Six operator applications a level and the vector passes between them."""
    b = f = 0
    for N in _schedule(c["N"]):
        ob, of = _op_work(c, N, prec)
        n = _dofs(c, N)
        b += 6 * ob + 30 * n * (8 if prec == "f64" else 4)
        f += 6 * of + 40 * n
    return b, f


def work(case):
    c = dict(case)
    if c["kind"] in ("op", "ipdg", "host"):
        b, f = _op_work(c, c["N"], c["prec"])
    elif c["kind"] == "vcycle":
        b, f = _vcycle_work(c, "f64")
    else:
        n = _dofs(c, c["N"])
        ob, of = _op_work(c, c["N"], "f64")
        if c["precon"] == "JACOBI":
            # about as many iterations as the box has nodes along two edges
            its, vb, vf = 2 * c["N"] * max(c["nx"], c["ny"], c["nz"]), 0, 0
        else:
            its = 8
            vb, vf = _vcycle_work(c, "f32" if c["prec"] == "mixed" else "f64")
        b, f = its * (ob + vb + 12 * 8 * n), its * (of + vf + 12 * n)
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------- the same in plain FP64
def _gll(N):
    """Gauss-Lobatto-Legendre points, weights and the derivative matrix."""
    P = np.polynomial.legendre.Legendre.basis(N)
    x = np.concatenate([[-1.0], np.sort(P.deriv().roots().real) if N > 1 else [], [1.0]])
    for _ in range(3):   # Newton on the interior points
        if N > 1:
            xi = x[1:-1]
            x[1:-1] = xi - P.deriv()(xi) / P.deriv(2)(xi)
    x = 0.5 * (x - x[::-1])
    w = 2.0 / (N * (N + 1) * P(x) ** 2)
    bw = np.array([1.0 / np.prod([x[j] - x[k] for k in range(N + 1) if k != j]) for j in range(N + 1)])
    D = np.zeros((N + 1, N + 1))
    for i in range(N + 1):
        for j in range(N + 1):
            if i != j:
                D[i, j] = bw[j] / bw[i] / (x[i] - x[j])
        D[i, i] = -D[i].sum()
    return x, w, D


def _mix(x):
    z = x + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _u01(seed, stream, key):
    """The documented uniform in [0, 1) keyed by (seed, stream, key): two splitmix64 steps."""
    with np.errstate(over="ignore"):
        s = _mix(np.array([seed ^ (stream << 56)], dtype=np.uint64))
        return (_mix(s + key.astype(np.uint64)) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


class _Mesh:
    """Nodes and dof numbering of a case's box; fields have the shape (nz, ny, nx, Nq, Nq, Nq)."""

    def __init__(self, c, seed):
        self.c, self.N = c, c["N"]
        nx, ny, nz = c["nx"], c["ny"], c["nz"]
        x1, self.w1, D = _gll(self.N)
        self.D = torch.tensor(D, device="cuda")
        vx, vy, vz = np.meshgrid(np.arange(nx + 1), np.arange(ny + 1), np.arange(nz + 1), indexing="ij")
        inner = (vx > 0) & (vx < nx) & (vy > 0) & (vy < ny) & (vz > 0) & (vz < nz) & (c["bc"] != -1)
        vid = (vx + (nx + 1) * (vy + (ny + 1) * vz)).astype(np.uint64)
        xyz = []
        for axis, (v, n) in enumerate(((vx, nx), (vy, ny), (vz, nz))):
            h = 2.0 / n
            p = -1.0 + h * v + np.where(inner, (2.0 * _u01(seed, axis, vid) - 1.0) * 0.1 * h, 0.0)
            xyz.append(torch.tensor(p.transpose(2, 1, 0).copy(), device="cuda"))   # [z][y][x]
        lo, hi = (torch.tensor(0.5 * (1 + s * x1), device="cuda") for s in (-1, 1))
        self.x, self.y, self.z = (self._trilinear(p, lo, hi) for p in xyz)
        self._number()

    @staticmethod
    def _trilinear(p, lo, hi):
        for axis in range(3):   # along z, y, x: the two vertices of every cell, weighted per node
            a = p.narrow(axis, 0, p.shape[axis] - 1).unsqueeze(-1)
            b = p.narrow(axis, 1, p.shape[axis] - 1).unsqueeze(-1)
            p = a * lo + b * hi
        return p

    def _number(self):
        """Dofs in the order of their first appearance in local node order; -1 where masked."""
        c, N = self.c, self.N
        ids, mask = [], []
        for n in (c["nx"], c["ny"], c["nz"]):
            g = torch.arange(n, device="cuda")[:, None] * N + torch.arange(N + 1, device="cuda")[None, :]
            total = n * N + 1
            mask.append((g == 0) | (g == total - 1) if c["bc"] == 1 else torch.zeros_like(g, dtype=torch.bool))
            ids.append(g % (total - 1) if c["bc"] == -1 else g)
        gx, gy, gz = ids
        L = [n * N + 1 for n in (c["nx"], c["ny"], c["nz"])]
        lat = (gx[None, None, :, None, None, :] + L[0] * (gy[None, :, None, None, :, None]
                                                         + L[1] * gz[:, None, None, :, None, None])).reshape(-1)
        off = (mask[0][None, None, :, None, None, :] | mask[1][None, :, None, None, :, None]
               | mask[2][:, None, None, :, None, None]).reshape(-1)
        local = torch.arange(lat.numel(), device="cuda")
        first = torch.full((L[0] * L[1] * L[2],), lat.numel(), dtype=torch.int64, device="cuda")
        first.scatter_reduce_(0, lat, torch.where(off, lat.numel(), local), "amin")
        is_first = first[lat] == local
        number = torch.cumsum(is_first, 0) - 1
        owner = first[lat].clamp_(max=lat.numel() - 1)
        self.g2l = torch.where(off, -1, number[owner])
        self.owner = local[is_first]
        self.n = int(self.owner.numel())

    @property
    def shape(self):
        return self.x.shape

    def to_dofs(self, field):
        return field.reshape(-1)[self.owner].contiguous()

    def scatter(self, q):
        return torch.where(self.g2l < 0, 0.0, q[self.g2l.clamp(min=0)]).view(self.shape)

    def gather(self, field):
        out = torch.zeros(self.n + 1, dtype=torch.float64, device="cuda")
        out.index_add_(0, torch.where(self.g2l < 0, self.n, self.g2l), field.reshape(-1))
        return out[:-1]

    def d(self, f, axis):
        """Derivative of a field along r (axis 0), s (1) or t (2)."""
        m = f.movedim(5 - axis, -1) @ self.D.T
        return m.movedim(-1, 5 - axis)

    def dT(self, f, axis):
        m = f.movedim(5 - axis, -1) @ self.D
        return m.movedim(-1, 5 - axis)

    def metric(self):
        """(grad r, grad s, grad t) as rows of three fields, and J."""
        x = [[self.d(v, a) for v in (self.x, self.y, self.z)] for a in range(3)]   # x[a][comp]

        def cross(a, b):
            return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]

        c0, c1, c2 = cross(x[1], x[2]), cross(x[2], x[0]), cross(x[0], x[1])
        J = x[0][0] * c0[0] + x[0][1] * c0[1] + x[0][2] * c0[2]
        return [[v / J for v in c] for c in (c0, c1, c2)], J

    def weights(self):
        w = torch.tensor(self.w1, device="cuda")
        return w[:, None, None] * w[None, :, None] * w[None, None, :]

    def lam(self, seed):
        c = self.c
        if c["lam"] != "field":
            return _LAMBDA[c["lam"]]
        e = np.arange(c["nx"] * c["ny"] * c["nz"])
        u1, u2 = 1.0 - _u01(seed, 4, e), _u01(seed, 5, e)
        v = np.exp(np.sqrt(-2.0 * np.log(u1)) * np.cos(2.0 * np.pi * u2))
        return torch.tensor(v, device="cuda").view(c["nz"], c["ny"], c["nx"], 1, 1, 1)


class _Continuous:
    def __init__(self, m, seed):
        self.m, self.lam = m, m.lam(seed)
        g, J = m.metric()
        self.wJ = J * m.weights()
        self.G = {(a, b): self.wJ * (g[a][0] * g[b][0] + g[a][1] * g[b][1] + g[a][2] * g[b][2])
                  for a in range(3) for b in range(a, 3)}

    def __call__(self, q):
        m, G = self.m, self.G
        u = m.scatter(q)
        du = [m.d(u, a) for a in range(3)]
        out = self.lam * self.wJ * u
        for a in range(3):
            out += m.dT(sum(G[min(a, b), max(a, b)] * du[b] for b in range(3)), a)
        return m.gather(out)

    def diagonal(self):
        """Diagonal of the assembled operator (its cross terms only meet at the node itself)."""
        m, G = self.m, self.G
        D2, dd = m.D * m.D, torch.diagonal(m.D)
        out = self.lam * self.wJ + torch.zeros_like(self.wJ)
        for a in range(3):
            out += (G[a, a].movedim(5 - a, -1) @ D2).movedim(-1, 5 - a)
        s = [dd.view([-1 if 2 - a == k else 1 for k in range(3)]) for a in range(3)]
        for a in range(3):
            for b in range(a + 1, 3):
                out += 2 * G[a, b] * s[a] * s[b]
        return m.gather(out)


def _interior_penalty(c, seed, q):
    """The symmetric interior-penalty operator, penalty 2 (N+1)(N+3) max(sJ/J)."""
    m = _Mesh(c, seed)
    N, periodic = m.N, c["bc"] == -1
    g, J = m.metric()
    W, lam = m.weights() * J, m.lam(seed)
    u = q.view(m.shape)
    du = [m.d(u, a) for a in range(3)]
    grad = [g[0][k] * du[0] + g[1][k] * du[1] + g[2][k] * du[2] for k in range(3)]
    acc = [W * v for v in grad]
    val = lam * W * u
    w1 = torch.tensor(m.w1, device="cuda")
    ww = w1[:, None] * w1[None, :]
    tau = 2.0 * (N + 1) * (N + 3)
    for a in range(3):
        axis, cells = 5 - a, 2 - a   # node axis and element axis of this direction
        nrm = torch.sqrt(g[a][0] ** 2 + g[a][1] ** 2 + g[a][2] ** 2)
        for hi in (0, 1):
            mine, theirs = (N, 0) if hi else (0, N)
            sgn, shift = (1.0, -1) if hi else (-1.0, 1)

            def own(f):
                return f.select(axis, mine)

            def other(f):
                return torch.roll(f.select(axis, theirs), shift, cells)

            edge = torch.zeros(own(u).shape[:3], dtype=torch.bool, device="cuda")
            if not periodic:
                edge.select(cells, edge.shape[cells] - 1 if hi else 0).fill_(True)
            edge = edge[..., None, None]
            h = nrm            # sJ / J = |grad| on this face
            hinv = torch.where(edge, own(h), torch.maximum(own(h), other(h)))
            n = [sgn * own(g[a][k]) / own(nrm) for k in range(3)]
            ws = own(nrm) * own(J) * ww
            gP = [torch.where(edge, own(v), other(v)) for v in grad]
            uP = torch.where(edge, -own(u), other(u))
            jump = uP - own(u)
            flux = sum(n[k] * (gP[k] + own(grad[k])) for k in range(3)) + tau * hinv * jump
            for k in range(3):
                acc[k].select(axis, mine).add_(0.5 * ws * n[k] * jump)
            val.select(axis, mine).sub_(0.5 * ws * flux)
    for a in range(3):
        val += m.dT(g[a][0] * acc[0] + g[a][1] * acc[1] + g[a][2] * acc[2], a)
    return val.reshape(-1)


def _solved(c, seed):
    """Conjugate gradients with Jacobi on the plain operator, to rounding."""
    m = _Mesh(c, seed)
    A = _Continuous(m, seed)
    u = m.to_dofs(_smooth(c, seed, m))
    b = m.gather(A.wJ * m.scatter(u))
    inv = 1.0 / A.diagonal()
    x, r = torch.zeros_like(b), b.clone()
    z = inv * r
    p, rz = z.clone(), torch.dot(r, z)
    stop = 1e-14 * float(b.norm())
    for it in range(4000):
        Ap = A(p)
        alpha = rz / torch.dot(p, Ap)
        x += alpha * p
        r -= alpha * Ap
        if it % 20 == 0 and float(r.norm()) < stop:
            break
        z = inv * r
        rz, old = torch.dot(r, z), rz
        p = z + (rz / old) * p
    return x


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "vcycle":
        return None   # the preconditioner is an algorithm, not a value with a closed form
    if c["kind"] == "solve":
        return {"x": _solved(c, seed)} if _dofs(c, c["N"]) < 1_500_000 else None
    if c["kind"] == "ipdg":
        n = c["nx"] * c["ny"] * c["nz"] * (c["N"] + 1) ** 3
    else:
        n = _dofs(c, c["N"])
    q = _uniform(n, seed, torch.float32 if c["prec"] in ("f32", "bf16g") else torch.float64).double()
    if c["kind"] == "ipdg":
        return {"Aq": _interior_penalty(c, seed, q)}
    Aq = _Continuous(_Mesh(c, seed), seed)(q)
    return {"Aq": Aq.cpu() if c["kind"] == "host" else Aq}
