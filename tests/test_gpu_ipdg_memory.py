"""Device memory of an IPDG object: the factors, the maps and vectors every object holds, and no
more scratch for the operator than a gradient and a value per node (32 bytes) and a map of
4 bytes per face node."""
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


@pytest.mark.parametrize("N", range(1, 9))
def test_bytes_held(N):
    n = 6
    s = box(**{"POLYNOMIAL DEGREE": N, "BOX NX": n, "BOX NY": n, "BOX NZ": n, "DISCRETIZATION": "IPDG"})
    keep = lpg.Elliptic(box())
    before = keep.info("device_bytes")
    e = lpg.Elliptic(s)
    held = e.info("device_bytes") - before
    E, Np, Nf = n ** 3, (N + 1) ** 3, 6 * (N + 1) ** 2
    factors = E * 8 * (7 * Np + 10 * Np + 5 * Nf)               # geo, vgeo, sgeo
    # vertices, boundary flags; numbering (4 + 4), weight (8), the vectors q, Aq, x, r (32) and PCG's work (32)
    common = E * (3 * 8 * 8 + 6 * 4) + E * Np * (16 + 64)
    small = 1 << 16                                             # 1-D bases, reduction scratch
    assert held <= factors + common + E * (32 * Np + 4 * Nf) + small, (held, factors, common)
    # and an application allocates nothing
    q = torch.ones(e.Nglobal, dtype=torch.float64, device="cuda")
    Aq = torch.zeros_like(q)
    e.Operator(q, Aq)
    assert e.info("device_bytes") - before == held
