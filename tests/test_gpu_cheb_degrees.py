"""The p-levels' Chebyshev smoother at degrees 0 to 3 (no step, one step that is first and last,
several): one preconditioner application against the oracle, in FP64, and in FP32 against FP64.
Bounds: those of the other preconditioner comparisons, 1e-9 (rounding amplified by the
estimated eigenvalues and the coarse solves) and 1e-4 (2^-24 times the same amplification)."""
import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg
from gpu_helpers import box, rel_err
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


@pytest.mark.parametrize("degree", [0, 1, 2, 3])
@pytest.mark.parametrize("N,degrees", [(7, "7,3,1"), (4, "4,2,1")])
def test_chebyshev_degrees(N, degrees, degree):
    s = box(**{"BOX NX": 4, "BOX NY": 3, "BOX NZ": 5, "POLYNOMIAL DEGREE": N, "LAMBDA": 1.0, "LINEAR SOLVER": "FPCG",
               "PRECONDITIONER": "MULTIGRID", "MULTIGRID DEGREES": degrees, "MULTIGRID CHEBYSHEV DEGREE": degree,
               "PARALMOND AGGREGATION": "SMOOTHED"})
    o = Oracle(s)
    out = {}
    for prec in ("FP64", "FP32"):
        e = lpg.Elliptic(dict(s, **{"PRECONDITIONER PRECISION": prec}))
        rh = np.random.default_rng(degree).standard_normal(e.Nglobal)
        z = torch.full((e.Nglobal,), float("nan"), dtype=torch.float64, device="cuda")
        e.precon(torch.tensor(rh, device="cuda"), z)
        torch.cuda.synchronize()
        out[prec] = z.cpu().numpy()
    assert rel_err(out["FP64"], o.precon(rh)) < 1e-9
    assert rel_err(out["FP32"], out["FP64"]) < 1e-4
