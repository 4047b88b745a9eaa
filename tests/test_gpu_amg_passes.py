"""The algebraic levels' passes (product and vector updates in one kernel) over Chebyshev
degrees and hierarchies with short and long rows: one preconditioner application against the
oracle. Both apply the same operations to the same matrices in another summation order: rounding
of a few hundred operations (1e-13), amplified by the coarsest level's inverse and the estimated
eigenvalues; 1e-9, the bound of the other preconditioner comparisons."""
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


@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("over", [
    {"BOX NX": 13, "BOX NY": 11, "BOX NZ": 12, "PARALMOND AGGREGATION": "SMOOTHED"},
    {"BOX NX": 12, "BOX NY": 9, "BOX NZ": 10, "PARALMOND AGGREGATION": "UNSMOOTHED"},
    {"BOX NX": 9, "BOX NY": 10, "BOX NZ": 11, "PARALMOND AGGREGATION": "SMOOTHED", "BOX BOUNDARY FLAG": -1},
], ids=["smoothed", "unsmoothed", "periodic"])
def test_amg_cycle_matches_oracle(over, degree):
    s = box(**{"POLYNOMIAL DEGREE": 1, "LAMBDA": 1.0, "LINEAR SOLVER": "FPCG", "PRECONDITIONER": "PARALMOND",
               "PARALMOND SMOOTHER": "CHEBYSHEV", "PARALMOND CHEBYSHEV DEGREE": degree, **over})
    e, o = lpg.Elliptic(s), Oracle(s)
    rh = np.random.default_rng(degree).standard_normal(e.Nglobal)
    r = torch.tensor(rh, device="cuda")
    z = torch.zeros_like(r)
    e.precon(r, z)
    torch.cuda.synchronize()
    assert rel_err(z.cpu().numpy(), o.precon(rh)) < 1e-9
