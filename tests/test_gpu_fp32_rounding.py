"""Roundings of the FP32 operator's last sum. On boxes much finer along t than along r and s the
t part is nearly all of the result, and what is added to it after the small parts costs one
rounding at the result's size. The mass term belongs to the small parts, so the error (against
the FP64 operator on the same input, relative 2-norm) does not depend on whether there is one. A
rounding more would raise it by 4 to 8 % (the result is good to about ten such roundings);
half of the least of that is allowed. N >= 3: at N = 2 the products with D's entries (1/2, 3/2, 2)
are nearly all exact, and a small rounding already shows."""
import numpy as np
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


def _error(N, **over):
    e = lpg.Elliptic(box(**{"POLYNOMIAL DEGREE": N, "BOX NX": 10, "BOX NY": 10, "BOX NZ": 24, **over}))
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    q = (torch.rand(e.Nglobal, generator=g, dtype=torch.float64, device="cuda") * 2 - 1).float()
    A32, A64 = torch.empty_like(q), torch.empty(e.Nglobal, dtype=torch.float64, device="cuda")
    e.OperatorF32(q, A32)
    e.Operator(q.double(), A64)
    torch.cuda.synchronize()
    return float((A32.double() - A64).norm() / A64.norm())


@pytest.mark.parametrize("N", range(3, 8))
def test_the_mass_term_adds_no_rounding(N):
    without = _error(N, LAMBDA=0.0)
    for over in ({"LAMBDA": 1.0}, {"LAMBDA FIELD": "LOGNORMAL", "LAMBDA SEED": 4}):
        assert _error(N, **over) <= 1.02 * without
