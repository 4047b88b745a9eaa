"""IPDG on mesh files whose boundary faces are not all tagged: a face without a neighbour and
without a positive tag is its own neighbour (q_P = q_M, grad q_P = grad q_M), in every
precision of the operator, as in the oracle."""
import numpy as np
import pytest
import torch

import libparanumal_gb300 as lpg
from gmsh_mesh import write_box
from gpu_helpers import rel_err
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    import __graft_entry__ as g
    g.build()
    torch.cuda.set_device(0)


def _partly_tagged(path):
    """-x untagged (its quadrilaterals left out of the file), +y with tag 0, the rest 1 or 2"""
    write_box(path, 3, 2, 3, rotate_seed=5, jitter=0.15, jitter_seed=3, tags=(77, 1, 2, 0, 1, 2))
    lines = open(path).read().split("\n")
    at = lines.index("$Elements") + 1
    body = [v for v in lines[at + 1:at + 1 + int(lines[at])] if v.split()[1:4] != ["3", "2", "77"]]
    lines[at:at + 1 + int(lines[at])] = [str(len(body))] + body
    open(path, "w").write("\n".join(lines))
    return path


@pytest.mark.parametrize("N", [1, 2, 4, 7, 8])
@pytest.mark.parametrize("lam", [0.0, 0.7])
def test_untagged_faces_match_oracle(tmp_path, N, lam):
    s = {"MESH FILE": _partly_tagged(str(tmp_path / "m.msh")), "POLYNOMIAL DEGREE": N, "LAMBDA": lam,
         "DISCRETIZATION": "IPDG", "LINEAR SOLVER": "PCG", "PRECONDITIONER": "NONE"}
    e, o = lpg.Elliptic(s), Oracle(s)
    q = np.random.default_rng(N).standard_normal(e.Nglobal)
    ref = o.operator(q)
    Aq = torch.zeros(e.Nglobal, dtype=torch.float64, device="cuda")
    qd = torch.tensor(q, device="cuda")
    e.Operator(qd, Aq)
    torch.cuda.synchronize()
    assert rel_err(Aq.cpu().numpy(), ref) < 1e-12   # the bar of the other operator comparisons
    e.OperatorDF64(qd, Aq)
    torch.cuda.synchronize()
    assert rel_err(Aq.cpu().numpy(), ref) < 1e-11
    q32 = q.astype(np.float32)
    A32 = torch.zeros(e.Nglobal, dtype=torch.float32, device="cuda")
    e.OperatorF32(torch.tensor(q32, device="cuda"), A32)
    torch.cuda.synchronize()
    assert rel_err(A32.cpu().numpy(), o.operator(q32.astype(np.float64))) < 1e-5
