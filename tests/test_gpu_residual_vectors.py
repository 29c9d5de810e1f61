"""What a residual-only pass reports stays what it reported when its element blocks are
formed afterwards: the rows before condensation, the element norms and the problems'
norms, bit for bit, and the pass's Rh is those rows.
"""
import os
import re

import numpy as np
import pytest

from hfem_b200.batch import BatchSolver
from hfem_b200.core import HDGSolver
from hfem_b200.gen.problem import ns2d_channel, ns2d_vortex, ns3d_fourier

CAPI = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hfem_b200", "csrc", "hfem_capi.cu")

PROBLEMS = {"2d_p2": lambda: ns2d_vortex(n=6, porder=2), "2d_p3_walls": lambda: ns2d_channel(n=3, porder=3),
            "3d_p1": lambda: ns3d_fourier(n=3, porder=1)}


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 3])
@pytest.mark.parametrize("name", list(PROBLEMS))
def test_vectors_of_the_pass_survive_forming_its_blocks(name, mode):
    s = HDGSolver(PROBLEMS[name]())
    s.set_precision(mode)
    s.getQ()
    s.computeResidualNorm()
    before = {k: s.download(k) for k in ("Ro", "ru2", "Rr")}
    s.download("K")
    for k, v in before.items():
        assert np.array_equal(s.download(k), v), k
    assert np.array_equal(s.download("Rh"), before["Ro"])
    s.close()


@pytest.mark.gpu
def test_problem_norms_do_not_depend_on_views():
    probs = [ns2d_vortex(n=n, porder=2, seed=n) for n in (3, 5)]
    a, b = BatchSolver(probs), BatchSolver(probs)
    a.s.getQ()
    b.s.getQ()
    a.s.assembleLinearSystem()
    b.s.assembleLinearSystem()
    b.s.device_tensor("K")
    a.s.computeResidualNorm()
    b.s.computeResidualNorm()
    na = a.rnorms()
    assert np.array_equal(na, b.rnorms())
    a.s.download("H")
    assert np.array_equal(na, a.rnorms())
    a.close()
    b.close()


def test_expired_waits_are_read_where_the_blocks_are_formed():
    """Source check: an expired wait of the element kernel launched by form_blocks fails that call."""
    src = re.sub(r"//[^\n]*", "", open(CAPI).read())
    body = src[src.index("int form_blocks("):]
    body = body[:body.index("\n}\n")]
    read = body.index("c->tc_err")
    sync = body.index("cudaStreamSynchronize", read)
    assert body.index("element_v[") < read < sync < body.index("wait_failure(c, err)")
