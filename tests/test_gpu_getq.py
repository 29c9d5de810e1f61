"""q recovery and assembly with a factor of the q equation other than 1 and a source on
it, against the oracle at the tolerance of the parity tests (1e-12 relative)."""
import numpy as np
import pytest

from hfem_b200.core import HDGSolver
from hfem_b200.gen.problem import ns2d_channel, ns2d_vortex, ns3d_fourier
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fc_q", [0.4, 2.5])
@pytest.mark.parametrize("make", [lambda: ns2d_vortex(n=3, porder=1), lambda: ns2d_channel(n=3, porder=3),
                                  lambda: ns3d_fourier(n=3, porder=2)], ids=["2d_p1", "2d_p3_walls", "3d_p2"])
def test_factor_of_the_q_equation(make, fc_q):
    prob = make()
    prob.fc_q = fc_q
    ncu = prob.master.nd + 2
    prob.sh[:, ncu:, :] = np.random.default_rng(3).standard_normal(prob.sh[:, ncu:, :].shape)
    o = Oracle(prob)
    ref = o.getq(prob.udg, prob.uh)
    s = HDGSolver(prob)
    s.getQ()
    udg, _ = s.get_solution()
    assert np.max(np.abs(udg - ref)) <= 1e-12 * np.max(np.abs(ref))
    a = o.assemble(ref, prob.uh)
    s.set_solution(ref, prob.uh, prob.sh)
    rn = s.assembleLinearSystem()
    for k in ("Hg", "DinvF"):
        assert np.max(np.abs(s.download(k) - a[k])) <= 1e-12 * np.max(np.abs(a[k])), k
    assert abs(rn - a["rnorm"]) <= 1e-12 * a["rnorm"]
    s.close()
