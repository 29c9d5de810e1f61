"""Element blocks at rough states: random u, q, uhat and source, so that every
column of the flux Jacobian and every gradient term carries its own value.

Tolerance as in the parity tests of smooth states: 1e-12 of the largest entry
for the blocks and for the residuals (whose terms have the blocks' scale).
"""
import numpy as np
import pytest

from hfem_b200.core import HDGSolver
from hfem_b200.gen.problem import as_euler, ns2d_channel, ns2d_vortex, ns3d_box, ns3d_fourier, with_models
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _shapes():
    for p, n in ((1, 7), (2, 4), (3, 3), (4, 3)):
        yield f"2d_p{p}", lambda p=p, n=n: ns2d_vortex(n=n, porder=p)
    for p in (1, 2, 3):
        yield f"3d_p{p}", lambda p=p: ns3d_fourier(n=3, porder=p)
    yield "2d_roe_suth_walls", lambda: with_models(ns2d_channel(n=3, porder=2), 2, 1)
    yield "3d_lf_suth_walls", lambda: with_models(ns3d_box(n=2, porder=2), 1, 1)
    yield "2d_euler", lambda: as_euler(ns2d_vortex(n=4, porder=3))


CASES = list(_shapes())


@pytest.mark.parametrize("make", [c[1] for c in CASES], ids=[c[0] for c in CASES])
def test_rough_state(make):
    prob = make()
    rng = np.random.default_rng(3)
    nd, ncu = prob.nd, prob.ncu
    u = prob.udg.copy()
    u[:, :ncu] *= 1.0 + 0.1 * rng.uniform(-1, 1, size=u[:, :ncu].shape)
    if prob.appname == 1:
        u[:, ncu:] = rng.uniform(-1, 1, size=u[:, ncu:].shape)
    uh = prob.uh * (1.0 + 0.1 * rng.uniform(-1, 1, size=prob.uh.shape))
    sh = prob.sh.copy()
    sh[:, :ncu] += rng.uniform(-1, 1, size=sh[:, :ncu].shape)
    ref = Oracle(prob).assemble(u, uh, sh, elem_blocks=True)
    s = HDGSolver(prob)
    s.set_solution(u, uh, sh)
    rn = s.assembleLinearSystem()
    rel = lambda a, b: np.max(np.abs(a - b)) / np.max(np.abs(b))  # noqa: E731
    assert rel(s.download("H"), ref["eH"]) < 1e-12
    assert rel(s.download("DinvF"), ref["DinvF"]) < 1e-12
    assert rel(s.download("Rr"), ref["Rr"]) < 1e-12
    assert rel(s.download("DinvRu"), ref["DinvRu"]) < 1e-12
    assert abs(rn - ref["rnorm"]) <= 1e-12 * ref["rnorm"]
    s.close()
