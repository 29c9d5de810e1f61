"""Element blocks of a residual-only pass, read after what they depend on has
changed: the blocks of that pass's state, bit for bit those read at once (the same
kernel on the same inputs), and after an assembly the assembly's.
"""
import ctypes as C

import numpy as np
import pytest
import torch

from hfem_b200.batched import MixedOrderAssembly
from hfem_b200.core import HDGSolver
from hfem_b200.gen.problem import ns2d_vortex, ns3d_fourier

pytestmark = pytest.mark.gpu

BLOCKS = ("H", "Rh", "K", "Dinv")


def _state(prob, seed):
    rng = np.random.default_rng(seed)
    f = lambda a: a * (1.0 + 0.05 * rng.uniform(-1, 1, size=a.shape))  # noqa: E731
    return f(prob.udg), f(prob.uh), prob.sh


def _set(s, prob):
    s.set_solution(*_state(prob, 2))


def _physics(s, prob):
    s.set_physics(np.asarray(prob.param) * 1.0, prob.tdep, 3.0 * prob.fc_u + 1.0, prob.fc_q, prob.time)


def _precision(s, prob):
    s._chk(s.lib.hfem_set_precision(s.h, 3), "set_precision")


def _update(s, prob):
    s._chk(s.lib.hfem_update(s.h, C.c_double(0.5)), "update")


CHANGES = {"set_solution": _set, "set_physics": _physics, "getq": lambda s, prob: s.getQ(),
           "precision": _precision, "update": _update}


@pytest.mark.parametrize("change", list(CHANGES))
@pytest.mark.parametrize("make", [lambda: ns2d_vortex(n=3, porder=2), lambda: ns3d_fourier(n=3, porder=1)],
                         ids=["2d_p2", "3d_p1"])
def test_blocks_of_the_pass(make, change):
    prob = make()
    s = HDGSolver(prob)
    s.set_solution(*_state(prob, 1))
    s.assembleLinearSystem()
    s._chk(s.lib.hfem_gmres(s.h, 2, 20, C.c_double(1e-3), 20, C.byref(C.c_int()), C.byref(C.c_int()), None, 0), "gmres")
    s.computeResidualNorm()
    ref = {k: s.download(k) for k in BLOCKS}
    s.computeResidualNorm()
    CHANGES[change](s, prob)
    for k in BLOCKS:
        assert np.array_equal(s.download(k), ref[k]), k
    s.close()


@pytest.mark.parametrize("what", ["K", "udg"])
def test_views_see_the_pass(what):
    prob = ns2d_vortex(n=3, porder=2)
    s = HDGSolver(prob)
    s.set_solution(*_state(prob, 1))
    s.assembleLinearSystem()
    ref = HDGSolver(prob)
    ref.set_solution(*_state(prob, 1))
    ref.computeResidualNorm()
    view = s.device_tensor(what)
    s.computeResidualNorm()
    if what == "udg":
        view.mul_(1.5)
        torch.cuda.synchronize()
        assert np.array_equal(s.download("K"), ref.download("K"))
    else:
        assert np.array_equal(view.cpu().numpy(), ref.download("K"))
    ref.close()
    s.close()


def test_graph_launch_after_a_residual():
    prob = ns2d_vortex(n=3, porder=2)
    m = MixedOrderAssembly([prob], tune=False)
    s = m.solvers[0]
    s = getattr(s, "s", s)
    m.launch()
    m.finish()
    ref = {k: s.download(k) for k in BLOCKS}
    s.computeResidualNorm()
    assert not np.array_equal(s.download("H"), ref["H"])
    s.computeResidualNorm()
    m.launch()
    m.stream.synchronize()
    for k in BLOCKS:
        assert np.array_equal(s.download(k), ref[k]), k
    m.close()
