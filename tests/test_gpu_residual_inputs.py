"""A residual-only pass costs no element pass unless its blocks are asked for: the calls
of a line search driven from outside (state, scalars, q, steps; state views held, as the
server holds them) launch none, and the blocks read after any chain of them are the
pass's, bit for bit those read at once.  Graphs: a launch replaces the blocks, a pass
the caller captured himself cannot be seen, so a context with one forms them at once.
"""
import ctypes as C

import numpy as np
import pytest
import torch

from hfem_b200.batch import BatchSolver
from hfem_b200.batched import MixedOrderAssembly, _lib
from hfem_b200.core import HDGSolver
from hfem_b200.gen.problem import ns2d_channel, ns2d_vortex, ns3d_fourier

pytestmark = pytest.mark.gpu

BLOCKS = ("H", "Rh", "K", "Dinv")
MAKE = {"2d_p1": lambda: ns2d_vortex(n=4, porder=1), "2d_p3_walls": lambda: ns2d_channel(n=3, porder=3),
        "3d_p2": lambda: ns3d_fourier(n=3, porder=2)}


def _state(prob, seed):
    rng = np.random.default_rng(seed)
    f = lambda a: a * (1.0 + 0.05 * rng.uniform(-1, 1, size=a.shape))  # noqa: E731
    return f(prob.udg), f(prob.uh), 0.01 * rng.standard_normal(prob.sh.shape)


def _scalars(s, prob):
    s.set_physics(np.asarray(prob.param) * 1.1, 0, 2.0 * prob.fc_u + 1.0, prob.fc_q, prob.time)


def _device_state(s, prob):
    st = [torch.as_tensor(np.ascontiguousarray(a), device="cuda") for a in _state(prob, 3)]
    s.set_solution_device(*[t.data_ptr() for t in st])
    torch.cuda.synchronize()


STEPS = {
    "update": lambda s, prob: s.updateSol(0.5),
    "solution": lambda s, prob: s.set_solution(*_state(prob, 2)),
    "device": _device_state,
    "scalars": _scalars,
    "getq": lambda s, prob: s.getQ(),
    "precision": lambda s, prob: s.set_precision(3),
    "models": lambda s, prob: s._chk(s.lib.hfem_set_models(s.h, 1, 1), "set_models"),
}
CHAINS = [("update",), ("getq", "solution"), ("scalars", "update", "getq", "device"), ("precision", "models", "solution"),
          ("device", "scalars", "getq", "solution")]


def _element_launches(s):
    return sum(v[1] for k, v in s.kernel_times().items() if k.startswith("element"))


@pytest.mark.parametrize("view", [None, "udg"])
@pytest.mark.parametrize("chain", CHAINS, ids="-".join)
@pytest.mark.parametrize("name", list(MAKE))
def test_no_element_pass_and_the_same_blocks(name, chain, view):
    prob = MAKE[name]()
    s = HDGSolver(prob)
    s.set_solution(*_state(prob, 1))
    s.assembleLinearSystem()
    s.gmres(precond=2, restart=20, tol=1e-3, maxit=20)
    s.computeResidualNorm()
    ref = {k: s.download(k) for k in BLOCKS}
    if view:
        s.device_tensor(view)
    s.set_timing(True)
    s.computeResidualNorm()
    for step in chain:
        STEPS[step](s, prob)
    assert _element_launches(s) == 0
    for k in BLOCKS:
        assert np.array_equal(s.download(k), ref[k]), k
    assert _element_launches(s) == 1
    s.close()


def test_line_searches_launch_no_element_kernel():
    """The batch's and the Newton driver's, with rejected steps and the state handed out."""
    probs = [ns2d_vortex(n=n, porder=2, seed=n) for n in (3, 4)]
    b = BatchSolver(probs)
    b.s.getQ()
    b.s.device_tensor("udg")
    b.s.assembleLinearSystem()
    b.gmres(tol=1e-2)
    b.s.set_timing(True)
    for alpha in (1.0, -0.5, -0.25):
        b.update(np.full(2, alpha))
        b.s.computeResidualNorm()
        b.rnorms()
    assert _element_launches(b.s) == 0
    b.close()
    prob = ns2d_vortex(n=4, porder=2)
    s = HDGSolver(prob)
    s.getQ()
    s.device_tensor("uh")
    s.set_timing(True)
    s.solveNonlinearProblem(newton_tol=1e-8, maxiter=3)
    n = s.kernel_times()
    assert n["residual"][1] > 0 and _element_launches(s) <= 3
    s.close()


def _blocks(s):
    return {k: s.download(k) for k in BLOCKS}


def _same(s, ref):
    for k in BLOCKS:
        assert np.array_equal(s.download(k), ref[k]), k


def test_launches_of_a_graph_replace_the_blocks():
    prob = ns2d_vortex(n=3, porder=2)
    m = MixedOrderAssembly([prob], tune=False)
    s = m.solvers[0].s
    m.launch()
    m.finish()
    ref = _blocks(s)
    s.computeResidualNorm()
    res = _blocks(s)
    assert not np.array_equal(res["H"], ref["H"])
    for _ in range(2):
        s.computeResidualNorm()
        m.launch()
        torch.cuda.synchronize()
        _same(s, ref)
        s.computeResidualNorm()
        _same(s, res)
    m.close()


def test_a_pass_captured_by_the_caller():
    """set_solution_device and assemble_async in the caller's own graph, captured while the
    blocks of a residual pass were still to be formed."""
    prob = ns2d_vortex(n=3, porder=2)
    lib = _lib()
    stream = torch.cuda.Stream()
    new = [torch.as_tensor(np.ascontiguousarray(a), device="cuda") for a in _state(prob, 5)]
    torch.cuda.synchronize()
    r = HDGSolver(prob)
    r.set_solution(*[t.cpu().numpy() for t in new])
    r.assembleLinearSystem()
    ref = _blocks(r)
    r.computeResidualNorm()
    ref_res = _blocks(r)
    r.close()
    s = HDGSolver(prob)
    s.set_stream(stream.cuda_stream)
    s.assembleLinearSystem()
    s.computeResidualNorm()
    res = _blocks(s)
    s.computeResidualNorm()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        s.set_solution_device(*[t.data_ptr() for t in new])
        s._chk(lib.hfem_assemble_async(s.h), "assemble_async")
    _same(s, res)
    g.replay()
    torch.cuda.synchronize()
    _same(s, ref)
    s.computeResidualNorm()
    g.replay()
    torch.cuda.synchronize()
    _same(s, ref)
    s.computeResidualNorm()
    _same(s, ref_res)
    s._chk(lib.hfem_assemble_finish(s.h, C.byref(C.c_double())), "finish")
    s.close()
