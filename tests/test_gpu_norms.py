"""Residual norms and pass outcome reduced on the device.

Norms are sums of n squares: any order is within n 2^-53 relative of the exact
sum, so device and numpy agree within 2 n 2^-53 (halved by the square root).
"""
import ctypes as C

import numpy as np
import pytest

from hfem_b200.batch import BatchSolver
from hfem_b200.core import HDGSolver, HfemError
from hfem_b200.gen.problem import as_euler, ns2d_channel, ns2d_vortex, ns3d_box, ns3d_fourier, with_models
from oracle import Oracle

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("prob", [ns2d_vortex(n=3, porder=1), ns2d_vortex(n=40, porder=2), ns3d_fourier(n=5, porder=1)],
                         ids=["18", "3200", "750"])
def test_residual_norm(prob):
    s = HDGSolver(prob)
    s.getQ()
    for norm in (s.assembleLinearSystem, s.computeResidualNorm, s.computeResidualNorm):
        rn = norm()
        rr, ru2 = s.download("Rr"), s.download("ru2")
        ref = np.sqrt(np.sum(ru2) + np.sum(rr ** 2))
        assert abs(rn - ref) <= (rr.size + ru2.size) * EPS * ref
    s.close()


RESIDUALS = {"2d_p1": lambda: ns2d_vortex(n=5, porder=1), "2d_p2": lambda: ns2d_vortex(n=4, porder=2),
             "2d_p3_walls_roe": lambda: with_models(ns2d_channel(n=3, porder=3), 2, 1),
             "2d_p4_euler": lambda: as_euler(ns2d_vortex(n=3, porder=4)), "3d_p1": lambda: ns3d_fourier(n=3, porder=1),
             "3d_p2_walls_lf": lambda: with_models(ns3d_box(n=2, porder=2), 1, 0),
             "3d_p3": lambda: ns3d_fourier(n=3, porder=3)}


@pytest.mark.parametrize("name", list(RESIDUALS))
def test_residual_only_pass(name):
    """Against the element kernel's residual (1e-13 of its largest entry: the same
    sums of at most a few hundred terms in another order), and the element blocks
    asked for after it against the oracle's (1e-12, as in the parity tests)."""
    prob = RESIDUALS[name]()
    s = HDGSolver(prob)
    s.getQ()
    rn = s.assembleLinearSystem()
    ref = {k: s.download(k) for k in ("Rr", "Ro", "ru2", "Rg", "DinvRu")}
    assert abs(s.computeResidualNorm() - rn) <= 1e-13 * rn
    for k in ("Rr", "Ro", "ru2"):
        assert np.max(np.abs(s.download(k) - ref[k])) <= 1e-13 * np.max(np.abs(ref[k]))
    for k in ("Rg", "DinvRu"):
        assert np.array_equal(s.download(k), ref[k])
    udg, uh = s.get_solution()
    o = Oracle(prob)
    for e in (0, prob.mesh.ne - 1):
        b = o.element(udg, uh, e)
        for k, r in (("Dinv", "D"), ("K", "K"), ("H", "H"), ("Rh", "Rh")):
            got = s.download(k).reshape(prob.mesh.ne, -1)[e]
            assert np.max(np.abs(got - b[r])) <= 1e-12 * max(np.max(np.abs(b[r])), np.max(np.abs(ref["Ro"])))
    s.close()


@pytest.mark.parametrize("nprob,sort", [(1, True), (5, True), (5, False), (40, False)])
def test_problem_norms_of_any_map(nprob, sort):
    probs = [ns2d_vortex(n=n, porder=2, seed=n) for n in (3, 6, 4)]
    b = BatchSolver(probs)
    me = b.union.mesh
    rng = np.random.default_rng(nprob)
    ep, fp = (rng.integers(0, nprob, size=k).astype(np.int32) for k in (me.ne, me.nf))
    if sort:
        ep, fp = np.sort(ep), np.sort(fp)
    ep[ep == 2], fp[fp == 2] = 0, 0                      # a problem with nothing (norm 0)
    if sort:
        ep, fp = np.sort(ep), np.sort(fp)
    params = np.tile(b.params[0], (nprob, 1))
    ip, dp = C.POINTER(C.c_int), C.POINTER(C.c_double)
    b.s._chk(b.lib.hfem_set_problem_map(b.s.h, nprob, ep.ctypes.data_as(ip), fp.ctypes.data_as(ip),
                                        params.ctypes.data_as(dp)), "set_problem_map")
    b.n = nprob
    b.s.getQ()
    b.s.assembleLinearSystem()
    for _ in range(2):
        got = b.rnorms()
        rr, ru2 = b.s.download("Rr").reshape(me.nf, -1), b.s.download("ru2")
        ref = np.sqrt([ru2[ep == p].sum() + (rr[fp == p] ** 2).sum() for p in range(nprob)])
        assert np.all(np.abs(got - ref) <= (rr.size + ru2.size) * EPS * ref)
        b.s.computeResidualNorm()
    b.close()


def test_first_singular_element_is_named():
    prob = ns2d_vortex(n=12, porder=1)
    s = HDGSolver(prob)
    udg = prob.udg.copy()
    udg[[283, 17, 150], 0] = np.nan
    s.set_solution(udg, prob.uh, prob.sh)
    with pytest.raises(HfemError, match="element 17: singular"):
        s.assembleLinearSystem()
    s.set_solution(prob.udg, prob.uh, prob.sh)
    assert np.isfinite(s.assembleLinearSystem())
    s.close()
