"""GMRES where the one-kernel cycle is not possible: on a stream that has part of the
SMs (a green context's), where its cooperative launch is refused, and for batches whose
CTAs would span more problems than it holds.  The kernels per step take over: same
iteration counts, histories within 1e-12 of the initial residual (both orthogonalise
twice, so each is that close to the exact one; tests/test_gpu_krylov.py).
"""
import numpy as np
import pytest

from hfem_b200.batch import BatchSolver
from hfem_b200.core import HDGSolver
from hfem_b200.gen.problem import ns2d_vortex, ns3d_fourier

pytestmark = pytest.mark.gpu


@pytest.fixture
def part_stream():
    """A stream on 32 of the device's SMs."""
    import torch
    drv = pytest.importorskip("cuda.bindings.driver")
    torch.zeros(1, device="cuda")

    def call(r):
        assert r[0] == drv.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]

    dev = call(drv.cuDeviceGet(0))
    sm = call(drv.cuDeviceGetDevResource(dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, nb, _ = call(drv.cuDevSmResourceSplitByCount(1, sm, 0, 32))
    assert nb == 1 and groups[0].sm.smCount < sm.sm.smCount
    desc = call(drv.cuDevResourceGenerateDesc([groups[0]], 1))
    ctx = call(drv.cuGreenCtxCreate(desc, dev, drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = call(drv.cuGreenCtxStreamCreate(ctx, drv.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield int(stream)
    drv.cuStreamDestroy(stream)
    drv.cuGreenCtxDestroy(ctx)


# block sizes 12 and 15: a cycle in one kernel; 50: a kernel per step
@pytest.mark.parametrize("make,restart,mode", [
    (lambda: ns2d_vortex(n=9, porder=2), 50, 0), (lambda: ns3d_fourier(n=4, porder=1), 7, 0),
    (lambda: ns3d_fourier(n=3, porder=3), 20, 0), (lambda: ns2d_vortex(n=9, porder=2), 50, 2),
], ids=["2d_p2", "3d_p1", "3d_p3", "2d_p2_f32"])
def test_on_part_of_the_sms(part_stream, make, restart, mode):
    prob = make()
    s = HDGSolver(prob)
    try:
        s.set_precision(mode)
        s.getQ()
        s.assembleLinearSystem()
        conv, hist = s.gmres(precond=2, restart=restart, tol=1e-10, maxit=300)
        x = s.download("x")
        s.set_stream(part_stream)
        conv2, hist2 = s.gmres(precond=2, restart=restart, tol=1e-10, maxit=300)
        x2 = s.download("x")
        s.set_stream(0)
        conv3, hist3 = s.gmres(precond=2, restart=restart, tol=1e-10, maxit=300)
    finally:
        s.set_stream(0)                 # the part's stream is destroyed before the context
        s.close()
    assert conv == conv2 == conv3 and len(hist) == len(hist2)
    assert np.max(np.abs(hist - hist2)) <= 1e-12
    assert np.array_equal(hist, hist3)
    assert np.max(np.abs(x - x2)) <= 1e-9 * np.max(np.abs(x))


def test_more_problems_per_cta_than_the_cycle_holds():
    kinds = [ns2d_vortex(n=3, porder=1, seed=k, re=60.0 * (k + 1)) for k in range(3)]
    few, many = BatchSolver(kinds), BatchSolver([kinds[i % 3] for i in range(1401)])
    out = []
    for b in (few, many):
        b.s.getQ()
        b.s.assembleLinearSystem()
        conv, its = b.gmres(restart=20, tol=1e-10, maxit=200)
        out.append((conv, its, b.s.download("x").reshape(b.n, -1)))
        b.close()
    (c0, i0, x0), (c1, i1, x1) = out
    assert np.all(c0 == 1) and np.all(c1 == 1)
    assert np.array_equal(i1, np.tile(i0, 467))
    assert np.max(np.abs(x1 - np.tile(x0, (467, 1)))) <= 1e-9 * np.max(np.abs(x0))
