"""The block matvec and the segmented GMRES at the sizes where they can go wrong.

* matvec: every block size (warp-per-row and CTA-per-row kernels), against a
  numpy sum over the downloaded blocks.  Bound: each entry sums ncol products,
  so both sides are within ncol 2^-53 |A||x| of the exact value.
* GMRES histories against the oracle's (modified Gram-Schmidt) within 1e-12 of
  the initial residual: the one-kernel cycle with the basis in shared memory and
  in L2, the kernels per step (restart above its limit, block size 50), vectors
  that are not a multiple of a piece, one piece and many, restarts of 1, below and
  above the 64-column chunks, an iteration limit, and no preconditioner.
"""
import numpy as np
import pytest

from hfem_b200.core import HDGSolver
from hfem_b200.gen.problem import ns2d_vortex, ns3d_fourier
from oracle import Oracle

pytestmark = pytest.mark.gpu

SHAPES = [(2, 1, 5), (2, 2, 4), (2, 3, 3), (2, 4, 3), (3, 1, 3), (3, 2, 3), (3, 3, 3)]


def _problem(nd, p, n):
    return ns2d_vortex(n=n, porder=p) if nd == 2 else ns3d_fourier(n=n, porder=p)


@pytest.mark.parametrize("nd,p,n", SHAPES)
def test_matvec(nd, p, n):
    import torch
    prob = _problem(nd, p, n)
    s = HDGSolver(prob)
    s.getQ()
    s.assembleLinearSystem()
    me, b = prob.mesh, prob.bsz
    Hg = s.download("Hg").reshape(-1, b, b).transpose(0, 2, 1)      # block k: [row, column]
    x = np.random.default_rng(7).standard_normal((me.nf, b))
    y = s.matvec(torch.as_tensor(x.ravel(), device="cuda")).cpu().numpy().reshape(me.nf, b)
    rows = np.repeat(np.arange(me.nf), np.diff(me.rowstart))
    ref, mag = np.zeros((me.nf, b)), np.zeros((me.nf, b))
    np.add.at(ref, rows, np.einsum("krc,kc->kr", Hg, x[me.colidx]))
    np.add.at(mag, rows, np.einsum("krc,kc->kr", np.abs(Hg), np.abs(x[me.colidx])))
    ncol = int(np.diff(me.rowstart).max()) * b
    assert np.all(np.abs(y - ref) <= 2 * (ncol + 2) * 2.0 ** -53 * mag)
    s.close()


@pytest.mark.parametrize("nd,p,n,precond,restart,maxit", [
    (2, 2, 3, 2, 50, 500), (2, 2, 9, 2, 50, 500), (2, 3, 7, 2, 1, 12), (2, 1, 24, 2, 7, 300), (2, 2, 6, -1, 70, 68),
    (2, 2, 20, 2, 80, 500), (2, 2, 6, 2, 120, 500), (2, 2, 42, 2, 50, 500), (2, 4, 5, 2, 3, 300), (3, 1, 4, 2, 50, 500), (3, 2, 3, 2, 20, 300), (3, 3, 3, 2, 50, 300),
])
def test_gmres_history(nd, p, n, precond, restart, maxit):
    prob = _problem(nd, p, n)
    s = HDGSolver(prob)
    s.getQ()
    s.assembleLinearSystem()
    Hg, Rg = s.download("Hg"), s.download("Rg")
    conv, hist = s.gmres(precond=precond, restart=restart, tol=1e-10, maxit=maxit)
    x = s.download("x")
    s.close()
    o = Oracle(prob)
    xr, flag, ref = o.gmres(Hg, Rg, o.bj_inverse(Hg) if precond == 2 else None, restart=restart, tol=1e-10,
                            maxit=maxit)
    assert conv == (1 if flag == 0 else 0) and len(hist) == len(ref)
    assert np.max(np.abs(hist - ref)) <= 1e-12
    assert np.max(np.abs(x - xr)) <= 1e-9 * np.max(np.abs(xr))
