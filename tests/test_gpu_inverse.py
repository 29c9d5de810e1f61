"""The element and block inverses through D^-1 and block-Jacobi GMRES.

Every order with a kernel of its own: D^-1 against the oracle's element matrix,
|D X - I| <= 32 n 2^-53 max(|D||X||D||X|), the form of the bound on Gauss-Jordan inverses,
with rows that need pivoting (a rough state) and element counts that leave a CTA's
last warps without a matrix.
"""
import numpy as np
import pytest

from hfem_b200.core import HDGSolver
from hfem_b200.gen.problem import ns2d_vortex, ns3d_fourier
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd,p,n", [(2, 1, 3), (2, 1, 7), (2, 2, 3), (2, 2, 5), (2, 3, 3), (2, 4, 3), (3, 1, 3),
                                    (3, 2, 3), (3, 3, 3)])
def test_dinv(nd, p, n):
    prob = ns2d_vortex(n=n, porder=p) if nd == 2 else ns3d_fourier(n=n, porder=p)
    rng = np.random.default_rng(p)
    u = prob.udg.copy()
    u[:, :prob.ncu] *= 1.0 + 0.2 * rng.uniform(-1, 1, size=u[:, :prob.ncu].shape)
    o = Oracle(prob)
    u = o.getq(u, prob.uh)
    s = HDGSolver(prob)
    s.set_solution(u, prob.uh, prob.sh)
    s.assembleLinearSystem()
    N = prob.n_local
    X = s.download("Dinv").reshape(prob.mesh.ne, N, N).transpose(0, 2, 1)
    for e in range(prob.mesh.ne):
        D = o.element(u, prob.uh, e)["D"].reshape(N, N).T
        bound = 32 * N * 2.0 ** -53 * (np.abs(D) @ np.abs(X[e]) @ np.abs(D) @ np.abs(X[e])).max()
        assert np.abs(D @ X[e] - np.eye(N)).max() <= bound
    s.close()
