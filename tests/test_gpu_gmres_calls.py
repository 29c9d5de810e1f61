"""What a GMRES call leaves in the caller's arrays."""
import ctypes as C

import numpy as np
import pytest

from hfem_b200.core import HDGSolver
from hfem_b200.gen.problem import ns2d_vortex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", [0, 2, -1])
@pytest.mark.parametrize("hist_len", [3, 400])
def test_history_past_the_iterations_is_left_alone(precond, hist_len):
    prob = ns2d_vortex(n=3, porder=2)
    s = HDGSolver(prob)
    s.getQ()
    s.assembleLinearSystem()
    conv, its = C.c_int(), C.c_int()
    hist = np.full(hist_len, -7.0)
    s._chk(s.lib.hfem_gmres(s.h, precond, 20, C.c_double(1e-6), 300, C.byref(conv), C.byref(its),
                            hist.ctypes.data_as(C.POINTER(C.c_double)), hist_len), "gmres")
    s.close()
    n = min(its.value, hist_len)
    assert conv.value == 1 and 3 < its.value < 300
    assert np.all(hist[:n] > 0.0) and np.all(hist[n:] == -7.0)
