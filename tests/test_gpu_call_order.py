"""Calls out of order are refused."""
import ctypes as C

import pytest

from hfem_b200.batched import _lib
from hfem_b200.core import HDGSolver, HfemError
from hfem_b200.gen.problem import ns2d_vortex

pytestmark = pytest.mark.gpu


def test_finish_without_an_assembly():
    """A bad call order, whatever the memory of a status record that no pass has written holds."""
    s = HDGSolver(ns2d_vortex(n=3, porder=1))
    assert _lib().hfem_assemble_finish(s.h, C.byref(C.c_double())) == -4
    with pytest.raises(HfemError):
        s.gmres()                       # ... and it did not count as one
    s._chk(_lib().hfem_assemble_async(s.h), "assemble_async")
    rn = C.c_double()
    assert _lib().hfem_assemble_finish(s.h, C.byref(rn)) == 0 and rn.value > 0.0
    s.close()
