"""Choice of the precision per element shape in a mixed-precision batch: every kernel
that differs between the modes is counted, on both sides (no GPU: kernel times given).
"""
import pytest

from hfem_b200.batched import MixedOrderAssembly


class _Solver:
    """Kernel times (ms, launches) of a pass in FP64 and in mixed precision."""

    def __init__(self, fp64, mixed):
        self.times, self.mode = {0: fp64, 1: mixed}, 0

    def set_precision(self, mode):
        self.mode = mode

    def assembleLinearSystem(self):
        return 1.0

    def set_timing(self, on=True):
        pass

    def kernel_times(self):
        return {k: (v, 2) for k, v in self.times[self.mode].items()}


class _Batch:
    def __init__(self, *times):
        self.s = _Solver(*times)


COMMON = {"inverse": 1.0, "scatter": 0.6, "pass_status": 0.0}


@pytest.mark.parametrize("fp64,mixed,pays", [
    # the condensation kernel alone is faster, with its lift and Rh passes it is not
    ({"element": 2.6, "schur_fused": 2.05}, {"element": 2.6, "lift_F": 0.59, "schur_tc": 1.54, "gemv_Rh": 0.15}, False),
    # the 3xTF32 element kernel costs more than the condensation saves
    ({"element": 2.6, "schur_fused": 2.9}, {"element": 3.6, "lift_F": 0.59, "schur_tc": 1.54, "gemv_Rh": 0.15}, False),
    # FP64 by the batched GEMMs, which have those passes too
    ({"element": 2.6, "lift_F": 0.59, "gemm_DinvF": 1.2, "gemm_schur": 2.3, "gemv_Rh": 0.15},
     {"element": 2.7, "lift_F": 0.59, "schur_tc": 1.54, "gemv_Rh": 0.15}, True),
    ({"element": 3.5, "schur_fused": 3.3}, {"element": 3.6, "lift_F": 0.59, "schur_tc": 1.54, "gemv_Rh": 0.15}, True),
])
def test_all_kernels_of_a_mode_count(fp64, mixed, pays):
    assert MixedOrderAssembly._tf32_pays(_Batch({**COMMON, **fp64}, {**COMMON, **mixed})) is pays
