"""The global step length on either side of the 2,048 blocks up to which the
gradient's last block finishes it (blocks of 64 cells in FP64, 256 in FP32)."""
import pytest

import test_gpu_step_length as base


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol,nx", [("PREC_FP64_EXACT", 1e-14, 2048),
                                              ("PREC_FP64_EXACT", 1e-14, 2049),
                                              ("PREC_FP64", 1e-14, 2048), ("PREC_FP64", 1e-14, 2049),
                                              ("PREC_FP32", 1e-6, 8192), ("PREC_FP32", 1e-6, 8193)])
def test_global_dt_at_the_edge(precision, tol, nx):
    base.test_global_dt(nx, 64, precision, tol)
