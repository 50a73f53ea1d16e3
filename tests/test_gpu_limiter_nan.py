"""Slopes next to a state that is not a number: a face whose own states are finite
but one of whose cells has no finite gradient takes that side's slope as zero, on
the production paths as on the exact one."""
import numpy as np
import pytest

from test_gpu_fp64_production import EPS, _mesh, _state


@pytest.mark.gpu
@pytest.mark.parametrize("limiter", [1, 2, 3])
@pytest.mark.parametrize("flux", [0, 1])
@pytest.mark.parametrize("sign", [0.0, -0.0])
def test_nan_cell(flux, limiter, sign):
    from mstcfd import Solver
    m, mesh = _mesh(13, 7, 5)
    arr = mesh.arrays()
    q = _state("smooth", arr["cell_ctr"], 1)
    at = int(np.argmin(np.abs(arr["cell_ctr"] - arr["cell_ctr"].mean(0)).sum(1)))
    q[at] = np.copysign(np.nan, sign)
    out = {}
    for prec in (0, 1, 2):
        s = Solver(mesh, precision=prec, flux=flux, order=2, limiter=limiter, reference_quirks=0,
                   dt=1e-5)
        s.set_state(q)
        s.solve()
        out[prec] = s.residual()
        s.close()
    ok = np.isfinite(out[0])
    assert 0 < (~ok).sum() < 40
    # the flux of a face that took the slope is off by a finite part of it; a
    # residual adds a few hundred roundings of its faces' fluxes
    S = np.zeros(m["n_cells"])
    for k in range(2):
        on = m["face_cells"][:, k] >= 0
        np.add.at(S, m["face_cells"][on, k], arr["face_area"][on])
    scale = np.abs(q[np.isfinite(q[:, 0])]).max() * 4.0
    for prec, eps in ((1, EPS), (2, np.finfo(np.float32).eps)):
        assert np.array_equal(np.isfinite(out[prec]), ok)
        assert np.all((np.abs(out[prec] - out[0]) <= 500 * eps * scale * S[:, None])[ok])
