"""FP32 slopes where the limiter's denominator lies beyond 2^126: an upwind
difference of 1e38 (van Leer) or 1.3e19 (van Albada, which squares it) against a
central one of 2e-3 gives the slope of the exact path, to FP32's rounding."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("limiter,far", [(2, 1e38), (3, 1.3e19), (2, 1e10), (3, 1e10)])
def test_2d(limiter, far):
    from mstcfd import Mesh, Solver, meshgen as mg
    m = mg.sod_strip(6, 1, length=6.0, height=1.0)
    mesh = Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                            m["n_cells"])
    x = mesh.arrays()["cell_ctr"][:, 0]
    order = np.argsort(x)
    # supersonic to the right: the face takes its left side's state
    q = np.tile([1.0, 3.0, 0.0, 2.5 + 4.5], (6, 1))
    i, j = order[2], order[3]
    q[order[1], 2], q[i, 2], q[j, 2], q[order[4], 2] = -far, 0.0, 2e-3, far
    face = [k for k, c in enumerate(m["face_cells"]) if set(c) == {i, j}][0]
    out = {}
    for prec in (0, 2):
        s = Solver(mesh, precision=prec, flux=0, order=2, limiter=limiter, reference_quirks=0,
                   dt=1e-5)
        s.set_state(q)
        s.solve()
        out[prec] = s.face_flux()[face, 0, 2]
        s.close()
    assert abs(out[0]) > 2e-3
    assert abs(out[2] - out[0]) <= 20 * np.finfo(np.float32).eps * abs(out[0])
