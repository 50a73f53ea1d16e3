"""3D states in and out, in file order, on either side of the sizes up to which the
host reorders them (512 cells out, 2,048 in): a state comes back as it went in, and
its residual is the same from every precision (FP32 states are always reordered
by the device)."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 7, 8, 9, 12, 13])
def test_state_order(n):
    from mstcfd import meshgen as mg
    from mstcfd.mesh3d import Mesh3D
    from mstcfd.solver3d import Solver3D
    m = mg.hex_box(n, jitter=0.1, seed=n)
    k = int(m["n_cells"])
    mesh = Mesh3D.from_dict(m)
    rng = np.random.default_rng(n)
    rho, p = rng.uniform(0.9, 1.1, (2, k))
    v = rng.uniform(-0.2, 0.2, (k, 3)) + [0.5, 0.0, 0.0]
    q = np.column_stack([rho, rho[:, None] * v, p / 0.4 + 0.5 * rho * (v * v).sum(1)])
    res = {}
    for precision, tol in (("exact", 0.0), ("fp64", 0.0), ("fp32", 2.0 ** -46)):
        s = Solver3D(mesh, precision=precision, order=1, limiter=0, inlet_q=q[0])
        s.set_state(2.0 * q)
        s.set_state(q)
        for _ in range(2):
            assert np.abs(s.state() - q).max() <= tol * np.abs(q).max()
        res[precision] = s.residual()
        s.close()
    # a few hundred roundings of the largest residual's faces
    scale = 10 * np.abs(res["exact"]).max()
    assert np.abs(res["fp64"] - res["exact"]).max() <= 500 * np.finfo(np.float64).eps * scale
    assert np.abs(res["fp32"] - res["exact"]).max() <= 500 * np.finfo(np.float32).eps * scale
