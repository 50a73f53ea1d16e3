"""The global step length where its reduction changes: one block, a partial last
block, either side of the 1,024 blocks up to which the gradient's last block
finishes it (blocks of 64 cells in FP64, 256 in FP32).  The fastest cell lies
first, in the middle or last; every call twice, for the ticket's reset.  On
a quadrilateral strip dt = cfl V / (|u| dy + |v| dx + a (dx + dy)).  Tolerances:
a few roundings of the wave speeds in the path's precision, and the node
coordinates' rounding over the cell width."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("PREC_FP64_EXACT", 1e-14), ("PREC_FP64", 1e-14),
                                           ("PREC_FP32", 1e-6)])
@pytest.mark.parametrize("nx,ny", [(2, 1), (65, 1), (1024, 64), (1025, 64), (4096, 64), (4097, 64)])
def test_global_dt(nx, ny, precision, tol):
    from mstcfd import Mesh, Solver, capi, meshgen as mg
    m = mg.sod_strip(nx, ny, length=1.0, height=0.5)
    mesh = Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                            m["n_cells"])
    n, dx, dy = nx * ny, 1.0 / nx, 0.5 / ny
    s = Solver(mesh, order=2, reference_quirks=0, time_scheme=capi.TIME_RK2, cfl=0.5,
               precision=getattr(capi, precision), flux=capi.FLUX_AUSM,
               limiter=capi.LIMITER_VANLEER, dt_mode=capi.DT_CFL_GLOBAL)
    rng = np.random.default_rng(n)
    for at in (0, n // 2, n - 1):
        r, p = 1 + 0.01 * rng.random(n), 1 + 0.01 * rng.random(n)
        u, v = 0.1 * rng.random(n), 0.1 * rng.random(n)
        u[at], p[at] = 0.9, 1.5
        q = np.stack([r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v)], 1)
        a = np.sqrt(1.4 * p / r)
        dt = (0.5 * dx * dy / (abs(u) * dy + abs(v) * dx + a * (dx + dy))).min()
        for _ in range(2):
            s.set_state(q)
            assert abs(s.step(1)["dt"] - dt) <= (tol + 1e-15 * max(nx, ny)) * dt
