"""Steps whose kernels are placed while the previous one still runs: many steps
in one call give the bits of the same steps called one at a time (each call ends
with the stream idle, so nothing overlaps there).  Sizes from one block to
several waves of them, every precision, both fluxes."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["PREC_FP64_EXACT", "PREC_FP64", "PREC_FP32"])
@pytest.mark.parametrize("flux", ["FLUX_AUSM", "FLUX_ROE"])
@pytest.mark.parametrize("nx,ny,steps", [(3, 2, 40), (37, 11, 40), (160, 90, 20), (700, 400, 4)])
def test_one_call_equals_single_steps(nx, ny, steps, flux, precision):
    from mstcfd import Mesh, Solver, capi, meshgen as mg
    m = mg.tri_box(nx, ny, 2.0, 1.0, jitter=0.2, seed=nx)
    mesh = Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                            m["n_cells"])
    s = Solver(mesh, order=2, reference_quirks=0, time_scheme=capi.TIME_RK2, cfl=0.3,
               precision=getattr(capi, precision), flux=getattr(capi, flux),
               limiter=capi.LIMITER_VANLEER, dt_mode=capi.DT_CFL_GLOBAL)
    rng = np.random.default_rng(ny)
    n = int(m["n_cells"])
    r, p = 1 + 0.2 * rng.random(n), 1 + 0.2 * rng.random(n)
    u, v = 0.5 + 0.1 * rng.standard_normal(n), 0.1 * rng.standard_normal(n)
    q = np.stack([r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v)], 1)
    s.set_state(q)
    for _ in range(steps):
        s.step(1)
    one = s.state()
    assert np.all(np.isfinite(one))
    for _ in range(3):
        s.set_state(q)
        s.step(steps)
        assert np.array_equal(s.state(), one)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["PREC_FP64_EXACT", "PREC_FP64", "PREC_FP32"])
@pytest.mark.parametrize("n,steps", [(2, 30), (7, 20), (24, 6)])
def test_one_call_equals_single_steps_3d(n, steps, precision):
    from mstcfd import capi, meshgen as mg
    from mstcfd.mesh3d import Mesh3D
    from mstcfd.solver3d import Solver3D
    m = mg.tet_box(n)
    s = Solver3D(Mesh3D.from_dict(m), precision=getattr(capi, precision), order=2, limiter=3,
                 cfl=0.3)
    rng = np.random.default_rng(n)
    k = int(m["n_cells"])
    r, p = 1 + 0.1 * rng.random(k), 1 + 0.1 * rng.random(k)
    v = 0.1 * rng.standard_normal((k, 3))
    v[:, 0] += 0.5
    q = np.concatenate([r[:, None], r[:, None] * v,
                        (p / 0.4 + 0.5 * r * (v * v).sum(1))[:, None]], 1)
    s.set_state(q)
    for _ in range(steps):
        s.step(1)
    one = s.state()
    assert np.all(np.isfinite(one))
    for _ in range(3):
        s.set_state(q)
        s.step(steps)
        assert np.array_equal(s.state(), one)
