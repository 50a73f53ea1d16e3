"""Chained launches against launches one after another: a context whose launches
are timed one by one starts each after the end of the one before, and its states,
residuals, norms and times have the same bits.  Sizes from one block to several
waves of them; every precision, both fluxes, the step lengths and schemes that
differ in their kernels, and 3D."""
import functools

import numpy as np
import pytest

PRECISIONS = ["PREC_FP64_EXACT", "PREC_FP64", "PREC_FP32"]
VISCOUS = dict(viscous=1, mu=1e-3, lambda_=-2e-3 / 3, kappa=2e-3, cv=1.7857)


@functools.lru_cache(maxsize=None)
def _mesh2d(nx, ny):
    from mstcfd import Mesh, meshgen as mg
    m = mg.tri_box(nx, ny, 2.0, 1.0, jitter=0.2, seed=nx)
    return Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                            m["n_cells"])


@functools.lru_cache(maxsize=None)
def _mesh3d(n):
    from mstcfd import meshgen as mg
    from mstcfd.mesh3d import Mesh3D
    m = mg.tet_box(n)
    return int(m["n_cells"]), Mesh3D.from_dict(m)


def _compare(s, q, steps, kernels, solve):
    out = []
    for on in (True, False, False, False):
        s.profile(on)
        s.set_state(q)
        n = s.step(steps)
        got = [s.state()]
        if solve:
            got += [n["l2_resid"], np.array([n["dt"], n["mass"]])]
            s.solve()
            got += [s.new_state(), s.residual()]
        if on:
            assert kernels <= set(s.profile_stats())
        out.append(got)
    assert all(np.all(np.isfinite(x)) for x in out[0])
    for o in out[1:]:
        for x, y in zip(o, out[0]):
            assert np.array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("flux", ["FLUX_AUSM", "FLUX_ROE"])
@pytest.mark.parametrize("nx,ny,steps", [(3, 2, 30), (37, 11, 30), (160, 90, 20), (700, 400, 4)])
@pytest.mark.parametrize("kw", [
    dict(order=2, dt_mode="DT_CFL_GLOBAL", time_scheme="TIME_RK2"),
    dict(order=2, dt_mode="DT_CFL_LOCAL", time_scheme="TIME_EULER", **VISCOUS),
    dict(order=1, dt_mode="DT_FIXED", time_scheme="TIME_RK2")])
def test_2d(nx, ny, steps, flux, precision, kw):
    from mstcfd import Solver, capi
    mesh = _mesh2d(nx, ny)
    kw = {k: getattr(capi, v) if isinstance(v, str) else v for k, v in kw.items()}
    s = Solver(mesh, reference_quirks=0, cfl=0.3, dt=1e-5, precision=getattr(capi, precision),
               flux=getattr(capi, flux), limiter=capi.LIMITER_VANLEER, **kw)
    rng = np.random.default_rng(ny)
    n = mesh.n_cells
    r, p = 1 + 0.2 * rng.random(n), 1 + 0.2 * rng.random(n)
    u, v = 0.5 + 0.1 * rng.standard_normal(n), 0.1 * rng.standard_normal(n)
    q = np.stack([r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v)], 1)
    kind = "f32" if precision == "PREC_FP32" else "f64"
    _compare(s, q, steps, {"k_flux_update<%s>" % kind}, True)
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("n,steps", [(2, 30), (7, 20), (24, 6)])
@pytest.mark.parametrize("order,viscous", [(1, 0), (2, 0), (2, 1)])
def test_3d(n, steps, precision, order, viscous):
    from mstcfd import capi
    from mstcfd.solver3d import Solver3D
    k, mesh = _mesh3d(n)
    s = Solver3D(mesh, precision=getattr(capi, precision), order=order, limiter=3,
                 cfl=0.3, **(VISCOUS if viscous else {}))
    rng = np.random.default_rng(n)
    r, p = 1 + 0.1 * rng.random(k), 1 + 0.1 * rng.random(k)
    v = 0.1 * rng.standard_normal((k, 3))
    v[:, 0] += 0.5
    q = np.concatenate([r[:, None], r[:, None] * v,
                        (p / 0.4 + 0.5 * r * (v * v).sum(1))[:, None]], 1)
    _compare(s, q, steps, {"k3_flux_update"}, False)
    s.close()
