"""FP32 runs in closed boxes keep their mass: no flux of it through walls.

The residuals of the FP32 paths are compensated sums of face fluxes that are
equal and opposite for a face's two cells, and a state is a pair of floats, so
what a step can lose is the pairs' rounding, 2^-46 of the mass per stage at
most, times the stages.  A wall's flux cancels exactly only if the rounded terms
of the mirrored states do; axis-aligned walls mirror without rounding."""
import numpy as np
import pytest

STEPS = 40
TOL = 2 * STEPS * 2.0 ** -46


def _state(n, dim, rng, columns=None):
    """Random moving state; with columns, constant within each (transverse
    velocity zero): faces between equal states must carry no mass either."""
    k = n if columns is None else columns.max() + 1
    r, p = 1 + 0.1 * rng.random(k), 1 + 0.1 * rng.random(k)
    v = 0.1 * rng.standard_normal((k, dim))
    if columns is not None:
        v[:, 1:] = 0.0
    q = np.concatenate([r[:, None], r[:, None] * v,
                        (p / 0.4 + 0.5 * r * (v * v).sum(1))[:, None]], 1)
    return q if columns is None else q[columns]


@pytest.mark.gpu
@pytest.mark.parametrize("flux", ["AUSM", "ROE"])
@pytest.mark.parametrize("by_column", [False, True])
@pytest.mark.parametrize("nx,ny", [(60, 12), (37, 1), (128, 3)])
def test_mass_2d(nx, ny, by_column, flux):
    from mstcfd import Mesh, Solver, capi, meshgen as mg
    m = mg.sod_strip(nx, ny, height=0.2, ends=mg.WALL)
    mesh = Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                            m["n_cells"])
    s = Solver(mesh, order=2, reference_quirks=0, time_scheme=capi.TIME_RK2, cfl=0.4,
               precision=capi.PREC_FP32, flux=getattr(capi, "FLUX_" + flux),
               limiter=capi.LIMITER_MINMOD, dt_mode=capi.DT_CFL_GLOBAL)
    q = _state(nx * ny, 2, np.random.default_rng(nx), np.repeat(np.arange(nx), ny)
               if by_column else None)
    s.set_state(q)
    s.step(STEPS)
    a, b = s.state()[:, 0].sum(), q[:, 0].sum()
    assert abs(a - b) <= TOL * b


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 8])
@pytest.mark.parametrize("limiter", [0, 3])
def test_mass_3d(n, limiter):
    from mstcfd import capi, meshgen as mg
    from mstcfd.mesh3d import Mesh3D
    from mstcfd.solver3d import Solver3D
    m = mg.hex_box(n, kinds=(mg.WALL,) * 6)
    s = Solver3D(Mesh3D.from_dict(m), precision=capi.PREC_FP32, order=2, limiter=limiter, cfl=0.4)
    q = _state(n ** 3, 3, np.random.default_rng(n))
    s.set_state(q)
    s.step(STEPS)
    a, b = s.state()[:, 0].sum(), q[:, 0].sum()
    assert abs(a - b) <= TOL * b
