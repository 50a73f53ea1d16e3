"""The CFL step of first-order FP32 runs follows the state: a Sod tube's steps are
those of the FP64 run, step by step and for jobs from host buffers, with the
smallest step of all cells and with each cell's own.

Tolerances: a step's length is a few roundings of the wave speeds in FP32, and a
state some steps on, of O(1), a few hundred of them."""
import numpy as np
import pytest

EPS = np.finfo(np.float32).eps
STEPS = 30


def _solver(precision, dt_mode, flux):
    from mstcfd import Mesh, Solver, capi, meshgen as mg
    m = mg.sod_strip(200, 2)
    mesh = Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                            m["n_cells"])
    s = Solver(mesh, order=1, reference_quirks=0, time_scheme=capi.TIME_RK2, cfl=0.5,
               precision=getattr(capi, precision), flux=getattr(capi, flux),
               dt_mode=getattr(capi, dt_mode))
    left = mesh.arrays()["cell_ctr"][:, 0] < 0.5
    z = np.zeros(len(left))
    return s, mg.primitive_to_q(np.where(left, 1.0, 0.125), z + 0.3, z, np.where(left, 1.0, 0.1))


@pytest.mark.gpu
@pytest.mark.parametrize("flux", ["FLUX_AUSM", "FLUX_ROE"])
@pytest.mark.parametrize("dt_mode", ["DT_CFL_GLOBAL", "DT_CFL_LOCAL"])
def test_steps_of_the_fp64_run(dt_mode, flux):
    out = {}
    for precision in ("PREC_FP64", "PREC_FP32"):
        s, q = _solver(precision, dt_mode, flux)
        s.set_state(q)
        dts = [s.step(1)["dt"] for _ in range(STEPS)]
        one = s.state()
        s.set_state(0.5 * q)
        s.set_state(q)
        s.step(STEPS)
        assert np.array_equal(s.state(), one)
        out[precision] = (np.array(dts), one)
    a, b = out["PREC_FP64"], out["PREC_FP32"]
    if dt_mode == "DT_CFL_GLOBAL":
        assert a[0].max() > 1.05 * a[0].min()  # the step does change
    assert np.all(np.abs(b[0] - a[0]) <= 50 * EPS * a[0])
    assert np.abs(b[1] - a[1]).max() <= 500 * EPS * np.abs(a[1]).max()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["PREC_FP64", "PREC_FP32"])
def test_host_jobs(precision):
    s, q = _solver(precision, "DT_CFL_GLOBAL", "FLUX_ROE")
    states = [q * [1.0, 1.0, 1.0, 1.0 + 0.4 * k] for k in range(3)]
    want = []
    for x in states:
        s.set_state(x)
        s.step(STEPS)
        want.append(s.state())
    s.set_state(q * [1.0, 1.0, 1.0, 5.0])
    got = [np.zeros_like(q) for _ in states]
    s.step_host_jobs([x.ctypes.data for x in states], [x.ctypes.data for x in got], nsteps=STEPS)
    for x, y in zip(got, want):
        assert np.array_equal(x, y)
