"""A context whose precision changes: its geometry and face buffer come with the
change, and every precision gives the bits of a context created with it."""
import itertools

import numpy as np
import pytest

NAMES = ("PREC_FP64_EXACT", "PREC_FP64", "PREC_FP32")


def _problem(nx, ny):
    from mstcfd import Mesh, meshgen as mg
    m = mg.tri_box(nx, ny, 2.0, 1.0, jitter=0.2, seed=nx)
    mesh = Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                            m["n_cells"])
    rng = np.random.default_rng(ny)
    n = int(m["n_cells"])
    r, p = 1 + 0.2 * rng.random(n), 1 + 0.2 * rng.random(n)
    u, v = 0.5 + 0.1 * rng.standard_normal(n), 0.1 * rng.standard_normal(n)
    return mesh, np.stack([r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v)], 1)


def _solver(mesh, precision, order):
    from mstcfd import Solver, capi
    return Solver(mesh, order=order, reference_quirks=0, time_scheme=capi.TIME_RK2, cfl=0.3,
                  precision=precision, flux=capi.FLUX_ROE, limiter=capi.LIMITER_VANLEER,
                  dt_mode=capi.DT_CFL_GLOBAL)


def _run(s, q):
    s.set_state(q)
    s.step(3)
    out = [s.state()]
    s.set_state(q)
    s.solve()
    return out + [s.new_state(), s.residual(), s.face_flux()]


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(3, 2), (300, 200)])
@pytest.mark.parametrize("first", NAMES)
def test_bits_of_a_fresh_context(nx, ny, first):
    from mstcfd import capi
    mesh, q = _problem(nx, ny)
    want = {}
    for name in NAMES:
        s = _solver(mesh, getattr(capi, name), 2)
        want[name] = _run(s, q)
        s.close()
    for order in itertools.permutations([n for n in NAMES if n != first]):
        s = _solver(mesh, getattr(capi, first), 2)
        for name in (first,) + order + (first,):
            s.set_params(precision=getattr(capi, name))
            for a, b in zip(_run(s, q), want[name]):
                assert np.array_equal(a, b), (name, order)
        s.close()


@pytest.mark.gpu
def test_state_is_carried_over():
    """FP64 to FP32 keeps the 48 bits of a float pair, FP32 to FP64 all of them."""
    from mstcfd import capi
    mesh, q = _problem(37, 11)
    s = _solver(mesh, capi.PREC_FP64, 2)
    s.set_state(q)
    s.set_params(precision=capi.PREC_FP32)
    a = s.state()
    assert np.abs(a - q).max() <= 2.0 ** -46 * np.abs(q).max()
    s.set_params(precision=capi.PREC_FP64_EXACT)
    assert np.array_equal(s.state(), a)
    s.close()
