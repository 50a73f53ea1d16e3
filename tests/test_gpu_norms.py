"""A step's norms where their reduction changes: a partial tile, either side of the
400 tiles of one block, several blocks with a partial last slice; every step twice,
for the ticket's reset.  Against the residual that mst_solve exports.

Tolerances: sums of n terms in FP64 (n eps), FP32 paths form the terms in FP32."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("precision,eps", [("PREC_FP64_EXACT", 2.0 ** -52), ("PREC_FP64", 2.0 ** -52),
                                           ("PREC_FP32", 2.0 ** -23)])
@pytest.mark.parametrize("nx,ny", [(3, 1), (127, 1), (400, 128), (400 * 128 + 1, 1), (1009, 101),
                                   (2048, 100)])
def test_norms(nx, ny, precision, eps):
    from mstcfd import Mesh, Solver, capi, meshgen as mg
    m = mg.sod_strip(nx, ny, length=1.0, height=0.5)
    mesh = Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                            m["n_cells"])
    s = Solver(mesh, order=1, reference_quirks=0, time_scheme=capi.TIME_EULER, dt=1e-9,
               precision=getattr(capi, precision), flux=capi.FLUX_ROE, dt_mode=capi.DT_FIXED)
    vol = mesh.arrays()["cell_vol"][:, None]
    rng = np.random.default_rng(nx)
    n = nx * ny
    for at in (0, n // 2, n - 1):
        r, p = 1 + 0.1 * rng.random(n), 1 + 0.1 * rng.random(n)
        u, v = 0.3 + 0.1 * rng.random(n), 0.1 * rng.random(n)
        p[at] = 3.0
        q = np.stack([r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v)], 1)
        s.set_state(q)
        s.solve()
        rv = s.residual() / vol
        l2 = np.sqrt((rv ** 2).mean(0))
        for _ in range(2):
            s.set_state(q)
            got = s.step(1)
            assert np.all(np.abs(got["l2_resid"] - l2) <= (20 + np.sqrt(n)) * eps * l2)
            mass = (vol[:, 0] * s.state()[:, 0]).sum()
            assert abs(got["mass"] - mass) <= n * 2.0 ** -46 * mass
            # (Time.cpp:72-73: the largest |change| over the old value, from 0)
            change = (np.abs(1e-9 * rv) / q).max(0).clip(min=0)
            big = change > 1e3 * eps
            assert np.all(np.abs(got["linf_change"] - change)[big] <= 1e3 * eps + 1e-2 * change[big])
    s.close()
