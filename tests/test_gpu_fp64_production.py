"""FP64 production path (fused multiply-add, shared reciprocals, one Riemann
solve per face) against the FP64_EXACT path on the same inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _mesh(nx, ny, seed):
    from mstcfd import Mesh
    from mstcfd import meshgen as mg
    m = mg.reorient(mg.tri_box(nx, ny, 4.0, 2.0, jitter=0.2, seed=seed), "random", seed=3)
    return m, Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                               m["n_cells"])


def _state(kind, xy, seed):
    from mstcfd import meshgen as mg
    if kind == "supersonic":  # both signs, |u| above and below the sound speed
        return mg.random_state(len(xy), seed=seed, umax=4.0)
    q = mg.smooth_state(xy, umax=2.5 if kind == "fast" else 0.8)
    if kind == "partly_uniform":  # zero and vanishing differences
        left = xy[:, 0] < 2.0
        q[left] = q[0]
        q[left, 2] = 1e-170 * (1 + xy[left, 1])
    return q


# (random states reconstruct to unphysical ones on some faces; the closed
# form of |A| dQ equals the exact path's R |L| R^-1 dQ only where the Roe
# average has a positive squared sound speed, so Roe takes the smooth ones)
@pytest.mark.parametrize("limiter,viscous", [(0, 0), (1, 0), (2, 0), (3, 0), (1, 1), (3, 1)])
@pytest.mark.parametrize("flux,kind", [(0, "smooth"), (0, "fast"), (0, "supersonic"),
                                       (0, "partly_uniform"), (1, "smooth"), (1, "fast"),
                                       (1, "partly_uniform")])
def test_fp64_residual_matches_exact(flux, limiter, viscous, kind):
    from mstcfd import Solver
    m, mesh = _mesh(13, 7, 5)
    arr = mesh.arrays()
    q = _state(kind, arr["cell_ctr"], 1)
    kw = dict(flux=flux, order=2, limiter=limiter, reference_quirks=0, dt=1e-5, viscous=viscous)
    if viscous:
        kw.update(mu=1e-3, lambda_=-2e-3 / 3, kappa=2e-3, cv=1.7857)
    out = {}
    for prec in (0, 1):
        s = Solver(mesh, precision=prec, **kw)
        s.set_state(q)
        s.solve()
        out[prec] = (s.residual(), s.face_flux())
        s.close()
    # a face's flux is a chain of a few hundred roundings of numbers of the
    # size of the largest flux; a cell adds its faces'
    # (an unlimited reconstruction of the random state may leave the physical
    # range: both paths then give no number on the same faces and cells)
    ok = [np.isfinite(out[0][i]) for i in range(2)]
    for i in range(2):
        assert np.array_equal(np.isfinite(out[1][i]), ok[i])
    F = np.abs(out[0][1][ok[1]]).max()
    S = np.zeros(m["n_cells"])
    for k in range(2):
        on = m["face_cells"][:, k] >= 0
        np.add.at(S, m["face_cells"][on, k], arr["face_area"][on])
    tol = 500 * EPS * F * S[:, None]
    assert np.all((np.abs(out[1][0] - out[0][0]) <= tol)[ok[0]])
    assert np.abs(out[1][1] - out[0][1])[ok[1]].max() <= 500 * EPS * F


@pytest.mark.parametrize("shape", ["tets", "hexes"])
@pytest.mark.parametrize("order,limiter,viscous", [(1, 0, 0), (2, 0, 0), (2, 1, 0), (2, 2, 0),
                                                   (2, 3, 0), (2, 2, 1)])
def test_fp64_residual3d_matches_exact(shape, order, limiter, viscous):
    """3D, with every boundary kind, on a mesh that ends inside a tile; the
    states come back in file order."""
    from mstcfd import meshgen as mg
    from mstcfd.mesh3d import Mesh3D
    from mstcfd.solver3d import Solver3D
    m = mg.tet_box(4, jitter=0.15, seed=2) if shape == "tets" else mg.hex_box(7, jitter=0.1, seed=2)
    rng = np.random.default_rng(4)
    n = int(m["n_cells"])
    rho, vel = rng.uniform(0.9, 1.1, n), rng.uniform(-0.4, 0.4, (n, 3)) + [0.5, 0.0, 0.0]
    p = rng.uniform(0.9, 1.1, n) / 1.4
    q = np.column_stack([rho, rho[:, None] * vel, p / 0.4 + 0.5 * rho * (vel ** 2).sum(1)])
    out = {}
    for prec in (0, 1, 2):
        s = Solver3D(Mesh3D.from_dict(m), precision=prec, order=order, limiter=limiter,
                     viscous=viscous, mu=1e-2, kappa=2e-2, inlet_q=q[0])
        s.set_state(q)
        # (float pairs hold 48 bits of a state)
        assert np.abs(s.state() - q).max() <= (0.0 if prec < 2 else 2.0 ** -46)
        out[prec] = s.residual()
        s.close()
    # as in 2D: a few hundred roundings of the largest face contribution,
    # here the largest residual of a cell times a few
    scale = np.abs(out[0]).max()
    assert np.abs(out[1] - out[0]).max() <= 500 * EPS * 10 * scale
    assert np.abs(out[2] - out[0]).max() <= 500 * np.finfo(np.float32).eps * 10 * scale
