"""A handle used right after its creation: what it uploads and clears is in place,
so its first results have the bits of its later ones."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["PREC_FP64_EXACT", "PREC_FP64", "PREC_FP32"])
@pytest.mark.parametrize("n", [2, 12])
def test_solver3d(n, precision):
    from mstcfd import capi, meshgen as mg
    from mstcfd.mesh3d import Mesh3D
    from mstcfd.solver3d import Solver3D
    m = mg.tet_box(n)
    mesh = Mesh3D.from_dict(m)
    rng = np.random.default_rng(n)
    k = int(m["n_cells"])
    r, p = 1 + 0.1 * rng.random(k), 1 + 0.1 * rng.random(k)
    v = 0.1 * rng.standard_normal((k, 3))
    q = np.concatenate([r[:, None], r[:, None] * v,
                        (p / 0.4 + 0.5 * r * (v * v).sum(1))[:, None]], 1)
    first = None
    for _ in range(6):
        s = Solver3D(mesh, precision=getattr(capi, precision), order=2, limiter=2, cfl=0.3)
        for _ in range(2):
            s.set_state(q)
            s.step(2)
            first = s.state() if first is None else first
            assert np.array_equal(s.state(), first)
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("block", [1, 4])
@pytest.mark.parametrize("dim", [3, 4000])
def test_sparse_system(dim, block):
    """The host memory of the tables is free for others once the handle exists."""
    from mstcfd.lusgs import SparseSystem
    rng = np.random.default_rng(dim)
    r = np.concatenate([np.arange(dim), rng.integers(0, dim, 4 * dim)]).astype(np.int32)
    c = np.concatenate([np.arange(dim), rng.integers(0, dim, 4 * dim)]).astype(np.int32)
    keep = (r != c) | (np.arange(len(r)) < dim)
    r, c = r[keep], c[keep]
    v = rng.uniform(0.1, 1.0, (len(r), block, block))
    v[r == c] += 40.0 * np.eye(block)
    b, x0 = rng.uniform(1, 2, dim * block), rng.uniform(1, 2, dim * block)
    first = None
    for k in range(8):
        s = SparseSystem(block, dim, r, c, None, v.ravel())
        junk = [np.full(n, -1.0) for n in (dim, 4 * dim, 64 * dim)]
        for _ in range(2):
            x, it = s.solve(b, x0)
            first = (x, it) if first is None else first
            assert np.array_equal(x, first[0]) and it == first[1]
        del junk
        s.close()
    assert np.all(np.isfinite(first[0]))


@pytest.mark.gpu
def test_batch():
    """Flags and lists that a batch sends while it solves -- phases, restarts, the
    cells left after a retirement -- are those of its next iterations."""
    from mstcfd import Mesh, batch, capi
    from mstcfd import meshgen as mg
    m = mg.wedge(6000, 9.0, seed=3)
    mesh = Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                            m["n_cells"])
    n = mesh.n_cells
    q0 = [mg.freestream(mach, n) for mach in (1.9, 2.2, 2.5, 2.8)]
    bad = q0[1].copy()
    bad[n // 2, 0] = np.nan
    cases = [(mesh, batch.case_params(mg.freestream(mach))) for mach in (1.9, 2.2, 2.5, 2.8)]
    first = None
    for _ in range(4):
        b = batch.Batch(cases, implicit=dict(max_iter=60, graph_iters=2, autotune=0, tol=1e-30,
                                             fp32_until=1e-1, fp32_window=10, sweep_fp32=1,
                                             restart_after=30),
                        flux=1, order=2, limiter=1, precision=capi.PREC_FP64)
        for _ in range(2):
            b.set_state([q0[0], bad, q0[2], q0[3]])
            b.set_fallback(q0)
            b.solve()
            out = b.state()
            first = out if first is None else first
            for x, y in zip(out, first):
                assert np.array_equal(x, y, equal_nan=True)
        b.close()


def _channel():
    from mstcfd import Mesh, meshgen as mg
    m = mg.tri_box(40, 30, 2.0, 1.0, jitter=0.2, seed=5, left=mg.INLET, right=mg.OUTLET,
                   bottom=mg.WALL, top=mg.WALL)
    return Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                            m["n_cells"])


@pytest.mark.gpu
def test_simple():
    from mstcfd.psolver import SimpleSolver, reference_initial
    mesh = _channel()
    p0, f0 = reference_initial(mesh, 1.0)
    first = None
    for _ in range(6):
        s = SimpleSolver(mesh, p0, f0)
        for _ in range(2):
            s.set_state(p0, f0)
            out = [s.step(1), *s.state()]
            first = out if first is None else first
            for x, y in zip(out, first):
                assert np.array_equal(x, y, equal_nan=True)
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("quirks", [0, 1])
def test_node_values(quirks):
    from mstcfd import Solver, capi, meshgen as mg
    mesh = _channel()
    q = mg.random_state(mesh.n_cells, seed=2)
    first = None
    for _ in range(6):
        s = Solver(mesh, order=1, reference_quirks=quirks, precision=capi.PREC_FP64)
        s.set_state(q)
        for _ in range(2):
            out = s.node_values()
            first = out if first is None else first
            for x, y in zip(out, first):
                assert np.array_equal(x, y)
        s.close()
