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
