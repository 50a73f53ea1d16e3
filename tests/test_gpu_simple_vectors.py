"""SIMPLE's Gauss-Seidel vectors where their place changes: both momentum
right-hand sides in the cluster's shared memory, only the pressure's, or neither
(200 KB a CTA: 12,800 and 25,600 rows on one CTA), and fewer rows than threads:
the oracle's bits."""
import numpy as np
import pytest

from oracle import pyoracle as po
from test_simple import _channel, _gpu_solver, same


@pytest.mark.gpu
@pytest.mark.parametrize("cluster,nx,ny", [(16, 4, 3), (2, 17, 15), (1, 80, 80), (1, 81, 80),
                                           (1, 128, 100), (1, 129, 100), (2, 129, 100)])
def test_bitwise(tmp_path, cluster, nx, ny):
    from mstcfd import meshgen as mg
    path = str(tmp_path / "chan.msh")
    mg.write_msh(path, _channel(nx, ny, nx))
    m = po.read_msh(path)
    rng = np.random.default_rng(ny)
    n = m.n_cells
    p0 = np.stack([rng.uniform(0.5, 1.5, n), rng.uniform(-0.3, 0.3, n),
                   rng.uniform(-0.3, 0.3, n), rng.uniform(0.8, 1.2, n) / 286.32], 1)
    p0[: n // 2, 1:3] = 0.0  # exact zeros in the residual rows' numerators
    f0 = np.tile(po.q_to_puvt(np.array(po.reference_inlet())[None])[0], (m.n_faces, 1))
    pv, fc, rows, inner, its = po.simple_step(m, p0, f0, 1)
    s, _ = _gpu_solver(path, p0, f0, cluster=cluster)
    grows = s.step(1)
    gpv, gfc = s.state()
    ginner, gits = s.rows()
    assert same(gpv, pv) and same(gfc, fc) and same(grows, rows)
    assert same(ginner, inner) and np.array_equal(gits, its)
