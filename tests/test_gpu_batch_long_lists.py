"""A batch whose compacted launches list more tiles than a grid has rows (65,535,
8.4M cells): after a quarter of the cases has retired the others go on as they do
alone."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("order,flux", [(1, 0), (2, 1)])
def test_listed_tiles_beyond_a_grid_dimension(order, flux):
    from mstcfd import Mesh, batch, capi
    from mstcfd import meshgen as mg
    m = mg.tri_box(390, 180, 2.0, 1.0, jitter=0.2, seed=4, left=mg.INLET, right=mg.OUTLET,
                   bottom=mg.WALL, top=mg.OUTLET)
    mesh = Mesh.from_arrays(m["node_xy"], m["face_nodes"], m["face_cells"], m["zones"],
                            m["n_cells"])
    n = int(m["n_cells"])
    j = 65536 * 128 // (3 * n) + 1  # 3 j cases of n cells: past 65,535 tiles of 128
    assert 3 * j * n > 65536 * 128
    inlet = mg.freestream(2.0)
    kw = dict(flux=flux, order=order, limiter=1, precision=capi.PREC_FP64)
    imp = dict(cfl0=20.0, cfl_max=20.0, omega=1.2, tol=1e-30, max_iter=8, graph_iters=2,
               autotune=0, freeze_tol=0.0)
    q0 = mg.freestream(2.0, n)
    bad = q0.copy()
    bad[n // 2, 0] = np.nan
    cp = batch.case_params(inlet)
    one = batch.Batch([(mesh, cp)], implicit=imp, **kw)
    one.set_state([q0])
    r1 = one.solve()
    want, l2 = one.state()[0], one.case_status()["last_l2"][0]
    one.close()
    b = batch.Batch([(mesh, cp)] * (4 * j), implicit=imp, **kw)
    b.set_state([bad if k % 4 == 1 else q0 for k in range(4 * j)])
    r = b.solve()
    st = b.case_status()
    assert r["iterations"] == r1["iterations"] == 8 and r["n_diverged"] == j
    for k, q in enumerate(b.state()):
        if k % 4 == 1:
            assert st["conv_iter"][k] == capi.CASE_DIVERGED
        else:
            assert np.array_equal(q, want) and st["last_l2"][k] == l2, k
    b.close()
