"""The network's products, aggregations and bias sums at the cell counts where
their work splits change (one cell, either side of a 64-row K tile, of a 128-row
tile and of a half-warp group), with cells that have no neighbours, more than
fit a half warp, and the padding rows of an earlier, larger graph: against the
oracle with the same BF16 rounding points, at the tolerances of a BF16 rounding
that falls the other way (test_mpnn.py)."""
import numpy as np
import pytest

from oracle import mpnn_ref as mr


def _graph(n, seed):
    """Random symmetric adjacency: a third of the cells isolated, cell 0 a hub."""
    rng = np.random.default_rng(seed)
    live = rng.permutation(n)[:max(1, 2 * n // 3)]
    a = rng.choice(live, 2 * n)
    b = rng.choice(live, 2 * n)
    hub = rng.choice(live, min(n, 41), replace=False) if n > 41 else live[:0]
    a, b = np.concatenate([a, np.zeros(len(hub), int)]), np.concatenate([b, hub])
    a, b = a[a != b], b[a != b]
    a, b = np.concatenate([a, b]), np.concatenate([b, a])
    order = np.lexsort((b, a))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.int32)
    feats = rng.standard_normal((n, mr.IN)).astype(np.float32)
    targ = (0.3 * rng.standard_normal((n, mr.OUT))).astype(np.float32)
    return feats, ptr, b[order].astype(np.int32), targ


def _rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-30)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 127, 129, 700, 20000])
def test_forward_backward_match_oracle(n):
    from mstcfd.mpnn import Network
    rng = np.random.default_rng(n)
    p = mr.unpack(mr.init_params(7))
    for i in (1, 3, 5, 7, 9):
        p[i] = 0.1 * rng.standard_normal(p[i].shape)
    w = mr.pack(p).astype(np.float32)
    net = Network(seed=1)
    net.set_params(w)
    for k, m in enumerate((n + 200, n)):  # the larger graph first: its rows stay behind
        feats, ptr, nbr, targ = _graph(m, n + k)
        net.set_graph(feats, ptr, nbr)
        net.set_targets(targ)
        y, loss, g = net.forward(), net.backward(), net.grads()
    ref = mr.Net(w.astype(np.float64), bf16_ops=True)
    yr = ref.forward(feats.astype(np.float64), ptr, nbr)
    lr, gr = ref.backward(yr, targ.astype(np.float64))
    assert _rel(y, yr) < 2e-3
    assert abs(loss - lr) <= 1e-3 * lr
    for i, (a, b) in enumerate(zip(mr.unpack(g), gr)):
        assert _rel(a, b) < 2e-2, i
    net.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [65, 700])
def test_infinite_and_nan_features(n):
    """Values that are not finite spread over the neighbours and no further."""
    from mstcfd.mpnn import Network
    feats, ptr, nbr, _ = _graph(n, 3)
    net = Network(seed=2)
    net.set_graph(feats, ptr, nbr)
    clean = net.forward()
    bad = n - 1
    feats[bad] = np.nan
    net.set_graph(feats, ptr, nbr)
    y = net.forward()
    reach = {bad}
    for _ in range(3):
        reach |= {int(c) for c in range(n) if reach & set(nbr[ptr[c]:ptr[c + 1]].tolist())}
    far = np.array(sorted(set(range(n)) - reach), int)
    assert np.array_equal(y[far], clean[far])
    net.close()
