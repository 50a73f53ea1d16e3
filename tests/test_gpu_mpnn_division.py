"""The network's division by a cell's degree, seen through the entry points.

Backward: one cell j whose first layer is open, one neighbour c of degree d, and
weights for which the gradient that j takes from c is a chosen FP32 number x per
column (three BF16 weights add up to its 24 bits): the encoder's bias gradient is
then x / d, and has to be the correctly rounded quotient.  Forward: an infinite
value of j reaches the mean of its neighbours, whatever their degrees, as an
infinity.  (The layers' max(y, 0) drops a NaN: an infinity that the division made
one would read as nothing.)"""
import numpy as np
import pytest

from oracle import mpnn_ref as mr

N = 512


def _params(**kw):
    p = {k: np.zeros(s, np.float32) for k, s in
         zip(("We", "be", "W0", "b0", "W1", "b1", "W2", "b2", "Wd", "bd"), mr.SHAPES)}
    for k, v in kw.items():
        p[k][...] = v
    return p


def _flat(p):
    return np.concatenate([v.ravel() for v in p.values()]).astype(np.float32)


def _graph(d):
    """Cell 0 lists cell 1; cell 1 lists d cells, cell 0 among them; the others
    list themselves."""
    lists = [[1], ([0] + list(range(2, d + 1)))[:d]] + [[k] for k in range(2, N)]
    ptr = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.int32)
    return ptr, np.concatenate(lists).astype(np.int32)


def _quotients(net, x, d, scale=1.0):
    """x / d by the network; scale: a power of two that the gradient of cell 1
    carries (x is what the weights hold)."""
    top = lambda v: (v.view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)  # noqa: E731
    hi = top(x)
    mid = top(x - hi)
    lo = x - hi - mid
    assert np.array_equal(top(lo), lo)
    p = _params(b0=1.0)
    p["We"][:, 0] = 2.0 ** -60 if scale == 1.0 else 2.0 ** -126
    for o, part in enumerate((hi, mid, lo)):
        p["W0"][o, mr.W:] = part
        p["Wd"][0, o] = 1.0
    net.set_params(_flat(p))
    feats = np.zeros((N, mr.IN), np.float32)
    feats[0, 0] = 1.0
    ptr, nbr = _graph(d)
    net.set_graph(feats, ptr, nbr)
    y = net.forward()
    assert np.all(y[1] == [3.0, 0, 0, 0]) and np.all(y[0] == [3.0, 0, 0, 0])
    t = y.copy()
    t[1, 0] -= np.float32(2 * N * scale)  # dY = 2 (y - t) / (4 N)
    net.set_targets(t)
    net.backward()
    return mr.unpack(net.grads())[1]


def _numerators(rng, d):
    """Significands: the ends, multiples of d and their neighbours, random ones."""
    k = np.array([2 ** 23, 2 ** 24 - 1, (2 ** 24 - 1) // max(d, 1) * max(d, 1)])
    k = np.concatenate([k, k[2:] - 1, np.minimum(k[2:] + 1, 2 ** 24 - 1)])
    k = np.concatenate([k, rng.integers(2 ** 23, 2 ** 24, mr.W - len(k))])
    k = np.where(k < 2 ** 23, 2 ** 23, k)
    return (k * 2.0 ** -23 * rng.choice([-1, 1], mr.W)).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("block", range(4))
def test_quotient_by_degree_is_correctly_rounded(block):
    from mstcfd.mpnn import Network
    net = Network(seed=1)
    rng = np.random.default_rng(block)
    x = _numerators(rng, 1)
    assert np.array_equal(_quotients(net, x, 1), x)  # the weights do hold x
    for d in list(range(1 + 64 * block, 65 + 64 * block)) + [3, 5, 7, 257, 300, 511][block:]:
        for _ in range(6 if d < 8 else 1):
            x = _numerators(rng, d)
            assert np.array_equal(_quotients(net, x, d), x / np.float32(d)), d
    net.close()


@pytest.mark.gpu
@pytest.mark.parametrize("d", [1, 3, 16, 17, 40, 256, 300])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_infinite_gradient(d, sign):
    from mstcfd.mpnn import Network
    net = Network(seed=1)
    x = np.zeros(mr.W, np.float32)
    x[[5, 77]] = sign * 2.0 ** 96  # times 2^100 in the product: an infinity
    g = _quotients(net, x, d, scale=2.0 ** 100)
    want = np.where(x != 0, sign * np.inf, 0.0)
    assert np.array_equal(g, want)
    net.close()


@pytest.mark.gpu
def test_neighbour_without_neighbours():
    """A listed cell whose own list is empty: x / 0 is infinite."""
    from mstcfd.mpnn import Network
    net = Network(seed=1)
    w = 2.0 ** -20
    net.set_params(_flat(_params(We=w, be=1.0, W0=w, b0=1.0, W1=w, b1=1.0, W2=w, b2=1.0, Wd=w)))
    net.set_graph(np.ones((N, mr.IN), np.float32), *_graph(0))
    t = net.forward()
    t[1] -= 1.0
    net.set_targets(t)
    net.backward()
    assert np.all(mr.unpack(net.grads())[1] == np.inf)
    net.close()


@pytest.mark.gpu
@pytest.mark.parametrize("d", [1, 3, 16, 17, 40, 256, 300])
def test_infinite_value_reaches_the_neighbours_only(d):
    from mstcfd.mpnn import Network
    net = Network(seed=1)
    p = _params()
    p["We"][0, 0] = 2.0 ** 100
    p["W0"][1, mr.W] = 1.0
    p["Wd"][0, 1] = 1.0
    p["bd"][:] = [1, 2, 3, 4]
    net.set_params(_flat(p))
    feats = np.zeros((N, mr.IN), np.float32)
    feats[0, 0] = 2.0 ** 100
    # cells 1 .. 3 list cell 0 among d; cell 4 lists cell 1
    lists = [[]] + [[0] + list(range(5, 4 + d)) for _ in range(3)] + [[1]] + [[]] * (N - 5)
    ptr = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.int32)
    net.set_graph(feats, ptr, np.concatenate(lists).astype(np.int32))
    y = net.forward()
    nan = np.nan
    assert np.array_equal(y[0], [nan] * 4, equal_nan=True)  # inf times zero weights
    assert np.array_equal(y[1:4], [[np.inf, nan, nan, nan]] * 3, equal_nan=True)
    assert np.array_equal(y[4:], [[1.0, 2.0, 3.0, 4.0]] * (N - 4))
    net.close()


@pytest.mark.gpu
def test_lists_before_their_start_are_refused():
    """A list that begins before the array is an error of the call, not a read."""
    from mstcfd import capi
    from mstcfd.mpnn import Network
    net = Network(seed=1)
    feats = np.zeros((3, mr.IN), np.float32)
    with pytest.raises(capi.MstError):
        net.set_graph(feats, [-4, 0, 1, 2], [1, 0])
    net.set_graph(feats, [0, 1, 2, 2], [1, 0])
    assert np.all(np.isfinite(net.forward()))
    net.close()
