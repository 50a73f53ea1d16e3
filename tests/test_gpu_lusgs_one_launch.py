"""The one-launch solve of scalar lusolver systems against the oracle, bit for
bit and with the same iteration count, where its work split changes: one row,
a row per CTA, rows with more than the four entries that stand at fixed places,
more rows in a level than the cluster has threads, systems without levels, and
either side of its largest system."""
import numpy as np
import pytest

from oracle import pyoracle as po

LAST = 224 * 1024 // 16 * 16  # most rows of the one-launch solve


def _system(dim, kind, seed):
    rng = np.random.default_rng(seed)
    r, c = [np.arange(dim)], [np.arange(dim)]
    if kind == "two":  # two levels of half the rows each
        lo = np.arange(0, dim // 2)
        r += [lo + dim - dim // 2, lo]
        c += [lo, lo + dim - dim // 2]
    elif kind == "random":  # up to 9 entries on either side, any distance, some repeated
        n = 9 * dim
        r.append(rng.integers(0, dim, n))
        c.append(rng.integers(0, dim, n))
        r[1], c[1] = r[1][r[1] != c[1]], c[1][r[1] != c[1]]
    rows, cols = np.concatenate(r).astype(np.int32), np.concatenate(c).astype(np.int32)
    off = rows != cols
    vals = np.where(off, -rng.uniform(0.1, 1.0, rows.size), 14.0 + rng.uniform(0, 1, rows.size))
    return rows, cols, np.zeros(rows.size, np.int32), vals, rng.uniform(1, 2, dim), \
        rng.uniform(1, 2, dim)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])  # ILUSGS, GS
@pytest.mark.parametrize("dim,kind", [
    (1, "diagonal"), (2, "two"), (17, "random"), (511, "random"), (8193, "two"),
    (3000, "random"), (8192, "diagonal"), (LAST, "two"), (LAST, "random"), (LAST + 1, "random")])
def test_bitwise(dim, kind, mode):
    from mstcfd.lusgs import SparseSystem
    rows, cols, ops, vals, b, x0 = _system(dim, kind, dim + mode)
    xo, ito = po.lu_scalar(mode, dim, rows, cols, ops, vals, b, x0)
    s = SparseSystem(1, dim, rows, cols, ops, vals)
    for _ in range(2):  # a second solve on the same system: the same answer
        x, it = s.solve(b, x0, method=1 if mode == 1 else 0)
        assert np.array_equal(x, xo) and it == ito
