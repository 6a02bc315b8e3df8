"""similar_nodes against numpy at the edges of its row classes: rows at and
around 8-lane steps (32, 64), the 256-entry limit, whole-warp steps, rows in
several 2^16 partitions, and thresholds on both sides of exact intersections."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 4, 5, 31, 32, 33, 63, 64, 65, 127, 128, 255, 256, 257, 258, 511, 513, 1025, 3000]


@pytest.fixture(scope="module")
def rows():
    rng = np.random.default_rng(9)
    n = 140001
    star = np.sort(np.concatenate([rng.choice(n, 5000, replace=False), np.arange(70000, 70400)]))
    star = np.unique(star)
    rows = [np.zeros(0, np.int64)] * n
    rows[77] = star
    for k, c in enumerate(SIZES):
        for v, frac in enumerate((0.0, 0.4, 1.0)):       # share of entries taken from the largest row
            a = rng.choice(star, int(c * frac), replace=False)
            b = rng.choice(n, c, replace=False)
            rows[1000 + 3001 * k + v] = np.unique(np.concatenate([a, b[:c - len(a)]]))
    rows[n - 1] = star[::2]
    rows[n - 2] = np.arange(200, 1500)                   # dense: a bitset row in the hybrids
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum([len(r) for r in rows])
    nbr = np.concatenate(rows).astype(np.uint32)
    both = np.bincount(np.repeat(np.arange(n), np.diff(off).astype(np.int64))[np.isin(nbr, star)], minlength=n)
    return off, nbr, both


@pytest.mark.parametrize("layout", ["hybrid", "uint", "bs", "pshort", "hybrid3"])
def test_similar_nodes_row_classes(eh, rows, layout):
    off, nbr, both = rows
    m = eh.Matrix.build(off, nbr, selection="all", layout=layout)
    for t in sorted({0, 1, 3, 4, 10, 30, 100, 255, 256, 4999, 5400, 6000} | set(both[both > 0]) | set(both[both > 0] - 1)):
        assert m.similar_nodes(int(t)) == int((both > t).sum()), t
