"""Counts on matrices of bitset and of pshort rows throughout: bitset rows of several
2 KB steps and of a step more or less a word, pshort rows of two partitions past the
dense core, long and short against the pivot.  Against the oracle; counts are
integers: the tolerance is 0.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 70000


@pytest.fixture(scope="module")
def graph():
    rng = np.random.default_rng(21)
    us, vs = [rng.integers(0, 500, 20000), rng.integers(66000, N, 30000)], [rng.integers(0, 500, 20000),
                                                                            rng.integers(0, 68000, 30000)]
    # Pivots whose rows span 127 .. 130 and 255 .. 258 word pairs (128 a step) and the whole range.
    for k, pairs in enumerate([1, 8, 9, 127, 128, 129, 130, 255, 256, 257, 546]):
        last = 128 * pairs - 1 - k
        for c in (2, 6, 40, 170):
            ids = np.unique(np.r_[rng.integers(0, last, c), last, np.arange(0, min(c, 60))])
            us.append(np.full(ids.size, N - 1 - 4 * k - (2, 6, 40, 170).index(c)))
            vs.append(ids[ids < N - 100])
            us[-1] = us[-1][:vs[-1].size]
    u, v = np.concatenate(us), np.concatenate(vs)
    keep = u != v
    key = np.unique(np.concatenate([u[keep] * N + v[keep], v[keep] * N + u[keep]]))
    off = np.zeros(N + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(key // N, minlength=N))
    return off, (key % N).astype(np.uint32)


@pytest.mark.parametrize("core", [0, 256, 32768])
@pytest.mark.parametrize("layout", ["bs", "pshort", "hybrid3"])
def test_long_rows(eh, oracle, graph, layout, core):
    low = eh.Matrix.build(*graph, "lower", layout)
    full = eh.Matrix.build(*graph, "all", layout)
    for m in (low, full):
        m.set_shape(96, 2048, 4, core)
    want = oracle.Matrix(*graph, oracle.SELECT_LOWER, oracle.HYBRID)
    assert low.count_triangles() == want.triangles()
    assert low.count_cliques(4) == want.cliques(4)
    assert full.count_lollipops() == oracle.Matrix(*graph, oracle.SELECT_ALL, oracle.HYBRID).lollipops()
