"""symbiosity against numpy's double quotients: thresholds on, just below and just
above ratios that occur, outside (0, 1), and rows at the edges of the lane (32),
warp (2,048) and CTA classes.  BFS from a hub whose level holds rows of every
class of its expansion.  Exact equality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 6, 7, 31, 32, 33, 64, 65, 96, 127, 255, 256, 257, 1000, 2047, 2048, 2049, 4096, 4097, 9000]
N = 66003


def csr(rows):
    off = np.zeros(N + 1, np.uint64)
    off[1:] = np.cumsum([len(r) for r in rows])
    return off, np.concatenate(rows).astype(np.uint32)


@pytest.fixture(scope="module")
def graph():
    rng = np.random.default_rng(3)
    out = [np.zeros(0, np.int64)] * N
    inn = [np.zeros(0, np.int64)] * N
    i = 0
    for c in SIZES:
        for d in {c, max(1, c // 2), min(40 * c, 20000)}:
            for share in (0.0, 0.34, 0.5, 1.0):
                a = rng.choice(N, c, replace=False)
                b = rng.choice(a, int(min(c, d) * share), replace=False)
                rest = np.setdiff1d(rng.choice(N, min(N, 2 * d + 8), replace=False), a)[:d - len(b)]
                out[5 * i], inn[5 * i] = np.sort(a), np.sort(np.concatenate([b, rest]))
                i += 1
    out[N - 1] = inn[N - 1] = np.arange(100, 3000)       # bitset rows in the hybrids
    both = np.array([len(np.intersect1d(a, b)) if len(a) and len(b) else 0 for a, b in zip(out, inn)])
    return out, inn, both


@pytest.mark.parametrize("layout", ["hybrid", "uint", "pshort"])
def test_symbiosity_thresholds(eh, graph, layout):
    out, inn, both = graph
    rows = eh.Matrix.build(*csr(out), selection="all", layout=layout)
    cols = eh.Matrix.build(*csr(inn), selection="all", layout=layout)
    with np.errstate(invalid="ignore"):
        ratio = both / (np.array([len(a) for a in out]) + [len(b) for b in inn] - both).astype(np.float64)
    seen = np.unique(ratio[ratio > 0])
    ts = {-1.0, 0.0, 1e-12, 2.0 ** -30, 0.25, 1 / 3, 0.5, 0.75, 1.0, 1.5, np.nextafter(1.0, 0), float("nan")}
    ts |= set(seen[::3]) | set(np.nextafter(seen[::3], 0)) | set(np.nextafter(seen[::3], 2))
    for t in ts:
        with np.errstate(invalid="ignore"):
            assert rows.symbiosity(cols, float(t)) == int((ratio > t).sum()), t


@pytest.mark.parametrize("layout", ["hybrid", "uint", "pshort"])
def test_bfs_row_classes(eh, oracle, graph, layout):
    out = [r.copy() for r in graph[0]]
    out[1] = np.flatnonzero([len(r) > 0 for r in out])   # one level over rows of every size
    off, nbr = csr(out)
    m = eh.Matrix.build(off, nbr, selection="all", layout=layout)
    o = oracle.Matrix(off, nbr, oracle.SELECT_ALL, oracle.LAYOUTS[layout])
    for start in (1, 0, 5, N - 1, N - 2):
        for depth in (1, 2, 0xEFFFFFF):
            assert m.bfs(start, depth) == o.n_path(start, depth)
