"""Pivots at the edges of every tier of the count kernels, against the oracle.

The graph has pivots of the sizes where the work changes hands (tiny chunks up
to 8 entries, one warp up to light_max, one CTA up to 512, units above, decoded
lists above 2,048; one- and two-word clique masks) and of rounds of 32, whose
entries reach past the membership windows (8,192 and 65,536 ids) and past the
dense core.  Counts are integers: the tolerance is 0.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 7, 8, 9, 16, 31, 32, 33, 63, 64, 65, 95, 96, 97, 128, 159, 160, 161, 255, 256, 257, 511, 512, 513, 1023,
         1024, 1025, 2047, 2048, 2049, 2500]
N = 72000


@pytest.fixture(scope="module")
def graph():
    rng = np.random.default_rng(5)
    near = rng.integers(0, 600, (2, 30000))              # a dense corner
    mid = np.stack([rng.integers(0, 20000, 150000), rng.integers(0, 3000, 150000)])
    far = np.stack([rng.integers(60000, N - 2 * len(SIZES), 120000), rng.integers(0, 66500, 120000)])
    us, vs = [near[0], mid[0], far[0]], [near[1], mid[1], far[1]]
    for k, c in enumerate(2 * SIZES):
        pivot = N - 1 - k                                # entries near, and near + far up to the pivot itself
        pool = np.arange(700) if k < len(SIZES) and c <= 700 else np.arange(pivot)
        if k >= len(SIZES) and c > 4:                    # neighbours of one far vertex among them
            pool = np.unique(np.concatenate([rng.choice(pool, 2 * c, replace=False), np.arange(66000, 66300),
                                             np.arange(0, 900)]))
        us.append(np.full(c, pivot))
        vs.append(rng.choice(pool, c, replace=False))
    u, v = np.concatenate(us), np.concatenate(vs)
    keep = u != v
    key = np.unique(np.concatenate([u[keep] * N + v[keep], v[keep] * N + u[keep]]))
    off = np.zeros(N + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(key // N, minlength=N))
    return off, (key % N).astype(np.uint32)


@pytest.fixture(scope="module")
def want(graph, oracle):
    low = oracle.Matrix(*graph, oracle.SELECT_LOWER, oracle.UINTEGER)
    full = oracle.Matrix(*graph, oracle.SELECT_ALL, oracle.UINTEGER)
    return dict(tri=low.triangles(), c4=low.cliques(4), c5=low.cliques(5), lol=full.lollipops())


@pytest.mark.parametrize("layout", ["hybrid", "uint", "pshort", "hybrid3"])
@pytest.mark.parametrize("shape", [None, (2, 7, 8, 0), (8, 1000, 1, 64), (64, 65536, 4, 1024), (160, 32, 8, 131072)])
def test_tier_edges(eh, graph, want, layout, shape):
    low = eh.Matrix.build(*graph, "lower", layout)
    full = eh.Matrix.build(*graph, "all", layout)
    if shape:
        low.set_shape(*shape)
        full.set_shape(*shape)
    assert low.count_triangles() == want["tri"]
    assert low.count_cliques(3) == want["tri"]
    assert low.count_cliques(4) == want["c4"]
    assert full.count_lollipops() == want["lol"]
    if shape is None:
        assert low.count_cliques(5) == want["c5"]


@pytest.mark.parametrize("layout", ["hybrid", "uint", "pshort"])
def test_batch_triangles_from_the_clique_masks(eh, oracle, layout):
    """Triangles and 4-cliques of a batch in one pass: complete graphs on both
    sides of the warp tier's 64 entries, and random ones."""
    torch = pytest.importorskip("torch")
    csrs = []
    for n in (2, 3, 4, 5, 32, 33, 34, 64, 65, 66, 67, 100, 600):
        off = np.arange(0, n * (n - 1) + 1, n - 1, dtype=np.uint64)
        nbr = np.concatenate([np.delete(np.arange(n), r) for r in range(n)]).astype(np.uint32)
        csrs.append((off, nbr))
    csrs += [eh.graph("er", 70 + k, n=1500 + 700 * k, edges=12000 * (k + 1)).csr()[:2] for k in range(3)]
    gr, off, nbr = eh.concat_graphs(csrs)
    b = eh.Batch(gr, off, nbr, layout=layout)
    out = torch.full((3, len(csrs)), -1, dtype=torch.int64, device="cuda")
    st = torch.cuda.Stream()
    for use_graph in (True, True, False, True):          # captured, replayed, direct
        out.fill_(-1)
        torch.cuda.synchronize()
        b.run(out[0].data_ptr(), out[1].data_ptr(), use_graph=use_graph, stream=st)
        st.synchronize()
        assert [int(x) for x in out[0][:4]] == [0, 1, 4, 10] and (out[1] >= 0).all()
    b.count(3, out[2].data_ptr(), stream=st)
    st.synchronize()
    lows = [oracle.Matrix(o, x, oracle.SELECT_LOWER, oracle.UINTEGER) for o, x in csrs]
    tri = [m.triangles() for m in lows]
    assert out[0].tolist() == tri and out[2].tolist() == tri
    assert out[1].tolist() == [m.cliques(4) for m in lows]


@pytest.mark.parametrize("layout", ["hybrid", "uint", "pshort"])
@pytest.mark.parametrize("kind", ["symmetric", "one entry missing", "one moved", "self-loop", "long rows below"])
def test_lollipops_by_triangles_only_where_symmetric(eh, oracle, graph, layout, kind):
    """Lollipops of a symmetric matrix without self-loops come from its
    triangles, weighted; anything else keeps the definition.  Both equal the
    oracle, twice in a row and at other shapes."""
    off, nbr = graph
    row = np.repeat(np.arange(N, dtype=np.int64), np.diff(off).astype(np.int64))
    key = row * N + nbr
    if kind == "one entry missing":
        key = np.delete(key, len(key) // 2)
    elif kind == "one moved":                            # as many entries below the diagonal as above
        free = np.setdiff1d(np.arange(1, 400) * N, key)
        key = np.append(np.delete(key, np.flatnonzero(nbr < row)[1234]), free[0])
    elif kind == "self-loop":
        key = np.append(key, 40 * N + 40)
    elif kind == "long rows below":                      # symmetric, but no pivot may hold 2,600 smaller neighbours
        far, some = np.int64(N - 200), np.arange(2600)
        key = np.concatenate([key, far * N + some, some * N + far])
    key = np.unique(key)
    off = np.zeros(N + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(key // N, minlength=N))
    nbr = (key % N).astype(np.uint32)
    m = eh.Matrix.build(off, nbr, "all", layout)
    want = oracle.Matrix(off, nbr, oracle.SELECT_ALL, oracle.UINTEGER).lollipops()
    assert m.count_lollipops() == want and m.count_lollipops() == want
    m.set_shape(8, 64, 8, 0)
    assert m.count_lollipops() == want
    m.set_shape(160, 64, 2, 4096)
    assert m.count_lollipops() == want
