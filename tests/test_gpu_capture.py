"""Single counts captured into a CUDA graph and replayed, against the blocking calls and
the oracle (exact).  A lollipop count needs the matrix's plan before the capture (here
from set_shape) and similar_nodes its largest row, but neither a first count."""
import pytest

pytestmark = pytest.mark.gpu


def captured(torch, launch):
    """Replays a captured launch(out pointer, stream) three times; returns the counts."""
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    g, st = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=st):
        launch(out.data_ptr(), st)
    got = []
    for _ in range(3):
        out.fill_(-1)
        g.replay()
        got.append(int(out.item()))
    return got


def small_graph(eh):
    return eh.graph("rmat", 31, scale=13, edges=90000).csr()[:2]


@pytest.mark.parametrize("layout", ["hybrid", "uint", "pshort"])
def test_lollipops_first_counted_in_a_capture(eh, oracle, layout):
    torch = pytest.importorskip("torch")
    off, nbr = small_graph(eh)
    want = oracle.Matrix(off, nbr, oracle.SELECT_ALL, oracle.LAYOUTS[layout]).lollipops()
    m = eh.Matrix.build(off, nbr, selection="all", layout=layout)
    m.set_shape(96, 2048, 4, 4096)
    assert captured(torch, lambda out, st: m.count_lollipops_async(out, stream=st)) == [want] * 3
    assert m.count_lollipops() == want
    assert captured(torch, lambda out, st: m.count_lollipops_async(out, stream=st)) == [want] * 3


@pytest.mark.parametrize("layout", ["hybrid", "uint", "pshort"])
def test_similar_nodes_first_counted_in_a_capture(eh, oracle, layout):
    torch = pytest.importorskip("torch")
    off, nbr = small_graph(eh)
    want = oracle.Matrix(off, nbr, oracle.SELECT_ALL, oracle.LAYOUTS[layout]).similar_nodes(10)
    m = eh.Matrix.build(off, nbr, selection="all", layout=layout)
    m.max_row_id()
    assert captured(torch, lambda out, st: m.similar_nodes_async(10, out, stream=st)) == [want] * 3
    assert m.similar_nodes(10) == want


@pytest.mark.parametrize("k", [0, 3, 4, 5])
def test_triangles_and_cliques_captured_after_a_count(eh, oracle, k):
    torch = pytest.importorskip("torch")
    off, nbr = small_graph(eh)
    o = oracle.Matrix(off, nbr, oracle.SELECT_LOWER, oracle.HYBRID)
    m = eh.Matrix.build(off, nbr, selection="lower", layout="hybrid")
    want = o.cliques(k) if k else o.triangles()
    assert (m.count_cliques(k) if k else m.count_triangles()) == want
    launch = ((lambda out, st: m.count_cliques_async(k, out, stream=st)) if k else
              (lambda out, st: m.count_triangles_async(out, stream=st)))
    assert captured(torch, launch) == [want] * 3
