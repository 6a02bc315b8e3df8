"""Counts of one matrix on several streams: the calls share the matrix's work queues, so
they run one after the other, and nothing of one is left for the next.  Exact."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def counted(eh):
    """A graph whose counts last longer than queueing them, with its blocking counts."""
    off, nbr = eh.graph("rmat", 41, scale=17, edges=1 << 21).csr()[:2]
    low = eh.Matrix.build(off, nbr, selection="lower", layout="hybrid")
    full = eh.Matrix.build(off, nbr, selection="all", layout="uint")
    launches = {
        "triangles": lambda out, st: low.count_triangles_async(out, stream=st),
        "cliques4": lambda out, st: low.count_cliques_async(4, out, stream=st),
        "lollipops": lambda out, st: full.count_lollipops_async(out, stream=st),
        "list": lambda out, st: low.list_triangles(0, 0, out, stream=st),
    }
    want = {"triangles": low.count_triangles(), "cliques4": low.count_cliques(4),
            "lollipops": full.count_lollipops(), "list": low.count_triangles()}
    return low, full, launches, want


def blocking(counted):
    low, full = counted[:2]
    return {"triangles": low.count_triangles(), "cliques4": low.count_cliques(4),
            "lollipops": full.count_lollipops(), "list": low.count_triangles()}


@pytest.mark.parametrize("kinds", [["triangles"], ["lollipops"], ["cliques4"], ["list"],
                                   ["triangles", "cliques4", "list"]])
def test_counts_queued_on_several_streams(counted, kinds):
    torch = pytest.importorskip("torch")
    _, _, launches, want = counted
    streams = [torch.cuda.Stream() for _ in range(3)] + [None]
    for rounds in (2, 24):
        out = torch.zeros(rounds, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        for r in range(rounds):
            launches[kinds[r % len(kinds)]](out[r:].data_ptr(), streams[r % len(streams)])
        torch.cuda.synchronize()
        assert out.tolist() == [want[kinds[r % len(kinds)]] for r in range(rounds)]
        assert blocking(counted) == want


def test_counts_on_streams_that_are_destroyed_while_they_run(counted):
    torch = pytest.importorskip("torch")
    _, _, launches, want = counted
    rt = torch.cuda.cudart()
    out = torch.zeros(32, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for r in range(32):  # a later stream may get an earlier one's handle
        st = C.c_void_p()
        assert int(rt.cudaStreamCreate(C.addressof(st))) == 0
        launches["triangles"](out[r:].data_ptr(), st.value)
        assert int(rt.cudaStreamDestroy(st.value)) == 0
    torch.cuda.synchronize()
    assert out.tolist() == [want["triangles"]] * 32
    assert blocking(counted) == want


@pytest.mark.parametrize("kind", ["triangles", "lollipops"])
def test_captured_counts_replayed_beside_direct_ones(counted, kind):
    torch = pytest.importorskip("torch")
    _, _, launches, want = counted
    one, other = torch.cuda.Stream(), torch.cuda.Stream()
    out = torch.zeros(2, dtype=torch.int64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=one):
        launches[kind](out.data_ptr(), one)
    for _ in range(8):
        out.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(one):
            graph.replay()
        launches[kind](out[1:].data_ptr(), other)
        torch.cuda.synchronize()
        assert out.tolist() == [want[kind]] * 2
    assert blocking(counted) == want
