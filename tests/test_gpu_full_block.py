"""Two adjacent rows that share a whole 2^16 block of ids below them: as pshort rows
their partition count wraps to 0 in the reference's uint16_t (intersection.hpp:857-865),
so the block's common neighbours are in no triangle, lollipop or 3-clique of the pair.
The other layouts count them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def hubs_and_block(hubs, first):
    """Symmetric CSR: `hubs` rows adjacent to each other and to 65,536 leaves, with the
    hubs' ids before the leaves' (aligned to a block) or after them."""
    leaf0 = 65536 if first else 0
    ids = np.arange(hubs, dtype=np.uint32) + (0 if first else 65536)
    leaves = np.arange(leaf0, leaf0 + 65536, dtype=np.uint32)
    n = 131072 if first else 65536 + hubs
    deg = np.zeros(n, np.uint64)
    deg[leaves], deg[ids] = hubs, 65536 + hubs - 1
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    nbr = np.zeros(int(off[-1]), np.uint32)
    for h in ids:
        nbr[int(off[h]):int(off[h + 1])] = np.sort(np.concatenate([leaves, ids[ids != h]]))
    at = int(off[leaf0])
    nbr[at:at + 65536 * hubs] = np.tile(ids, 65536)
    return off, nbr


@pytest.mark.parametrize("first", [False, True])
@pytest.mark.parametrize("hubs", [2, 3])
@pytest.mark.parametrize("layout", ["pshort", "hybrid3", "hybrid", "uint"])
def test_shared_full_block(eh, oracle, layout, hubs, first):
    torch = pytest.importorskip("torch")
    off, nbr = hubs_and_block(hubs, first)
    low = eh.Matrix.build(off, nbr, selection="lower", layout=layout)
    olow = oracle.Matrix(off, nbr, oracle.SELECT_LOWER, oracle.LAYOUTS[layout])
    full = eh.Matrix.build(off, nbr, selection="all", layout=layout)
    ofull = oracle.Matrix(off, nbr, oracle.SELECT_ALL, oracle.LAYOUTS[layout])
    assert low.count_triangles() == olow.triangles()
    assert low.count_cliques(3) == olow.cliques(3)
    assert full.count_lollipops() == ofull.lollipops()
    want = np.unique(olow.list_cliques(3).reshape(-1, 3), axis=0)
    d = torch.zeros((len(want) + 1, 3), dtype=torch.int32, device="cuda")
    total = torch.zeros(1, dtype=torch.int64, device="cuda")
    low.list_cliques(3, d.data_ptr(), len(want) + 1, total.data_ptr())
    assert int(total.item()) == len(want)
    assert np.array_equal(np.unique(d[:len(want)].cpu().numpy().view(np.uint32), axis=0), want)


def test_the_wrap_shows_in_the_oracle(oracle):
    off, nbr = hubs_and_block(2, False)
    counts = [oracle.Matrix(off, nbr, oracle.SELECT_LOWER, oracle.LAYOUTS[x]).triangles() for x in ("pshort", "uint")]
    assert counts == [0, 65536]
