"""Pivots of a batch at the edges of its warp kernel, against the oracle: sizes around
32 and 64 entries, entries that share one slot of the pivot's hash table, rows with no
entry, rows too long to stream, bitset and uint rows of one pivot.  Counts are
integers: the tolerance is 0.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 4, 8, 15, 16, 17, 31, 32, 33, 34, 48, 62, 63, 64, 65, 70]


def csr(n, u, v):
    keep = u != v
    key = np.unique(np.concatenate([u[keep] * n + v[keep], v[keep] * n + u[keep]]))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return off, (key % n).astype(np.uint32)


def colliding(rng, n=70000):
    """Pivots whose entries have few slots between them; edges among those entries."""
    slot = ((np.arange(n, dtype=np.uint64) * 0x9e3779b1) & 0xffffffff) >> 22
    u, v = [], []
    for k, c in enumerate(SIZES):
        pool = np.flatnonzero((slot % 512 == k) & (np.arange(n) < n - 100))
        ids = rng.choice(pool, c, replace=False)
        a, b = np.triu_indices(c, 1)
        some = rng.random(a.size) < 0.5
        u += [np.full(c, n - 1 - k), ids[a[some]]]
        v += [ids, ids[b[some]]]
    return csr(n, np.concatenate(u), np.concatenate(v))


def mixed(rng, n=6000):
    """A dense corner, sparse rows, a row of 2,000 entries (4,000) and pivots over all of them."""
    corner, wide = rng.integers(0, 150, (2, 6000)), np.stack([rng.integers(0, 5900, 30000), rng.integers(0, 3000, 30000)])
    u, v = [corner[0], wide[0], np.full(2000, 4000)], [corner[1], wide[1], rng.choice(4000, 2000, replace=False)]
    for k, c in enumerate(3 * SIZES):
        pool = [np.arange(150), np.arange(5900), np.r_[0:100, 3900:4001]][k // len(SIZES)]
        ids = rng.choice(pool, c, replace=False)
        if k >= 2 * len(SIZES):
            ids = np.unique(np.r_[ids[1:], 4000])
        u.append(np.full(ids.size, n - 1 - k))
        v.append(ids)
    return csr(n, np.concatenate(u), np.concatenate(v))


@pytest.mark.parametrize("layout", ["hybrid", "uint", "pshort"])
def test_batch_pivots_of_every_kind(eh, oracle, layout):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(9)
    a, b = np.triu_indices(70, 1)
    csrs = [colliding(rng), mixed(rng), csr(70, a, b), (np.zeros(1, np.uint64), np.zeros(0, np.uint32))]
    batch = eh.Batch(*eh.concat_graphs(csrs), layout=layout)
    out = torch.zeros((3, len(csrs)), dtype=torch.int64, device="cuda")
    stream = torch.cuda.Stream()
    batch.run(out[0].data_ptr(), out[1].data_ptr(), use_graph=True, stream=stream)
    stream.synchronize()
    batch.count(3, out[2].data_ptr())
    torch.cuda.synchronize()
    want = [oracle.Matrix(o, x, oracle.SELECT_LOWER, oracle.HYBRID) for o, x in csrs]
    assert out[0].tolist() == [m.triangles() for m in want]
    assert out[1].tolist() == [m.cliques(4) for m in want]
    assert out[2].tolist() == out[0].tolist()
