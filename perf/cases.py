"""The calls whose speed this framework is judged by: pattern counts over seeded graphs.

Each case is one call (or, for "oneshot", one build-count-free sequence) that a
program makes through the public entry points.  The graphs are made on the GPU
from the seed alone: R-MAT graphs (a, b, c, d = 0.57, 0.19, 0.19, 0.05) on any
number of vertices, graphs of planted cliques over a uniform background, and
batches of G(n, M) and preferential-attachment graphs, all relabelled by
descending degree as the loaders do.

Listing calls (tuples in no particular order) are not here: two runs of one
call give differently ordered buffers.
"""
import math

import numpy as np
import torch

import simdgraphprocessing_gb300 as eh

DEV = "cuda"
RMAT = (0.57, 0.19, 0.19)


def listed():
    return [
        # A graph of the size of the reference's own test graph (4,039 vertices, 88 K edges), counted by the
        # blocking call: what a small query costs.
        dict(name="triangles_small", kind="triangles", n=4039, edges=88234, layout="hybrid", tuned=False, sync=True),
        # The uint workload: 2^16 vertices, 1 M edges.
        dict(name="triangles_uint_s16", kind="triangles", n=1 << 16, edges=1000000, layout="uint", tuned=False,
             sync=False),
        # A resident graph whose owner ran the tuner before counting.
        dict(name="triangles_tuned_s20", kind="triangles", n=1 << 20, edges=16 << 20, layout="hybrid", tuned=True,
             sync=False),
        # The headline graph (scale 22, edge factor 16), counted as built, without tuning, as the drop-in apps do.
        dict(name="triangles_s22", kind="triangles", n=1 << 22, edges=16 << 22, layout="hybrid", tuned=False,
             sync=False),
        # 4-cliques on a skewed graph: pivots of every size, all tiers.
        dict(name="cliques4_1m", kind="cliques", n=1000003, edges=16000000, k=4, layout="hybrid"),
        # 4-cliques on dense communities: large bitset pivots.
        dict(name="cliques4_planted", kind="planted_cliques", n=1 << 18, edges=1 << 20, cliques=256, lo=64, hi=512,
             k=4, layout="hybrid"),
        # Lollipops on full rows: hub pivots of 10^5 entries.
        dict(name="lollipops_s20", kind="lollipops", n=1 << 20, edges=16 << 20, layout="hybrid"),
        # Rows like the largest one, uint layout (the reference's default for this app).
        dict(name="similar_uint_s21", kind="similar", n=1 << 21, edges=16 << 21, threshold=10, layout="uint"),
        # Out-rows against in-rows of a half-reciprocal directed graph.
        dict(name="symbiosity_s21", kind="symbiosity", n=1 << 21, edges=16 << 21, threshold=0.5, layout="hybrid"),
        # Breadth-first search from the largest row of a directed graph.
        dict(name="bfs_s21", kind="bfs", n=1 << 21, edges=16 << 21, layout="uint"),
        # A batch of graphs of uneven size: triangles and 4-cliques of each, replayed as one CUDA graph.
        dict(name="batch_256", kind="batch", graphs=256, lo=200, hi=50000, layout="hybrid"),
        # A graph met once: pinned host CSR -> build -> count -> free, as the apps' own main() goes.
        dict(name="oneshot_1500k", kind="oneshot", n=1500000, edges=24000000, layout="hybrid"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["triangles", "triangles", "triangles", "cliques", "planted_cliques", "lollipops", "similar",
                       "symbiosity", "bfs", "batch", "oneshot"])
    if kind == "batch":
        return dict(kind=kind, graphs=_log_int(rng, 8, 256), lo=200, hi=_log_int(rng, 2000, 50000),
                    layout=rng.choice(["hybrid", "uint"]))
    if kind == "planted_cliques":
        n = _log_int(rng, 1 << 14, 1 << 18)
        return dict(kind=kind, n=n, edges=4 * n, cliques=max(1, n >> 10), lo=64, hi=rng.choice([128, 300, 512]), k=4,
                    layout=rng.choice(["hybrid", "uint"]))
    if kind == "triangles":
        n = _log_int(rng, 4000, 1 << 22)
        edges = int(n * rng.uniform(8, 16))
        layouts = ["hybrid", "hybrid", "uint", "pshort"] + (["bitset"] if n <= 1 << 16 else [])
        return dict(kind=kind, n=n, edges=edges, layout=rng.choice(layouts), tuned=n <= 1 << 20 and rng.random() < 0.3,
                    sync=rng.random() < 0.3)
    if kind == "cliques":
        k = rng.choice([4, 4, 5])
        n = _log_int(rng, 4000, (1 << 20) if k == 4 else (1 << 15))
        return dict(kind=kind, n=n, edges=int(n * rng.uniform(8, 16)), k=k, layout=rng.choice(["hybrid", "uint", "pshort"]))
    n = _log_int(rng, 1 << 14, (1 << 20) if kind in ("lollipops", "oneshot") else 1 << 21)
    c = dict(kind=kind, n=n, edges=int(n * rng.uniform(8, 16)), layout=rng.choice(["hybrid", "uint", "pshort"]))
    if kind == "similar":
        c["threshold"] = rng.choice([4, 10, 30])
    if kind == "symbiosity":
        c["threshold"] = rng.choice([0.1, 0.5])
    return c


# ---- graphs, from the seed alone ----

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _rmat_pairs(n, edges, g):
    """`edges` R-MAT draws on ceil(log2 n) levels; ids outside [0, n) are folded back into it."""
    a, b, c = RMAT
    u = torch.zeros(edges, dtype=torch.int64, device=DEV)
    v = torch.zeros(edges, dtype=torch.int64, device=DEV)
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(edges, device=DEV, generator=g)
        down = r >= a + b
        u.mul_(2).add_(down)
        v.mul_(2).add_(((r >= a) & (r < a + b)) | (r >= a + b + c))
    return u.remainder_(n), v.remainder_(n)


def _csr(n, src, dst):
    """Sorted, deduplicated CSR of the directed pairs: (offsets i64[n + 1], nbrs i64[m])."""
    keys = torch.unique_consecutive(torch.sort(src * n + dst)[0])
    rows = torch.div(keys, n, rounding_mode="floor")
    offs = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    offs[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return offs, keys - rows * n


def _degree_ordered(n, u, v, group=None):
    """Undirected edges without self-loops or duplicates, relabelled by descending degree (ties by id; within
    its group when given): (lo, hi) with lo < hi."""
    keep = u != v
    u, v = u[keep], v[keep]
    keys = torch.unique_consecutive(torch.sort(torch.minimum(u, v) * n + torch.maximum(u, v))[0])
    u = torch.div(keys, n, rounding_mode="floor")
    v = keys - u * n
    deg = torch.bincount(u, minlength=n) + torch.bincount(v, minlength=n)
    rank = (1 << 32) - 1 - deg
    if group is not None:
        rank = rank + (group << 32)
    order = torch.sort(rank, stable=True)[1]
    new = torch.empty_like(order)
    new[order] = torch.arange(n, device=DEV)
    u, v = new[u], new[v]
    return torch.minimum(u, v), torch.maximum(u, v)


def _undirected(case, seed):
    """(n, lo, hi) of the case's degree-ordered undirected graph."""
    g = _gen(seed)
    n = case["n"]
    if case["kind"] != "planted_cliques":
        u, v = _rmat_pairs(n, case["edges"], g)
        return (n,) + _degree_ordered(n, u, v)
    us = [torch.randint(n, (case["edges"],), device=DEV, generator=g)]
    vs = [torch.randint(n, (case["edges"],), device=DEV, generator=g)]
    span = math.log((case["hi"] + 1) / case["lo"])
    sizes = (case["lo"] * torch.exp(torch.rand(case["cliques"], device=DEV, generator=g) * span)).long().tolist()
    for s in sizes:
        members = torch.randperm(n, device=DEV, generator=g)[:s]
        at = torch.triu_indices(s, s, 1, device=DEV)
        us.append(members[at[0]])
        vs.append(members[at[1]])
    return (n,) + _degree_ordered(n, torch.cat(us), torch.cat(vs))


def _directed(case, seed):
    """(n, src, dst): the half-reciprocal orientation of an undirected graph (symbiosity), or R-MAT draws (bfs)."""
    if case["kind"] == "symbiosity":
        n, lo, hi = _undirected(case, seed)
        r = torch.rand(lo.numel(), device=DEV, generator=_gen(seed + 1))
        fwd, bwd = r < 0.75, (r < 0.5) | (r >= 0.75)
        return n, torch.cat([lo[fwd], hi[bwd]]), torch.cat([hi[fwd], lo[bwd]])
    n = case["n"]
    u, v = _rmat_pairs(n, case["edges"], _gen(seed))
    keep = u != v
    return n, u[keep], v[keep]


def _batch_edges(case, seed):
    """(n, lo, hi, graph boundaries): even graphs G(n, M), odd ones preferential attachment (each new edge's far
    end is an end of an earlier edge), sizes log-uniform, mean degree uniform in 4..64."""
    g = _gen(seed)
    cpu = np.random.RandomState(seed & 0x7FFFFFFF)
    count = case["graphs"]
    sizes = np.exp(cpu.uniform(math.log(case["lo"]), math.log(case["hi"] + 1), count)).astype(np.int64)
    half = np.maximum(1, np.rint(cpu.uniform(4, 64, count) / 2)).astype(np.int64)  # edges per vertex
    bounds = np.concatenate([[0], np.cumsum(sizes)])
    n = int(bounds[-1])
    m = sizes * half
    gid = torch.repeat_interleave(torch.arange(count, device=DEV), torch.from_numpy(m).to(DEV))
    first = torch.from_numpy(np.concatenate([[0], np.cumsum(m)[:-1]])).to(DEV)[gid]
    e = torch.arange(int(m.sum()), device=DEV) - first  # edge index within its graph
    size, per, base = (torch.from_numpy(x).to(DEV)[gid] for x in (sizes, half, bounds[:-1]))
    r1 = torch.rand(e.numel(), device=DEV, generator=g, dtype=torch.float64)
    r2 = torch.rand(e.numel(), device=DEV, generator=g, dtype=torch.float64)
    er = gid % 2 == 0
    src = torch.where(er, (r1 * size).long(), torch.div(e, per, rounding_mode="floor"))
    # Preferential attachment: slot r of 2e + 1 earlier ends; even slots are sources, odd slots copy an edge's far end.
    slot = (r2 * (2 * e + 1)).long()
    ref = slot.clone()
    while True:
        odd = (ref % 2 == 1) & ~er
        if not bool(odd.any()):
            break
        ref = torch.where(odd, slot[first + torch.div(ref, 2, rounding_mode="floor") * odd], ref)
    dst = torch.where(er, (r2 * size).long(), torch.div(torch.div(ref, 2, rounding_mode="floor"), per,
                                                        rounding_mode="floor"))
    group = torch.repeat_interleave(torch.arange(count, device=DEV), torch.from_numpy(sizes).to(DEV))
    lo, hi = _degree_ordered(n, base + src, base + dst, group)
    return n, lo, hi, bounds


def _matrix(n, offs, nbrs, selection, layout):
    o, b = offs.contiguous(), nbrs.to(torch.int32)
    m = eh.Matrix.build_device(n, o.data_ptr(), b.data_ptr(), selection=selection, layout=layout)
    torch.cuda.synchronize()
    return m


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case, out=torch.zeros(1, dtype=torch.int64, device=DEV))
    if kind == "batch":
        n, lo, hi, bounds = _batch_edges(case, seed)
        offs, nbrs = _csr(n, torch.cat([lo, hi]), torch.cat([hi, lo]))
        s["batch"] = eh.Batch(bounds.astype(np.uint64), offs.cpu().numpy().astype(np.uint64),
                              nbrs.to(torch.int32).cpu().numpy().view(np.uint32), layout=case["layout"])
        s["out"] = torch.zeros((2, case["graphs"]), dtype=torch.int64, device=DEV)
        s["stream"] = torch.cuda.Stream()
        return s
    if kind in ("symbiosity", "bfs"):
        n, src, dst = _directed(case, seed)
        s["m"] = _matrix(n, *_csr(n, src, dst), "all", case["layout"])
        if kind == "bfs":
            s["start"] = s["m"].max_row_id()
        else:
            s["cols"] = _matrix(n, *_csr(n, dst, src), "all", case["layout"])
        return s
    n, lo, hi = _undirected(case, seed)
    offs, nbrs = _csr(n, torch.cat([lo, hi]), torch.cat([hi, lo]))
    if kind == "oneshot":
        # torch's pinned tensors, filled from the device, as numpy views for the build call
        s["keep"] = (torch.empty(n + 1, dtype=torch.int64, pin_memory=True),
                     torch.empty(nbrs.numel(), dtype=torch.int32, pin_memory=True))
        s["keep"][0].copy_(offs)
        s["keep"][1].copy_(nbrs.to(torch.int32))
        torch.cuda.synchronize()
        s["offs"], s["nbrs"] = s["keep"][0].numpy().view(np.uint64), s["keep"][1].numpy().view(np.uint32)
        return s
    s["m"] = _matrix(n, offs, nbrs, "all" if kind in ("lollipops", "similar") else "lower", case["layout"])
    if case.get("tuned"):
        s["m"].tune()
    return s


def run(s):
    kind = s["kind"]
    if kind == "triangles" and s["sync"]:
        return s["m"].count_triangles()
    if kind == "triangles":
        s["m"].count_triangles_async(s["out"].data_ptr())
    elif kind in ("cliques", "planted_cliques"):
        s["m"].count_cliques_async(s["k"], s["out"].data_ptr())
    elif kind == "lollipops":
        s["m"].count_lollipops_async(s["out"].data_ptr())
    elif kind == "similar":
        s["m"].similar_nodes_async(s["threshold"], s["out"].data_ptr())
    elif kind == "symbiosity":
        s["m"].symbiosity_async(s["cols"], s["threshold"], s["out"].data_ptr())
    elif kind == "bfs":
        return s["m"].bfs(s["start"])
    elif kind == "batch":
        s["batch"].run(s["out"][0].data_ptr(), s["out"][1].data_ptr(), use_graph=True, stream=s["stream"])
        return [s["out"][0], s["out"][1]]
    else:
        m = eh.Matrix.build(s["offs"], s["nbrs"], selection="lower", layout=s["layout"])
        return m.count_triangles()
    return s["out"]


def work(case):
    """Bytes of the graph's adjacency (4 per selected entry) and row index (16 per row), read once."""
    kind = case["kind"]
    if kind == "batch":
        span = math.log(case["hi"] / case["lo"])
        n = case["graphs"] * (case["hi"] - case["lo"]) / span  # mean of the log-uniform sizes
        return {"bytes": int(4 * 17 * n + 16 * n + 16 * case["graphs"]), "flops": 0}
    n, edges = case["n"], case["edges"]
    if kind == "planted_cliques":
        span = math.log(case["hi"] / case["lo"])
        edges += int(case["cliques"] * (case["hi"] ** 2 - case["lo"] ** 2) / (4 * span))
    entries = {"lollipops": 2, "similar": 2, "symbiosity": 3, "oneshot": 2}.get(kind, 1) * edges
    rows = 2 * n if kind == "symbiosity" else n
    return {"bytes": 4 * entries + 16 * rows + 8, "flops": 0}


# ---- the same numbers from plain torch ----

def _triangles(n, lo, hi):
    """Yields the triangles (i, j, k), i > j > k, a block of pivots at a time."""
    keys = torch.sort(hi * n + lo)[0]
    rows = torch.div(keys, n, rounding_mode="floor")
    nbr = keys - rows * n
    # Entry e of row i is paired with the entries before it.
    start = torch.searchsorted(rows, rows)
    before = torch.arange(keys.numel(), device=DEV) - start
    ends = torch.cumsum(before, 0)
    total = int(ends[-1]) if keys.numel() else 0
    block, at = 1 << 25, 0
    while at < total:
        q = torch.arange(at, min(total, at + block), device=DEV)
        e = torch.searchsorted(ends, q, right=True)
        x = nbr[start[e] + q - (ends[e] - before[e])]
        want = nbr[e] * n + x
        pos = torch.searchsorted(keys, want).clamp_(max=keys.numel() - 1)
        hit = keys[pos] == want
        yield rows[e][hit], nbr[e][hit], x[hit]
        at += block


def exact(case, seed):
    kind = case["kind"]
    if kind in ("cliques", "planted_cliques") or case.get("edges", 0) > 20 << 20 and kind in ("triangles", "lollipops"):
        return None
    as_out = (lambda x: torch.tensor([int(x)], dtype=torch.int64))
    if kind == "batch":
        n, lo, hi, bounds = _batch_edges(case, seed)
        b = torch.from_numpy(bounds).to(DEV)
        tri = torch.zeros(case["graphs"], dtype=torch.int64, device=DEV)
        for i, _, _ in _triangles(n, lo, hi):
            tri += torch.bincount(torch.searchsorted(b, i, right=True) - 1, minlength=case["graphs"])
        return [tri, None]  # 4-cliques have no plain value here
    if kind == "bfs":
        n, src, dst = _directed(case, seed)
        offs, nbrs = _csr(n, src, dst)
        at = torch.zeros(n, dtype=torch.bool, device=DEV)
        at[int(torch.argmax(offs[1:] - offs[:-1]))] = True
        seen, level = at.clone(), 0
        rows = torch.repeat_interleave(torch.arange(n, device=DEV), offs[1:] - offs[:-1])
        while True:
            nxt = torch.zeros_like(seen)
            nxt[nbrs[at[rows]]] = True
            nxt &= ~seen
            if not bool(nxt.any()):
                return level, int(seen.sum())
            seen |= nxt
            at, level = nxt, level + 1
    if kind == "symbiosity":
        n, src, dst = _directed(case, seed)
        out = torch.unique(src * n + dst)
        inn = torch.unique(dst * n + src)
        rows = torch.div(out, n, rounding_mode="floor")
        both = torch.bincount(rows[torch.isin(out, inn, assume_unique=True)], minlength=n)
        total = torch.bincount(rows, minlength=n) + torch.bincount(torch.div(inn, n, rounding_mode="floor"), minlength=n)
        return as_out((both.double() / (total - both).double() > case["threshold"]).sum())
    n, lo, hi = _undirected(case, seed)
    if kind == "similar":
        deg = torch.bincount(lo, minlength=n) + torch.bincount(hi, minlength=n)
        star = int(torch.argmax(deg))
        near = torch.zeros(n, dtype=torch.bool, device=DEV)
        near[hi[lo == star]] = True
        near[lo[hi == star]] = True
        both = torch.bincount(lo[near[hi]], minlength=n) + torch.bincount(hi[near[lo]], minlength=n)
        return as_out((both > case["threshold"]).sum())
    if kind == "lollipops":
        deg = torch.bincount(lo, minlength=n) + torch.bincount(hi, minlength=n)
        return as_out(sum(int(deg[i].sum() + deg[j].sum() + deg[k].sum()) for i, j, k in _triangles(n, lo, hi)))
    count = sum(int(i.numel()) for i, _, _ in _triangles(n, lo, hi))
    return count if kind == "oneshot" or case["sync"] else as_out(count)

