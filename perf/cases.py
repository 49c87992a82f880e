"""Workloads of the graph kernels, for timing and for comparing results.

Every case is one call that a program with a resident graph makes through the
public entry points (include/ursa_gpu.h, ursa_b200.batch), over the graph
families of the benchmark's configurations: R-MAT (a/b/c = .57/.19/.19,
self-loops and duplicates dropped) and Poisson out-degrees with uniform
targets, from a thousand nodes to R-MAT-22.  Result buffers are allocated once
and kept, as a program that calls again and again does: device arrays where
the entry point writes device memory, pinned host arrays where it returns
host data.
"""

import ctypes as C
import math

import numpy as np
import torch

from ursa_b200 import PageRankParams, Topology, _lib
from ursa_b200.batch import GraphBatch

A, B, CC = 0.57, 0.19, 0.19  # R-MAT quadrant probabilities
DIRECTIONS = {"out": 0, "in": 1, "both": 2}


def listed():
    return [
        # The smallest analytics call: the 1,000-node graph of average degree
        # 10 that the reference's own leaderboard is quoted on.
        {"name": "pagerank_1k", "op": "pagerank", "graph": "poisson", "n": 1000, "ef": 10, "max_iter": 30},
        # The headline: PageRank to 1e-6 on the resident R-MAT-22.
        {"name": "pagerank_rmat22", "op": "pagerank", "graph": "rmat", "n": 1 << 22, "ef": 16, "max_iter": 100},
        # A new edge table already on the device: CSR build, transpose,
        # PageRank and the end of the topology (an ingested snapshot).
        {"name": "ingest_rmat22", "op": "ingest", "graph": "rmat", "n": 1 << 22, "ef": 16, "max_iter": 100},
        # Interactive traversal of a small graph, along in-edges too: latency
        # and launches, at a size that fits nothing evenly.
        {"name": "bfs_50k", "op": "bfs", "graph": "rmat", "n": 50_021, "ef": 13, "dir": "both"},
        # Single-source traversal of the large graph.
        {"name": "bfs_rmat22", "op": "bfs", "graph": "rmat", "n": 1 << 22, "ef": 16, "dir": "out"},
        # Weak components of the large graph.
        {"name": "components_rmat22", "op": "components", "graph": "rmat", "n": 1 << 22, "ef": 16},
        # Triangle counts: an ordinary graph and a large one with hubs.
        {"name": "triangles_rmat16", "op": "triangles", "graph": "rmat", "n": 1 << 16, "ef": 16},
        {"name": "triangles_rmat20", "op": "triangles", "graph": "rmat", "n": 1 << 20, "ef": 16},
        # Weighted distances on a graph like the weighted benchmark's (an odd
        # node count); the weights are a host column, as the reference's
        # slice is.
        {"name": "dijkstra_1m", "op": "dijkstra", "graph": "poisson", "n": 1_000_003, "ef": 16, "dir": "out"},
        # Centrality: sampled betweenness (four passes of 64 sources), and
        # closeness from every node.
        {"name": "betweenness_poisson20", "op": "betweenness", "graph": "poisson", "n": 1 << 20, "ef": 16, "sources": 256},
        {"name": "closeness_rmat16", "op": "closeness", "graph": "rmat", "n": 1 << 16, "ef": 16},
        # Many small graphs in one launch: PageRank, components and triangles.
        {"name": "batch_1000", "op": "batch", "count": 1000, "max_iter": 30},
    ]


def _between(rng, lo, hi):
    """An integer in [lo, hi], uniform over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["pagerank", "ingest", "bfs", "components", "triangles", "dijkstra", "betweenness", "closeness",
                     "batch"])
    if op == "batch":
        return {"op": op, "count": _between(rng, 50, 1000), "max_iter": rng.choice([10, 30])}
    case = {"op": op, "graph": rng.choice(["rmat", "poisson"]), "ef": rng.randint(4, 20)}
    hi = 1 << 22
    if op == "closeness":
        hi = 1 << 15
    elif op in ("triangles", "dijkstra", "betweenness"):
        hi = 1 << 20
    case["n"] = _between(rng, 1000, hi)
    if hi == 1 << 22:
        case["ef"] = min(case["ef"], 16)
    if op in ("pagerank", "ingest"):
        case["max_iter"] = rng.choice([10, 30, 100])
    elif op in ("bfs", "dijkstra"):
        case["dir"] = rng.choice(["out", "out", "in", "both"])
    elif op == "betweenness":
        case["ef"] = min(case["ef"], 16)
        case["sources"] = min(case["n"], rng.choice([16, 64, 100, 256]))
    elif op == "triangles":
        case["ef"] = min(case["ef"], 16)
    return case


# ------------------------------------------------------------------ inputs


def _rmat_bit(src, dst, r):
    """One more bit of every endpoint from the uniform draws r."""
    lower = r >= A + B  # the row half
    right = ((r >= A) & ~lower) | (r >= A + B + CC)  # the column half
    return src * 2 + lower, dst * 2 + right


def _edges(case, seed):
    """(src, dst) u32 columns on the GPU, in the graph's row order."""
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)
    n, ef = case["n"], case["ef"]
    if case["graph"] == "poisson":
        deg = torch.poisson(torch.full((n,), float(ef), device="cuda"), generator=g).long()
        src = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
        dst = torch.randint(0, n, (src.numel(),), device="cuda", generator=g)
        return src.int(), dst.int()
    bits = max(1, (n - 1).bit_length())
    m = n * ef
    src = torch.zeros(m, dtype=torch.int64, device="cuda")
    dst = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(bits):
        src, dst = _rmat_bit(src, dst, torch.rand(m, device="cuda", generator=g))
    keep = (src != dst) & (src < n) & (dst < n)
    key = torch.unique(src[keep] * n + dst[keep])
    key = key[torch.randperm(key.numel(), device="cuda", generator=g)]
    return (key // n).int(), (key % n).int()


def _batch(case, seed):
    """Small R-MAT graphs of the batch benchmark's sizes: log-normal node
    counts (median 2,000, clipped to 100..50,000), 8..32 draws per node.  Returns (nodes per graph, first node
    per graph, src, dst) on the GPU; the edges of one graph follow the other
    and carry ids of the whole batch."""
    count = case["count"]
    rng = np.random.default_rng(100)  # sizes belong to the case
    n = np.clip(np.rint(2000.0 * np.exp(rng.standard_normal(count))), 100, 50_000).astype(np.int64)
    n = torch.from_numpy(n).cuda()
    ef = torch.from_numpy(rng.integers(8, 33, count)).cuda()
    first = torch.cumsum(n, 0) - n
    g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)
    bits = torch.ceil(torch.log2(n.double())).long()
    graph = torch.repeat_interleave(torch.arange(count, device="cuda"), n * ef)
    src = torch.zeros_like(graph)
    dst = torch.zeros_like(graph)
    ebits = bits[graph]
    for b in range(int(bits.max())):
        s, d = _rmat_bit(src, dst, torch.rand(graph.numel(), device="cuda", generator=g))
        src = torch.where(b < ebits, s, src)
        dst = torch.where(b < ebits, d, dst)
    en = n[graph]
    keep = (src != dst) & (src < en) & (dst < en)
    total = int(n.sum())
    at = first[graph]
    key = torch.unique((src + at)[keep] * total + (dst + at)[keep])
    return n, first, key // total, key % total


def _weights(m, seed):
    """f32 weights in [1, 10) widened to f64, one per edge row (host)."""
    g = torch.Generator().manual_seed(seed * 104729 + 5)
    return (1.0 + 9.0 * torch.rand(m, generator=g)).double()


def _source(src, seed):
    """The source of one of the graph's rows (a node with an out-edge)."""
    return int(src[(seed * 1_000_003 + 12_345) % src.numel()])


def _pinned(n, dtype):
    return torch.empty(n, dtype=dtype).pin_memory()


class _DeviceArray:
    """A library-owned device buffer, as torch.as_tensor takes it."""

    def __init__(self, ptr, n, kind):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (ptr, False), "version": 2}


def _prepare_batch(case, seed):
    n, first, src, dst = _batch(case, seed)
    graph = torch.bucketize(src, first, right=True) - 1
    m = torch.bincount(graph, minlength=case["count"])
    cols = [(x - first[graph]).int().cpu().numpy().view(np.uint32) for x in (src, dst)]
    batch = GraphBatch(n.cpu().numpy(), m.cpu().numpy(), *cols)
    params = PageRankParams(0.85, case["max_iter"], 1e-6)
    total = batch.n_nodes()
    out = [torch.as_tensor(_DeviceArray(p, total, kind), device="cuda")
           for p, kind in zip(batch.device_results(), ("<f8", "<i4", "<i4"))]
    torch.cuda.synchronize()
    return {"op": "batch", "batch": batch, "params": params, "out": out}


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        return _prepare_batch(case, seed)
    n = case["n"]
    src, dst = _edges(case, seed)
    st = {"op": op, "n": n, "seed": seed}
    torch.cuda.synchronize()
    if op == "ingest":
        st.update(src=src, dst=dst)
    else:
        st["topo"] = Topology.build_device(n, src, dst)
    if op in ("pagerank", "ingest"):
        st["params"] = PageRankParams(0.85, case["max_iter"], 1e-6)
        st["out"] = torch.empty(n, dtype=torch.float64, device="cuda")
    elif op == "bfs":
        st.update(source=_source(src, seed), dir=DIRECTIONS[case["dir"]], out=_pinned(n, torch.int32))
    elif op in ("components", "triangles"):
        st["out"] = _pinned(n, torch.int32)
    elif op == "dijkstra":
        st.update(source=_source(src, seed), dir=DIRECTIONS[case["dir"]], out=_pinned(n, torch.float64),
                  weights=_weights(src.numel(), seed).pin_memory())
    elif op == "betweenness":
        st.update(sample=case["sources"] / n, out=_pinned(n, torch.float64))
    else:
        st["out"] = torch.empty(n, dtype=torch.float64, device="cuda")
    if op == "triangles":
        st["topo"].prepare(transpose=True, undirected=True)
    torch.cuda.synchronize()
    return st


def run(st):
    L, op, out = _lib.load(), st["op"], st["out"]
    if op == "ingest":
        topo = Topology.build_device(st["n"], st["src"], st["dst"])
        _lib.check(L.ursa_gpu_pagerank_device(topo.handle, C.byref(st["params"]), out.data_ptr(), None, None))
        topo.free()
        return out
    if op == "batch":
        st["batch"].run(st["params"])
        return out
    h = st["topo"].handle
    if op == "pagerank":
        _lib.check(L.ursa_gpu_pagerank_device(h, C.byref(st["params"]), out.data_ptr(), None, None))
    elif op == "bfs":
        _lib.check(L.ursa_gpu_bfs_distances(h, st["source"], st["dir"], out.data_ptr()))
    elif op == "components":
        _lib.check(L.ursa_gpu_connected_components_weak(h, out.data_ptr()))
    elif op == "triangles":
        _lib.check(L.ursa_gpu_triangle_count(h, out.data_ptr()))
    elif op == "dijkstra":
        w = st["weights"]
        _lib.check(L.ursa_gpu_dijkstra_distances(h, w.data_ptr(), w.numel(), st["source"], st["dir"], out.data_ptr()))
    elif op == "betweenness":
        _lib.check(L.ursa_gpu_betweenness(h, 1, st["sample"], 1, st["seed"], out.data_ptr()))
    else:
        _lib.check(L.ursa_gpu_closeness_device(h, out.data_ptr(), None, None))
    return out


def work(case):
    """Compulsory bytes of one pass (the graph once in u32 CSR form, the
    result once) and its arithmetic; m is the expected edge count."""
    op = case["op"]
    if op == "batch":  # about 3,200 nodes and 48,000 edges a graph
        n, m = 3200.0 * case["count"], 48_000.0 * case["count"]
        return {"bytes": 4.0 * m + 8.0 * n + 16.0 * n, "flops": 2.0 * m * 10}
    n = case["n"]
    m = n * case["ef"] * (0.97 if case["graph"] == "rmat" else 1.0)
    csr = 4.0 * m + 4.0 * (n + 1)
    if op == "pagerank":
        return {"bytes": csr + 4.0 * n + 8.0 * n, "flops": 2.0 * m * min(case["max_iter"], 15)}
    if op == "ingest":  # the edge table in, both CSRs (targets and edge rows) and the ranks out
        return {"bytes": 8.0 * m + 16.0 * m + 8.0 * (n + 1) + 8.0 * n, "flops": 2.0 * m * min(case["max_iter"], 15)}
    if op in ("bfs", "dijkstra"):
        both = 2.0 if case["dir"] == "both" else 1.0
        per = 12.0 if op == "dijkstra" else 4.0
        return {"bytes": per * m * both + 4.0 * (n + 1) * both + (8.0 if op == "dijkstra" else 4.0) * n,
                "flops": m * both if op == "dijkstra" else 0.0}
    if op == "components":
        return {"bytes": csr + 4.0 * n, "flops": 0.0}
    if op == "triangles":  # the undirected CSR
        return {"bytes": 8.0 * m + 4.0 * (n + 1) + 4.0 * n, "flops": 0.0}
    if op == "betweenness":
        k = case["sources"]
        return {"bytes": csr + 8.0 * n, "flops": 4.0 * m * k}
    return {"bytes": csr + 8.0 * n, "flops": 0.0}


# ------------------------------------------- the same results in 64 bits


def _exact_pagerank(case, src, dst):
    n, d = case["n"], 0.85
    deg = torch.bincount(src, minlength=n).double()
    dst_sorted, order = torch.sort(dst)
    src_sorted = src[order]
    lens = torch.bincount(dst_sorted, minlength=n)
    rank = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    div = torch.where(deg > 0, deg, torch.ones_like(deg))
    for _ in range(case["max_iter"]):
        base = (1.0 - d) / n + d * float(rank[deg == 0].sum()) / n
        share = (rank / div)[src_sorted]
        nxt = base + d * torch.segment_reduce(share, "sum", lengths=lens, unsafe=True)
        delta = float((nxt - rank).abs().sum())
        rank = nxt
        if delta < 1e-6:
            break
    return rank


def _oriented(case, src, dst):
    """(from, to) of every step the traversal may take."""
    if case["dir"] == "in":
        return dst, src
    if case["dir"] == "both":
        return torch.cat([src, dst]), torch.cat([dst, src])
    return src, dst


def _exact_batch(case, seed):
    """Ranks and components; triangle counts are whole numbers."""
    n, first, src, dst = _batch(case, seed)
    count, total, d = case["count"], int(n.sum()), 0.85
    graph = torch.repeat_interleave(torch.arange(count, device="cuda"), n)
    nf = n.double()
    deg = torch.bincount(src, minlength=total).double()
    div = torch.where(deg > 0, deg, torch.ones_like(deg))
    rank = (1.0 / nf)[graph]
    live = torch.ones(count, dtype=torch.bool, device="cuda")
    for _ in range(case["max_iter"]):
        zero = torch.zeros(count, dtype=torch.float64, device="cuda")
        lost = zero.index_add(0, graph, torch.where(deg == 0, rank, 0.0))
        base = (1.0 - d) / nf + d * lost / nf
        nxt = base[graph] + d * torch.zeros_like(rank).index_add(0, dst, (rank / div)[src])
        delta = zero.index_add(0, graph, (nxt - rank).abs())
        rank = torch.where(live[graph], nxt, rank)
        live &= delta >= 1e-6
        if not bool(live.any()):
            break
    label = _exact_components(total, src, dst)
    return [rank, (label - first[graph]).int(), None]


def _exact_bfs(case, src, dst, source):
    a, b = _oriented(case, src, dst)
    dist = torch.full((case["n"],), -1, dtype=torch.int32, device="cuda")
    dist[source] = 0
    level = 0
    while True:
        hit = b[(dist[a] == level) & (dist[b] < 0)]
        if hit.numel() == 0:
            return dist
        level += 1
        dist[hit] = level


def _exact_dijkstra(case, src, dst, source, w):
    a, b = _oriented(case, src, dst)
    w = torch.cat([w, w]) if case["dir"] == "both" else w
    dist = torch.full((case["n"],), math.inf, dtype=torch.float64, device="cuda")
    dist[source] = 0.0
    while True:  # the least fixed point of the left-to-right sums
        nxt = dist.scatter_reduce(0, b, dist[a] + w, "amin")
        if torch.equal(nxt, dist):
            return dist
        dist = nxt


def _exact_components(n, src, dst):
    label = torch.arange(n, device="cuda")
    while True:  # smallest member by hooking and pointer jumping
        la, lb = label[src], label[dst]
        low = torch.minimum(la, lb)
        nxt = label.scatter_reduce(0, la, low, "amin").scatter_reduce(0, lb, low, "amin")
        nxt = nxt[nxt]
        nxt = nxt[nxt]
        if torch.equal(nxt, label):
            return label
        label = nxt


def _sampled_sources(n, k, seed):
    """The first k of the seeded Fisher-Yates order (SplitMix64 draws)."""
    mask = (1 << 64) - 1
    state = (seed ^ 0xD1B54A32D192ED03) & mask
    order = list(range(n))
    for i in range(n - 1, 0, -1):
        state = (state + 0x9E3779B97F4A7C15) & mask
        z = state
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (i + 1)
        order[i], order[j] = order[j], order[i]
    return order[:k]


def _csr(rows, cols, n, dtype):
    rows, order = torch.sort(rows, stable=True)
    crow = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    crow[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    ones = torch.ones(rows.numel(), dtype=dtype, device="cuda")
    return torch.sparse_csr_tensor(crow, cols[order], ones, (n, n))


def _exact_betweenness(case, src, dst, seed):
    n = case["n"]
    k = max(1, min(n, math.ceil(n * (case["sources"] / n))))
    sources = _sampled_sources(n, k, seed)
    fwd = _csr(dst, src, n, torch.float64)  # row v: the sources of v's in-edges
    bwd = _csr(src, dst, n, torch.float64)
    total = torch.zeros(n, dtype=torch.float64, device="cuda")
    for at in range(0, k, 32):
        s = torch.tensor(sources[at:at + 32], device="cuda")
        cols = torch.arange(s.numel(), device="cuda")
        level = torch.full((n, s.numel()), -1, dtype=torch.int16, device="cuda")
        sigma = torch.zeros((n, s.numel()), dtype=torch.float64, device="cuda")
        level[s, cols] = 0
        sigma[s, cols] = 1.0
        depth = 0
        while True:
            reach = fwd @ torch.where(level == depth, sigma, 0.0)
            new = (reach > 0) & (level < 0)
            if not bool(new.any()):
                break
            depth += 1
            level[new] = depth
            sigma = torch.where(new, reach, sigma)
        delta = torch.zeros_like(sigma)
        for lv in range(depth, 0, -1):
            coeff = torch.where(level == lv, (1.0 + delta) / sigma, 0.0)
            delta = torch.where(level == lv - 1, delta + sigma * (bwd @ coeff), delta)
        delta[s, cols] = 0.0
        total += delta.sum(1)
    return total * (n / k)  # an estimate over all n sources


def _exact_closeness(case, src, dst):
    n = case["n"]
    adj = _csr(dst, src, n, torch.float32)
    out = torch.zeros(n, dtype=torch.float64, device="cuda")
    for at in range(0, n, 2048):
        s = torch.arange(at, min(n, at + 2048), device="cuda")
        cols = torch.arange(s.numel(), device="cuda")
        front = torch.zeros((n, s.numel()), device="cuda")
        front[s, cols] = 1.0
        seen = front > 0
        reach = torch.zeros(s.numel(), dtype=torch.float64, device="cuda")
        total = torch.zeros_like(reach)
        depth = 0
        while True:
            new = ((adj @ front) > 0) & ~seen
            got = new.sum(0).double()
            if float(got.sum()) == 0:
                break
            depth += 1
            reach += got
            total += depth * got
            seen |= new
            front = new.float()
        out[s] = torch.where(total > 0, reach / total, torch.zeros_like(total))
    return out


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        return _exact_batch(case, seed)
    src, dst = (x.long() for x in _edges(case, seed))
    if op in ("pagerank", "ingest"):
        return _exact_pagerank(case, src, dst)
    if op == "bfs":
        return _exact_bfs(case, src, dst, _source(src, seed))
    if op == "dijkstra":
        return _exact_dijkstra(case, src, dst, _source(src, seed), _weights(src.numel(), seed).cuda())
    if op == "components":
        return _exact_components(case["n"], src, dst).int()
    if op == "betweenness":
        return _exact_betweenness(case, src, dst, seed)
    if op == "closeness":
        return _exact_closeness(case, src, dst)
    return None  # triangle counts are whole numbers
