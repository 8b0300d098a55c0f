"""Performance cases: the work users of the library have it do, through the
Python mirror of the C ABI, from single small traversals to the headline
SSSP + PageRank step.

A case names an operation (`op`), a graph family and its size, and the
operation's options.  The case fixes the graph up to its numbering (R-MAT
with a/b/c = 0.57/0.19/0.19, symmetrised, without loops and duplicates,
unused ids removed; or a 4-neighbour lattice with 5 % diagonal shortcuts), so
that its sizes do not depend on the seed; the seed picks the numbering (ids
shifted round, so neighbouring ids stay neighbours), the weights (integers
1..64 per undirected edge), the sources and the seeds.  Graphs are drawn on
the GPU, handed to the library as host CSR arrays and uploaded.  Results go
to page-locked arrays that the caller keeps from run to run where the entry
point takes one (`out=`), else to the arrays the entry point makes.
"""
import math

import numpy as np
import torch

import multigraph_gb300 as mg

DAMPING = 0.85
UNREACHED = 0x64646464


def listed():
    return [
        # one traversal of a small graph: an interactive query, where launches,
        # synchronisations and the readback are the cost
        dict(name="bfs_rmat12", op="bfs", family="rmat", scale=12, ef=16),
        # components of the 65,536-vertex R-MAT graph of the BFS / CC configuration
        dict(name="cc_rmat16", op="cc", family="rmat", scale=16, ef=16),
        # ranks of an ordinary mid-size graph, some 16 short sweeps
        dict(name="pagerank_rmat16", op="pagerank", family="rmat", scale=16, ef=16, variant="topology", tol=1e-6),
        # one traversal of a graph whose columns fill the L2 cache
        dict(name="bfs_rmat20", op="bfs", family="rmat", scale=20, ef=16),
        # the headline step: SSSP from one vertex and PageRank to L1 change 1e-6
        dict(name="step_rmat22", op="step", family="rmat", scale=22, ef=16, tol=1e-6),
        # a new set of edge weights uploaded, then one SSSP (the serving loop
        # of a graph whose costs change)
        dict(name="update_rmat20", op="update", family="rmat", scale=20, ef=16),
        # betweenness of one source on a road-like lattice: hundreds of short
        # levels, path counts past 2^90 (sides such that they stay in the
        # 64-bit range, here and below)
        dict(name="bc_lattice", op="bc", family="lattice", rows=320, cols=311),
        # betweenness summed over many sources: 32 sources a traversal on a
        # power-law graph, and on a lattice
        dict(name="bc_multi_rmat20", op="bc_multi", family="rmat", scale=20, ef=16, sources=256),
        dict(name="bc_multi_lattice", op="bc_multi", family="lattice", rows=480, cols=397, sources=32),
        # personalised ranks of a batch of seeds, two groups of 32
        dict(name="ppr_rmat20", op="ppr", family="rmat", scale=20, ef=16, seeds=64, tol=1e-6),
        # one training step on edge weights: new float weights, weighted
        # PageRank, its adjoint, the gradient back on the host
        dict(name="train_rmat19", op="train", family="rmat", scale=19, ef=16, tol=1e-7),
        # BFS and components of a batch of uneven graphs in one arena
        dict(name="graphs_30", op="graphs", family="rmat", count=30, lo=10, hi=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any operation, sizes spread over the logarithm of the
    range, edge factors 6..24, lattices with odd sides."""
    op = rng.choice(["bfs", "bfs", "cc", "sssp", "pagerank", "pagerank", "step", "update", "bc", "bc_multi", "ppr",
                     "train", "graphs"])
    if op == "graphs":
        lo = rng.randint(6, 11)
        return dict(op=op, family="rmat", count=rng.randint(3, 32), lo=lo, hi=rng.randint(lo + 1, 15))
    case = dict(op=op)
    lattice = op in ("bfs", "cc", "sssp", "pagerank", "bc", "bc_multi") and rng.random() < 0.35
    if lattice:
        area = _log_int(rng, 2_000, {"bc": 100_000, "bc_multi": 160_000}.get(op, 2_000_000))
        rows = max(8, int(math.sqrt(area) * rng.uniform(0.6, 1.5)))
        case.update(family="lattice", rows=rows, cols=max(8, area // rows))
    else:
        top = {"step": 21, "train": 19, "bc_multi": 20, "ppr": 20}.get(op, 21)
        case.update(family="rmat", scale=rng.randint(9, top), ef=rng.randint(6, 24))
        if case["scale"] >= 20:
            case["ef"] = min(case["ef"], 16)
    if op == "pagerank":
        case.update(variant=rng.choice(["topology", "topology", "data"]), tol=rng.choice([1e-5, 1e-6]))
    elif op in ("step", "ppr"):
        case["tol"] = rng.choice([1e-5, 1e-6])
    elif op == "train":
        case["tol"] = rng.choice([1e-6, 1e-7])
    if op == "bc_multi":
        case["sources"] = rng.randint(2, 32 if lattice else 160)
    if op == "ppr":
        case["seeds"] = rng.randint(1, 64)
    return case


# ---------------------------------------------------------------------------
# graphs
# ---------------------------------------------------------------------------
def _generator(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFF)
    return g


def _csr(src, dst, bits, seed):
    """Symmetrised, loop-free, duplicate-free CSR of the id pairs with unused
    ids removed and the others shifted round by a distance from the seed:
    (row offsets, columns) as int32 on the GPU, columns ascending."""
    used = torch.zeros(1 << bits, dtype=torch.bool, device="cuda")
    keep = src != dst
    src, dst = src[keep], dst[keep]
    used[src] = True
    used[dst] = True
    n = int(used.sum())
    new = (torch.cumsum(used, 0) - 1 + np.random.default_rng(seed).integers(n)) % n
    src, dst = new[src], new[dst]
    key = torch.unique(torch.cat([(src << bits) | dst, (dst << bits) | src]))
    del src, dst, keep
    row = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(key >> bits, minlength=n), 0, out=row[1:])
    return row.int(), (key & ((1 << bits) - 1)).int()


def _rmat(scale, ef, seed, copy=0):
    gen = _generator(17 + copy, 7 * scale + ef)
    m = ef << scale
    src = torch.zeros(m, dtype=torch.int64, device="cuda")
    dst = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(m, generator=gen, device="cuda")
        src.mul_(2).add_(r >= 0.76)
        dst.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    return _csr(src, dst, scale, seed)


def _lattice(rows, cols, seed):
    gen = _generator(17, 5 * rows + cols)
    ids = torch.arange(rows * cols, device="cuda").view(rows, cols)
    pairs = [(ids[:, :-1], ids[:, 1:]), (ids[:-1, :], ids[1:, :])]
    short = torch.rand(rows - 1, cols - 1, generator=gen, device="cuda") < 0.05
    pairs.append((ids[:-1, :-1][short], ids[1:, 1:][short]))
    src = torch.cat([p[0].reshape(-1) for p in pairs])
    dst = torch.cat([p[1].reshape(-1) for p in pairs])
    return _csr(src, dst, max(1, (rows * cols - 1).bit_length()), seed)


def _graph(case, seed):
    if case["family"] == "lattice":
        return _lattice(case["rows"], case["cols"], seed)
    return _rmat(case["scale"], case["ef"], seed)


def _batch(case):
    """Scale and edge factor of each graph of a batch."""
    rng = np.random.default_rng(case["count"])
    return list(zip(rng.integers(case["lo"], case["hi"] + 1, case["count"]).tolist(),
                    rng.integers(8, 33, case["count"]).tolist()))


def _rows_of(row):
    """The row of every CSR entry."""
    return torch.repeat_interleave(torch.arange(len(row) - 1, device="cuda"), (row[1:] - row[:-1]).long())


def _weights(row, col, seed):
    """Integer weights 1..64, one per undirected edge."""
    u, v = _rows_of(row), col.long()
    z = torch.minimum(u, v) * 2654435761 + torch.maximum(u, v) * 40503 + int(seed) * 97
    z = (z ^ (z >> 15)) * 2246822519 & 0x7FFFFFFFFFFF
    return (1 + ((z ^ (z >> 13)) & 63)).int()


def _float_weights(row, col, seed):
    """Float weights in (0, 1], one per CSR entry."""
    return 1.0 - torch.rand(len(col), generator=_generator(seed, 11), device="cuda")


def _sources(col, count, seed):
    """Vertices met by following random edges (so they sit in the large part
    of the graph)."""
    at = torch.randint(len(col), (count,), generator=_generator(seed, 3), device="cuda")
    return col[at].cpu().numpy()


def _host(row, col, wt=None):
    return mg.HostGraph.from_csr(row.cpu().numpy(), col.cpu().numpy(), None if wt is None else wt.cpu().numpy())


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


# ---------------------------------------------------------------------------
def prepare(case, seed):
    op = case["op"]
    s = dict(case=case)
    if op == "graphs":
        parts = [_rmat(k, ef, seed + i, copy=i) for i, (k, ef) in enumerate(_batch(case))]
        s["sources"] = [int(_sources(col, 1, seed + i)[0]) for i, (_, col) in enumerate(parts)]
        hosts = [_host(row, col) for row, col in parts]
        s["batch"] = mg.Batch(hosts)
        for h in hosts:
            h.free()
        return s
    row, col = _graph(case, seed)
    n = len(row) - 1
    host = _host(row, col, _weights(row, col, seed) if op in ("sssp", "step", "update") else None)
    s["graph"] = mg.Graph(host)
    if op in ("bfs", "sssp", "bc", "step", "update"):
        s["source"] = int(_sources(col, 1, seed)[0])
    if op in ("bfs", "cc", "sssp", "step", "update"):
        s["labels"] = _pinned((n,), torch.int32)
    if op in ("pagerank", "step", "train"):
        s["rank"] = _pinned((n,), torch.float32)
    if op == "update":
        s["next"] = _host(row, col, _weights(row, col, seed + 1))
        s["next"].pin()
    if op == "bc_multi":
        s["sources"] = _sources(col, case["sources"], seed)
        s["scores"] = _pinned((n,), torch.float32)
    if op == "ppr":
        s["seeds"] = _sources(col, case["seeds"], seed)
        s["ranks"] = _pinned((case["seeds"], n), torch.float32)
    if op == "train":
        s["weights"] = _float_weights(row, col, seed).cpu().numpy()
        s["loss"] = torch.randn(n, generator=_generator(seed, 13), device="cuda").cpu().numpy()
    host.free()
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "graphs":
        levels, _ = s["batch"].bfs(s["sources"])
        labels, _ = s["batch"].cc()
        return levels, labels
    g = s["graph"]
    if op == "bfs":
        return g.bfs(s["source"], out=s["labels"])[0]
    if op == "sssp":
        return g.sssp(s["source"], out=s["labels"])[0]
    if op == "cc":
        return g.cc(out=s["labels"])[0]
    if op == "pagerank":
        variant = mg.PR_DATA if case["variant"] == "data" else mg.PR_TOPOLOGY
        return g.pagerank(variant, out=s["rank"], tol=case["tol"])[0]
    if op == "step":
        dist, _ = g.sssp(s["source"], out=s["labels"])
        rank, _ = g.pagerank(mg.PR_TOPOLOGY, out=s["rank"], tol=case["tol"])
        return dist, rank
    if op == "update":
        g.reload(s["next"])
        return g.sssp(s["source"], out=s["labels"])[0]
    if op == "bc":
        return g.bc(s["source"])[0]
    if op == "bc_multi":
        return g.bc_multi(s["sources"], out=s["scores"])[0]
    if op == "ppr":
        return g.ppr_batch(s["seeds"], out=s["ranks"], tol=case["tol"])[0]
    if op == "train":
        g.set_float_weights(s["weights"])
        x, _ = g.wpagerank(out=s["rank"], tol=case["tol"])
        (grad, lam), _ = g.wpagerank_backward(s["loss"], tol=10 * case["tol"])
        return x, grad, lam
    raise ValueError(op)


# ---------------------------------------------------------------------------
def _sizes(case):
    """Vertices and directed edges after loops, duplicates and unused ids are
    gone (R-MAT: fitted to drawn graphs, within a few per cent)."""
    if case["family"] == "lattice":
        n = case["rows"] * case["cols"]
        return n, int(4.1 * n)
    if "count" in case:
        return tuple(map(sum, zip(*[_sizes(dict(family="rmat", scale=k, ef=ef)) for k, ef in _batch(case)])))
    k, ef = case["scale"], case["ef"]
    return int(2 ** k * min(1.0, 0.93 - 0.0163 * k) * (ef / 16) ** 0.25), int(2 ** k * 2 * ef * (1 - 0.95 * 0.868 ** k))


SWEEPS = {1e-5: 13, 1e-6: 16, 1e-7: 20}   # sweeps to the L1 change, about


def work(case):
    """Each edge array read once per sweep of an iterative method (it does
    not stay on the chip), once per traversal or direction otherwise; each
    vertex value read and written once per sweep."""
    n, m = _sizes(case)
    op = case["op"]
    sweep = 4 * m + 16 * n
    if op == "graphs":
        return dict(bytes=2 * 4 * n * 2 + 4 * m, flops=0)
    if op in ("bfs", "cc"):
        return dict(bytes=4 * m + 8 * n, flops=0)
    if op == "sssp":
        return dict(bytes=8 * m + 8 * n, flops=0)
    if op == "update":
        return dict(bytes=8 * m + 16 * m + 12 * n + 8 * m, flops=0)
    if op == "pagerank":
        return dict(bytes=sweep * SWEEPS[case["tol"]], flops=m * SWEEPS[case["tol"]])
    if op == "step":
        return dict(bytes=sweep * SWEEPS[case["tol"]] + 8 * m + 8 * n, flops=m * SWEEPS[case["tol"]])
    if op == "bc":
        return dict(bytes=8 * m + 32 * n, flops=4 * m)
    if op == "bc_multi":
        groups = -(-case["sources"] // 32)
        return dict(bytes=groups * 8 * m + case["sources"] * 24 * n, flops=4 * m * case["sources"])
    if op == "ppr":
        groups, k = -(-case["seeds"] // 32), SWEEPS[case["tol"]]
        return dict(bytes=k * (groups * 4 * m + case["seeds"] * 12 * n), flops=k * m * case["seeds"])
    k = 3 * SWEEPS[case["tol"]]   # train: forward and adjoint sweeps
    return dict(bytes=k * (8 * m + 16 * n) + 4 * m * 4, flops=2 * k * m)


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------
def _scatter(n, dst, val):
    return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, dst, val)


def _pagerank64(row, col, tol):
    n = len(row) - 1
    u, v = _rows_of(row), col.long()
    deg = (row[1:] - row[:-1]).double()
    x = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    while True:
        nx = (1 - DAMPING) / n + DAMPING * _scatter(n, v, (x / deg)[u])
        change = float((nx - x).abs().sum())
        x = nx
        if change <= tol:
            return x


def _adjacency(row, col):
    n = len(row) - 1
    ones = torch.ones(len(col), dtype=torch.float64, device="cuda")
    return torch.sparse_csr_tensor(row.long(), col.long(), ones, size=(n, n))


def _brandes64(row, col, sources):
    """Levels, path counts and dependencies of the sources, a column each."""
    n, k = len(row) - 1, len(sources)
    a = _adjacency(row, col)
    src = torch.as_tensor(np.asarray(sources, dtype=np.int64), device="cuda")
    lanes = torch.arange(k, device="cuda")
    level = torch.full((n, k), -1, dtype=torch.int32, device="cuda")
    sigma = torch.zeros((n, k), dtype=torch.float64, device="cuda")
    level[src, lanes], sigma[src, lanes] = 0, 1.0
    d = 0
    while True:
        t = a @ torch.where(level == d, sigma, 0.0)
        new = (level < 0) & (t > 0)
        if not bool(new.any()):
            break
        d += 1
        level[new] = d
        sigma = torch.where(new, t, sigma)
    delta = torch.zeros_like(sigma)
    for at in range(d, 0, -1):
        t = a @ torch.where(level == at, (1.0 + delta) / sigma, 0.0)
        delta = torch.where(level == at - 1, sigma * t, delta)
    return level, sigma, delta


def exact(case, seed):
    op = case["op"]
    if op in ("bfs", "sssp", "cc", "update", "graphs") or case.get("variant") == "data":
        return None
    row, col = _graph(case, seed)
    n = len(row) - 1
    if op == "pagerank":
        return _pagerank64(row, col, case["tol"])
    if op == "step":
        return None, _pagerank64(row, col, case["tol"])
    if op == "bc":
        _, sigma, delta = _brandes64(row, col, _sources(col, 1, seed))
        return None, sigma[:, 0], delta[:, 0]
    if op == "bc_multi":
        sources = _sources(col, case["sources"], seed)
        total = torch.zeros(n, dtype=torch.float64, device="cuda")
        for k in range(0, len(sources), 32):
            part = sources[k:k + 32]
            delta = _brandes64(row, col, part)[2]
            delta[torch.as_tensor(part.astype(np.int64), device="cuda"), torch.arange(len(part), device="cuda")] = 0.0
            total += delta.sum(1)
        return total
    if op == "ppr":
        a = _adjacency(row, col)
        deg = (row[1:] - row[:-1]).double()[:, None]
        seeds = _sources(col, case["seeds"], seed)
        out = torch.empty((len(seeds), n), dtype=torch.float64, device="cuda")
        for k in range(0, len(seeds), 32):
            part = torch.as_tensor(seeds[k:k + 32].astype(np.int64), device="cuda")
            e = torch.zeros((n, len(part)), dtype=torch.float64, device="cuda")
            e[part, torch.arange(len(part), device="cuda")] = 1.0
            x = e.clone()
            while True:
                nx = (1 - DAMPING) * e + DAMPING * (a @ (x / deg))
                change = float((nx - x).abs().sum(0).max())
                x = nx
                if change <= case["tol"]:
                    break
            out[k:k + 32] = x.t()
        return out
    # train: weighted PageRank, its adjoint and the edge gradient
    u, v = _rows_of(row), col.long()
    w = _float_weights(row, col, seed).double()
    total = _scatter(n, u, w)
    p = w / total[u]
    x = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    while True:
        nx = (1 - DAMPING) / n + DAMPING * _scatter(n, v, p * x[u])
        change = float((nx - x).abs().sum())
        x = nx
        if change <= case["tol"]:
            break
    g = torch.randn(n, generator=_generator(seed, 13), device="cuda").double()
    limit = 10 * case["tol"] * float(g.abs().sum())
    lam = g.clone()
    while True:
        nl = g + DAMPING * _scatter(n, u, p * lam[v])
        change = float((nl - lam).abs().sum())
        lam = nl
        if change <= limit:
            break
    back = _scatter(n, u, p * lam[v])
    grad = DAMPING * (x / total)[u] * (lam[v] - back[u])
    return x, grad, lam
