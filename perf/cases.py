"""The calls that a program on this framework spends its time in, with the
sizes they are made at: PageRank, SpMV, BFS (one root and 64 bit-sliced),
SSSP (one source and a batch), WCC, batched personalised PageRank, and the
layout build every one of them starts from.

Graphs are RMAT (a=.57, b=.19, c=.19) or uniform random edge lists made on the
GPU from the seed and handed over as device pairs.  Results stay on the device
where a program would read them there (out = "device"), or land in an array of
the host: a new one ("host") or a page-locked one that the program keeps
("pinned").
"""
import ctypes
import functools

import numpy as np
import torch

import everythinggraph_gb300 as eg

_GOLDEN = 0x9E3779B97F4A7C15


def listed():
    return [
        # global PageRank of a crawl- or follower-sized graph, ten iterations,
        # on the schedule the autotuner keeps at this size
        dict(name="pagerank_rmat24", op="pagerank", graph="rmat", n=1 << 24, m=1 << 28, undirected=False,
             iterations=10, tolerance=0.0, dangling=False, schedule=12, out="device"),
        # PageRank of a small community graph to convergence: launches and host round trips
        dict(name="pagerank_10k", op="pagerank", graph="rmat", n=10007, m=120000, undirected=True,
             iterations=50, tolerance=1e-6, dangling=True, schedule=0, out="host"),
        # sparse matrix times dense vector, x larger than the L2 cache
        dict(name="spmv_er25_f32", op="spmv", graph="er", n=1 << 25, m=1 << 30, undirected=False, kind="f32",
             out="device"),
        # compensated row sums on a skewed matrix of odd size
        dict(name="spmv_1m5_comp", op="spmv", graph="rmat", n=1500007, m=24000111, undirected=False,
             kind="f32_comp", out="host"),
        # one breadth-first search over a large social graph
        dict(name="bfs_rmat24u", op="bfs", graph="rmat", n=1 << 24, m=1 << 28, undirected=True, loop="host",
             out="device"),
        # one breadth-first search over a small graph: latency of a call
        dict(name="bfs_5k", op="bfs", graph="rmat", n=5003, m=40000, undirected=True, loop="default", out="host"),
        # 64 searches at once (centrality estimates, landmark distances)
        dict(name="bfs_multi_rmat20u", op="bfs_multi", graph="rmat", n=1 << 20, m=1 << 24, undirected=True, k=64,
             out="pinned"),
        # shortest paths from one source, integer weights
        dict(name="sssp_rmat23", op="sssp", graph="rmat", n=1 << 23, m=1 << 27, undirected=False, rule="hash",
             out="device"),
        # shortest paths from 64 sources at once
        dict(name="sssp_multi_1m", op="sssp_multi", graph="rmat", n=1000003, m=16000057, undirected=False, k=64,
             rule="hash", out="pinned"),
        # connected components
        dict(name="wcc_6m", op="wcc", graph="rmat", n=6000011, m=96000007, undirected=True, out="device"),
        # 32 personalised PageRank queries (recommendation), 1 to 8 seeds each
        dict(name="ppr_rmat20u", op="ppr", graph="rmat", n=1 << 20, m=1 << 24, undirected=True, queries=32,
             tolerance=1e-5, out="pinned"),
        # edge list to CSR and CSC: what a program pays for each graph it loads
        dict(name="build_rmat22u", op="build", graph="rmat", n=1 << 22, m=1 << 26, undirected=True, out="device"),
    ]


def draw(rng):
    def size(lo, hi):  # spread over the logarithm, odd ones among them
        return int(2 ** rng.uniform(lo, hi))

    op = rng.choice(["pagerank", "pagerank", "spmv", "spmv", "bfs", "bfs", "bfs_multi", "sssp", "sssp_multi", "wcc",
                     "ppr", "build"])
    top = {"pagerank": 24, "spmv": 24, "bfs": 23.9, "bfs_multi": 20, "sssp": 23, "sssp_multi": 19.9, "wcc": 23,
           "ppr": 20, "build": 22}[op]
    n = size(10, top)
    graph = "er" if rng.random() < 0.25 else "rmat"
    undirected = op in ("wcc", "build", "bfs", "bfs_multi", "ppr") or rng.random() < 0.3
    m = int(n * rng.uniform(4, 8 if undirected and op not in ("wcc", "build", "bfs", "bfs_multi") else 16))
    case = dict(op=op, graph=graph, n=n, m=m, undirected=undirected,
                out="device" if n > 1 << 21 else "host")
    if op == "pagerank":
        stop = rng.random() < 0.5
        case.update(iterations=50 if stop else 10, tolerance=1e-6 if stop else 0.0, dangling=stop,
                    schedule=12 if n > 1 << 21 and not stop else 0)
    elif op == "spmv":
        case.update(kind=rng.choice(["f32", "f32", "f32_comp", "f64", "u32_pull", "u32_push"]))
    elif op == "bfs":
        case.update(loop="host" if n > 1 << 22 else "default")
    elif op == "bfs_multi":
        case.update(k=rng.choice([4, 17, 32, 64]), out="pinned")
    elif op == "sssp":
        case.update(rule=rng.choice(["hash", "ref", "f32"]))
    elif op == "sssp_multi":
        case.update(k=rng.choice([4, 33, 64]), rule=rng.choice(["hash", "f32"]), out="pinned")
    elif op == "ppr":
        case.update(queries=rng.choice([3, 20, 32]), tolerance=1e-5, out="pinned")
    return case


# ------------------------------------------------------------------ inputs
def _endpoints(case, seed):
    """(src, dst) int32 tensors of the edge list."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 1000003 + 17)
    n, m = case["n"], case["m"]
    if case["graph"] == "er":
        return tuple(torch.randint(0, n, (m,), generator=gen, device="cuda", dtype=torch.int32) for _ in range(2))
    scale = max(1, (n - 1).bit_length())
    src = torch.empty(m, dtype=torch.int32, device="cuda")
    dst = torch.empty(m, dtype=torch.int32, device="cuda")
    step = 1 << 25
    for lo in range(0, m, step):
        c = min(step, m - lo)
        s = torch.zeros(c, dtype=torch.int64, device="cuda")
        d = torch.zeros(c, dtype=torch.int64, device="cuda")
        for _ in range(scale):
            r = torch.rand(c, generator=gen, device="cuda")
            s.mul_(2).add_(r >= 0.76)
            d.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        if n != 1 << scale:  # onto [0, n), the order of the ids kept
            s = (s * n) >> scale
            d = (d * n) >> scale
        src[lo:lo + c] = s
        dst[lo:lo + c] = d
    return src, dst


def _pairs(case, seed):
    src, dst = _endpoints(case, seed)
    out = torch.empty((case["m"], 2), dtype=torch.int32, device="cuda")
    out[:, 0] = src
    out[:, 1] = dst
    return out


def _x(case, seed):
    rng = np.random.default_rng([int(seed), 5])
    if case["kind"].startswith("u32"):
        return rng.integers(0, 1 << 20, case["n"], dtype=np.uint32)
    return rng.random(case["n"], dtype=np.float32)


def _seed_lists(case, seed):
    """1 to 8 seeds for each query, drawn over all vertices."""
    rng = np.random.default_rng([int(seed), 9])
    return [rng.integers(0, case["n"], int(rng.integers(1, 9))).astype(np.uint32) for _ in range(case["queries"])]


@functools.lru_cache(maxsize=1)
def _context():
    return eg.Context(0)


class _DeviceArray:
    """A device array of a graph, for torch.as_tensor: the tensor keeps this
    object, and so the graph that owns the memory."""

    def __init__(self, graph, ptr, count, typestr):
        self.graph = graph
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _on_device(graph, which, count, typestr="<i4"):
    return torch.as_tensor(_DeviceArray(graph, graph.device_ptr(which), count, typestr), device="cuda")


def prepare(case, seed):
    ctx = _context()
    op, n = case["op"], case["n"]
    pairs = _pairs(case, seed)
    torch.cuda.synchronize()
    state = {"case": case, "ctx": ctx}
    if op == "build":  # the edge list is in hand, the graph is not
        state["pairs"] = pairs
        return state
    g = ctx.from_device_pairs(n, pairs.data_ptr(), case["m"], case["undirected"])
    g.build(eg.CSR | eg.CSC)
    del pairs
    torch.cuda.empty_cache()
    state["graph"] = g
    if op == "pagerank":
        g.set_row_schedule(case["schedule"])
    elif op == "spmv":
        x = eg.pinned_empty(n, np.uint32 if case["kind"].startswith("u32") else np.float32)
        x[:] = _x(case, seed)
        state["x"] = x
    elif op in ("bfs", "sssp"):
        state["root"] = int(g.sample_roots(1, seed)[0])
    elif op in ("bfs_multi", "sssp_multi"):
        state["roots"] = g.sample_roots(case["k"], seed)
        state["dst"] = eg.pinned_empty((case["k"], n), np.int32 if op == "bfs_multi" else np.uint32)
    elif op == "ppr":
        lists = _seed_lists(case, seed)
        state["offsets"] = np.concatenate([[0], np.cumsum([len(s) for s in lists])]).astype(np.uint32)
        state["seeds"] = np.concatenate(lists)
        state["dst"] = eg.pinned_empty((case["queries"], n), np.float32)
        o = eg.L.PprOpts()
        o.damping, o.max_iters = 0.85, 50
        for q in range(32):
            o.tolerance[q] = case["tolerance"]
        state["opts"] = o
    if op in ("sssp", "sssp_multi"):
        state["weights"] = eg.weights(case["rule"], seed=int(seed) + 6, lo=1, hi=255)
    return state


# ------------------------------------------------------------------ one pass
def _ptr(a):
    return ctypes.c_void_p(a.ctypes.data)


def run(state):
    case = state["case"]
    op, n, on_device = case["op"], case["n"], case["out"] == "device"
    if op == "build":
        m = 2 * case["m"] if case["undirected"] else case["m"]
        state["graph"] = g = state["ctx"].from_device_pairs(n, state["pairs"].data_ptr(), case["m"],
                                                            case["undirected"])
        g.build(eg.CSR | eg.CSC)
        return [_on_device(g, eg.L.EG_DEV_CSR_PTR, n + 1), _on_device(g, eg.L.EG_DEV_CSR_COL, m),
                _on_device(g, eg.L.EG_DEV_CSC_PTR, n + 1), _on_device(g, eg.L.EG_DEV_CSC_COL, m)]
    g = state["graph"]
    if op == "pagerank":
        rank, _ = g.pagerank(iterations=case["iterations"], tolerance=case["tolerance"], dangling=case["dangling"],
                             copy_out=not on_device)
        return _on_device(g, eg.L.EG_DEV_RANK, n, "<f4") if on_device else rank
    if op == "spmv":
        y, _ = g.spmv(state["x"], case["kind"], value_seed=3, copy_out=not on_device)
        if on_device:
            return _on_device(g, eg.L.EG_DEV_SPMV_Y, n,
                              {"f64": "<f8", "f32": "<f4", "f32_comp": "<f4"}.get(case["kind"], "<i4"))
        return y.view(np.int32) if y.dtype == np.uint32 else y
    if op == "bfs":
        level, _ = g.bfs(state["root"], host_loop=True if case["loop"] == "host" else None, copy_out=not on_device)
        return _on_device(g, eg.L.EG_DEV_LEVEL, n) if on_device else level
    if op == "bfs_multi":
        st = eg.L.BfsStats()
        eg.L.check(eg.lib().eg_bfs_multi(g._h, _ptr(state["roots"]), case["k"], _ptr(state["dst"]), ctypes.byref(st)))
        return state["dst"]
    if op == "sssp":
        dist, _ = g.sssp(state["root"], state["weights"], copy_out=not on_device)
        return _on_device(g, eg.L.EG_DEV_DIST, n) if on_device else dist.view(np.int32)
    if op == "sssp_multi":
        st = eg.L.SsspStats()
        eg.L.check(eg.lib().eg_sssp_multi(g._h, _ptr(state["roots"]), case["k"], ctypes.byref(state["weights"]),
                                          _ptr(state["dst"]), ctypes.byref(st)))
        return state["dst"].view(np.int32)
    if op == "wcc":
        label, _ = g.wcc(copy_out=not on_device)
        return _on_device(g, eg.L.EG_DEV_LABEL, n) if on_device else label
    if op == "ppr":
        st = eg.L.PprStats()
        eg.L.check(eg.lib().eg_ppr_multi(g._h, _ptr(state["seeds"]), _ptr(state["offsets"]), case["queries"],
                                         ctypes.byref(state["opts"]), _ptr(state["dst"]), ctypes.byref(st)))
        return state["dst"]
    raise ValueError(op)


def work(case):
    op, n = case["op"], case["n"]
    m = 2 * case["m"] if case["undirected"] else case["m"]  # adjacency entries
    k = case.get("k", 1)
    if op == "pagerank":  # per iteration: an index and a contribution per entry, four words per vertex
        its = 10  # about what the runs to 1e-6 need, too
        return {"bytes": its * (8 * m + 16 * n), "flops": its * 2 * m}
    if op == "spmv":  # index and value per entry (u32: no value); x read, row starts read, y written
        y = 8 if case["kind"] == "f64" else 4
        return {"bytes": (4 if case["kind"].startswith("u32") else 8) * m + (8 + y) * n, "flops": 2 * m}
    if op == "bfs":  # one list entry per vertex, row starts, levels
        return {"bytes": 12 * n, "flops": 0}
    if op == "bfs_multi":  # every list once, the levels
        return {"bytes": 4 * m + 4 * n + 4 * n * k, "flops": 0}
    if op in ("sssp", "sssp_multi"):  # target and weight of every edge, row starts, distances
        return {"bytes": 8 * m + 4 * n + 4 * n * k, "flops": 0}
    if op == "wcc":  # two list entries per vertex, row starts, labels
        return {"bytes": 16 * n, "flops": 0}
    if op == "ppr":  # about 12 sweeps: an index per entry, two rows of the queries' values per vertex; the ranks out
        q = case["queries"]
        return {"bytes": 12 * (4 * m + 8 * n * q) + 4 * n * q, "flops": 12 * m * q}
    return {"bytes": 8 * case["m"] + 2 * (4 * m + 4 * n), "flops": 0}  # build: pairs in, two adjacencies out


# ------------------------------------------------------------------ 64-bit values
def _directed(case, seed):
    """(src, dst) of every adjacency entry."""
    src, dst = _endpoints(case, seed)
    if case["undirected"]:
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    return src, dst


def _scatter_rows(src, dst, x, scale_of=None):
    """y[v] = sum over entries (u, v) of x[u] (times scale_of(u, v)), in float64."""
    y = torch.zeros_like(x)
    step = max(1 << 16, (1 << 26) // (x.shape[1] if x.dim() > 1 else 1))
    for lo in range(0, len(src), step):
        s, d = src[lo:lo + step].long(), dst[lo:lo + step].long()
        t = x[s]
        y.index_add_(0, d, t if scale_of is None else t * scale_of(s, d))
    return y


def _mix(z):
    """SplitMix64's output function on int64 tensors (wrapping)."""
    def signed(c):
        return c - (1 << 64) if c >= 1 << 63 else c

    def shr(v, k):
        return (v >> k) & ((1 << (64 - k)) - 1)

    z = z + signed(_GOLDEN)
    z = (z ^ shr(z, 30)) * signed(0xBF58476D1CE4E5B9)
    z = (z ^ shr(z, 27)) * signed(0x94D049BB133111EB)
    return z ^ shr(z, 31)


def _edge_value(seed):
    """The value rule of the fp32 and fp64 kinds: 24 hashed bits of the endpoint pair."""
    base = _mix(torch.tensor([seed], dtype=torch.int64, device="cuda"))

    def value(u, v):
        pair = (torch.minimum(u, v) << 32) | torch.maximum(u, v)
        return ((_mix(_mix(base ^ pair)) >> 40) & 0xFFFFFF).double() / 16777216.0

    return value


def exact(case, seed):
    op, n = case["op"], case["n"]
    if op == "spmv" and not case["kind"].startswith("u32"):
        src, dst = _directed(case, seed)
        return _scatter_rows(src, dst, torch.from_numpy(_x(case, seed)).cuda().double(), _edge_value(3))
    if op not in ("pagerank", "ppr"):
        return None  # whole numbers
    src, dst = _directed(case, seed)
    deg = torch.zeros(n, dtype=torch.float64, device="cuda")
    for lo in range(0, len(src), 1 << 26):
        s = src[lo:lo + (1 << 26)].long()
        deg += torch.bincount(s, minlength=n)
    none = deg == 0
    inv = torch.where(none, torch.zeros_like(deg), 1.0 / deg)
    d = float(np.float32(0.85))
    if op == "pagerank":
        rank = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
        for _ in range(case["iterations"]):
            spread = d * float(rank[none].sum()) / n if case["dangling"] else 0.0
            new = (1.0 - d) / n + spread + d * _scatter_rows(src, dst, rank * inv)
            change = float((new - rank).abs().sum())
            rank = new
            if case["tolerance"] > 0 and change < case["tolerance"]:
                break
        return rank
    q = case["queries"]
    home = torch.zeros((n, q), dtype=torch.float64, device="cuda")
    for i, s in enumerate(_seed_lists(case, seed)):
        home[:, i].index_add_(0, torch.from_numpy(s.astype(np.int64)).cuda(),
                              torch.full((len(s),), 1.0 / len(s), dtype=torch.float64, device="cuda"))
    rank = home.clone()
    live = torch.ones(q, dtype=torch.bool, device="cuda")
    for _ in range(50):
        back = (1.0 - d) + d * rank[none].sum(0)
        new = back * home + d * _scatter_rows(src, dst, rank * inv[:, None])
        change = (new - rank).abs().sum(0)
        rank = torch.where(live, new, rank)
        live = live & ~(change < case["tolerance"])
        if not bool(live.any()):
            break
    return rank.t().contiguous()
