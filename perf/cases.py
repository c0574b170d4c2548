"""Performance cases: the calls a user of this library makes, over their range.

An index is built in two calls: the kNN graph of a base (GNN-Descent), then a
prune of that graph to one of the index types. A built index is searched. Each
case is one such call through tagore_b200.capi, on inputs drawn from a seed:

  knn     capi.gnn_descent_host on a pinned FP32 base in host memory
  prune   capi.pruning (an index type) or capi.pruning_cfs (a mode and metric)
          on a kNN graph that is already on the device
  search  capi.search over a pruned index

Bases are the Gaussian mixtures of tagore_b200/synth.py, drawn on the GPU, with
components of equal size in random id order.

What is compared. A prune and a search are functions of their inputs, bit for
bit: every buffer they write comes back and has to be the same. GNN-Descent is
not: its reverse samples are the first that arrive, so two runs of one build
keep slightly different ids. The ids are therefore not compared; the whole
sorted distance array is, against another run's within a tolerance and against
the exact kNN distances in 64 bits, which is the graph's recall as a number.
"""
import math

import numpy as np
import torch

from tagore_b200 import capi

SEARCH_SEED = 0x5EED


def _knn(name, data, n, d, comps, k, iters, rescale=1):
    return dict(name=name, call="knn", data=data, n=n, d=d, comps=comps, k=k, iters=iters,
                rescale=rescale)


def _prune(name, data, n, d, comps, k, fd, what, thre=1.0, topm=64):
    return dict(name=name, call="prune", data=data, n=n, d=d, comps=comps, k=k, fd=fd, what=what,
                thre=thre, topm=topm)


def _search(name, data, n, d, comps, nq, L, k):
    return dict(name=name, call="search", data=data, n=n, d=d, comps=comps, nq=nq, L=L, k=k)


def listed():
    return [
        # a small shard or a test build: launches and fixed costs count
        _knn("knn_5k_x128", "sift", 5003, 128, 4, 32, 10),
        # a width the 16-byte row rules do not take (d % 8 != 0)
        _knn("knn_50k_x100", "sift", 50_000, 100, 32, 48, 10),
        # one cluster of the clustered large-index build at its median size:
        # 8 + 8 iterations, no rescale
        _knn("knn_165k_x96", "deep", 165_118, 96, 84, 64, 16, rescale=0),
        # the headline base, 10 iterations; K 64, because at the headline's 96 a
        # few rows end in another component in one run and not in the next
        _knn("knn_1m_x128", "sift", 1_000_000, 128, 256, 64, 10),
        # wide rows, a quarter of the GIST-like configuration
        _knn("knn_250k_x960", "gist", 250_000, 960, 128, 64, 12),
        # NSG of a small shard
        _prune("nsg_10k_x128", "sift", 10_007, 128, 6, 32, 24, "NSG"),
        # the headline configuration's prune
        _prune("cfs_path_1m_x128", "sift", 1_000_000, 128, 256, 96, 32, "path/dist"),
        # the Deep-like configuration's prune, a quarter of its points
        _prune("vamana_500k_x96", "deep", 500_009, 96, 256, 64, 32, "Vamana", thre=1.2),
        # the GIST-like configuration's two prunes
        _prune("nssg_100k_x960", "gist", 100_000, 960, 51, 64, 32, "NSSG", thre=0.5),
        _prune("dpg_60k_x960", "gist", 60_000, 960, 30, 64, 32, "DPG"),
        # the rank prune at the headline size
        _prune("cagra_1m_x128", "sift", 1_000_000, 128, 256, 96, 32, "CAGRA"),
        # evaluating a built index: 10,000 held-out queries
        _search("search_100k_x128", "sift", 100_000, 128, 64, 10_000, 128, 10),
    ]


WIDTHS = [16, 32, 48, 64, 96, 100, 112, 128, 136, 200, 256, 384, 512, 768, 960, 1024]
PRUNES = [("NSG", 1.0), ("Vamana", 1.2), ("NSSG", 0.5), ("CAGRA", 1.0), ("DPG", 1.0),
          ("path/dist", 1.0), ("path/dist", 1.2), ("path/angle", 0.5), ("2-hop/dist", 1.0),
          ("2-hop/angle", 0.5), ("1-hop/rank", 1.0)]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["knn", "knn", "prune", "prune", "prune", "search"])
    d = rng.choice(WIDTHS)
    data = "gist" if d > 200 else rng.choice(["sift", "deep"])
    top = max(4000, min(400_000, 100_000_000 // d))
    n = _log_int(rng, 3000, top)
    comps = max(1, n // rng.randrange(1000, 3000))
    if call == "knn":
        c = _knn("", data, n, d, comps, rng.randrange(32, 65), rng.randrange(10, 17),
                 rescale=rng.randrange(2))
    elif call == "prune":
        what, thre = rng.choice(PRUNES)
        k = rng.randrange(24, 97)
        fd = rng.randrange(16, min(k, 64) + 1)
        if what == "DPG":
            fd = rng.randrange(max(16, k // 2), min(k - 1, 64) + 1)  # fd < k <= 2 fd + 1
        c = _prune("", data, n, d, comps, k, fd, what, thre, rng.choice([32, 64, 100]))
    else:
        L = rng.randrange(32, 201)
        c = _search("", data, min(n, 200_000), rng.choice([7, 50] + WIDTHS), comps,
                    _log_int(rng, 1, 10_000), L, rng.randrange(1, min(L, 100) + 1))
    del c["name"]
    return c


# ---- inputs ----

SIGMA = {"sift": 20.0, "gist": 0.05, "deep": 0.35}
FACTOR = {"sift": 0.01, "gist": 1.0, "deep": 10.0}  # the power-of-ten rescale of such a base


def _centers(data, comps, d, g):
    u = torch.rand(comps, d, generator=g, device="cuda")
    return u * 128.0 if data == "sift" else u if data == "gist" else u * 2.0 - 1.0


def _draw_rows(data, centers, label, g):
    x = torch.randn(label.numel(), centers.shape[1], generator=g, device="cuda")
    x.mul_(SIGMA[data]).add_(centers[label])
    if data == "sift":
        return x.clamp_(0, 255).round_()
    if data == "gist":
        return x.clamp_(0, 1)
    return torch.nn.functional.normalize(x, dim=1)


def _base(case, seed, nq=0):
    """(base, queries, grid): grid[c] lists component c's ids, padded with -1."""
    n, comps = case["n"], case["comps"]
    g = torch.Generator("cuda").manual_seed(seed)
    centers = _centers(case["data"], comps, case["d"], g)
    perm = torch.randperm(n, generator=g, device="cuda")
    m = -(-n // comps)
    grid = torch.full((m * comps,), -1, dtype=torch.int64, device="cuda")
    grid[:n] = perm
    label = torch.empty(n, dtype=torch.int64, device="cuda")
    label[perm] = torch.arange(n, device="cuda") % comps
    base = _draw_rows(case["data"], centers, label, g)
    queries = None
    if nq:
        queries = _draw_rows(case["data"], centers,
                             torch.randint(comps, (nq,), generator=g, device="cuda"), g)
    return base, queries, grid.view(m, comps).t().contiguous(), g


def _exact_rows(x, grid, k):
    """Ids (n x k) of each row's k nearest other rows of its component. The
    components lie far apart, so these are its k nearest of all rows."""
    n, d = x.shape
    comps, m = grid.shape
    out = torch.empty(n, k, dtype=torch.int64, device="cuda")
    step = max(1, (1 << 28) // (m * max(m, d)))
    for c in range(0, comps, step):
        ids = grid[c:c + step]
        pad = ids < 0
        rows = x[ids.clamp_min(0)].float()
        sq = (rows * rows).sum(2)
        dist = sq[:, :, None] + sq[:, None, :] - 2.0 * torch.bmm(rows, rows.transpose(1, 2))
        dist.masked_fill_(pad[:, None, :], float("inf"))
        dist.diagonal(dim1=1, dim2=2).fill_(float("inf"))
        near = dist.topk(k, dim=2, largest=False).indices
        near = torch.gather(ids[:, None, :].expand(-1, m, -1), 2, near)
        out[ids[~pad]] = near[~pad]
    return out


def _pair_dist(x, ids, dtype):
    """Squared distances of row i to rows ids[i], summed in `dtype`."""
    n, k = ids.shape
    out = torch.empty(n, k, dtype=dtype, device="cuda")
    step = max(1, (1 << 27) // (k * x.shape[1]))
    for i in range(0, n, step):
        a = x[i:i + step].to(dtype)[:, None, :]
        out[i:i + step] = (a - x[ids[i:i + step]].to(dtype)).square_().sum(2)
    return out


def _graph(x, grid, k, g):
    """A kNN graph as GNN-Descent leaves it: sorted rows of the k + k/16
    nearest with k/16 of them, at random, missed."""
    ids = _exact_rows(x, grid, min(k + max(1, k // 16), grid.shape[1] - 2))
    keep = torch.rand(ids.shape, generator=g, device="cuda").topk(k, dim=1).indices
    ids = torch.gather(ids, 1, keep.sort(dim=1).values)
    dist, at = _pair_dist(x, ids, torch.float32).sort(dim=1, stable=True)
    return torch.gather(ids, 1, at).to(torch.int32), dist


def _half(case, base):
    return (base * FACTOR[case["data"]]).half()


class _Device:
    """A kNN graph in buffers of the caller's own, and the pristine graph a
    program that makes several indexes of it keeps aside."""

    def __init__(self, half, ids, dist):
        n, k = ids.shape
        new = lambda *shape: torch.zeros(*shape, dtype=torch.int32, device="cuda")
        self.ids, self.dist, self.data = ids, dist, half
        self.graph, self.nd = new(n, k), torch.zeros(n, k, device="cuda")
        self.rgraph, self.rd = new(n * 128), torch.zeros(n * 128, device="cuda")
        self.rnum, self.hybrid = new(n), new(n * 128)
        self.center = half.float().mean(0).half()
        self.norms = half.float().square().sum(1)
        st = capi.KnnState(n=n, dim=half.shape[1], k=k, device=torch.cuda.current_device(),
                           norm_factor=1.0)
        for name, t in (("graph", self.graph), ("reverse_graph", self.rgraph),
                        ("data", self.data), ("nei_distance", self.nd),
                        ("reverse_distance", self.rd), ("reverse_num", self.rnum),
                        ("center", self.center), ("hybrid_list", self.hybrid),
                        ("norms", self.norms)):
            setattr(st, name, t.data_ptr())
        self.state = capi.State(st)

    def prune(self, case):
        self.graph.copy_(self.ids)
        self.nd.copy_(self.dist)
        self.rnum.zero_()
        what = case["what"]
        if "/" in what:
            mode, metric = what.split("/")
            return capi.pruning_cfs(self.state, case["fd"], mode, metric, topm=case["topm"],
                                    thre=case["thre"])
        return capi.pruning(self.state, case["fd"], what, topm=case["topm"], thre=case["thre"])


def _use_stream(stream):
    capi.check(capi.lib().tagore_set_stream(stream.cuda_stream))


def prepare(case, seed):
    stream = torch.cuda.Stream()
    s = {"case": case, "stream": stream}
    if case["call"] == "knn":
        base = _base(case, seed)[0]
        s["pinned"] = torch.empty(base.shape, pin_memory=True)
        s["pinned"].copy_(base)
        s["base"] = s["pinned"].numpy()
        s["seed"] = seed
    elif case["call"] == "prune":
        base, _, grid, g = _base(case, seed)
        half = _half(case, base)
        s["dev"] = _Device(half, *_graph(half, grid, case["k"], g))
    else:
        base, queries, grid, g = _base(case, seed, case["nq"])
        n, k = case["n"], 32
        half = _half(case, base)
        if case["d"] % 4:  # the prune takes widths that are multiples of 4
            half = torch.nn.functional.pad(half, (0, -case["d"] % 4))
        dev = _Device(half.contiguous(), *_graph(half, grid, k, g))
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            _use_stream(stream)
            s["ep"] = dev.prune(dict(what="NSG", fd=24, topm=48, thre=1.0))
        rows = dev.graph.to(torch.int64)
        deg = rows[:, 0]
        offs = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        offs[1:] = deg.cumsum(0)
        s["offs"] = offs
        s["adj"] = rows[:, 1:][torch.arange(k - 1, device="cuda") < deg[:, None]].to(torch.int32)
        s["base"], s["queries"] = base, queries.contiguous()
    torch.cuda.synchronize()
    return s


class _Array:
    """A device buffer of the library as torch sees it."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False),
                                         "version": 2}


def run(s):
    case = s["case"]
    with torch.cuda.stream(s["stream"]):
        _use_stream(s["stream"])
        if case["call"] == "knn":
            s.pop("graph", None)  # the program is done with the graph of its last build
            st = capi.gnn_descent_host(s["base"], case["k"], case["iters"],
                                       rescale=case["rescale"], seed=s["seed"])
            s["graph"] = st
            return torch.as_tensor(_Array(st.st.nei_distance, (case["n"], case["k"]), st),
                                   device="cuda")
        if case["call"] == "prune":
            dev = s["dev"]
            ep = dev.prune(case)
            return {"ep": ep, "graph": dev.graph, "nei_distance": dev.nd,
                    "reverse_graph": dev.rgraph, "reverse_distance": dev.rd,
                    "reverse_num": dev.rnum, "hybrid_list": dev.hybrid}
        return capi.search(s["base"], s["offs"], s["adj"], s["ep"], s["queries"], case["L"],
                           case["k"], seed=SEARCH_SEED, stream=s["stream"].cuda_stream)


# ---- what a pass cannot do without ----

def work(case):
    n, d, k = case["n"], case["d"], case["k"]
    if case["call"] == "knn":
        # the FP32 base in, the rows out; one exact distance per edge
        return {"bytes": 4 * n * d + 8 * n * k, "flops": 3 * n * k * d}
    if case["call"] == "prune":
        fd, what = case["fd"], case["what"]
        # kNN rows and distances in, pruned rows and reverse edges out
        io = 8 * n * k + 4 * n * (fd + 1) + 8 * n * fd
        if what in ("CAGRA", "1-hop/rank"):
            return {"bytes": io, "flops": n * k * k}  # detour counts: one test per (list, id)
        rows = k * (k - 1) / 2 if what == "DPG" else 480  # rows scored per node
        return {"bytes": io + 2 * n * d, "flops": 3 * n * d * rows}
    # the queries in and ids out; L expansions of about 14 neighbours, each row
    # of the base read at most once
    rows = case["nq"] * case["L"] * 14
    return {"bytes": 4 * d * (min(n, rows) + case["nq"]) + 8 * case["nq"] * k,
            "flops": 3 * rows * d}


def tolerance(case):
    # Two runs of one build differ in the ids they miss: up to 0.0038 of the
    # distances' 2-norm, and single entries by up to 0.25 of the value (0.7 where
    # a row of 1M still held a far component).
    if case["call"] == "knn":
        return {"rel": 0.015, "max": 0.95}
    return "exact"


def exact(case, seed):
    """The exact kNN distances of the FP16 base, in 64 bits."""
    if case["call"] != "knn":
        return None
    base, _, grid, _ = _base(case, seed)
    factor, ten = np.float32(1.0), np.float32(10.0)
    if case["rescale"]:
        # vector 0's mean |x| brought into [0.5, 5] by powers of ten
        ave = float(base[0].double().abs().mean())
        while ave < 0.5:
            ave, factor = ave * 10, factor * ten
        while ave > 5:
            ave, factor = ave / 10, factor / ten
    half = (base * factor.item()).half()
    ids = _exact_rows(half, grid, min(case["k"] + 4, grid.shape[1] - 2))
    return _pair_dist(half, ids, torch.float64).sort(dim=1).values[:, :case["k"]].contiguous()
