"""What a program has the range-search library do, as measurable cases.

A case is one call (or one rebuild followed by a call) through the Python binding of the C ABI:

  search   Index.search, boxes and results on the GPU, ascending ids per query
  lookup   Index.search, one or a few boxes from numpy, ids back in numpy
  host     Index.search, a batch from numpy, ids left in the library's pinned host arena
  plain    Index.search with the one-query-per-block traversal
  counts   Index.counts, hit counts only
  plan     Plan.run_device, the captured pipeline that the serving loop replays
  refresh  BuildPlan.run over new positions, then a batch of queries on the new index
  build    Index.build of a new index, then a batch of queries on it

Results of a build are the answers of the queries that follow it: the index itself is opaque on the
device.  Ids are returned sorted, the default; without the sort their order is not defined.
"""
from __future__ import annotations

import importlib.util
import math
import pathlib
import sys

import numpy as np
import torch

ROOT = pathlib.Path(__file__).resolve().parent.parent
PKG = ROOT / "query-co-processing-on-heterogeneous-architectures_b200"

CLUSTERS, SIGMA = 64, 0.02  # the clustered sets: 64 Gaussians in the unit cube
KEYS = {"norm": 0, "ref": 1, "kmeans": 2}
KMEANS_ITERS = 10


def _load():
    if "qcp_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("qcp_b200", PKG / "__init__.py",
                                                      submodule_search_locations=[str(PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["qcp_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["qcp_b200"]


def _case(op, data, n, dims, q, vol, fanout=128, centre="data", grouped=False, key="norm"):
    """vol: lowest and highest box volume (log-uniform between them); for 8-D style boxes of one
    side length per dimension see `sides` in _boxes."""
    return {"op": op, "data": data, "n": n, "dims": dims, "q": q, "vol_lo": vol[0], "vol_hi": vol[1],
            "fanout": fanout, "centre": centre, "grouped": grouped, "key": key}


def listed():
    side8 = (0.125 ** 8, 0.125 ** 8)
    return [
        # an interactive lookup: one box, the ids wanted in host memory
        dict(_case("lookup", "uniform", 1_000_000, 3, 1, (1e-4, 1e-4)), name="lookup_1m_one_box"),
        # a small batch on a small index (about 100 hits each): launches and round trips
        dict(_case("search", "uniform", 1_000_000, 3, 1000, (1e-4, 1e-4), centre="uniform"), name="search_1m_1k"),
        # one serving batch: 64 requests of mixed volume on the captured pipeline
        dict(_case("plan", "clusters", 16_000_000, 3, 64, (1e-7, 1e-3)), name="plan_16m_64"),
        # the headline batch: clustered points, 10,000 cubes, about 10^9 ids
        dict(_case("search", "clusters", 16_000_000, 3, 10_000, (1e-6, 1e-2)), name="search_16m_clusters_10k"),
        # map tiles: many small squares over uniform 2-D points (about 640 hits each)
        dict(_case("search", "uniform", 64_000_000, 2, 100_000, (1e-5, 1e-5), centre="uniform"),
             name="search_64m_2d_100k"),
        # high-dimensional rectangles: a few hits per box, the traversal is the work
        dict(_case("search", "rects", 32_000_000, 8, 50_000, side8, centre="uniform"), name="search_32m_rect8d_50k"),
        # a batch from and to host memory; objects arrive cluster by cluster, so ids follow space
        dict(_case("host", "clusters", 2_000_003, 3, 5000, (1e-7, 1e-3), fanout=64, grouped=True),
             name="host_2m_grouped_5k"),
        # selectivity estimates: how many objects each box holds
        dict(_case("counts", "clusters", 16_000_000, 3, 10_000, (1e-6, 1e-2)), name="counts_16m_10k"),
        # moving objects: a captured rebuild of the whole index each tick, then that tick's queries
        dict(_case("refresh", "clusters", 16_000_000, 3, 1000, (1e-6, 1e-4)), name="refresh_16m"),
        # a new index from scratch: rectangles, the largest fan-out, an odd count
        dict(_case("build", "rects", 5_000_011, 4, 1000, (1e-5, 1e-5), fanout=256, centre="uniform"),
             name="build_5m_rect4d"),
        # a new index with k-means-clustered keys, for skewed data
        dict(_case("build", "clusters", 1_000_003, 3, 1000, (1e-6, 1e-4), key="kmeans"), name="build_1m_kmeans"),
        # the one-query-per-block traversal
        dict(_case("plain", "clusters", 2_000_000, 3, 1000, (1e-6, 1e-3)), name="plain_2m_1k"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["lookup", "search", "search", "search", "search", "plan", "host", "counts", "refresh", "build",
                     "plain"])
    data = rng.choice(["uniform", "clusters", "clusters", "rects"])
    dims = rng.choice([2, 3, 3, 8] if op == "search" else [2, 3, 3, 4, 5])
    top = {"lookup": 16e6, "search": 64e6, "plan": 16e6, "host": 4e6, "counts": 32e6, "refresh": 16e6, "build": 8e6,
           "plain": 4e6}[op]
    if dims > 3:
        top = min(top, 16e6)
    n = int(_log(rng, 2e4, top)) | 1
    q = {"lookup": int(_log(rng, 1, 16)), "search": int(_log(rng, 100, 50_000)), "plan": int(_log(rng, 4, 1024)),
         "host": int(_log(rng, 100, 8000)), "counts": int(_log(rng, 100, 20_000)), "refresh": 1000, "build": 1000,
         "plain": int(_log(rng, 50, 1500))}[op]
    # hits per query if the data were uniform; clustered data is denser around its objects
    cap = min(n / 8, {"search": 2e8, "host": 4e6, "plan": 2e6, "plain": 4e6}.get(op, 1e6) / q / 4)
    hits = _log(rng, 1, max(2.0, cap))
    vol = max(hits / n, 1e-7 if dims <= 3 else 0.05 ** dims)
    if data == "clusters":
        vol /= 16
    wide = rng.choice([1.0, 10.0])
    key = rng.choice(["norm", "ref", "kmeans"]) if op == "build" and dims <= 3 and data != "rects" else "norm"
    if key == "kmeans":
        n = min(n, 1_000_001)
    # leaves of five coordinate and id runs are used with the smaller and the larger fan-out
    runs = dims * (2 if data == "rects" else 1) + 1
    return _case(op, data, n, dims, q, (vol / wide, vol), fanout=rng.choice([64, 128, 128, 256] if runs != 5 else [64, 256]),
                 centre="data" if data == "clusters" else rng.choice(["data", "uniform"]),
                 grouped=data == "clusters" and rng.random() < 0.3, key=key)


# -- inputs ---------------------------------------------------------------------------------------
# The number of ids that come back depends on the data, and results are compared by shape: so a case
# has one set of objects and boxes, and the seed says in which order the program holds them (which
# gives every object another id and every box another place) and which coordinate is which axis.
def _objects(case, g):
    n, d = case["n"], case["dims"]
    dev = "cuda"
    if case["data"] == "uniform":
        return torch.rand((n, d), generator=g, device=dev), None
    if case["data"] == "rects":
        lo = torch.rand((n, d), generator=g, device=dev)
        side = torch.empty((n, d), device=dev).exponential_(1.0 / 0.002, generator=g)
        return torch.cat([lo, lo + side], 1), None
    centres = torch.rand((CLUSTERS, d), generator=g, device=dev)
    which = torch.randint(0, CLUSTERS, (n,), generator=g, device=dev)
    pts = torch.randn((n, d), generator=g, device=dev) * SIGMA + centres[which]
    return pts.clamp_(0.0, float(np.nextafter(np.float32(1.0), np.float32(0.0)))), which


def _boxes(case, objs, g):
    q, d, dev = case["q"], case["dims"], "cuda"
    if case["centre"] == "data":
        c = objs[torch.randint(0, case["n"], (q,), generator=g, device=dev)][:, :d]
    else:
        c = torch.rand((q, d), generator=g, device=dev)
    lo, hi = math.log(case["vol_lo"]), math.log(case["vol_hi"])
    vol = torch.exp(torch.rand((q, 1), generator=g, device=dev) * (hi - lo) + lo)
    half = vol ** (1.0 / d) * 0.5
    if case["data"] == "rects":  # sides of their own per dimension, between 0.4 and 1.6 of the mean
        half = half * (0.4 + 1.2 * torch.rand((q, d), generator=g, device=dev))
    return torch.cat([c - half, c + half], 1)


def _inputs(case, seed):
    n, d, q = case["n"], case["dims"], case["q"]
    g = torch.Generator(device="cuda")
    g.manual_seed(1234)
    objs, which = _objects(case, g)
    boxes = _boxes(case, objs, g)
    g.manual_seed(int(seed) * 7919 + 17)
    order = torch.randperm(n, generator=g, device="cuda")
    if case["grouped"]:  # cluster by cluster, the clusters and each one's objects in any order
        rank = torch.randperm(CLUSTERS, generator=g, device="cuda")
        order = order[torch.sort(rank[which[order]], stable=True).indices]
    axes = torch.randperm(d, generator=g, device="cuda")
    pair = torch.cat([axes, axes + d])
    objs = objs[order][:, pair if case["data"] == "rects" else axes].contiguous()
    return objs, boxes[torch.randperm(q, generator=g, device="cuda")][:, pair].contiguous()


def _plan_hits(case):
    return int(max(1 << 20, 4 * _hits(case) + case["q"] * 4096))


def prepare(case, seed):
    qcp = _load()
    objs, boxes = _inputs(case, seed)
    op = case["op"]
    rect = case["data"] == "rects"
    s = {"case": case, "qcp": qcp, "boxes": boxes}
    if op in ("lookup", "host", "counts"):
        s["host_boxes"] = boxes.cpu().numpy()
    if op == "build":
        s["objs"] = objs
    elif op == "refresh":
        s["objs"] = objs
        s["plan"] = qcp.BuildPlan(case["n"], case["dims"], is_rect=rect, fanout=case["fanout"])
    else:
        torch.cuda.synchronize()
        s["index"] = qcp.Index.build(objs, dims=case["dims"], is_rect=rect, fanout=case["fanout"], n=case["n"])
        if op == "plan":
            s["plan"] = qcp.Plan(s["index"], case["q"], _plan_hits(case))
    return s


# -- a pass ---------------------------------------------------------------------------------------
class _Owner:
    """A library result and what it hangs on; given back when the last array over it is gone."""

    def __init__(self, result, *parents):
        self.result, self.parents = result, parents

    def __del__(self):
        self.result.release()


class _DeviceView:
    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (int(ptr), False), "version": 3}


class _HostView:
    def __init__(self, owner, array):
        self.owner = owner
        self.__array_interface__ = dict(array.__array_interface__)


def _on_device(owner, offsets, ids, q, total):
    o = torch.as_tensor(_DeviceView(owner, offsets, q + 1, "<i8"), device="cuda")
    if not total:
        return o, torch.zeros(0, dtype=torch.int32, device="cuda")
    return o, torch.as_tensor(_DeviceView(owner, ids, total, "<i4"), device="cuda")


def _search(s, index, *parents, algo="batched"):
    q = s["case"]["q"]
    r = index.search(s["boxes"], algo=algo, q=q, result_mem=s["qcp"].MEM_DEVICE)
    return _on_device(_Owner(r, index, *parents), r.offsets, r.ids, q, r.total_hits)


def run(s):
    case, qcp = s["case"], s["qcp"]
    op = case["op"]
    if op == "search":
        return _search(s, s["index"])
    if op == "plain":
        return _search(s, s["index"], algo="plain")
    if op == "lookup":
        r = s["index"].search(s["host_boxes"])
        return r.offsets, r.ids
    if op == "host":
        r = s["index"].search(s["host_boxes"], copy=False)
        own = _Owner(r, s["index"])
        return np.asarray(_HostView(own, r.offsets)), np.asarray(_HostView(own, r.ids))
    if op == "counts":
        return s["index"].counts(s["host_boxes"])
    if op == "plan":
        q, total, offsets, ids = s["plan"].run_device(s["boxes"], q=case["q"])
        return _on_device((s["plan"], s["index"]), offsets, ids, q, total)
    if op == "refresh":
        return _search(s, s["plan"].run(s["objs"]), s["plan"])
    index = qcp.Index.build(s["objs"], dims=case["dims"], is_rect=case["data"] == "rects", fanout=case["fanout"],
                            n=case["n"], key_mode=KEYS[case["key"]],
                            kmeans_iters=KMEANS_ITERS if case["key"] == "kmeans" else 0)
    return _search(s, index)


# -- what a pass cannot do without ----------------------------------------------------------------
def _hits(case):
    """Expected ids of all queries together."""
    n, d = case["n"], case["dims"]
    steps, total = 64, 0.0
    for i in range(steps):
        f = (i + 0.5) / steps
        vol = case["vol_lo"] * (case["vol_hi"] / case["vol_lo"]) ** f
        side = vol ** (1.0 / d)
        if case["data"] == "clusters":
            # objects of the centre's own cluster within side / 2 of it, and a share of the others
            total += n / CLUSTERS * math.erf(side / (4 * SIGMA)) ** d + n * min(1.0, vol)
        else:
            total += n * min(1.0, vol)
    return case["q"] * total / steps


def work(case):
    n, d, q, F = case["n"], case["dims"], case["q"], case["fanout"]
    row = 4 * d * (2 if case["data"] == "rects" else 1)
    hits = _hits(case)
    # a query: its box, the coordinates of one node's objects (each object once), its ids read and written
    b = 8.0 * d * q + 8.0 * q + min(n, q * F) * row
    if case["op"] != "counts":
        b += 4.0 * min(n, hits) + 4.0 * hits
    flops = 0.0
    if case["op"] in ("refresh", "build"):
        # objects read, then written in key order with their ids and keys, and the nodes' boxes
        b += n * (2.0 * row + 4 + 8) + 8.0 * d * n / (F - 1)
        if case["key"] == "kmeans":
            flops = 3.0 * d * n * min(1024, n) * KMEANS_ITERS
    return {"bytes": b, "flops": flops}


def exact(case, seed):
    """The same answers by testing every object against every box, where that is quick."""
    if case["n"] * case["q"] * case["dims"] > 2e10 or _hits(case) > 5e7:
        return None
    objs, boxes = _inputs(case, seed)
    d = case["dims"]
    lo, hi = objs[:, :d].double(), objs[:, -d:].double()
    counts, ids = [], []
    for b in boxes.double():
        hit = torch.nonzero(((b[:d] <= hi) & (b[d:] >= lo)).all(1)).reshape(-1)
        counts.append(hit.numel())
        ids.append(hit.to(torch.int32))
    if case["op"] == "counts":
        return np.array(counts, np.uint64)
    offsets = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    ids = torch.cat(ids).cpu().numpy()
    if case["op"] in ("lookup", "host"):
        return offsets.astype(np.uint64), ids
    return offsets, ids
