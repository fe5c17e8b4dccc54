"""The counts that a user of this package has it do, as cases that can be timed and compared.

A case is one call (or one burst of requests) through the public entry points on a synthetic graph:

  device    TriangleCounter.count_device on a CSR that is already on the GPU
  host      TriangleCounter.count on numpy arrays: copies in, count, copies out
  batch     TriangleCounter.count_batch_device on a union of many graphs
  plan      the same union counted by a captured Plan
  dag       TriangleCounter.count_dag_device on one rank's oriented lists with ghosts (katric's local phase)
  strategy  count_device with one of the reference's intersection methods
  serve     a burst of requests to a Server, submitted and waited for

The graphs are of the three families the package generates on the host (G(n,m), RMAT with
(0.57, 0.19, 0.19, 0.05), 2D random geometric in Morton order), built here with torch on the GPU so that
a new graph takes well under a second: undirected, simple, both directions stored, lists sorted by id.
Sizes come from a case; which edges a graph has comes from the seed alone.
"""
import math
import random

import numpy as np
import torch

from katric_gb300 import Config, Graph, Server, TriangleCounter

GNM, RMAT, RGG = "gnm", "rmat", "rgg"
FAMILIES = (GNM, RMAT, RGG)
ABC = (0.57, 0.19, 0.19)  # RMAT quadrant probabilities a, b, c


# ---- the cases ------------------------------------------------------------------------------------


def listed():
    return [
        # one small uniform graph on the device: latency and launches (the smallest workload of the benchmark)
        dict(name="device-gnm-2e14", kind="device", family=GNM, n=1 << 14, degree=16.0, per_vertex=True),
        # an everyday request handed over as numpy arrays: 2^16 skewed edges, the median served graph
        dict(name="host-rmat-8e3", kind="host", family=RMAT, n=8191, degree=16.0, per_vertex=True),
        # a mid-sized skewed graph of an odd size on the device
        dict(name="device-rmat-1e6", kind="device", family=RMAT, n=1_000_003, degree=32.0, per_vertex=True),
        # the headline: RMAT scale 24, edge factor 16
        dict(name="device-rmat-2e24", kind="device", family=RMAT, n=1 << 24, degree=32.0, per_vertex=True),
        # a triangle-dense local graph of ordinary size
        dict(name="device-rgg-2e20", kind="device", family=RGG, n=1 << 20, degree=32.0, per_vertex=True),
        # the large triangle-dense graph: 2^24 points, average degree 32
        dict(name="device-rgg-2e24", kind="device", family=RGG, n=1 << 24, degree=32.0, per_vertex=True),
        # a skewed graph from host memory and back, copies and all: what shmetric's call site does
        dict(name="host-rmat-2e21", kind="host", family=RMAT, n=1 << 21, degree=24.0, per_vertex=True),
        # many graphs of uneven sizes in one launch sequence, default options
        dict(name="batch-512", kind="batch", graphs=512, log2_min=8.0, log2_max=17.0, degree_min=4.0, degree_max=64.0,
             mix=4, small_outdegree=0),
        # a captured plan over a smaller batch with the owner bound the autotuner picks for this workload
        dict(name="plan-96", kind="plan", graphs=96, log2_min=8.0, log2_max=16.0, degree_min=4.0, degree_max=64.0, mix=5,
             small_outdegree=48),
        # one rank of two: oriented lists of its vertices and ghosts
        dict(name="dag-rmat-7e5", kind="dag", family=RMAT, n=700_001, degree=32.0),
        # the reference's default strategy (merge) chosen by name
        dict(name="merge-rgg-2e18", kind="strategy", family=RGG, n=1 << 18, degree=24.0, method="merge"),
        # a burst of requests of the served size distribution, none of them resident
        dict(name="serve-30", kind="serve", requests=30, median_m=1 << 16, sigma=2.0, mix=6),
    ]


def draw(rng):
    def log_uniform(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["device"] * 5 + ["host"] * 2 + ["batch", "plan", "dag", "strategy", "serve"])
    family = rng.choice(FAMILIES)
    degree = round(rng.uniform(4.0, 64.0), 2)
    if kind in ("device", "host", "dag"):
        n = log_uniform(256, 1 << (24 if kind == "device" else 22))
        if family == RMAT:
            degree = min(degree, 40.0)
        # no dearer than the headline: fewer vertices where the drawn degree is high
        n = min(n, int((1 << (28 if kind == "device" and family != RMAT else 27)) / degree))
        case = dict(kind=kind, family=family, n=n, degree=degree)
        if kind != "dag":
            case["per_vertex"] = rng.random() < 0.7
        return case
    if kind in ("batch", "plan"):
        graphs = log_uniform(16, 512 if kind == "batch" else 192)
        return dict(kind=kind, graphs=graphs, log2_min=8.0, log2_max=round(rng.uniform(11.0, 17.0), 2), degree_min=4.0,
                    degree_max=round(rng.uniform(16.0, 64.0), 1), mix=rng.randrange(1 << 20),
                    small_outdegree=rng.choice([0, 0, 32, 48]))
    if kind == "strategy":
        return dict(kind=kind, family=family, n=log_uniform(256, 1 << 18), degree=round(rng.uniform(4.0, 32.0), 2),
                    method=rng.choice(["merge", "merge", "binary-search", "hybrid", "binary"]))
    return dict(kind="serve", requests=rng.randint(4, 40), median_m=log_uniform(1 << 13, 1 << 17),
                sigma=round(rng.uniform(0.5, 2.0), 2), mix=rng.randrange(1 << 20))


# ---- graphs on the GPU ----------------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _unique_sorted(keys):
    keys = keys.sort().values
    if keys.numel():
        keep = torch.ones_like(keys, dtype=torch.bool)
        torch.ne(keys[1:], keys[:-1], out=keep[1:])
        keys = keys[keep]
    return keys


def _simple_edges(u, v, n):
    """Distinct undirected edges without loops, as sorted keys u * n + v with u < v."""
    keys = torch.minimum(u, v).mul_(n).add_(torch.maximum(u, v))
    return _unique_sorted(keys[u != v])


def _uniform_edges(first, n, samples, gen):
    """Uniform pairs inside graph i's vertices [first[i], first[i] + n[i])."""
    base = torch.repeat_interleave(first, samples)
    span = torch.repeat_interleave(n, samples).double()
    ends = []
    for _ in range(2):
        r = torch.rand(base.numel(), generator=gen, device="cuda", dtype=torch.float64)
        ends.append(torch.minimum((r * span).long(), span.long() - 1) + base)
    return ends


def _rmat_edges(first, n, samples, gen):
    scales = [max(1, math.ceil(math.log2(x))) for x in n.tolist()]
    total = int(samples.sum())
    scale = torch.repeat_interleave(torch.tensor(scales, device="cuda"), samples) if len(set(scales)) > 1 else None
    u = torch.zeros(total, dtype=torch.int64, device="cuda")
    v = torch.zeros(total, dtype=torch.int64, device="cuda")
    for level in range(max(scales)):
        p = torch.rand(total, generator=gen, device="cuda")
        bu = p >= ABC[0] + ABC[1]
        bv = ((p >= ABC[0]) & ~bu) | (p >= sum(ABC))
        if scale is None:
            u.mul_(2).add_(bu)
            v.mul_(2).add_(bv)
        else:
            on = scale > level
            u = torch.where(on, 2 * u + bu, u)
            v = torch.where(on, 2 * v + bv, v)
    size = torch.repeat_interleave(n, samples)
    inside = (u < size) & (v < size)
    base = torch.repeat_interleave(first, samples)[inside]
    return [u[inside] + base, v[inside] + base]


def _spread16(x):
    """Bits of a 16-bit number moved to the even positions."""
    for shift, mask in ((8, 0x00FF00FF), (4, 0x0F0F0F0F), (2, 0x33333333), (1, 0x55555555)):
        x = (x | (x << shift)) & mask
    return x


def _rgg_edges(first, n, degree, gen):
    """Points uniform in a unit square per graph, ids in Morton order, edges below the radius."""
    graphs = torch.arange(len(n), device="cuda")
    who = torch.repeat_interleave(graphs, n)
    x = torch.rand(who.numel(), generator=gen, device="cuda", dtype=torch.float64)
    y = torch.rand(who.numel(), generator=gen, device="cuda", dtype=torch.float64)
    code = _spread16((x * 65536).long()) | (_spread16((y * 65536).long()) << 1) | (who << 32)
    code, order = code.sort()
    x, y = x[order], y[order]
    r = torch.sqrt(degree / (math.pi * n.double())).clamp(max=1.0)
    # cells are aligned squares of side 2^-k >= radius: contiguous in Morton order
    k = torch.floor(-torch.log2(r)).clamp(0, 16).long()
    kp, r2 = k[who], (r * r)[who]
    ids = torch.arange(who.numel(), device="cuda")
    start_of = first - (torch.cumsum(n, 0) - n)  # from a point's rank here to its vertex id
    got = []
    step = 1 << 20
    for a in range(0, who.numel(), step):
        s = slice(a, min(a + step, who.numel()))
        kk = kp[s]
        side = 1 << kk
        cx, cy = (x[s] * side).long(), (y[s] * side).long()
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                ox, oy = cx + dx, cy + dy
                ok = (ox >= 0) & (oy >= 0) & (ox < side) & (oy < side)
                shift = 2 * (16 - kk)
                cell = (_spread16(ox.clamp(min=0)) | (_spread16(oy.clamp(min=0)) << 1)) << shift
                cell = cell | (who[s] << 32)
                lo = torch.searchsorted(code, cell)
                hi = torch.searchsorted(code, cell + (1 << shift))
                lo = torch.maximum(lo, ids[s] + 1)  # each pair once
                count = ((hi - lo).clamp(min=0)) * ok
                i = torch.repeat_interleave(ids[s], count)
                at = torch.cumsum(count, 0) - count
                j = torch.arange(i.numel(), device="cuda") + torch.repeat_interleave(lo - at, count)
                near = (x[i] - x[j]) ** 2 + (y[i] - y[j]) ** 2 < r2[i]
                i, j = i[near], j[near]
                off = start_of[who[i]]
                got.append((i + off, j + off))
    return [torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got])]


def _edges(family, first, n, degree, gen):
    if family == RGG:
        return _rgg_edges(first, n, degree, gen)
    samples = (n.double() * degree / 2).round().long()
    return (_uniform_edges if family == GNM else _rmat_edges)(first, n, samples, gen)


def _edge_keys(specs, seed):
    """Sorted keys (u * n + v, u < v) of the disjoint union of graphs [(family, n, degree)], and their first vertices."""
    sizes = torch.tensor([s[1] for s in specs], device="cuda")
    first = torch.cumsum(sizes, 0) - sizes
    n = int(sizes.sum())
    gen = _generator(seed)
    us, vs = [], []
    for family in FAMILIES:
        at = [i for i, s in enumerate(specs) if s[0] == family]
        if at:
            degree = torch.tensor([specs[i][2] for i in at], device="cuda", dtype=torch.float64)
            u, v = _edges(family, first[at], sizes[at], degree, gen)
            us.append(u)
            vs.append(v)
    u, v = (us[0], vs[0]) if len(us) == 1 else (torch.cat(us), torch.cat(vs))
    return _simple_edges(u, v, n), n, torch.cat([first, torch.tensor([n], device="cuda")])


def _csr(keys, n):
    """CSR of undirected edge keys, both directions, lists sorted by id."""
    u = torch.div(keys, n, rounding_mode="floor")
    both = torch.cat([keys, (keys - u * n) * n + u]).sort().values
    return _lists(both, n)


def _lists(keys, n):
    """first_out and head of sorted keys tail * n + head."""
    tail = torch.div(keys, n, rounding_mode="floor")
    head = (keys - tail * n).to(torch.int32)
    first_out = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(tail, minlength=n), 0, out=first_out[1:])
    return first_out, head


def _oriented(keys, n):
    """Sorted keys of the edges turned from the smaller to the larger (degree, id)."""
    u = torch.div(keys, n, rounding_mode="floor")
    v = keys - u * n
    degree = torch.bincount(u, minlength=n) + torch.bincount(v, minlength=n)
    swap = degree[u] > degree[v]  # u < v: equal degrees stay
    return torch.where(swap, v * n + u, keys).sort().values


def _rank_lists(keys, n):
    """What rank 0 of two holds after katric's preprocessing: the edges that touch its half of the vertices, oriented
    by the whole graph's (degree, id).  Its vertices come first, then the other half as ghosts."""
    local = n // 2
    turned = _oriented(keys, n)
    u = torch.div(turned, n, rounding_mode="floor")
    v = turned - u * n
    return turned[(u < local) | (v < local)]


def _specs(case):
    """(family, n, degree) of every graph of a case: the same for every seed."""
    if "family" in case:
        return [(case["family"], case["n"], case["degree"])]
    r = random.Random(case["mix"])
    got = []
    if case["kind"] == "serve":
        for i in range(case["requests"]):
            m = min(max(r.lognormvariate(math.log(case["median_m"]), case["sigma"]), 1000.0), 2.0 ** 22)
            degree = r.uniform(4.0, 64.0)
            got.append((FAMILIES[i % 3], max(64, round(2 * m / degree)), degree))
    else:
        for i in range(case["graphs"]):
            n = round(2 ** r.uniform(case["log2_min"], case["log2_max"]))
            got.append((FAMILIES[i % 3], n, r.uniform(case["degree_min"], case["degree_max"])))
    return got


# ---- what a program keeps between calls -----------------------------------------------------------

_kept = {}


def _counter():
    if "counter" not in _kept:
        _kept["counter"] = TriangleCounter(0)
    return _kept["counter"]


def _server():
    if "server" not in _kept:
        _kept["server"] = Server(memory_budget=8 << 30, max_batch_nnz=1 << 24)
    return _kept["server"]


def prepare(case, seed):
    kind = case["kind"]
    keys, n, first = _edge_keys(_specs(case), seed)
    state = {"kind": kind, "counter": _counter()}
    if kind == "dag":
        keys = _rank_lists(keys, n)
        state["fo"], state["head"] = _lists(keys, n)
    else:
        state["fo"], state["head"] = _csr(keys, n)
    state["n"], state["nnz"] = n, state["head"].numel()
    state["conf"] = Config(intersection_method=case.get("method", "auto"),
                           small_outdegree=case.get("small_outdegree", 0))
    if kind in ("host", "serve"):
        fo = state.pop("fo").cpu().numpy().view(np.uint64)
        head = state.pop("head").cpu().numpy().view(np.uint32)
        if kind == "host":
            state.update(fo=fo, head=head, per_vertex=case["per_vertex"])
            return state
        at = first.tolist()
        state["graphs"] = [Graph(fo[a:b + 1] - fo[a], head[int(fo[a]):int(fo[b])] - np.uint32(a))
                           for a, b in zip(at[:-1], at[1:])]
        state["server"] = _server()
        return state
    state["totals"] = torch.zeros(max(1, len(first) - 1), dtype=torch.int64, device="cuda")
    if case.get("per_vertex", True):
        state["pv"] = torch.zeros(n, dtype=torch.int64, device="cuda")
    if kind in ("batch", "plan"):
        state["first"], state["graphs"] = first, len(first) - 1
    if kind == "plan":
        state["plan"] = state["counter"].plan_batch(
            state["fo"].data_ptr(), state["head"].data_ptr(), n, state["nnz"], first.data_ptr(), state["graphs"],
            state["totals"].data_ptr(), state["pv"].data_ptr(), state["conf"])
    return state


def run(state):
    kind, c = state["kind"], state["counter"]
    if kind == "host":
        total, pv = c.count(state["fo"], state["head"], state["conf"], per_vertex=state["per_vertex"])
        return [total] if pv is None else [total, pv.view(np.int64)]
    if kind == "serve":
        ids = [state["server"].submit(g, borrow=True) for g in state["graphs"]]
        got = [state["server"].wait(i) for i in ids]
        return [np.array([g[0] for g in got], dtype=np.int64)] + [g[1].view(np.int64) for g in got]
    stream = torch.cuda.current_stream().cuda_stream
    pv = state.get("pv")
    if kind == "plan":
        state["plan"].launch(stream)
    elif kind == "batch":
        c.count_batch_device(state["fo"].data_ptr(), state["head"].data_ptr(), state["n"], state["nnz"],
                             state["first"].data_ptr(), state["graphs"], state["totals"].data_ptr(), pv.data_ptr(),
                             state["conf"], stream)
    else:
        call = c.count_dag_device if kind == "dag" else c.count_device
        call(state["fo"].data_ptr(), state["head"].data_ptr(), state["n"], state["nnz"], state["totals"].data_ptr(),
             pv.data_ptr() if pv is not None else None, state["conf"], stream)
    return [state["totals"]] if pv is None else [state["totals"], pv]


def work(case):
    """Bytes of one pass: first_out and head read once, the totals and per-vertex counts written once."""
    specs = _specs(case)
    n = sum(s[1] for s in specs)
    nnz = sum(s[1] * s[2] for s in specs)
    if case["kind"] == "dag":  # half of the directions, and about three quarters of the edges (one end local)
        nnz *= 3 / 8
    per_vertex = 8 * n if case.get("per_vertex", True) else 0
    return {"bytes": int(8 * (n + 1) + 4 * nnz + per_vertex + 8 * len(specs)), "flops": 0}


# ---- the same counts with plain torch -------------------------------------------------------------


def _count_plain(keys, n):
    """(triangles, per-vertex counts) of undirected edge keys by wedge lookup, or None where that takes too long."""
    turned = _oriented(keys, n)
    tail = torch.div(turned, n, rounding_mode="floor")
    head = turned - tail * n
    first_out, _ = _lists(turned, n)
    wedges = first_out[head + 1] - first_out[head]
    if int(wedges.sum()) > 1_500_000_000:
        return None
    ends = torch.cumsum(wedges, 0)
    pv = torch.zeros(n, dtype=torch.int64, device="cuda")
    total, a, step = 0, 0, 1 << 26
    while a < turned.numel():
        done = int(ends[a - 1]) if a else 0
        b = max(a + 1, int(torch.searchsorted(ends, done + step, right=True)))
        count = wedges[a:b]
        e = torch.repeat_interleave(torch.arange(a, min(b, turned.numel()), device="cuda"), count)
        at = torch.cumsum(count, 0) - count
        third = head[torch.arange(e.numel(), device="cuda") + torch.repeat_interleave(first_out[head[a:b]] - at, count)]
        probe = tail[e] * n + third
        place = torch.searchsorted(turned, probe).clamp(max=turned.numel() - 1)
        hit = turned[place] == probe
        for corner in (tail[e[hit]], head[e[hit]], third[hit]):
            pv += torch.bincount(corner, minlength=n)
        total += int(hit.sum())
        a = b
    return total, pv


def exact(case, seed):
    keys, n, first = _edge_keys(_specs(case), seed)
    if case["kind"] == "dag":
        turned = _rank_lists(keys, n)
        u = torch.div(turned, n, rounding_mode="floor")
        v = turned - u * n
        keys = _simple_edges(u, v, n)
    got = _count_plain(keys, n)
    if got is None:
        return None
    total, pv = got
    if case["kind"] in ("batch", "plan", "serve"):
        prefix = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cumsum(pv, 0)])
        totals = torch.div(prefix[first[1:]] - prefix[first[:-1]], 3, rounding_mode="floor")
        if case["kind"] == "serve":
            at = first.tolist()
            return [totals] + [pv[a:b] for a, b in zip(at[:-1], at[1:])]
        return [totals, pv]
    totals = total if case["kind"] == "host" else torch.tensor([total], device="cuda")
    return [totals, pv] if case.get("per_vertex", True) else [totals]
