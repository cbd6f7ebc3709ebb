"""Measured workloads of the R-tree library, through its public Python entry
points: bulk loads, window-query batches of every form, and text ingest.

Boxes and windows follow curtree_b200/datasets.py (unit-square draws scaled by
2^15, positional ids), drawn on the GPU so that preparing a case is quick.

Pair lists come back in the canonical (window, box id) order of
`canonicalize`, the order in which the reference's drivers put a result
before they use it; batches of hundreds of millions of pairs and more come
back as the per-window counts and digests of `PairDigest`, as such results
are checked in earnest (the order of the pairs themselves is unspecified and
differs from run to run).
"""
import math
import tempfile

import numpy as np
import torch

import curtree_b200 as C
from curtree_b200 import datasets as D

SCALE = 2.0 ** 15
FANOUTS = (8, 10, 10, 16, 16, 32, 3, 7, 20, 48)


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # An interactive lookup: a handful of windows against a small tree.
        # Launches and latency are all of it.
        dict(name="lookup_16", kind="query", boxes="uniform", n=100_003, fanout=10,
             windows="uniform", nq=16, hi=1e-2),
        # The reference's own small case: 1M boxes, 10k windows, fanout 10,
        # the drop-in query and its pairs in canonical order.
        dict(name="batch_10k", kind="query", boxes="uniform", n=1_000_000, fanout=10,
             windows="uniform", nq=10_000, hi=1e-2),
        # The plain per-batch form with window offsets over windows of very
        # uneven size.
        dict(name="plain_mixed_20k", kind="plain", boxes="uniform", n=3_000_017, fanout=16,
             windows="mixed", nq=20_011, lo=1e-5, hi=2e-2),
        # A large batch of small windows (about ten hits each) through the
        # drop-in query: the persistent form with library defaults.
        dict(name="small_windows_1m", kind="query", boxes="uniform", n=10_000_000, fanout=10,
             windows="uniform", nq=1_000_000, hi=1e-3),
        # The headline batch's distribution (sides 1e-5 .. 1e-1, half of the
        # windows centred on boxes), replayed as a graph plan with the
        # autotuner's options, 1.3e9 pairs.
        dict(name="plan_mixed_250k", kind="plan", boxes="uniform", n=10_000_000, fanout=16,
             windows="mixed", nq=250_000, lo=1e-5, hi=1e-1, warps=16, chunk=1024, stage=2),
        # Road-like geometry (thin boxes along segments, half of the windows
        # points, a tenth covering more than 1% of the domain), streamed
        # through one output buffer.
        dict(name="stream_road_40k", kind="stream", boxes="road", n=5_000_011, fanout=16,
             windows="road", nq=40_009, cap=1 << 29),
        # Drop-in, in-place bulk loads: a small set, where launches count, and
        # the reference's small case.
        dict(name="load_20k", kind="load", boxes="uniform", n=20_011, fanout=10),
        dict(name="load_1m", kind="load", boxes="uniform", n=1_000_000, fanout=10),
        # Out-of-place bulk loads into the caller's arrays: the headline tree,
        # and the large clustered set with duplicates and points.
        dict(name="build_10m", kind="build", boxes="uniform", n=10_000_000, fanout=16),
        dict(name="build_clustered_100m", kind="build", boxes="clustered", n=100_000_000, fanout=10),
        # Reading the reference's MBR text format from a file.
        dict(name="ingest_400k", kind="ingest", boxes="uniform", n=400_009),
    ]


def _log(rng, lo, hi):
    """A whole number log-uniform in [lo, hi], odd and even alike."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "plain", "plan", "stream", "load", "build", "build", "ingest"])
    f = rng.choice(FANOUTS)
    if kind == "query":
        if rng.random() < 0.5:  # small and ordinary batches, sides up to 1e-2
            n, nq = _log(rng, 10_000, 3_000_000), _log(rng, 1, 30_000)
            return dict(kind=kind, boxes="uniform", n=n, fanout=f, windows="uniform", nq=nq, hi=1e-2)
        # large batches of small windows
        n, nq = _log(rng, 1_000_000, 10_000_000), _log(rng, 32_768, 1_000_000)
        return dict(kind=kind, boxes=rng.choice(["uniform", "clustered"]), n=n, fanout=f,
                    windows="uniform", nq=nq, hi=1e-3)
    if kind == "plain":
        return dict(kind=kind, boxes="uniform", n=_log(rng, 10_000, 5_000_000), fanout=f,
                    windows="mixed", nq=_log(rng, 10, 40_000), lo=1e-5, hi=rng.choice([1e-3, 1e-2, 2e-2]))
    if kind == "plan":
        w = rng.choice([8, 16, 32])
        return dict(kind=kind, boxes="uniform", n=_log(rng, 1_000_000, 10_000_000), fanout=f,
                    windows="mixed", nq=_log(rng, 1_000, 250_000), lo=1e-5, hi=1e-1, warps=w,
                    chunk=rng.choice([1024, 4096]), stage=rng.choice([0, 2, 3]))
    if kind == "stream":
        return dict(kind=kind, boxes="road", n=_log(rng, 500_000, 5_000_000), fanout=f,
                    windows="road", nq=_log(rng, 2_000, 40_000), cap=1 << 29)
    if kind == "load":
        return dict(kind=kind, boxes="uniform", n=_log(rng, 2, 3_000_000), fanout=f)
    if kind == "build":
        return dict(kind=kind, boxes=rng.choice(["uniform", "clustered", "clustered", "road"]),
                    n=_log(rng, 100_000, 60_000_000), fanout=f)
    return dict(kind=kind, boxes="uniform", n=_log(rng, 1_000, 400_000))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * (int(seed) + 1))
    return g


def _rand(g, n):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _sides(cx, cy, w, h):
    """Boxes [c - w/2, c + w/2] rounded once to fp32, scaled by 2^15."""
    f = lambda v: v.to(torch.float32) * SCALE
    n = cx.numel()
    return C.BBox(f(cx - w / 2), f(cy - h / 2), f(cx + w / 2), f(cy + h / 2),
                  torch.arange(n, dtype=torch.int32, device="cuda"))


def _concat(parts):
    cat = lambda name: torch.cat([getattr(p, name) for p in parts])
    b = C.BBox(cat("xmin"), cat("ymin"), cat("xmax"), cat("ymax"), cat("id"))
    b.id = torch.arange(b.sz, dtype=torch.int32, device="cuda")
    return b


def _uniform(g, n):
    return _sides(_rand(g, n), _rand(g, n), _rand(g, n) * 1e-3, _rand(g, n) * 1e-3)


def _clustered(g, n):
    """1000 Gaussians (sigma log-uniform in [1e-4, 1e-2]) plus 10% uniform
    background, log-normal sides, 1% points, 1% exact duplicates."""
    mu = torch.rand(1000, 2, generator=g, device="cuda", dtype=torch.float64)
    sig = torch.exp(math.log(1e-4) + math.log(100.0) * _rand(g, 1000))
    parts = []
    for a in range(0, n, 20_000_000):
        m = min(20_000_000, n - a)
        k = torch.randint(0, 1000, (m,), generator=g, device="cuda")
        norm = lambda: torch.randn(m, generator=g, device="cuda", dtype=torch.float64)
        x, y = mu[k, 0] + sig[k] * norm(), mu[k, 1] + sig[k] * norm()
        bg = (_rand(g, m) < 0.1) | (x < 0) | (x >= 1) | (y < 0) | (y >= 1)
        x, y = torch.where(bg, _rand(g, m), x), torch.where(bg, _rand(g, m), y)
        point = _rand(g, m) < 0.01
        w = torch.exp(math.log(1e-4) + norm()).masked_fill_(point, 0.0)
        h = torch.exp(math.log(1e-4) + norm()).masked_fill_(point, 0.0)
        b = _sides(x, y, w, h)
        src = torch.arange(m, device="cuda")
        src = torch.where(_rand(g, m) < 0.01, torch.randint(0, m, (m,), generator=g, device="cuda"), src)
        parts.append(C.BBox(b.xmin[src], b.ymin[src], b.xmax[src], b.ymax[src], b.id))
    return parts[0] if len(parts) == 1 else _concat(parts)


def _road(g, n):
    """Centres along 100 random segments, Pareto(1.5) long sides, aspect
    ratios up to 1e4."""
    p = torch.rand(100, 4, generator=g, device="cuda", dtype=torch.float64)
    parts = []
    for a in range(0, n, 20_000_000):
        m = min(20_000_000, n - a)
        k = torch.randint(0, 100, (m,), generator=g, device="cuda")
        t = _rand(g, m)
        jitter = lambda: 1e-4 * torch.randn(m, generator=g, device="cuda", dtype=torch.float64)
        x = (p[k, 0] + t * (p[k, 2] - p[k, 0]) + jitter()).clamp_(0.0, 1.0 - 1e-9)
        y = (p[k, 1] + t * (p[k, 3] - p[k, 1]) + jitter()).clamp_(0.0, 1.0 - 1e-9)
        long = (1e-6 * (1.0 - _rand(g, m)) ** (-1.0 / 1.5)).clamp_(max=0.5)
        short = long / torch.exp(_rand(g, m) * math.log(1e4))
        flat = _rand(g, m) < 0.5
        parts.append(_sides(x, y, torch.where(flat, long, short), torch.where(flat, short, long)))
    return parts[0] if len(parts) == 1 else _concat(parts)


def _boxes(case, g):
    return {"uniform": _uniform, "clustered": _clustered, "road": _road}[case["boxes"]](g, case["n"])


def _windows(case, g, b):
    nq = case["nq"]
    x, y = _rand(g, nq), _rand(g, nq)
    if case["windows"] == "uniform":
        s = _rand(g, nq) * case["hi"]
    elif case["windows"] == "mixed":
        s = torch.exp(math.log(case["lo"]) + _rand(g, nq) * math.log(case["hi"] / case["lo"]))
        pick = torch.randint(0, b.sz, (nq,), generator=g, device="cuda")
        at = lambda lo, hi: (lo[pick].double() + hi[pick].double()) / 2 / SCALE
        on_box = _rand(g, nq) < 0.5
        x, y = torch.where(on_box, at(b.xmin, b.xmax), x), torch.where(on_box, at(b.ymin, b.ymax), y)
    else:  # road: half points, 40% small, 10% large
        u = _rand(g, nq)
        small = torch.exp(math.log(1e-5) + _rand(g, nq) * math.log(100.0))
        large = 0.1 + 0.2 * _rand(g, nq)
        s = torch.where(u < 0.5, torch.zeros_like(u), torch.where(u < 0.9, small, large))
    return _sides(x, y, s, s)


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    b = _boxes(case, g)
    st = dict(case=case, kind=kind)
    if kind == "ingest":
        text = D.mbr_csv_text(b.to_host(), seed=int(seed) + 1)
        st["file"] = tempfile.NamedTemporaryFile(prefix="mbr_", suffix=".csv")
        st["file"].write(text)
        st["file"].flush()
        return st
    if kind == "build":
        st["boxes"] = b
        return st
    if kind == "load":
        st["source"], st["boxes"] = b, C.BBox.empty(b.sz)
        return st
    st["windows"] = _windows(case, g, b)
    st["boxes"], st["rt"] = C.build_into(b, case["fanout"])
    if kind == "plan":
        opts = dict(warps_per_cta=case["warps"], chunk=case["chunk"], stage_levels=case["stage"])
        pairs = C.query_stats(st["rt"], st["boxes"], st["windows"])["hits"]
        cap = C.query_capacity(pairs, chunk=case["chunk"])
        st["fid"] = torch.empty(cap, dtype=torch.int32, device="cuda")
        st["tid"] = torch.empty(cap, dtype=torch.int32, device="cuda")
        st["result"] = C.new_result_block()
        st["plan"] = C.Plan(st["rt"], st["boxes"], st["windows"], st["fid"], st["tid"],
                            st["result"], **opts)
    elif kind in ("query", "plain"):  # the program's own arrays for the pairs, -1 past the last one
        cap = _room(case)
        st["fid"], st["tid"] = (torch.full((cap,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
        if kind == "plain":
            st["result"] = C.new_result_block()
            st["offsets"] = torch.zeros(case["nq"] + 1, dtype=torch.int64, device="cuda")
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
class _Span:
    """A device array the library allocated, for torch's view of it; the view
    keeps its owner alive."""

    def __init__(self, owner, ptr, n, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (int(ptr), False),
                                         "version": 2}


def _view(owner, ptr, n, kind="<i4"):
    if n == 0:
        return torch.empty(0, dtype=torch.int32 if kind == "<i4" else torch.float32, device="cuda")
    return torch.as_tensor(_Span(owner, ptr, n, kind), device="cuda")


def _box_list(b):
    return [b.xmin, b.ymin, b.xmax, b.ymax, b.id]


def _node_list(rt):
    s, n = rt.s, rt.sz
    return ([_view(rt, p, n, "<f4") for p in (s.xmin, s.ymin, s.xmax, s.ymax)] +
            [_view(rt, p, n) for p in (s.pos, s.len)])


def run(st):
    kind = st["kind"]
    if kind == "query":  # drop-in query; the pairs into the program's arrays, in canonical order
        pairs = C.bfs_frontier(st["rt"], st["boxes"], st["windows"])
        n = pairs.sz
        fid, tid = st["fid"][:n], st["tid"][:n]
        fid.copy_(_view(pairs, pairs.s.fid, n))
        tid.copy_(_view(pairs, pairs.s.tid, n))
        C.canonicalize(fid, tid)
        return {"pairs": n, "fid": st["fid"], "tid": st["tid"]}
    if kind == "plain":  # into the program's arrays, in canonical order within the windows' offsets
        C.query_into(st["rt"], st["boxes"], st["windows"], st["fid"], st["tid"], st["result"],
                     st["offsets"], C.CRT_QUERY_PLAIN)
        n = C.read_result(st["result"])["count"]
        C.canonicalize(st["fid"][:n], st["tid"][:n])
        return {"pairs": n, "fid": st["fid"], "tid": st["tid"], "offsets": st["offsets"]}
    if kind == "plan":
        st["plan"].launch()
        n = C.read_result(st["result"])["count"]
        d = C.PairDigest(st["windows"].sz)
        d.add(st["fid"], st["tid"], n=n)
        return {"pairs": n, "counts": d.counts, "hashes": d.hashes, "bad": d.bad}
    if kind == "stream":
        d = C.PairDigest(st["windows"].sz)
        got = C.query_stream(st["rt"], st["boxes"], st["windows"],
                             lambda fid, tid, first: d.add(fid, tid, first), capacity=st["case"]["cap"])
        return {"pairs": got["pairs"], "counts": d.counts, "hashes": d.hashes, "bad": d.bad}
    if kind == "load":  # in place: the boxes arrive in the arrays that the load then sorts
        for dst, src in zip(_box_list(st["boxes"]), _box_list(st["source"])):
            dst.copy_(src)
        rt = C.RTree(st["case"]["fanout"])
        C.build_rtree(st["boxes"], rt)
        return {"boxes": _box_list(st["boxes"]), "nodes": _node_list(rt)}
    if kind == "build":
        out, rt = C.build_into(st["boxes"], st["case"]["fanout"])
        return {"boxes": _box_list(out), "nodes": _node_list(rt)}
    return {"boxes": _box_list(C.read_mbr_csv(st["file"].name))}


# ---------------------------------------------------------------------------
# Work and exact values
# ---------------------------------------------------------------------------
def _expected_pairs(case):
    """Pairs per batch from the distributions' moments (uniform density)."""
    n, nq = case["n"], case["nq"]
    if case["windows"] == "road":
        return nq * (0.1 * n * 0.0433)  # mean square of the large sides
    if case["windows"] == "uniform":
        s1, s2 = case["hi"] / 2, case["hi"] ** 2 / 3
    else:
        r = math.log(case["hi"] / case["lo"])
        s1, s2 = (case["hi"] - case["lo"]) / r, (case["hi"] ** 2 - case["lo"] ** 2) / (2 * r)
    w = 5e-4 if case["boxes"] == "uniform" else 1.65e-4  # mean box side
    return nq * n * (s2 + 2 * s1 * w + w * w)


def _room(case):
    """Pairs to make room for: the expected count and eight deviations of a sum
    of windows that may each meet the densest spot."""
    most = case["n"] * (1e-3 if case["boxes"] == "clustered" else (case["hi"] + 1e-3) ** 2)
    return int(1.2 * _expected_pairs(case) + 8 * math.sqrt(case["nq"]) * most) + 4096


def _nodes(n, fanout):
    total = 0
    while n > 1:
        n = -(-n // fanout)
        total += n
    return total


def work(case):
    n = case["n"]
    if case["kind"] == "ingest":  # about 65 bytes of text in, 20 bytes of box out
        return {"bytes": 85.0 * n, "flops": 0}
    if case["kind"] in ("build", "load"):  # boxes in, boxes and nodes out
        return {"bytes": 40.0 * n + 24.0 * _nodes(n, case["fanout"]), "flops": 0}
    # windows in, hit boxes read once, pairs out (counts and digests where the
    # pairs are consumed by the digest, which reads them again)
    p = _expected_pairs(case)
    digest = case["kind"] in ("plan", "stream")
    b = 16.0 * case["nq"] + 20.0 * min(p, n) + 8.0 * p
    return {"bytes": b + (8.0 * p + 16.0 * case["nq"] if digest else 0), "flops": 0}


def _dilate(v):
    for s, m in ((8, 0x00FF00FF), (4, 0x0F0F0F0F), (2, 0x33333333), (1, 0x55555555)):
        v = (v | (v << s)) & m
    return v


def _exact_tree(b, fanout):
    """The bulk load in plain torch: stable sort by Morton key of the truncated
    centre, then min/max over runs of `fanout`."""
    q = lambda lo, hi: ((lo + hi) / 2).to(torch.float64).clamp(min=0, max=2.0 ** 32 - 1).to(torch.int64) & 0xFFFF
    key = (_dilate(q(b.ymin, b.ymax)) << 1) | _dilate(q(b.xmin, b.xmax))
    key = torch.where(key >= 2 ** 31, key - 2 ** 32, key)
    order = torch.sort(key, stable=True).indices
    boxes = [t[order].double() for t in _box_list(b)[:4]] + [b.id[order]]
    levels, child, first = [], boxes[:4], None
    while child[0].numel() > 1:
        n = child[0].numel()
        m = -(-n // fanout)
        pad = m * fanout - n
        red = []
        for i, t in enumerate(child):
            fill = math.inf if i < 2 else -math.inf
            t = torch.cat([t, torch.full((pad,), fill, dtype=t.dtype, device=t.device)]).view(m, fanout)
            red.append(t.amin(1) if i < 2 else t.amax(1))
        start = torch.arange(m, device="cuda") * fanout
        levels.append(red + [start, (n - start).clamp(max=fanout)])
        child = red
    total = sum(l[0].numel() for l in levels)
    at, below = total, total  # leaf-parents point past the nodes, at box slots
    for l in levels:
        l[4] = l[4] + below
        at -= l[0].numel()
        below = at
    if not levels:
        return {"boxes": boxes, "nodes": [None] * 6}
    nodes = [torch.cat([l[i] for l in reversed(levels)]) for i in range(6)]
    return {"boxes": boxes, "nodes": nodes[:4] + [t.int() for t in nodes[4:]]}


def exact(case, seed):
    """Sorted boxes and nodes of a load; the other cases' outputs are whole
    numbers, or (ingest) the text's own values rounded once."""
    if case["kind"] in ("load", "build"):
        return _exact_tree(_boxes(case, _gen(seed)), case["fanout"])
    if case["kind"] == "ingest":
        st = prepare(case, seed)
        v = np.loadtxt(st["file"].name, delimiter=",", usecols=(0, 1, 2, 3, 4), ndmin=2)
        box = [np.minimum(v[:, 0], v[:, 2]), np.minimum(v[:, 1], v[:, 3]),
               np.maximum(v[:, 0], v[:, 2]), np.maximum(v[:, 1], v[:, 3])]
        return {"boxes": box + [v[:, 4].astype(np.int32)]}
    return None
