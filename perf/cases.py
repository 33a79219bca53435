"""The work that a user of this library has it do, as measurable cases.

Every case goes through the public entry points: the Python classes of
``parallel_distance_oracle_gb300.pado`` and, where a program keeps page-locked
or device arrays of its own, the C ABI behind them.  Graphs are the generators'
of this repository (R-MAT, Erdos-Renyi, grids with long-range edges) with its
benchmark's parameters, drawn here on the GPU from a seed so that inputs are
quick to make.  All outputs are whole numbers (labels, distances, ids), so no
case has an inexact reference.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from parallel_distance_oracle_gb300 import _lib, graphs, pado

# A service that prepares graph after graph keeps this much scratch reserved.
SCRATCH_KEEP = 2 << 30


# ---------------------------------------------------------------------------
# What is measured.
# ---------------------------------------------------------------------------

def listed():
    return [
        # Labeling, smallest: one small social-like graph, as when a program
        # labels a neighbourhood on request.  Launches and set-up decide.
        {"name": "label_tiny", "op": "label", "graph": "rmat", "scale": 10, "factor": 8, "weighted": False,
         "roots": 50, "batch": 1024, "ranked": False},
        # Labeling, headline: the benchmark's R-MAT s20/ef16 from a ranked
        # page-locked CSR to exported labels and bit-parallel rows.
        {"name": "label_rmat20", "op": "label", "graph": "rmat", "scale": 20, "factor": 16, "weighted": False,
         "roots": 64, "batch": 1024, "ranked": True},
        # Labeling, long lists: a sparse random graph of odd size in original
        # ids with its vertex order, the many-graph workload's larger kind.
        {"name": "label_er", "op": "label", "graph": "er", "n": 20011, "factor": 6, "weighted": False,
         "roots": 50, "batch": 512, "ranked": False},
        # Weighted labeling: the benchmark's R-MAT s18/ef8, weights 1..100.
        {"name": "label_weighted18", "op": "label", "graph": "rmat", "scale": 18, "factor": 8, "weighted": True,
         "roots": 0, "batch": 512, "ranked": True},
        # Many graphs labeled together, half Erdos-Renyi and half grids.
        {"name": "label_many", "op": "many", "graphs": 64, "n_lo": 1000, "n_hi": 12000, "factor": 6,
         "shortcuts": 0.02, "roots": 50, "batch": 1024},
        # One pair per call, the reference's query_distance, sixteen in turn.
        {"name": "query_one", "op": "query", "graph": "rmat", "scale": 14, "factor": 8, "weighted": False,
         "roots": 50, "batch": 1024, "pairs": 16, "device": False, "single": True, "zipf": 0.0},
        # The benchmark's 10M uniform pairs on the headline index, in device
        # memory.
        {"name": "query_rmat20", "op": "query", "graph": "rmat", "scale": 20, "factor": 16, "weighted": False,
         "roots": 64, "batch": 1024, "pairs": 10_000_000, "device": True, "single": False,
         "zipf": 0.0},
        # Weighted pairs from and to host arrays, an odd count.
        {"name": "query_weighted", "op": "query", "graph": "rmat", "scale": 16, "factor": 8, "weighted": True,
         "roots": 0, "batch": 512, "pairs": 1_000_003, "device": False, "single": False,
         "zipf": 0.0},
        # Serving: requests of 1 to 65,536 pairs, Zipf(1.1) endpoints, over
        # several label sets, all in flight at once.
        {"name": "serve_mix", "op": "serve", "sets": 8, "n_lo": 1000, "n_hi": 12000, "requests": 64,
         "k_hi": 65536, "zipf": 1.1, "batch_pairs": 1 << 18, "slots": 8},
        # Graph ingest, the benchmark's 16.8M raw samples in device memory.
        {"name": "ingest_rmat20", "op": "ingest", "scale": 20, "edges": 16 << 20, "weighted": False,
         "dedupe": False, "device": True},
        # Graph ingest of a weighted host edge list with repeats merged.
        {"name": "ingest_weighted", "op": "ingest", "scale": 17, "edges": 1_200_007, "weighted": True,
         "dedupe": True, "device": False},
        # Both graph reductions of an edge list in device memory.
        {"name": "reduce_rmat19", "op": "reduce", "scale": 19, "edges": 8 << 20},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["label", "label", "wlabel", "many", "query", "query", "serve", "ingest", "ingest", "reduce"])
    if op == "label":
        kind = rng.choice(["rmat", "er", "grid"])
        c = {"op": "label", "graph": kind, "weighted": False, "roots": rng.choice([16, 50, 64]),
             "batch": rng.choice([256, 512, 1000, 1024, 2048]), "ranked": rng.random() < 0.5}
        if kind == "rmat":
            c |= {"scale": rng.randint(10, 19), "factor": rng.choice([4, 8, 16])}
        elif kind == "er":
            c |= {"n": int(_log_uniform(rng, 1000, 25000)), "factor": rng.choice([4, 6, 10])}
        else:
            # no distance of a grid with shortcuts this size reaches the uint8 limit
            c |= {"n": int(_log_uniform(rng, 1000, 25000)), "factor": 0.02}
        return c
    if op == "wlabel":
        return {"op": "label", "graph": "rmat", "scale": rng.randint(9, 18), "factor": rng.choice([4, 8]),
                "weighted": True, "roots": 0, "batch": rng.choice([256, 512, 1000]), "ranked": rng.random() < 0.5}
    if op == "many":
        return {"op": "many", "graphs": rng.randint(16, 64), "n_lo": 1000, "n_hi": int(_log_uniform(rng, 2000, 12000)),
                "factor": 6, "shortcuts": 0.02, "roots": rng.choice([16, 50]), "batch": rng.choice([512, 1024])}
    if op == "query":
        weighted = rng.random() < 0.4
        single = rng.random() < 0.2
        return {"op": "query", "graph": "rmat", "scale": rng.randint(12, 16 if weighted else 19),
                "factor": 8 if weighted else rng.choice([8, 16]), "weighted": weighted,
                "roots": 0 if weighted else rng.choice([50, 64]), "batch": 512 if weighted else 1024,
                "pairs": rng.randint(8, 32) if single else int(_log_uniform(rng, 16, 4_000_000)),
                "device": not single and rng.random() < 0.5, "single": single, "zipf": rng.choice([0.0, 1.1])}
    if op == "serve":
        return {"op": "serve", "sets": rng.randint(2, 8), "n_lo": 1000, "n_hi": int(_log_uniform(rng, 2000, 12000)),
                "requests": rng.randint(16, 64), "k_hi": int(_log_uniform(rng, 64, 65536)), "zipf": 1.1,
                "batch_pairs": 1 << 18, "slots": rng.choice([4, 8])}
    scale = rng.randint(12, 20)
    edges = int(min(_log_uniform(rng, 2, 16), 16) * (1 << scale)) + rng.randint(0, 100)
    edges = min(edges, 16 << 20)
    if op == "ingest":
        return {"op": "ingest", "scale": scale, "edges": edges, "weighted": rng.random() < 0.5,
                "dedupe": rng.random() < 0.5, "device": rng.random() < 0.5}
    return {"op": "reduce", "scale": min(scale, 19), "edges": min(edges, 8 << 20)}


# ---------------------------------------------------------------------------
# Graphs, made on the GPU.
# ---------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _rmat_samples(scale, m, gen):
    """m R-MAT samples (a, b, c = .57, .19, .19) on 2**scale vertices."""
    u = torch.zeros(m, dtype=torch.int64, device="cuda")
    v = torch.zeros(m, dtype=torch.int64, device="cuda")
    for bit in range(scale):
        r = torch.rand(m, generator=gen, device="cuda")
        u |= (r >= 0.76).long() << bit
        v |= (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).long() << bit
    return u, v


def _clean(n, u, v):
    """Undirected edges (lo, hi), self-loops and repeats dropped."""
    key = torch.unique((torch.minimum(u, v) * n + torch.maximum(u, v))[u != v])
    return torch.div(key, n, rounding_mode="floor"), key % n


def _edges(case, gen):
    if case["graph"] == "rmat":
        n = 1 << case["scale"]
        u, v = _rmat_samples(case["scale"], n * case["factor"], gen)
    elif case["graph"] == "er":
        n = case["n"]
        m = n * case["factor"] // 2
        u = torch.randint(n, (m,), generator=gen, device="cuda")
        v = torch.randint(n, (m,), generator=gen, device="cuda")
    else:
        n = case["n"]
        cols = math.isqrt(n - 1) + 1
        i = torch.arange(n, device="cuda")
        right = i[(i % cols != cols - 1) & (i + 1 < n)]
        down = i[i + cols < n]
        k = int(round(case["factor"] * (len(right) + len(down))))
        u = torch.cat([right, down, torch.randint(n, (k,), generator=gen, device="cuda")])
        v = torch.cat([right + 1, down + cols, torch.randint(n, (k,), generator=gen, device="cuda")])
    return (n, *_clean(n, u, v))


def _host(t, view):
    """A page-locked host copy of a device tensor, as a numpy array."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy().view(view)


def _graph(case, gen):
    """(CSRGraph, rank): original ids with ascending lists and their degree
    order, or, when the case says so, ranked ids with descending lists."""
    n, lo, hi = _edges(case, gen)
    w = None
    if case["weighted"]:
        w = torch.randint(1, 101, lo.shape, generator=gen, device="cuda", dtype=torch.uint8)
        w = torch.cat([w, w])
    src, dst = torch.cat([lo, hi]), torch.cat([hi, lo])
    deg = torch.bincount(src, minlength=n)
    order = torch.sort(-deg, stable=True).indices
    rank = torch.empty_like(order)
    rank[order] = torch.arange(n, device="cuda")
    if case["ranked"]:
        src, dst, deg = rank[src], n - 1 - rank[dst], deg[order]
    key, perm = torch.sort(src * n + dst)
    adj = key % n
    if case["ranked"]:
        adj = n - 1 - adj
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(deg, 0, out=off[1:])
    g = graphs.CSRGraph(n, _host(off, np.uint64), _host(adj.int(), np.uint32),
                        None if w is None else _host(w[perm], np.uint8))
    return g, None if case["ranked"] else _host(rank.int(), np.uint32)


def _endpoints(n, k, zipf, order, gen):
    """k vertices: uniform, or Zipf over the degree rank (`order[r]`: the
    vertex of rank r)."""
    if not zipf:
        return torch.randint(n, (k,), generator=gen, device="cuda").int()
    cdf = torch.cumsum(torch.arange(1, n + 1, device="cuda", dtype=torch.float64) ** -zipf, 0)
    r = torch.searchsorted(cdf, torch.rand(k, generator=gen, device="cuda", dtype=torch.float64) * cdf[-1])
    return order[r.clamp_(max=n - 1)].int()


def _order(rank):
    """order[r] = vertex of rank r, on the device."""
    r = torch.from_numpy(rank.view(np.int32)).cuda().long()
    order = torch.empty_like(r)
    order[r] = torch.arange(len(r), device="cuda")
    return order


def _spread(count, lo, hi):
    """count whole numbers spread evenly over the logarithm of [lo, hi], in an
    order that mixes small and large."""
    x = [int(lo * (hi / lo) ** ((i + 0.5) / count)) for i in range(count)]
    return [x[i] for i in np.random.RandomState(count).permutation(count)]


def _many_cases(case, factor=6, shortcuts=0.02, roots=50):
    return [{"graph": "er" if i % 2 == 0 else "grid", "n": n, "factor": factor if i % 2 == 0 else shortcuts,
             "weighted": False, "ranked": False, "roots": roots}
            for i, n in enumerate(_spread(case["graphs"], case["n_lo"], case["n_hi"]))]


# ---------------------------------------------------------------------------
# Preparation: what a program has in hand before the call.
# ---------------------------------------------------------------------------

class _ExportBuffers:
    """Page-locked arrays that a program keeps for exported labels, with room
    for the label sets of the given cases one after another; a label set that
    does not fit its part gets arrays of its own."""

    def __init__(self, cases):
        self.n = [_vertices(c) for c in cases]
        self.roots = [c["roots"] for c in cases]
        self.room = [_room(c) for c in cases]
        weighted = cases[0]["weighted"]
        nk = sum(n * k for n, k in zip(self.n, self.roots))

        def pinned(count, dtype):
            return torch.zeros(max(count, 1), dtype=dtype, pin_memory=True)
        self.all = {"off": pinned(sum(self.n) + len(cases), torch.int64), "hub": pinned(sum(self.room), torch.int32),
                    "dist": pinned(sum(self.room), torch.int16 if weighted else torch.uint8)}
        if nk:
            self.all |= {"bp_dist": pinned(nk, torch.uint8), "bp_sets": pinned(2 * nk, torch.int64)}

    def export(self, indexes):
        """Every index's labels, offsets within its own part."""
        o = l = b = 0
        for i, index in enumerate(indexes):
            n, nk, tot = self.n[i], self.n[i] * self.roots[i], index.info().num_labels
            hub, dist = self.all["hub"][l:], self.all["dist"][l:]
            if tot > self.room[i]:
                hub = self.all["hub%d" % i] = torch.zeros(tot, dtype=hub.dtype, pin_memory=True)
                dist = self.all["dist%d" % i] = torch.zeros(tot, dtype=dist.dtype, pin_memory=True)
            _lib.check(_lib.lib.pado_export(index._need(), _p(self.all["off"][o:]), _p(hub), _p(dist),
                                            _p(self.all["bp_dist"][b:]) if nk else None,
                                            _p(self.all["bp_sets"][2 * b:]) if nk else None))
            o, l, b = o + n + 1, l + self.room[i], b + nk
        return dict(self.all)


def _p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _build(case, g, rank):
    if case["weighted"]:
        return pado.WeightedVertexCentricPLL(g, rank, batch=case["batch"])
    return pado.VertexCentricPLL(g, rank, bp_roots=case["roots"], batch=case["batch"])


def prepare(case, seed):
    gen = _gen(seed)
    _lib.check(_lib.lib.pado_set_scratch_cache(SCRATCH_KEEP))
    st = {"case": case}
    if case["op"] == "label":
        g, rank = _graph(case, gen)
        st |= {"g": g, "rank": rank, "out": _ExportBuffers([case])}
    elif case["op"] == "many":
        subs = _many_cases(case, case["factor"], case["shortcuts"], case["roots"])
        gr = [_graph(s, gen) for s in subs]
        st |= {"g": [g for g, _ in gr], "rank": [r for _, r in gr], "out": _ExportBuffers(subs)}
    elif case["op"] == "query":
        g, rank = _graph(case | {"ranked": False}, gen)
        st["index"] = _build(case, g, rank)
        order = _order(rank)
        a = _endpoints(g.n, case["pairs"], case["zipf"], order, gen)
        b = _endpoints(g.n, case["pairs"], case["zipf"], order, gen)
        if case["device"]:
            st |= {"a": a, "b": b, "out": torch.empty(case["pairs"], device="cuda",
                                                      dtype=torch.int16 if case["weighted"] else torch.uint8)}
        else:
            st |= {"a": a.cpu().numpy().view(np.uint32), "b": b.cpu().numpy().view(np.uint32)}
    elif case["op"] == "serve":
        subs = _many_cases(case | {"graphs": case["sets"]})
        gr = [_graph(s, gen) for s in subs]
        st["server"] = pado.Server(40 << 30, max_batch_pairs=case["batch_pairs"], slots=case["slots"])
        for ix in pado.build_many([g for g, _ in gr], [r for _, r in gr], bp_roots=50, batch=1024):
            st["server"].add(ix)
        ids = torch.randint(case["sets"], (case["requests"],), generator=gen, device="cuda").tolist()
        ks = _spread(case["requests"], 1, case["k_hi"])
        orders = [_order(r) for _, r in gr]
        st["requests"] = []
        for i, k in zip(ids, ks):
            ab = _endpoints(gr[i][0].n, 2 * k, case["zipf"], orders[i], gen).cpu().numpy().view(np.uint32)
            st["requests"].append((i, ab[:k], ab[k:]))
    else:
        n, m = 1 << case["scale"], case["edges"]
        u, v = (x.int() for x in _rmat_samples(case["scale"], m, gen))
        w = None
        if case.get("weighted"):
            w = torch.randint(1, 101, (m,), generator=gen, device="cuda", dtype=torch.uint8)
        st["n"] = n
        if case["op"] == "ingest" and not case["device"]:
            u, v, w = u.cpu(), v.cpu(), None if w is None else w.cpu()
        if case["op"] == "ingest":
            st |= {"u": u, "v": v, "w": w, "off": torch.zeros(n + 1, dtype=torch.int64, device=u.device),
                   "adj": torch.zeros(2 * m, dtype=torch.int32, device=u.device),
                   "w_out": None if w is None else torch.zeros(2 * m, dtype=torch.uint8, device=u.device),
                   "rank": torch.zeros(n, dtype=torch.int32, device=u.device)}
        else:
            st |= {"u": u, "v": v, "gone": torch.zeros(n, dtype=torch.uint8, device="cuda"),
                   "kept": torch.zeros(m, dtype=torch.int64, device="cuda"),
                   "twin": torch.zeros(n, dtype=torch.uint8, device="cuda"),
                   "new_id": torch.zeros(n, dtype=torch.int32, device="cuda"),
                   "kept2": torch.zeros(m, dtype=torch.int64, device="cuda")}
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------

def run(st):
    case, lib = st["case"], _lib.lib
    if case["op"] == "label":
        index = _build(case, st["g"], st["rank"])
        out = st["out"].export([index])
        index.close()
        return out
    if case["op"] == "many":
        indexes = pado.build_many(st["g"], st["rank"], bp_roots=case["roots"], batch=case["batch"])
        out = st["out"].export(indexes)
        for index in indexes:
            index.close()
        return out
    if case["op"] == "query":
        if case["device"]:
            st["index"].query_device(st["a"].data_ptr(), st["b"].data_ptr(), st["out"].data_ptr(), case["pairs"],
                                     torch.cuda.current_stream().cuda_stream)
            return st["out"]
        if case["single"]:
            return [st["index"].query_distance(a, b) for a, b in zip(st["a"].tolist(), st["b"].tolist())]
        return st["index"].query(st["a"], st["b"])
    if case["op"] == "serve":
        srv = st["server"]
        tickets = [srv.submit(i, a, b) for i, a, b in st["requests"]]
        return [srv.wait(t)[0] for t in tickets]
    n, m = st["n"], case["edges"]
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    if case["op"] == "ingest":
        entries = C.c_uint64()
        args = (m, _p(st["u"]), _p(st["v"]), _p(st["w"]), n, _lib.PADO_INGEST_DEDUPE if case["dedupe"] else 0,
                _p(st["off"]), _p(st["adj"]), _p(st["w_out"]), _p(st["rank"]), C.byref(entries))
        _lib.check(lib.pado_graph_ingest_device(*args, stream) if case["device"] else lib.pado_graph_ingest(*args))
        # entries past the count keep what the program's arrays held
        return {"off": st["off"], "adj": st["adj"], "w": st["w_out"], "rank": st["rank"],
                "entries": int(entries.value)}
    k1, k2, nout = C.c_uint64(), C.c_uint64(), C.c_uint32()
    _lib.check(lib.pado_reduce_degree1_device(m, _p(st["u"]), _p(st["v"]), n, _p(st["gone"]), _p(st["kept"]),
                                              C.byref(k1), stream))
    _lib.check(lib.pado_reduce_equivalent_device(m, _p(st["u"]), _p(st["v"]), n, _p(st["twin"]), _p(st["new_id"]),
                                                 _p(st["kept2"]), C.byref(k2), C.byref(nout), stream))
    return {"deleted": st["gone"], "kept": st["kept"], "kept_count": int(k1.value), "redundant": st["twin"],
            "new_id": st["new_id"], "kept_equivalent": st["kept2"], "kept_equivalent_count": int(k2.value),
            "n_out": int(nout.value)}


# ---------------------------------------------------------------------------
# What a pass cannot do without.
# ---------------------------------------------------------------------------

def _vertices(case):
    return 1 << case["scale"] if case["graph"] == "rmat" else case["n"]


def _entries(case):
    """Directed adjacency entries after cleaning, about."""
    n = _vertices(case)
    if case["graph"] == "grid":
        return int(4 * n * (1 + case["factor"]))
    # R-MAT repeats samples: 31.4M entries of 33.6M at s20/ef16
    return int((1.87 if case["graph"] == "rmat" else 1.0) * n * case["factor"])


# Labels per vertex measured on these generators (R-MAT by scale, the larger
# of edge factors 8 and 16; Erdos-Renyi of average degree 6 by size), with
# K = 50 to 64 and B = 1024, weighted B = 512.
_PER_VERTEX = {
    "rmat": [(10, 0.67), (12, 0.93), (14, 1.73), (16, 4.92), (18, 19.6), (20, 68.7)],
    "weighted": [(10, 10.7), (12, 15.0), (14, 22.3), (16, 31.9), (18, 50.4)],
    "er": [(math.log2(1000), 5.0), (math.log2(5000), 130.0), (math.log2(20011), 661.0), (math.log2(50000), 1749.0)],
}


def _labels(case):
    """The label count of a case's graph, about."""
    n = _vertices(case)
    if case["graph"] == "grid":
        return 0.0286 * n ** 1.89
    x, y = zip(*_PER_VERTEX["weighted" if case["weighted"] else case["graph"]])
    per = math.exp(np.interp(math.log2(n), x, np.log(y)))
    return per * n * (math.sqrt(case["factor"] / 6) if case["graph"] == "er" else 1.0)


def _room(case):
    """Entries a program keeps for a case's labels: a margin over the count it
    expects, more for the small random graphs, whose counts spread more, and
    with few bit-parallel roots, which prune less."""
    margin = 1.2 if case["graph"] == "rmat" else 1.6
    return int(_labels(case) * margin * (1.0 if case["weighted"] or case["roots"] >= 50 else 1.6)) + 8192


def work(case):
    if case["op"] == "label":
        n, m = _vertices(case), _entries(case)
        csr = 8 * (n + 1) + (5 if case["weighted"] else 4) * m + (0 if case["ranked"] else 4 * n)
        return {"bytes": int(csr + 8 * (n + 1) + (6 if case["weighted"] else 5) * _labels(case)
                             + 17 * n * case["roots"]), "flops": 0}
    if case["op"] == "many":
        # mean of a log-uniform size, half of the graphs of each kind
        r = math.log(case["n_hi"] / case["n_lo"])

        def mean(p):
            return (case["n_hi"] ** p - case["n_lo"] ** p) / (p * r)
        per = mean(1) * (8 + 4 + 8 + 17 * case["roots"]) + 4 * mean(1) * 5 + 5 * (0.0463 * mean(1.91)
                                                                                + 0.0143 * mean(1.89))
        return {"bytes": int(case["graphs"] * per), "flops": 0}
    if case["op"] == "query":
        per = 2 * (6 if case["weighted"] else 5) * _labels(case) / _vertices(case) + 34 * case["roots"] + 40
        return {"bytes": int(case["pairs"] * (per + (10 if case["weighted"] else 9))), "flops": 0}
    if case["op"] == "serve":
        r = math.log(case["n_hi"] / case["n_lo"])
        lists = 0.06 * (case["n_hi"] ** 0.9 - case["n_lo"] ** 0.9) / (0.9 * r)
        pairs = case["requests"] * max(1.0, (case["k_hi"] - 1) / math.log(case["k_hi"]))
        return {"bytes": int(pairs * (9 + 40 + 34 * 50 + 10 * lists)), "flops": 0}
    n, m = 1 << case["scale"], case["edges"]
    if case["op"] == "ingest":
        wb = 1 if case["weighted"] else 0
        return {"bytes": int(m * (8 + wb) + 2 * m * (4 + wb) + 12 * n + 8), "flops": 0}
    return {"bytes": int(2 * (8 * m + n + 8 * m) + 4 * n), "flops": 0}
