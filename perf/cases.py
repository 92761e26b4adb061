"""Counting work of a user of the engine, through its Python binding.

Every case names a kind of call and a seeded synthetic graph: R-MAT (a, b, c =
.57, .19, .19), Erdos-Renyi or Chung-Lu.  A graph handle is what a program
keeps between counts; task queues and relabelled copies are built by the first
count on it and belong to that pass.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gpm-artifact_b200"))
import gpm  # noqa: E402

# query shapes of the labelled workload: (vertices, edges)
SHAPES = {
    "triangle": (3, [(0, 1), (1, 2), (2, 0)]),
    "cycle4": (4, [(0, 1), (1, 2), (2, 3), (3, 0)]),
    "diamond": (4, [(0, 1), (0, 2), (0, 3), (1, 2), (2, 3)]),
    "house": (5, [(0, 1), (0, 4), (1, 2), (1, 4), (2, 3), (3, 4)]),
}
LABELS, ZIPF = 8, 1.2


def listed():
    return [
        # a small sparse graph counted again and again: latency and launches
        {"name": "tc_er16k", "kind": "tc", "mode": "v", "graph": "er", "n": 16384, "deg": 16.0},
        # the drop-in solver's edge-centric count of a skewed graph
        {"name": "tc_rmat20_edge", "kind": "tc", "mode": "e", "graph": "rmat", "scale": 20, "deg": 32.0},
        # the headline: asynchronous count of a large skewed graph
        {"name": "tc_rmat22", "kind": "tc_async", "graph": "rmat", "scale": 22, "deg": 32.0},
        # a service that receives a CSR in pinned host memory and answers with its count
        {"name": "tc_host_rmat20", "kind": "tc_host", "graph": "rmat", "scale": 20, "deg": 32.0},
        # the reference's driver program: edge list in, orient, count once
        {"name": "load_count_cl300k", "kind": "load_count", "graph": "cl", "n": 300007, "deg": 24.0, "gamma": 2.3},
        {"name": "clique4_rmat20", "kind": "clique", "k": 4, "graph": "rmat", "scale": 20, "deg": 32.0},
        {"name": "clique5_rmat19", "kind": "clique", "k": 5, "graph": "rmat", "scale": 19, "deg": 32.0},
        {"name": "motif4_rmat18", "kind": "motif", "k": 4, "graph": "rmat", "scale": 18, "deg": 32.0},
        # motifs of many graphs of uneven size in one replayed launch
        {"name": "motif_batch48", "kind": "motif_batch", "graph": "cl", "count": 48, "n": 200000},
        # one labelled query at a time
        {"name": "match_cycle4_rmat19", "kind": "match", "shapes": "cycle4", "labels": "0 0 3 1", "graph": "rmat",
         "scale": 19, "deg": 32.0},
        # several labelled queries on one graph in one launch
        {"name": "match_batch_rmat17", "kind": "match_batch", "shapes": "triangle diamond house cycle4",
         "labels": "3 4 1 1 0 0 0 0 0 4 1 0 0 0 3 1", "graph": "rmat", "scale": 17, "deg": 32.0},
        # a named pattern of the G2Miner / Pattern solvers, enumerated per edge
        {"name": "pattern_p7_cl4k", "kind": "pattern", "pattern": "P7", "graph": "cl", "n": 4099, "deg": 12.0,
         "gamma": 2.4},
    ]


def _between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_graph(rng, nmin, nmax):
    """An R-MAT, Erdos-Renyi or Chung-Lu graph of about nmin..nmax vertices."""
    what = rng.choice(["rmat", "rmat", "er", "cl"])
    n = _between(rng, nmin, nmax)
    g = {"graph": what, "deg": round(rng.uniform(8, 32), 2)}
    if what == "rmat":
        g["scale"] = round(math.log2(n))
        g["deg"] = 2.0 * rng.randint(4, 16)
    else:
        g["n"] = int(n) | 1
        if what == "cl":
            g["gamma"] = round(rng.uniform(2.2, 2.8), 3)
    return g


def _draw_labels(rng, k):
    """k labels by their frequency in the data graph, one of them at least not of the two commonest."""
    weights = [1.0 / (i + 1) ** ZIPF for i in range(LABELS)]
    while True:
        got = rng.choices(range(LABELS), weights, k=k)
        if max(got) > 1:
            return got


def draw(rng):
    kind = rng.choice(["tc", "tc", "tc_async", "tc_async", "tc_host", "load_count", "clique", "clique", "motif", "motif_batch",
                       "match", "match", "match_batch", "pattern"])
    c = {"kind": kind}
    if kind == "tc":
        c["mode"] = rng.choice(["v", "e"])
        c.update(_draw_graph(rng, 1 << 10, 1 << 20))
    elif kind == "tc_async":
        c.update(_draw_graph(rng, 1 << 14, 1 << 22))
    elif kind == "tc_host":
        c.update(_draw_graph(rng, 1 << 12, 1 << 20))
    elif kind == "load_count":
        c.update(_draw_graph(rng, 1 << 10, 300000))
    elif kind == "clique":
        c["k"] = rng.choice([4, 4, 5])
        c.update(_draw_graph(rng, 1 << 12, 1 << (20 if c["k"] == 4 else 19)))
    elif kind == "motif":
        c["k"] = rng.choice([3, 4, 4])
        c.update(_draw_graph(rng, 1 << 12, 1 << 18))
    elif kind == "motif_batch":
        c.update({"graph": "cl", "count": rng.randint(5, 48), "n": int(_between(rng, 5000, 200000))})
    elif kind == "match":
        s = rng.choice(sorted(SHAPES))
        top = {"triangle": 19, "cycle4": 18, "diamond": 18, "house": 15}[s]
        c.update({"shapes": s, "labels": " ".join(map(str, _draw_labels(rng, SHAPES[s][0]))), "graph": "rmat",
                  "scale": rng.randint(12, top), "deg": 2.0 * rng.randint(6, 16)})
    elif kind == "match_batch":
        shapes = [rng.choice(["triangle", "cycle4", "diamond"]) for _ in range(rng.randint(2, 5))]
        labels = [x for s in shapes for x in _draw_labels(rng, SHAPES[s][0])]
        c.update({"shapes": " ".join(shapes), "labels": " ".join(map(str, labels)), "graph": "rmat",
                  "scale": rng.randint(12, 16), "deg": 2.0 * rng.randint(6, 16)})
    else:
        c["pattern"] = rng.choice(["P1", "P4", "P5", "P7", "P8"])
        c.update({"graph": rng.choice(["er", "cl"]), "n": int(_between(rng, 500, 2000)) | 1,
                  "deg": round(rng.uniform(6, 12), 2), "gamma": 2.5})
    return c


def _sizes(case):
    """Vertices and drawn edges (loops and duplicates among them) of the case's graph."""
    n = 1 << case["scale"] if case["graph"] == "rmat" else case["n"]
    return n, int(round(n * case["deg"] / 2))


def _edges(case, seed):
    """The case's graph as a host edge list."""
    n, m = _sizes(case)
    if case["graph"] == "rmat":
        return gpm.gen_rmat(case["scale"], int(case["deg"]) // 2, seed=seed)
    if case["graph"] == "er":
        return gpm.gen_er(n, m, seed=seed)
    return gpm.gen_chung_lu(n, case["gamma"], case["deg"], seed=seed)


def _graph(case, seed):
    """The same graph on the device, symmetric."""
    n, m = _sizes(case)
    if case["graph"] == "rmat":
        return gpm.Graph.rmat(case["scale"], int(case["deg"]) // 2, seed=seed)
    if case["graph"] == "er":
        return gpm.Graph.generate(1, n, m, seed=seed)
    return gpm.Graph.generate(2, n, 0, a=case["gamma"], b=case["deg"], seed=seed)


def _members(case, seed):
    """Member sizes, exponents and mean degrees of a batch of Chung-Lu graphs."""
    rng = np.random.default_rng(seed)
    k = case["count"]
    n = np.exp(rng.uniform(math.log(1000), math.log(case["n"]), k)).astype(np.int64)
    n[0] = case["n"]  # the largest member is there with every seed
    return n, rng.uniform(2.1, 2.8, k), rng.uniform(8, 64, k)


def _queries(case):
    labels = [int(x) for x in case["labels"].split()]
    out = []
    for name in case["shapes"].split():
        k, edges = SHAPES[name]
        own, labels = labels[:k], labels[k:]
        out.append(gpm.Query(k, [a for a, _ in edges], [b for _, b in edges], own))
    return out


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "load_count":
        st["edges"] = _edges(case, seed)
        return st
    if kind == "motif_batch":
        n, gamma, deg = _members(case, seed)
        st["b"] = gpm.Batch.chung_lu(n, gamma, deg, seed=seed)
        return st
    g = _graph(case, seed)
    if kind == "tc_host":
        off, idx = g.csr()
        g.close()
        st["n"] = len(off) - 1
        st["off"], st["idx"] = torch.from_numpy(off).pin_memory(), torch.from_numpy(idx).pin_memory()
        return st
    if kind in ("tc", "tc_async", "clique"):
        g.orient()
    if kind == "tc_async":
        st["out"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    if kind in ("match", "match_batch"):
        g.set_labels(gpm.gen_zipf_labels(g.info().n, LABELS, ZIPF, seed=seed))
        st["q"] = _queries(case)
    if kind == "match_batch":
        st["b"] = gpm.MatchBatch(g, st["q"])
    st["g"] = g
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "tc":
        return st["g"].tc(gpm.V_CENTRIC if case["mode"] == "v" else gpm.E_CENTRIC)
    if kind == "tc_async":
        st["g"].tc_async(gpm.TC_AUTO, torch.cuda.current_stream().cuda_stream, st["out"].data_ptr())
        return st["out"]
    if kind == "tc_host":
        return gpm.tc_host_csr_ptrs(st["n"], st["off"].data_ptr(), st["idx"].data_ptr(), gpm.TC_AUTO, 0)
    if kind == "load_count":
        n, src, dst = st["edges"]
        g = gpm.Graph.from_edges(n, src, dst).orient()
        t = g.tc(gpm.V_CENTRIC)
        g.close()
        return t
    if kind == "clique":
        return st["g"].clique(case["k"])
    if kind == "motif":
        return st["g"].motif(case["k"]).view(np.int64)
    if kind == "motif_batch":
        return st["b"].motif(use_graph=True).view(np.int64)
    if kind == "match":
        return st["g"].match(st["q"][0])
    if kind == "match_batch":
        return st["b"].run(use_graph=True).view(np.int64)
    result, counters = st["g"].pattern(case["pattern"])
    return [result, counters.view(np.int64)]


def work(case):
    """Bytes of the stored lists (offsets 8 per vertex, ids 4 per entry), each read once, and of the counts.
    Nothing is computed in floating point."""
    kind = case["kind"]
    if kind == "motif_batch":
        n, _, deg = _members(case, 1)
        verts, entries, counts = int(n.sum()), int((n * deg).sum()), 8 * case["count"]
    else:
        verts, m = _sizes(case)
        entries = m if kind in ("tc", "tc_async", "clique") else 2 * m
        counts = {"motif": 6, "pattern": 7, "match_batch": len(case.get("shapes", "").split())}.get(kind, 1)
    if kind in ("match", "match_batch"):
        verts = 1.5 * verts  # a 4-byte label each
    return {"bytes": int(8 * verts + 4 * entries + 8 * counts), "flops": 0}


def exact(case, seed):
    """Triangles of a small graph from its dense adjacency matrix: sum(A A . A) / 6."""
    if case["kind"] not in ("tc", "tc_async", "tc_host", "load_count") or _sizes(case)[0] > 20000:
        return None
    n, src, dst = _edges(case, seed)
    a = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    u, v = (torch.from_numpy(x.astype(np.int64)).cuda() for x in (src, dst))
    a[u, v] = 1
    a[v, u] = 1
    a.fill_diagonal_(0)
    t = int(((a @ a) * a).sum().round().item()) // 6
    return torch.tensor([t]) if case["kind"] == "tc_async" else t
