"""Counted queries whose plan sizes a set in place of walking it (a vertex that
is adjacent neither to the vertex mapped last nor to another such vertex), and
4-cycles: every count must equal the oracle's, the number of embeddings listed
by gpm_match_list, and the batched count."""
import numpy as np
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu

SHAPES = {
    "diamond": (4, [(0, 1), (0, 2), (0, 3), (1, 2), (2, 3)]),
    "cycle4": (4, [(0, 1), (1, 2), (2, 3), (3, 0)]),
    "star3": (4, [(0, 1), (0, 2), (0, 3)]),
    "path4": (4, [(0, 1), (1, 2), (2, 3)]),
    "tailed": (4, [(0, 1), (1, 2), (2, 0), (2, 3)]),
    "house": (5, [(0, 1), (0, 4), (1, 2), (1, 4), (2, 3), (3, 4)]),
    "k23": (5, [(0, 2), (0, 3), (0, 4), (1, 2), (1, 3), (1, 4)]),
    "book3": (5, [(0, 1), (0, 2), (1, 2), (0, 3), (1, 3), (0, 4), (1, 4)]),
    "tree6": (6, [(0, 1), (1, 2), (1, 3), (3, 4), (3, 5)]),
    "pyramid6": (6, [(0, 1), (0, 2), (0, 3), (0, 4), (0, 5), (1, 2), (2, 3), (3, 4), (4, 5), (5, 1)]),
    "cycle6": (6, [(0, 1), (1, 2), (2, 3), (3, 4), (4, 5), (5, 0)]),
}
# label tuples: all equal, all different, and every mix of two that pairs the
# set vertices with mapped ones
LABELS = ["000000", "012012", "001100", "010101", "011000", "012201"]


@pytest.mark.parametrize("wide", [False, True], ids=["partitioned", "labels_from_64"])
@pytest.mark.parametrize("graph", ["sparse", "dense", "hubs"])
def test_factored_counts(graph, wide):
    if graph == "sparse":
        n, s, d = gpm.gen_er(400, 1200, seed=5)
    elif graph == "dense":
        n, s, d = gpm.gen_er(45, 420, seed=6)
    else:
        n, s, d = gpm.gen_chung_lu(700, 2.1, 5.0, seed=7)
    lab = gpm.gen_zipf_labels(n, 3, 1.2, seed=8) + (70 if wide else 0)
    off, idx = orc.build_csr(n, s, d)
    g = gpm.Graph.from_edges(n, s, d, labels=lab)
    queries, want = [], []
    for name, (k, edges) in SHAPES.items():
        e = np.array(edges, np.int32)
        qo, qi = orc.build_csr(k, e[:, 0], e[:, 1])
        for t in LABELS:
            ql = np.array([int(c) for c in t[:k]], np.int32) + (70 if wide else 0)
            if graph != "sparse" and name in ("tree6", "cycle6") and len(set(ql)) < 3:
                continue  # hundreds of millions of embeddings for the CPU to walk
            q = gpm.Query(k, e[:, 0], e[:, 1], ql)
            w = orc.match(off, idx, lab, qo, qi, ql)
            assert g.match(q) == w, (name, t)
            if w <= 20000:
                emb = g.match_list(q, w + 1)
                assert len(emb) == w and len(np.unique(emb, axis=0)) == w, (name, t)
            queries.append(q)
            want.append(w)
    b = gpm.MatchBatch(g, queries)
    assert b.run(use_graph=False)[:, 0].tolist() == want
    assert b.run(use_graph=True)[:, 0].tolist() == want


def test_members_joined_by_edges():
    """Member ids that split a component: a count goes to the member of the
    root of the plan that enumerates, as with one task per row."""
    n, s, d = gpm.gen_er(60, 200, seed=3)
    lab = gpm.gen_zipf_labels(n, 2, 1.2, seed=3)
    g = gpm.Graph.from_edges(n, s, d, labels=lab)
    mem = (np.arange(n) % 3).astype(np.int32)
    for k, edges in (SHAPES["diamond"], SHAPES["cycle4"]):
        e = np.array(edges, np.int32)
        q = gpm.Query(k, e[:, 0], e[:, 1], [1, 0, 0, 0])
        emb = g.match_list(q, 10 ** 6)
        got = gpm.MatchBatch(g, [q], member=mem, nmembers=3).run()[0]
        # the root is the rarest label's vertex (ties: higher degree, then lower id)
        assert got.tolist() == np.bincount(mem[emb[:, 0]], minlength=3).tolist()
