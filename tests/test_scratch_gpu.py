"""Counts whose faster way needs scratch that cannot be had: they take the way
that does without it."""
import contextlib

import numpy as np
import pytest

import gpm

pytestmark = pytest.mark.gpu

MIB = 1 << 20


@contextlib.contextmanager
def _left(mib):
    """All device memory but about `mib` MiB taken."""
    import torch
    gpm.trim()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - mib * MIB, dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < (mib + 4) * MIB
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def test_cycle_query_without_label_classes():
    g = gpm.Graph.rmat(19, 16, seed=3)
    g.set_labels(np.where(np.arange(1 << 19) % 4096 == 0, 1, 0).astype(np.int32) + (np.arange(1 << 19) % 4096 == 1) * 2)
    q = gpm.Query(4, [0, 1, 2, 3], [1, 2, 3, 0], [1, 2, 1, 2])
    want = g.match(q, limit=1 << 40)  # walked
    with _left(48):
        assert g.match(q) == want
    assert g.match(q) == want


def test_rows_that_cannot_be_extended():
    """One root, 30 hubs, 100,000 leaves under each hub, one vertex under all
    leaves: 30 pairs, whose extension takes 36 MB."""
    hubs, leaves = 30, 100000
    n = 1 + hubs + leaves + 1
    leaf = np.arange(1 + hubs, 1 + hubs + leaves)
    s = np.concatenate([np.zeros(hubs), np.repeat(np.arange(1, 1 + hubs), leaves), leaf]).astype(np.int32)
    d = np.concatenate([np.arange(1, 1 + hubs), np.tile(leaf, hubs), np.full(leaves, n - 1)]).astype(np.int32)
    lab = np.full(n, 2, np.int32)
    lab[0], lab[1:1 + hubs], lab[n - 1] = 0, 1, 3
    g = gpm.Graph.from_edges(n, s, d, labels=lab)
    q = gpm.Query(4, [0, 1, 2], [1, 2, 3], [0, 1, 2, 3])
    assert g.match(q, limit=1 << 40) == hubs * leaves
    with _left(20):
        assert g.match(q, limit=1 << 40) == hubs * leaves


def test_heavy_edges_without_their_list():
    g = gpm.Graph.generate(1, 200000, 13000000, seed=5)
    assert g.info().max_degree * 2 > 192
    want = g.pattern("P7")
    with _left(40):
        got = g.pattern("P7")
    assert got[0] == want[0] > 0 and got[1].tolist() == want[1].tolist()


@pytest.mark.parametrize("k,scale,levels", [(3, 20, range(230, 310, 10)), (5, 18, range(44, 90, 6)), (4, 20, range(150, 310, 20))])
def test_cliques_with_little_memory(k, scale, levels):
    """Room for the rows' slabs, but not for the hubs' bitmaps beside them."""
    g = gpm.Graph.rmat(scale, 16, seed=4).orient()
    want = g.clique(k)
    for mib in levels:
        g.drop_plans()
        with _left(mib):
            assert g.clique(k) == want, mib
