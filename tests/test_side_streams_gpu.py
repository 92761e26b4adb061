"""Plans with kernels on a side stream, last run inside a CUDA graph's capture,
then released: the counts are right and the next call finds no error left by
the release."""
import math

import numpy as np
import pytest

import gpm

pytestmark = pytest.mark.gpu


def _complete(n):
    return [a.astype(np.int32) for a in np.triu_indices(n, 1)]


def _check(out, sizes):
    for g, n in enumerate(sizes):  # of the induced motifs a complete graph has cliques alone
        assert out[g].tolist() == [0, math.comb(n, 3), 0, 0, 0, 0, 0, math.comb(n, 4)], n


@pytest.mark.parametrize("after", ["destroy", "autotune"])
def test_batch_with_large_clique_tasks(after):
    """700 vertices give out-lists above 512 neighbours, the small ones the
    other kernels' tasks beside them."""
    sizes = [700, 40, 5, 90]
    edges = [_complete(n) for n in sizes]
    b = gpm.Batch.from_edges([(n, *e) for n, e in zip(sizes, edges)])
    _check(b.motif(use_graph=True), sizes)
    _check(b.motif(use_graph=True), sizes)
    if after == "autotune":
        b.autotune()
        _check(b.motif(use_graph=True), sizes)
    b.close()
    g = gpm.Graph.from_edges(90, *edges[3]).orient()
    assert g.clique(4) == math.comb(90, 4)


def test_captured_count_with_a_dense_core():
    import torch
    g = gpm.Graph.rmat(15, 32, seed=2).orient()
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    g.tc_async(gpm.TC_BITMAP, 0, out.data_ptr())
    torch.cuda.synchronize()
    want = out.item()
    assert g.plan_stats()[4] > 0  # dense segments
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        g.tc_async(gpm.TC_BITMAP, torch.cuda.current_stream().cuda_stream, out.data_ptr())
    out.fill_(-1)
    graph.replay()
    assert out.item() == want > 0
    del graph
    g.close()
    h = gpm.Graph.from_edges(90, *_complete(90)).orient()
    assert h.tc() == math.comb(90, 3) and h.clique(5) == math.comb(90, 5)
