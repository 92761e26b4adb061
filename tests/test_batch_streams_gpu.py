"""Runs of one batch handed to several streams without waiting in between:
each gives the counts of a run by itself, and so does the next one.  The
members are large enough for the 4-cycle counters that span several windows of
keys, and for those past the shared ones."""
import numpy as np
import pytest

import gpm

pytestmark = pytest.mark.gpu


def _overlap(run_async, want, legacy=False):
    import torch
    streams = [torch.cuda.Stream() for _ in range(3)]
    if legacy:  # the legacy default stream between two others
        streams[1] = torch.cuda.default_stream()
    out = torch.zeros(12, want.size, dtype=torch.int64, device="cuda")
    for r in range(4):
        out.fill_(-1)
        torch.cuda.synchronize()
        for i in range(12):
            run_async(i % 4 == 3, streams[i % 3].cuda_stream, out[i].data_ptr())
        torch.cuda.synchronize()
        for i in range(12):
            assert np.array_equal(out[i].cpu().numpy().view(np.uint64), want.ravel()), (r, i)


def test_motif_batch():
    b = gpm.Batch.chung_lu([120000, 3000, 60000], [2.1, 2.4, 2.2], [12.0, 20.0, 16.0], seed=3)
    want = b.motif(use_graph=False)
    assert (want == b.motif(use_graph=True)).all() and want[:, 5].all()
    _overlap(b.motif_async, want)
    _overlap(b.motif_async, want, legacy=True)
    assert (want == b.motif(use_graph=False)).all()


def test_match_batch():
    n, s, d = gpm.gen_rmat(17, 8, seed=5)
    g = gpm.Graph.from_edges(n, s, d, labels=(np.arange(n) % 2).astype(np.int32))
    qs = [gpm.Query(4, [0, 1, 2, 3], [1, 2, 3, 0], lab) for lab in ([0, 0, 1, 1], [0, 1, 0, 1])]
    qs.append(gpm.Query(3, [0, 1, 2], [1, 2, 0], [0, 1, 1]))
    b = gpm.MatchBatch(g, qs)
    want = b.run(use_graph=False)
    assert want[:, 0].tolist() == [g.match(q) for q in qs] and want.all()
    assert (want == b.run(use_graph=True)).all()
    _overlap(b.run_async, want)
    _overlap(b.run_async, want, legacy=True)
    assert (want == b.run(use_graph=False)).all()
