"""Graph construction at the edges of its key width and of its gaps: vertex
counts around powers of two, long runs of vertices without neighbours, no
entries at all; and the degrees an oriented graph remembers."""
import numpy as np
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 1023, 1024, 1025, 70001])
@pytest.mark.parametrize("m", [0, 1, 40, 3000])
def test_build_matches_oracle(n, m):
    rng = np.random.default_rng(n * 7 + m)
    # ids beyond both ends are dropped; the largest pair of ids is the key next to the sentinel
    s = rng.integers(-1, n + 1, m).astype(np.int32)
    d = rng.integers(-1, n + 1, m).astype(np.int32)
    s = np.concatenate([s, [n - 1, n - 1, 0]]).astype(np.int32)
    d = np.concatenate([d, [n - 1, max(n - 2, 0), n - 1]]).astype(np.int32)
    ok = (s >= 0) & (d >= 0) & (s < n) & (d < n)
    off, idx = orc.build_csr(n, s[ok], d[ok])
    got = gpm.Graph.from_edges(n, s, d).csr()
    assert got[0].tolist() == off.tolist() and got[1].tolist() == idx.tolist()
    a = np.unique(np.stack([s, d], 1)[ok & (s != d)], axis=0)
    o, i = gpm.Graph.from_edges(n, s, d, symmetrize=False).csr()
    assert i.tolist() == a[:, 1].tolist() and np.diff(o).tolist() == np.bincount(a[:, 0], minlength=n).tolist()


def test_long_gaps():
    n = 3_000_001
    s = np.array([5, 5, 1_500_000, n - 1], np.int32)
    d = np.array([1_000_000, 7, 40, 6], np.int32)
    off, idx = gpm.Graph.from_edges(n, s, d).csr()
    want_off, want_idx = orc.build_csr(n, s, d)
    assert np.array_equal(off, want_off) and np.array_equal(idx, want_idx)


@pytest.mark.parametrize("how", ["symmetric", "one_way", "csr", "relabelled", "twice"])
def test_counts_after_orientation(how):
    """The rank order takes the degrees from the orientation where the graph
    was built symmetric, and counts them otherwise."""
    n, s, d = gpm.gen_rmat(11, 12, seed=6)
    off, idx = orc.build_csr(n, s, d)
    if how == "one_way":
        g = gpm.Graph.from_edges(n, s, d, symmetrize=False).orient()
    elif how == "csr":
        g = gpm.Graph.from_csr(off, idx).orient()
    else:
        g = gpm.Graph.from_edges(n, s, d).orient(relabel=how == "relabelled")
        if how == "twice":
            g.orient()
    doff, didx = g.csr()
    want = orc.tc(doff, didx)
    import torch
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    g.tc_async(gpm.TC_BITMAP, torch.cuda.current_stream().cuda_stream, out.data_ptr())
    assert int(out.item()) == want
    if how in ("symmetric", "csr", "relabelled"):
        assert want == orc.tc(*orc.orient(off, idx))
        assert g.clique(4) == orc.clique(*orc.orient(off, idx), 4)
