"""k-cliques where the row layouts change: out-lists around 64 (warp or CTA
task), 65 members of a row (warp or CTA compaction), rows beyond a small CTA's
shared memory, beyond a large one's (slab), and lists much longer than the rest
of an out-list.  Counts against the oracle or a closed form."""
import math

import numpy as np
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 31, 33, 64, 65, 66, 67, 97, 129, 200, 420, 700])
def test_complete_graph(n):
    u, v = np.triu_indices(n, 1)
    g = gpm.Graph.from_edges(n, u, v).orient()
    for k in (3, 4, 5):
        assert g.clique(k) == math.comb(n, k), k
    if n <= 67:
        assert g.clique(6) == math.comb(n, 6)


def test_slab_rows():
    """Vertices with 2000 out-neighbours that are joined sparsely, so that
    their rows are far larger than shared memory."""
    rng = np.random.default_rng(7)
    m = 2000
    e = rng.integers(0, m, size=(60000, 2))
    hub = np.stack([np.full(m, m), np.arange(m)], 1)
    # pendant edges keep the hub's neighbours above it in degree order
    pend = np.stack([np.repeat(np.arange(m), 2100), m + 1 + np.tile(np.arange(2100), m)], 1)
    e = np.concatenate([e, hub, pend]).astype(np.int32)
    n = m + 1 + 2100
    g = gpm.Graph.from_edges(n, e[:, 0], e[:, 1])
    off, idx = orc.build_csr(n, e[:, 0], e[:, 1])
    doff, didx = orc.orient(off, idx)
    g.orient()
    assert g.info().max_degree >= 1900
    assert g.clique(4) == orc.clique(doff, didx, 4)
    assert g.clique(5) == orc.clique(doff, didx, 5)


@pytest.mark.parametrize("k", [4, 5])
@pytest.mark.parametrize("scale,ef", [(9, 40), (11, 24), (13, 12)])
def test_skewed(scale, ef, k):
    n, s, d = gpm.gen_rmat(scale, ef, seed=scale)
    off, idx = orc.build_csr(n, s, d)
    doff, didx = orc.orient(off, idx)
    g = gpm.Graph.from_edges(n, s, d).orient()
    assert g.clique(k) == orc.clique(doff, didx, k)
