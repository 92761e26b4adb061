"""Cliques of six to eight vertices on rows of every layout: a hub over m
vertices joined sparsely, with a few complete subgraphs among them, m from a
warp task's to rows far past shared memory.  Against the oracle."""
import numpy as np
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [40, 65, 100, 300, 500, 560, 1025, 2000])
def test_hub_over_planted_cliques(m):
    rng = np.random.default_rng(m)
    e = [rng.integers(0, m, size=(8 * m, 2))]
    for size in (7, 8, 10, 12):
        v = rng.choice(m, size, replace=False)
        iu, iv = np.triu_indices(size, 1)
        e.append(np.stack([v[iu], v[iv]], 1))
    e.append(np.stack([np.full(m, m), np.arange(m)], 1))
    # pendant vertices keep the hub's neighbours above it in degree order
    pend = m + 100
    e.append(np.stack([np.repeat(np.arange(m), pend), m + 1 + np.tile(np.arange(pend), m)], 1))
    e = np.concatenate(e).astype(np.int32)
    n = m + 1 + pend
    doff, didx = orc.orient(*orc.build_csr(n, e[:, 0], e[:, 1]))
    g = gpm.Graph.from_edges(n, e[:, 0], e[:, 1]).orient()
    assert g.info().max_degree >= m - 1
    for k in (3, 6, 7, 8):
        want = orc.clique(doff, didx, k)
        assert g.clique(k) == want > 0, k


@pytest.mark.parametrize("k", [6, 7, 8])
def test_many_tasks(k):
    """Out-lists on both sides of a warp task's 64, thousands of tasks."""
    rng = np.random.default_rng(k)
    n, s, d = gpm.gen_er(3000, 190000, seed=k)
    e = [np.stack([s, d], 1)]
    for _ in range(40):
        v = rng.choice(n, 11, replace=False)
        iu, iv = np.triu_indices(11, 1)
        e.append(np.stack([v[iu], v[iv]], 1))
    e = np.concatenate(e).astype(np.int32)
    doff, didx = orc.orient(*orc.build_csr(n, e[:, 0], e[:, 1]))
    lens = np.diff(doff)
    assert (lens > 64).sum() > 500 and (lens <= 64).sum() > 500
    g = gpm.Graph.from_edges(n, e[:, 0], e[:, 1]).orient()
    want = orc.clique(doff, didx, k)
    for _ in range(3):
        assert g.clique(k) == want > 0
