"""Sums over edges in blocks of 1 to 32 vertices: batches of many small members,
so that a block holds edges of several, and dense members, against the oracle."""
import numpy as np
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members,top", [(1, 300), (60, 14), (500, 40), (1500, 40), (8000, 45)])
def test_members(members, top):
    rng = np.random.default_rng(members)
    graphs, want = [], []
    for _ in range(members):
        n = int(rng.integers(1, top + 1)) if members > 1 else top
        iu, iv = np.triu_indices(n, 1)
        k = rng.random(len(iu)) < rng.choice([0.05, 0.3, 1.0])
        s, d = iu[k].astype(np.int32), iv[k].astype(np.int32)
        graphs.append((n, s, d))
    b = gpm.Batch.from_edges(graphs)
    got = b.motif(use_graph=False)
    for i in rng.choice(members, min(members, 60), replace=False):
        n, s, d = graphs[i]
        off, idx = orc.build_csr(n, s, d)
        doff, didx = orc.orient(off, idx)
        want = orc.motif3(off, idx, orc.tc(doff, didx)).tolist() + orc.motif4(off, idx).tolist()
        assert got[i].tolist() == want, i
