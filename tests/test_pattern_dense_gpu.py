"""Named patterns where all edges are alike, where a few are not, and where the
bound between them lies, against the oracle."""
import numpy as np
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu


def _dense(n, p, seed):
    iu, iv = np.triu_indices(n, 1)
    k = np.random.default_rng(seed).random(len(iu)) < p
    return n, iu[k].astype(np.int32), iv[k].astype(np.int32)


def _hubs(n, hubs, p, seed):
    """A dense random graph and a few vertices joined to nearly all."""
    _, s, d = _dense(n, p, seed)
    hs, hd = np.divmod(np.arange(hubs * n), n)
    keep = hs != hd
    return n, np.concatenate([s, hs[keep].astype(np.int32)]), np.concatenate([d, hd[keep].astype(np.int32)])


GRAPHS = {
    "complete": lambda: _dense(40, 2.0, 1),
    "dense": lambda: _dense(70, 0.7, 2),
    "half": lambda: _dense(90, 0.4, 3),
    "hubs": lambda: _hubs(120, 4, 0.12, 4),
    "one_hub": lambda: _hubs(110, 1, 0.2, 5),
}


@pytest.mark.parametrize("graph", sorted(GRAPHS))
def test_patterns(graph):
    n, s, d = GRAPHS[graph]()
    off, idx = orc.build_csr(n, s, d)
    g = gpm.Graph.from_edges(n, s, d)
    for p in range(1, 9):
        assert g.pattern(f"P{p}")[0] == orc.pattern_g2miner(off, idx, p), p
