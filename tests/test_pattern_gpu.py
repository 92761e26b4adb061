"""Named patterns on graphs whose edges fall on both sides of the rule that
shares an edge out over several warps: a hub joined to a rim (its edges heavy,
the rim's light), a power-law graph, and one with light edges alone."""
import numpy as np
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu


def wheel(k):
    hub = np.stack([np.full(k, k), np.arange(k)], 1)
    rim = np.stack([np.arange(k), (np.arange(k) + 1) % k], 1)
    chords = np.stack([np.arange(0, k, 3), (np.arange(0, k, 3) + 5) % k], 1)
    e = np.concatenate([hub, rim, chords]).astype(np.int32)
    return k + 1, e[:, 0], e[:, 1]


GRAPHS = {
    "wheel45": lambda: wheel(45),
    "wheel190": lambda: wheel(190),
    "power": lambda: gpm.gen_chung_lu(260, 2.1, 7.0, seed=3),
    "light": lambda: gpm.gen_er(120, 300, seed=4),
}


@pytest.mark.parametrize("graph", sorted(GRAPHS))
def test_patterns_against_oracle(graph):
    n, s, d = GRAPHS[graph]()
    off, idx = orc.build_csr(n, s, d)
    g = gpm.Graph.from_edges(n, s, d)
    for p in (2, 3, 5, 6, 7, 8):
        assert g.pattern("P%d" % p)[0] == orc.pattern_g2miner(off, idx, p), p
