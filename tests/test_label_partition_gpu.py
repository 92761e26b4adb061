"""The label partition of long and short lists: matches on graphs whose hubs'
lists pass one warp's and one CTA share's size, with 1, 2, 63 and 64 labels."""
import numpy as np
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nl", [1, 2, 33, 63, 64])
@pytest.mark.parametrize("hub", [1023, 1024, 1025, 5000, 16385])
def test_hub_lists(hub, nl):
    n = hub + 3
    rng = np.random.default_rng(hub + nl)
    spokes = np.stack([np.full(hub, hub), np.arange(hub)], 1)
    rim = np.stack([np.arange(hub - 1), np.arange(1, hub)], 1)
    e = np.concatenate([spokes, rim[rng.random(hub - 1) < 0.3], [[hub, hub + 1]]]).astype(np.int32)
    lab = rng.integers(0, nl, n).astype(np.int32)
    lab[0] = nl - 1
    g = gpm.Graph.from_edges(n, e[:, 0], e[:, 1], labels=lab)
    off, idx = orc.build_csr(n, e[:, 0], e[:, 1])
    for shape in ([(0, 1), (1, 2), (2, 0)], [(0, 1), (1, 2)], [(0, 1)]):
        qe = np.array(shape, np.int32)
        k = int(qe.max()) + 1
        qo, qi = orc.build_csr(k, qe[:, 0], qe[:, 1])
        for ql in ([int(lab[hub])] + [0] * (k - 1), [int(lab[hub]), nl - 1, 0][:k], [0, int(lab[hub]), nl - 1][:k]):
            want = orc.match(off, idx, lab, qo, qi, np.array(ql, np.int32))
            assert g.match(gpm.Query(k, qe[:, 0], qe[:, 1], ql)) == want, (shape, ql)
