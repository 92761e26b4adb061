"""gpm_tc chooses its kernel by the graph and by the counts made on it: every
one of a row of counts, before and after the plan is built, equals the other
variants' and the oracle's, in both modes, on oriented and symmetric lists."""
import numpy as np
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu

GRAPHS = {
    "tiny": lambda: gpm.gen_er(40, 90, seed=1),
    "rmat10": lambda: gpm.gen_rmat(10, 16, seed=2),
    "rmat12": lambda: gpm.gen_rmat(12, 10, seed=2),
    "rmat13": lambda: gpm.gen_rmat(13, 16, seed=2),
    # more tail tasks than eight per resident warp
    "er200k": lambda: gpm.gen_er(200003, 1400000, seed=3),
    "hubs": lambda: gpm.gen_chung_lu(30001, 2.1, 40.0, seed=4),
    # short lists around the merging kernel's limit, a last warp of one vertex
    "er65": lambda: gpm.gen_er(65, 200, seed=5),
    "er5k": lambda: gpm.gen_er(4737, 40000, seed=6),
    "clique25": lambda: (25, *(x.astype(np.int32) for x in np.triu_indices(25, 1))),
    "clique26": lambda: (26, *(x.astype(np.int32) for x in np.triu_indices(26, 1))),
}


@pytest.mark.parametrize("oriented", [True, False])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_every_count_of_a_row(name, oriented):
    import torch
    n, s, d = GRAPHS[name]()
    off, idx = orc.build_csr(n, s, d)
    g = gpm.Graph.from_edges(n, s, d)
    if oriented:
        off, idx = orc.orient(off, idx)
        g.orient()
    want = orc.tc(off, idx)
    out = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    for i in range(24):
        assert g.tc(gpm.E_CENTRIC if i % 2 else gpm.V_CENTRIC) == want, i
        g.tc_async(gpm.TC_HASH, stream, out.data_ptr())
        assert int(out.item()) == want, i
    for variant in (gpm.TC_BITMAP, gpm.TC_AUTO, gpm.TC_AUTO):
        out.fill_(-1)
        g.tc_async(variant, stream, out.data_ptr())
        assert int(out.item()) == want, variant
    g.drop_plans()
    assert g.tc() == want


def test_no_entries():
    g = gpm.Graph.from_edges(5, [1], [1])
    assert [g.tc() for _ in range(3)] == [0, 0, 0]
    assert g.orient().tc(gpm.E_CENTRIC) == 0
