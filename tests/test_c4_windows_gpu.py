"""4-cycle counters of giant tasks against the oracle: the hash table and the
windows it stands in for, with a cursor per list and without, in one window and
several, narrow and wide (graphs of more than 400,000 vertices)."""
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu

GRAPHS = {
    "one_window": lambda: gpm.gen_chung_lu(3000, 2.1, 12.0, seed=1),
    "two_windows": lambda: gpm.gen_chung_lu(70001, 2.2, 6.0, seed=2),
    "at_the_line": lambda: gpm.gen_chung_lu(400000, 2.4, 2.5, seed=3),
    "wide": lambda: gpm.gen_chung_lu(400001, 2.4, 2.5, seed=3),
    "wide_several": lambda: gpm.gen_chung_lu(500001, 2.4, 3.0, seed=4),
}


@pytest.mark.parametrize("graph", sorted(GRAPHS))
def test_every_way_against_the_oracle(graph, monkeypatch):
    n, s, d = GRAPHS[graph]()
    want = orc.motif4(*orc.build_csr(n, s, d)).tolist()
    assert want[3] > 0
    monkeypatch.setenv("GPM_C4_BIG_MIN", "0")  # tasks from a bound of 256 on
    for hash_max in (None, "0", "1000"):
        for cursors in (None, "0", "40"):
            for name, value in (("GPM_C4_HASH_MAX", hash_max), ("GPM_C4_CURSORS", cursors)):
                monkeypatch.delenv(name, raising=False) if value is None else monkeypatch.setenv(name, value)
            g = gpm.Graph.from_edges(n, s, d)
            for _ in range(2):
                assert g.motif(4).tolist() == want, (hash_max, cursors)
