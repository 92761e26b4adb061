"""4-cycle counters of the giant tasks: one window of keys and many, every list
with a cursor, some and none, with 2-hop bounds down to a handful; and 4-cycle
queries on classes larger than the shared counters.  Against the other
kernels' counts."""
import numpy as np
import pytest

import gpm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", ["rmat", "cl", "star"])
def test_windows_and_cursors(graph, monkeypatch):
    if graph == "rmat":
        n, s, d = gpm.gen_rmat(16, 4, seed=3)
    elif graph == "cl":
        n, s, d = gpm.gen_chung_lu(600001, 2.2, 6.0, seed=4)  # a dozen windows
    else:  # two hubs over 70,000 common neighbours: 32-bit counters, one pair
        n = 300002
        s = np.concatenate([np.arange(70000), np.arange(70000)]).astype(np.int32)
        d = np.concatenate([np.full(70000, n - 2), np.full(70000, n - 1)]).astype(np.int32)
    want = None
    for cursors in (None, "0", "1000"):
        for big in (None, "0"):
            for name, value in (("GPM_C4_CURSORS", cursors), ("GPM_C4_BIG_MIN", big)):
                monkeypatch.delenv(name, raising=False) if value is None else monkeypatch.setenv(name, value)
            g = gpm.Graph.from_edges(n, s, d)
            got = g.motif(4).tolist()
            assert got == g.motif(4).tolist()  # counters are left at zero
            want = want or got
            assert got == want, (cursors, big)
    if graph == "star":
        assert want[3] == 70000 * 69999 // 2


@pytest.mark.parametrize("nl", [1, 2])
def test_cycle_query_on_large_classes(nl):
    """Classes of more vertices than shared counters: over all label tuples the
    embeddings add up to eight per (non-induced) 4-cycle, and a rotated query
    counts the same."""
    n, s, d = gpm.gen_rmat(17, 5, seed=5)
    lab = (np.arange(n) % nl).astype(np.int32)
    g = gpm.Graph.from_edges(n, s, d, labels=lab)
    m = g.motif(4)
    total, got = 8 * int(m[3] + m[4] + 3 * m[5]), {}
    for t in np.ndindex(*[nl] * 4):
        q = gpm.Query(4, [0, 1, 2, 3], [1, 2, 3, 0], list(t))
        got[t] = g.match(q)
        assert g.match(q) == got[t]
    assert sum(got.values()) == total
    for t, c in got.items():
        assert c == got[t[1:] + t[:1]] == got[t[::-1]], t
