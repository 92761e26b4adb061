"""Long runs of vertices without neighbours: the offsets at the edges of the
pieces they are filled in, and the time a long unused end takes."""
import time

import numpy as np
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [0, 1, 8190, 8191, 8192, 8193])
def test_runs_around_a_piece(first):
    at = np.cumsum([first, 1, 2, 33, 8190, 8191, 8192, 8193, 8194, 16383, 16384, 16385, 40000])
    n = int(at[-1]) + 1
    for tail in (0, 1, 8190, 8191, 8192, 8193, 20000):
        s, d = at[:-1].astype(np.int32), at[1:].astype(np.int32)
        want_off, want_idx = orc.build_csr(n + tail, s, d)
        off, idx = gpm.Graph.from_edges(n + tail, s, d).csr()
        assert np.array_equal(off, want_off) and np.array_equal(idx, want_idx), tail


def test_time_of_an_unused_end():
    """One edge and 2^27 - 2 unused ids take no longer than 2^21 edges among
    as many ids, which read and write more."""
    n = 1 << 27
    x = np.arange(0, n - 64, 64, dtype=np.int32)

    def build(s, d):
        best = 1e9
        for _ in range(6):
            t = time.perf_counter()
            g = gpm.Graph.from_edges(n, s, d)
            best = min(best, time.perf_counter() - t)
            g.close()
        return best

    spread = build(x, x + 1)
    assert build(x[:1], x[:1] + 1) < 2 * spread
