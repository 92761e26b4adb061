"""Named patterns on more than 2^31 stored entries, with the heavy edges among
the last ones."""
import numpy as np
import pytest

import gpm

pytestmark = pytest.mark.gpu


def test_heavy_edges_past_2_31():
    """A long cycle, which holds no pattern with a triangle, and behind it a
    dense random graph, which alone gives the same counts."""
    import torch
    gpm.trim()
    torch.cuda.empty_cache()
    host = [int(line.split()[1]) >> 20 for line in open("/proc/meminfo") if line.startswith("MemAvailable")][0]
    if host < 60 or torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("needs 60 GB of host and 80 GB of device memory")
    k, n = 130, (1 << 30) + 5  # vertices of the dense graph and of the cycle
    iu, iv = np.triu_indices(k, 1)
    keep = np.random.default_rng(5).random(len(iu)) < 0.85
    small = gpm.Graph.from_edges(k, iu[keep], iv[keep])
    soff, sidx = small.csr()
    idx = np.empty(2 * n + len(sidx), np.int32)
    idx[0:2 * n:2] = np.arange(-1, n - 1, dtype=np.int32)  # each vertex's two neighbours, ascending
    idx[1:2 * n:2] = np.arange(1, n + 1, dtype=np.int32)
    idx[0:2] = 1, n - 1
    idx[2 * n - 2:2 * n] = 0, n - 2
    idx[2 * n:] = sidx + n
    off = np.concatenate([np.arange(n, dtype=np.int64) * 2, 2 * n + soff])
    g = gpm.Graph.from_csr(off, idx)
    del idx, off
    for p in ("P7", "P8"):
        got, want = g.pattern(p), small.pattern(p)
        assert got[0] == want[0] > 0 and got[1].tolist() == want[1].tolist(), p
    g.close()
    gpm.trim()
