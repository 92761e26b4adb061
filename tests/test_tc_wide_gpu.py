"""The triangle plan on more than 2^32 stored keys."""
import numpy as np
import pytest

import gpm

pytestmark = pytest.mark.gpu


def test_more_than_2_32_keys():
    """A directed ring where every vertex points at the next 1024: each of
    them closes a triangle with every later one."""
    import torch
    gpm.trim()
    torch.cuda.empty_cache()
    host = [int(line.split()[1]) >> 20 for line in open("/proc/meminfo") if line.startswith("MemAvailable")][0]
    if host < 60 or torch.cuda.mem_get_info()[0] < 150 << 30:
        pytest.skip("needs 60 GB of host and 150 GB of device memory")
    d, n = 1024, (1 << 22) + 3
    step = np.arange(1, d + 1, dtype=np.int32)
    idx = np.empty((n, d), np.int32)
    for a in range(0, n - d, 1 << 16):
        b = min(n - d, a + (1 << 16))
        idx[a:b] = np.arange(a, b, dtype=np.int32)[:, None] + step
    idx[n - d:] = np.sort((np.arange(n - d, n)[:, None] + step) % n, axis=1)
    assert idx.size > 1 << 32
    g = gpm.Graph.from_csr(np.arange(n + 1, dtype=np.int64) * d, idx.reshape(-1))
    del idx
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    g.tc_async(gpm.TC_BITMAP, 0, out.data_ptr())
    assert out.item() == n * d * (d - 1) // 2
    g.close()
    gpm.trim()
