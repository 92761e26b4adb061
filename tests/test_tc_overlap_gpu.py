"""Triangle counts of one handle that overlap on the GPU: a synchronous count
made while asynchronous ones run on a stream of the caller's, in every pairing
of kernels, and first counts on two streams where nothing is kept between
launches.  Both counts, and the next one, equal the oracle's."""
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu

GRAPHS = {
    "tiny": lambda: gpm.gen_er(300, 4000, seed=1),          # binary search
    "short": lambda: gpm.gen_er(60001, 420000, seed=2),     # merged lists
    "even": lambda: gpm.gen_er(20003, 330000, seed=3),      # hash kernel, few counts
    "skewed": lambda: gpm.gen_rmat(15, 16, seed=4),         # rank plan, dense core
}


def _case(name):
    n, s, d = GRAPHS[name]()
    doff, didx = orc.orient(*orc.build_csr(n, s, d))
    return gpm.Graph.from_edges(n, s, d).orient(), orc.tc(doff, didx)


@pytest.mark.parametrize("variant", ["TC_AUTO", "TC_HASH", "TC_BITMAP", "TC_BSEARCH"])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_synchronous_beside_asynchronous(name, variant):
    import torch
    g, want = _case(name)
    side = torch.cuda.Stream()  # does not wait for the default stream
    out = torch.zeros(8, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for i in range(16):
        for j in range(8):  # one after another on their stream, so the last runs beside the synchronous count
            g.tc_async(getattr(gpm, variant), side.cuda_stream, out[j:].data_ptr())
        assert g.tc(i % 2) == want, i
        side.synchronize()
        assert out.tolist() == [want] * 8, i
        assert g.tc(i % 2) == want, i


@pytest.mark.parametrize("name", ["tiny", "short"])
def test_first_counts_on_two_streams(name):
    import torch
    g, want = _case(name)
    streams = [torch.cuda.Stream() for _ in range(4)]
    out = torch.zeros(4, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(10):
        out.fill_(-1)
        torch.cuda.synchronize()
        for i, s in enumerate(streams):
            g.tc_async(gpm.TC_AUTO, s.cuda_stream, out[i:].data_ptr())
        torch.cuda.synchronize()
        assert out.tolist() == [want] * 4
