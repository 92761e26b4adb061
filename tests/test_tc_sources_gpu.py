"""The per-entry sources of the binary-search count, which its first call
fills: on one stream for counts on others at once, and inside a capture for
counts outside of it before the first replay."""
import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu


def _case(seed):
    n, s, d = gpm.gen_er(150, 4000, seed=seed)
    doff, didx = orc.orient(*orc.build_csr(n, s, d))
    return gpm.Graph.from_edges(n, s, d).orient(), orc.tc(doff, didx)


@pytest.mark.parametrize("variant", ["TC_BSEARCH", "TC_MERGE", "TC_AUTO"])
def test_first_counts_on_several_streams(variant):
    import torch
    streams = [torch.cuda.Stream() for _ in range(4)]
    for seed in range(8):
        g, want = _case(seed)
        out = torch.full((5,), -1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        for i, s in enumerate(streams):
            g.tc_async(getattr(gpm, variant), s.cuda_stream, out[i:].data_ptr())
        assert g.tc(gpm.E_CENTRIC) == want
        torch.cuda.synchronize()
        assert out[:4].tolist() == [want] * 4


@pytest.mark.parametrize("variant,warm", [("TC_BSEARCH", None), ("TC_AUTO", "TC_BITMAP"), ("TC_AUTO", "TC_AUTO")])
def test_first_count_inside_a_capture(variant, warm):
    import torch
    g, want = _case(3)
    _case(4)[0].close()  # leaves idle blocks behind
    out = torch.full((2,), -1, dtype=torch.int64, device="cuda")
    side = torch.cuda.Stream()
    if warm:
        g.tc_async(getattr(gpm, warm), side.cuda_stream, out.data_ptr())
        side.synchronize()
        out.fill_(-1)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed" if warm is None else "global"):
        g.tc_async(getattr(gpm, variant), torch.cuda.current_stream().cuda_stream, out.data_ptr())
    g.tc_async(gpm.TC_BSEARCH, side.cuda_stream, out[1:].data_ptr())
    side.synchronize()
    assert out.tolist() == [-1, want]
    for _ in range(3):
        out.fill_(-1)
        graph.replay()
        assert g.tc(gpm.E_CENTRIC) == want
        torch.cuda.synchronize()
        assert out[0].item() == want
    del graph
