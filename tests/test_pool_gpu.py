"""Released device memory: kept for later calls only when nothing of a caller's
can still use it, within its bound, and sound with several threads, streams and
captures."""
import threading

import pytest

import gpm
import _oracle as orc

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


def _empty_pool():
    g = gpm.Graph.from_edges(2, [0], [1])
    g.drop_plans()  # gives the idle blocks back
    g.close()


@pytest.mark.parametrize("how", ["stream", "capture"])
def test_memory_a_callers_stream_may_use_is_not_kept(how):
    """The handle is closed while its last count still runs on the caller's
    stream, and new graphs are built at once."""
    import torch
    side = torch.cuda.Stream()
    n, s, d = gpm.gen_rmat(14, 16, seed=3)
    want = orc.tc(*orc.orient(*orc.build_csr(n, s, d)))
    out = torch.zeros(2, dtype=torch.int64, device="cuda")
    first = gpm.Graph.rmat(18, 16, seed=1).orient()
    big = first.tc()
    first.close()
    for _ in range(3):
        _empty_pool()
        torch.cuda.synchronize()
        g = gpm.Graph.rmat(18, 16, seed=1).orient()
        g.tc_async(gpm.TC_BITMAP, side.cuda_stream, out.data_ptr())
        side.synchronize()
        _empty_pool()
        torch.cuda.synchronize()
        before = _free()
        if how == "capture":
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                g.tc_async(gpm.TC_BITMAP, torch.cuda.current_stream().cuda_stream, out.data_ptr())
        out.fill_(-1)
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            graph.replay() if how == "capture" else g.tc_async(gpm.TC_BITMAP, side.cuda_stream, out.data_ptr())
        g.close()
        # 6.9 M list entries with their plan: everything is with the driver again
        assert _free() - before > 80 * MIB
        h = gpm.Graph.from_edges(n, s, d).orient()
        h.tc_async(gpm.TC_BITMAP, 0, out[1:].data_ptr())
        torch.cuda.synchronize()
        assert out.tolist() == [big, want]
        h.close()
        if how == "capture":
            del graph


def test_bound():
    """Lists of embeddings want one block of a size of their own each."""
    import torch
    g = gpm.Graph.from_edges(3, [0, 1], [1, 2], labels=[0, 0, 0])
    q = gpm.Query(2, [0], [1], [0, 0])
    _empty_pool()
    torch.cuda.synchronize()
    start = _free()
    for mib in (700, 800, 900, 1000, 1100, 1200, 1300, 1400):
        buf = torch.empty(mib * MIB // 4, dtype=torch.int32)
        written = gpm.c_uint64()
        gpm.check(gpm.lib.gpm_match_list(g.h, q.h, mib * MIB // 8, gpm.c_void_p(buf.data_ptr()), written))
        assert written.value == 4
        assert start - _free() < 4096 * MIB + 64 * MIB
    assert start - _free() > 2048 * MIB
    _empty_pool()
    assert start - _free() < 64 * MIB


def test_trim_without_a_handle():
    import torch
    gpm.trim()
    torch.cuda.synchronize()
    start = _free()
    g = gpm.Graph.rmat(17, 16, seed=1).orient()
    want = g.tc()
    g.close()
    assert start - _free() > 64 * MIB  # kept for the next graph
    gpm.trim()
    assert start - _free() < 32 * MIB
    g = gpm.Graph.rmat(17, 16, seed=1).orient()
    assert g.tc() == want


@pytest.mark.parametrize("mib", [3100, 4400])
def test_the_last_of_the_memory(mib):
    """A buffer that fits, but not rounded up to a size of the pool's."""
    import torch
    g = gpm.Graph.from_edges(3, [0, 1], [1, 2], labels=[0, 0, 0])
    q = gpm.Query(2, [0], [1], [0, 0])
    assert g.match(q) == 4  # the label partition is there
    buf = torch.empty(mib * MIB // 4, dtype=torch.int32)
    _empty_pool()
    torch.cuda.synchronize()
    held = torch.empty(_free() - (mib + 64) * MIB, dtype=torch.uint8, device="cuda")
    written = gpm.c_uint64()
    try:
        assert mib * MIB < _free() < (mib + 130) * MIB
        gpm.check(gpm.lib.gpm_match_list(g.h, q.h, mib * MIB // 8, gpm.c_void_p(buf.data_ptr()), written))
    finally:
        del held
        torch.cuda.empty_cache()
    assert written.value == 4


def test_threads_and_streams():
    """Graphs built, counted on a stream of the thread's own, and closed, in
    several threads at once."""
    import torch
    cases = []
    for i in range(4):
        n, s, d = gpm.gen_rmat(11 + i % 2, 16, seed=i)
        doff, didx = orc.orient(*orc.build_csr(n, s, d))
        cases.append((n, s, d, orc.tc(doff, didx), orc.clique(doff, didx, 4)))
    torch.cuda.synchronize()
    errors = []

    def work(i):
        try:
            n, s, d, want, want4 = cases[i]
            st = torch.cuda.Stream()
            out = torch.zeros(1, dtype=torch.int64, device="cuda")
            for r in range(12):
                g = gpm.Graph.from_edges(n, s, d).orient()
                g.tc_async(gpm.TC_BITMAP if r % 2 else gpm.TC_HASH, st.cuda_stream, out.data_ptr())
                if r % 3:
                    assert g.clique(4) == want4, (i, r)
                g.close()  # the count may still be running
                st.synchronize()
                assert out.item() == want, (i, r)
        except BaseException as e:  # reported by the test's own thread
            errors.append((i, e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors


def test_release_beside_another_threads_capture():
    """A count, its release and the reuse of its memory leave a capture of
    another thread intact."""
    import torch
    n, s, d = gpm.gen_rmat(12, 16, seed=9)
    want = orc.tc(*orc.build_csr(n, s, d))
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    got = []

    def work():
        for _ in range(5):
            g = gpm.Graph.from_edges(n, s, d)
            got.append(g.tc())
            g.close()

    graph, st = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(st):
        graph.capture_begin(capture_error_mode="thread_local")
        x.add_(1)
        t = threading.Thread(target=work)
        t.start()
        t.join()
        x.add_(1)
        graph.capture_end()
    assert got == [want] * 5
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 1000
