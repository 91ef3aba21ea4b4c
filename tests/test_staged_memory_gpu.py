"""Device memory of staged batches: who may still read it when it is freed, what
outlives the context, and what a context keeps (run on the B200: pytest -m gpu)."""
import ctypes as C
import threading

import numpy as np
import pytest

from mbs_fast_b200 import abi
from mbs_fast_b200.handler import GpuHandlerPO, lib
from tests import synthetic as S


def _acc(g):
    import torch
    return torch.zeros(g.n_dirs * 16, dtype=torch.float64, device="cuda:0")


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_free_beside_another_threads_capture(mode):
    """A batch freed while another thread has a capture open: the capture goes
    on, its replay is right, and the batch's memory serves the next one."""
    import torch
    g, w = S.grid(4, 20), S.wave()
    h = GpuHandlerPO(g, w)
    b = S.batch(40, 60, 12.0, 5)
    ref = _acc(g)
    st = h.stage(b)
    h.diffract_staged(st, ref.data_ptr(), precision=abi.FP64)
    torch.cuda.synchronize()
    x = torch.zeros(1 << 16, device="cuda:0")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode=mode):
        x.add_(1)
        t = threading.Thread(target=st.free)
        t.start()
        t.join()
        x.add_(1)
    graph.replay()
    torch.cuda.synchronize()
    assert float(x.min()) == float(x.max()) == 2.0
    acc = _acc(g)
    st = h.stage(b)
    h.diffract_staged(st, acc.data_ptr(), precision=abi.FP64)
    torch.cuda.synchronize()
    assert torch.equal(acc, ref)
    st.free()
    h.close()


@pytest.mark.gpu
def test_free_while_several_streams_read():
    """Readers on more streams than are tracked, and a captured reader whose
    replay is in flight: the freed memory is staged again at once, and every
    result is that of the first batch."""
    import torch
    g, w = S.grid(16, 100), S.wave()
    h = GpuHandlerPO(g, w)
    b, other = S.batch(30, 60, 12.0, 5), S.batch(30, 60, 12.0, 6)
    ref = _acc(g)
    st = h.stage(b)
    h.diffract_staged(st, ref.data_ptr(), precision=abi.FP64)
    torch.cuda.synchronize()
    st.free()
    for n_streams in (1, 3, 20):
        st = h.stage(b)
        streams = [torch.cuda.Stream() for _ in range(n_streams)]
        accs = [_acc(g) for _ in streams]
        torch.cuda.synchronize()
        for i, (s, a) in enumerate(zip(streams, accs)):
            if i:
                s.wait_stream(streams[i - 1])     # the calls share the context's partial sums
            h.diffract_staged(st, a.data_ptr(), precision=abi.FP64, stream=s.cuda_stream, stats=False)
        st.free()
        st2 = h.stage(other)
        torch.cuda.synchronize()
        assert all(torch.equal(a, ref) for a in accs)
        st2.free()
    st = h.stage(b)
    acc = _acc(g)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        h.diffract_staged(st, acc.data_ptr(), precision=abi.FP64,
                          stream=torch.cuda.current_stream().cuda_stream, stats=False)
    graph.replay()
    st.free()                                     # waits for the replay
    st2 = h.stage(other)
    torch.cuda.synchronize()
    assert torch.equal(acc, ref)
    st2.free()
    del graph
    h.close()


@pytest.mark.gpu
def test_batches_outlive_their_context():
    """Staged, re-filled and repeated batches freed after their handler was
    closed, over and over: nothing is left behind (64 MiB for the driver's own
    blocks)."""
    import torch
    g, w = S.grid(4, 20), S.wave()
    small, large = S.batch(10, 30, 12.0, 5), S.batch(200, 60, 12.0, 6)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(12):
        h = GpuHandlerPO(g, w)
        acc = _acc(g)
        a, r = h.stage(large), h.stage(small)
        h.restage(r, large)
        v = h.stage_repeat(a, [3, 1], [0.5, 0.5])
        h.diffract_staged(v, acc.data_ptr())
        h.diffract_staged(r, acc.data_ptr())
        torch.cuda.synchronize()
        h.close()
        v.free()
        r.free()
        a.free()
    del acc
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] > before - (64 << 20)


def _room(h, per_orient=10_000, n=400_000):
    """Orientations of one large aperture each that mbs_po_select_batch says fit."""
    bo = np.arange(n + 1, dtype=np.int64)
    vo = bo * per_orient
    b = abi.Beams()
    b.n_orient, b.n_beams, b.n_verts = n, n, int(vo[-1])
    b.beam_offsets, b.vert_offsets = abi.ptr(bo, C.c_int64), abi.ptr(vo, C.c_int64)
    out = C.c_int()
    assert lib().mbs_po_select_batch(h.ctx, C.byref(b), 0, n * 10, 0.88, C.byref(out)) == 0
    assert out.value < n
    return out.value


@pytest.mark.gpu
def test_kept_memory_counts_as_free():
    """A freed batch's memory is free to the next one: mbs_po_select_batch
    answers as if it had gone back to the device, and no more than 256 MiB stays
    (to 2 MiB a block for the driver's granularity)."""
    import torch
    h = GpuHandlerPO(S.grid(4, 20), S.wave())
    b = S.batch(1000, 100, 12.0, 5)               # about 130 MB of records
    st = h.stage(b)                               # the upload area has its size now
    full = torch.cuda.mem_get_info()[0]
    held = _room(h)
    st.free()
    kept = torch.cuda.mem_get_info()[0] - full
    freed = _room(h)
    # an orientation of 10,000 vertices takes 1.13 MB
    assert (freed - held) * 1.13e6 > 0.8 * 0.88 * 1.2e8
    sts = [h.stage(b) for _ in range(4)]
    low = torch.cuda.mem_get_info()[0]
    for s in sts:
        s.free()
    back = torch.cuda.mem_get_info()[0] - low
    assert kept < 1e7                             # the one freed batch was kept
    assert back > 2 * 1.2e8 - (4 << 21)           # of four, those beyond 256 MiB went back
    h.close()
