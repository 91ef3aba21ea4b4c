"""Calls on staged batches and launch shapes on synthetic batches, against the CPU
oracle (run on the B200: pytest -m gpu): the allocation-free call, repeated and
re-filled batches, the azimuth-interpolated call and the other launch shapes."""
import numpy as np
import pytest

import oracle
from mbs_fast_b200 import abi
from mbs_fast_b200.beams import BeamBatch
from mbs_fast_b200.handler import GpuHandlerPO
from tests import synthetic as S

# The gates of tests/test_device_paths_gpu.py.
FP64_L2 = 1e-8
GATE = {abi.FP64: FP64_L2, abi.FP32C: 2e-5}


def _l2(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _acc(g, fill=0.0):
    import torch
    return torch.full((g.n_dirs * 16,), fill, dtype=torch.float64, device="cuda:0")


def _np(t, g):
    return t.cpu().numpy().reshape(g.n_az, g.n_zen + 1, 16)


@pytest.mark.gpu
@pytest.mark.parametrize("n_zen", [40, 383, 500, 4000])
@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32C])
def test_noalloc(n_zen, precision):
    """The allocation-free call on a fresh handler: a tail alone, whole tiles, a
    tail beside them, and a grid whose scratch holds fewer chunks; both sums,
    twice in a row and in a captured graph; no device memory is taken.  Its
    chunk sums are grouped differently: 1e-12 against the staged call."""
    import torch
    g, w = S.grid(5, n_zen), S.wave()
    b = S.ragged(70, 9, 12.0, n_zen)
    warm = GpuHandlerPO(g, w)                   # loads the module and its array
    ws = warm.stage(b)
    warm.diffract_staged_noalloc(ws, _acc(g).data_ptr(), _acc(g).data_ptr(), precision=precision)
    warm.diffract_staged_noalloc(ws, _acc(g).data_ptr(), precision=precision)
    torch.cuda.synchronize()
    ws.free()
    warm.close()
    h = GpuHandlerPO(g, w)
    st = h.stage(b)
    M, N, P = _acc(g), _acc(g), _acc(g)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        h.diffract_staged_noalloc(st, M.data_ptr(), N.data_ptr(), precision=precision)
        h.diffract_staged_noalloc(st, P.data_ptr(), precision=precision)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    R, RN, RP = _acc(g), _acc(g), _acc(g)
    h.diffract_staged(st, R.data_ptr(), RN.data_ptr(), precision=precision)
    h.diffract_staged(st, RP.data_ptr(), precision=precision)
    torch.cuda.synchronize()
    for got, want in ((M, R), (N, RN), (P, RP)):
        assert _l2(got.cpu(), 2 * want.cpu()) < 1e-12
    assert _l2(_np(RP, g), oracle.po_diffract(b, g, w)) < GATE[precision]
    graph = torch.cuda.CUDAGraph()
    Q = _acc(g)
    with torch.cuda.graph(graph):
        h.diffract_staged_noalloc(st, Q.data_ptr(), precision=precision,
                                  stream=torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(Q, P)
    del graph
    st.free()
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("index", [[0], [2, 2, 2], [3, 1, 0, 3], [0, 4, 1], list(range(6)) * 20])
def test_repeated_batches(index):
    """Orientations repeated, out of order and with gaps, re-weighted: as a
    batch made of them; a view of a view; the source still as it was."""
    import torch
    g, w = S.grid(4, 130), S.wave()
    b = S.ragged(6, 12, 12.0, 4)
    weight = np.random.default_rng(len(index)).uniform(0.2, 1.5, len(index))
    parts = []
    for i, wt in zip(index, weight):
        one = b.select(i, 1)
        one.orient_weight = np.array([wt])
        parts.append(one)
    want = oracle.po_diffract(BeamBatch.concat(parts), g, w)
    h = GpuHandlerPO(g, w)
    src = h.stage(b)
    before = _acc(g)
    h.diffract_staged(src, before.data_ptr(), precision=abi.FP64)
    v = h.stage_repeat(src, index, weight)
    for precision in (abi.FP64, abi.FP32C):
        acc = _acc(g)
        h.diffract_staged(v, acc.data_ptr(), precision=precision)
        torch.cuda.synchronize()
        assert _l2(_np(acc, g), want) < GATE[precision]
    v.free()
    after = _acc(g)
    h.diffract_staged(src, after.data_ptr(), precision=abi.FP64)
    torch.cuda.synchronize()
    assert torch.equal(before, after)
    src.free()
    h.close()


@pytest.mark.gpu
def test_refilled_batches():
    """A batch re-filled with larger, smaller, empty and refused ones, in its
    first block and in the pool, with another batch staged between: always what
    the batch staged anew gives."""
    import torch
    g, w = S.grid(4, 60), S.wave()
    h = GpuHandlerPO(g, w)
    small, mid, large = S.ragged(3, 5, 8.0, 1), S.ragged(20, 40, 12.0, 2), S.ragged(200, 80, 12.0, 3)
    st = h.stage(mid)
    for b in (small, mid, large, small, mid.select(0, 0), large, mid):
        h.restage(st, b)
        other = h.stage(mid)
        acc, ref = _acc(g), _acc(g)
        fresh = h.stage(b)
        h.diffract_staged(st, acc.data_ptr(), precision=abi.FP64)
        h.diffract_staged(fresh, ref.data_ptr(), precision=abi.FP64)
        torch.cuda.synchronize()
        assert torch.equal(acc, ref)
        if b.n_orient in (3, 20):
            assert _l2(_np(acc, g), oracle.po_diffract(b, g, w)) < FP64_L2
        other.free()
        fresh.free()
    bad = small.select(0, 3)
    bad.vert_offsets = bad.vert_offsets.copy()
    bad.vert_offsets[1] = 1                     # an aperture of one vertex
    with pytest.raises(RuntimeError):
        h.restage(st, bad)
    acc = _acc(g)
    h.diffract_staged(st, acc.data_ptr(), precision=abi.FP64)
    torch.cuda.synchronize()
    assert not acc.any()                        # holds no orientations until re-filled
    h.restage(st, small)
    h.diffract_staged(st, acc.data_ptr(), precision=abi.FP64)
    torch.cuda.synchronize()
    assert _l2(_np(acc, g), oracle.po_diffract(small, g, w)) < FP64_L2
    st.free()
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n_low,n_full,n_zen", [(5, 5, 20), (6, 17, 70), (16, 48, 400)])
def test_azimuth_interpolated_call(n_low, n_full, n_zen):
    """The azimuth-interpolated host call after another call on the context (its
    sums are stored over what the last one left), both sums: the direct grid
    interpolated by the oracle."""
    full, w = S.grid(n_full, n_zen), S.wave()
    low = S.grid(n_low, n_zen)
    b = S.ragged(9, 20, 12.0, n_full)
    h = GpuHandlerPO(full, w)
    hl = GpuHandlerPO(low, w)
    for precision in (abi.FP64, abi.FP32C):
        M = h.new_mueller()
        assert h.handle_orientations_to_local_gpu(b, M, precision=precision)
        got, got_n = h.diffract_fft_phi(b, low, n_full, precision, noshadow=True)
        again, _ = h.diffract_fft_phi(b, low, n_full, precision, noshadow=True)
        L, LN = hl.new_mueller(), hl.new_mueller()
        assert hl.handle_orientations_to_local_gpu(b, L, LN, precision=precision)
        assert np.array_equal(got, again)
        assert _l2(got, oracle.phi_upsample_fft(L, n_full)) < 1e-12
        assert _l2(got_n, oracle.phi_upsample_fft(LN, n_full)) < 1e-12
    h.close()
    hl.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision,variant", [(abi.FP64, v) for v in range(5)] + [(abi.FP32C, v) for v in range(6)])
def test_launch_shapes(precision, variant):
    """Every launch shape with more beams than a stage holds (64 to 128), empty
    and single-beam orientations, near-forward rows, and row counts around the
    shapes' tiles."""
    w = S.wave()
    for n_zen, beams in ((10, 150), (130, 63), (200, 65)):
        b, g = S.ragged(4, beams, 12.0, 3 * beams), S.grid(3, n_zen, plates=True)
        h = GpuHandlerPO(g, w)
        h.set_variant(precision, variant)
        M = h.new_mueller()
        assert h.handle_orientations_to_local_gpu(b, M, precision=precision)
        h.close()
        assert _l2(M, oracle.po_diffract(b, g, w)) < GATE[precision]
