"""The device paths at the sizes where their work splits change, on synthetic
batches, against the CPU oracle (run on the B200: pytest -m gpu)."""
import numpy as np
import pytest

import oracle
from mbs_fast_b200 import abi
from mbs_fast_b200.handler import GpuHandlerPO
from tests import synthetic as S

# FP64 against the oracle: both carry vertex phases of up to 1.3e3 rad with
# rounding errors near 2e-13 rad; the gate of the traced FP64 parity tests
# (tests/test_parity_gpu.py).
FP64_L2 = 1e-8


def _l2(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.gpu
@pytest.mark.parametrize("n_orient,beams", [(1, 2), (1, 33), (3, 70), (9, 31), (20, 64), (40, 8), (2, 700)])
def test_polar_rows(n_orient, beams):
    """Polar rows: one warp to a whole CTA per orientation, ragged and empty
    orientations, with and without the sums over internal beams."""
    b = S.ragged(n_orient, beams, 20.0, 3 + n_orient + beams)
    g, w = S.grid(5, 3), S.wave()
    M0, N0 = oracle.po_diffract(b, g, w, noshadow=True)
    h = GpuHandlerPO(g, w)
    M, N, P = h.new_mueller(), h.new_mueller(), h.new_mueller()
    assert h.handle_orientations_to_local_gpu(b, M, N, precision=abi.FP64)
    assert h.handle_orientations_to_local_gpu(b, P, precision=abi.FP64)
    h.close()
    for t in (0, 3):
        assert _l2(M[:, t], M0[:, t]) < FP64_L2
        assert _l2(P[:, t], M0[:, t]) < FP64_L2
        assert _l2(N[:, t], N0[:, t]) < FP64_L2
        assert all(np.array_equal(M[0, t], M[p, t]) for p in range(5))
    assert _l2(M, M0) < FP64_L2


@pytest.mark.gpu
@pytest.mark.parametrize("n_orient", [1, 7, 13, 65, 130])
@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32C])
def test_small_batches_split_into_single_orientations(n_orient, precision):
    """Few orientations on a small grid: one to a few orientations per chunk,
    up to 64 chunk planes, ragged beam counts, empty orientations.  FP32C: the
    gate of the traced FP32C parity tests on the whole grid's L2."""
    b = S.ragged(n_orient, 9, 15.0, 100 + n_orient)
    g, w = S.grid(3, 6), S.wave()
    M0, N0 = oracle.po_diffract(b, g, w, noshadow=True)
    h = GpuHandlerPO(g, w)
    M, N, P = h.new_mueller(), h.new_mueller(), h.new_mueller()
    assert h.handle_orientations_to_local_gpu(b, M, N, precision=precision)
    assert h.handle_orientations_to_local_gpu(b, P, precision=precision)
    h.close()
    gate = FP64_L2 if precision == abi.FP64 else 2e-5
    assert _l2(M, M0) < gate and _l2(P, M0) < gate
    assert _l2(N, N0) < (gate if precision == abi.FP64 else 1e-4)


@pytest.mark.gpu
@pytest.mark.parametrize("n_sizes", [1, 3, 65])
def test_small_multisize_batches(n_sizes):
    """Chunk planes shared by the sizes: up to 64 in all, then one per size."""
    b = S.batch(4, 6, 5.0, 7, raw=True, absorbing=True)
    g, w = S.grid(3, 5), S.wave(True)
    scales = np.geomspace(0.5, 3.0, n_sizes)
    h = GpuHandlerPO(g, w)
    ms = [h.new_mueller() for _ in scales]
    assert h.handle_orientations_to_local_gpu_multik(b, 0, 4, scales, w.wave_index, ms)
    h.close()
    for s, M in list(zip(scales, ms))[::16] + [(scales[-1], ms[-1])]:
        assert _l2(M, oracle.po_diffract(oracle.scale_batch(b, s, w.wave_index, w.abs_coeff), g, w)) < FP64_L2


def _with_nv(n_beams, nv, size, seed):
    """One orientation whose beams are regular-ish polygons of nv vertices
    (the generator's polygons stop at 8)."""
    b = S.batch(1, n_beams, size, seed)
    rng = np.random.default_rng(seed)
    n = b.n_beams
    ang = (np.arange(nv)[None, :] + rng.uniform(-0.3, 0.3, (n, nv))) * (2 * np.pi / nv)
    r = size * rng.uniform(0.05, 0.6, (n, 1))
    x, y = r * np.cos(ang), 0.6 * r * np.sin(ang)
    dx, dy = np.roll(x, -1, 1) - x, np.roll(y, -1, 1) - y
    b.vert_offsets = np.arange(n + 1, dtype=np.int64) * nv
    c = lambda a: np.ascontiguousarray(a.ravel())
    b.vx, b.vy, b.slope_yx, b.slope_xy = c(x), c(y), c(dy / dx), c(dx / dy)
    b.edge_flags = np.full(n * nv, 3, np.uint8)
    g = b.beam_geom.copy()
    g[:, abi.G_AREA] = 0.5 * np.sum(x * np.roll(y, -1, 1) - np.roll(x, -1, 1) * y, 1)
    b.beam_geom = g
    return b


@pytest.mark.gpu
@pytest.mark.parametrize("n_beams,nv", [(1, 3), (15, 31), (16, 8), (17, 9), (33, 4), (160, 31)])
def test_packed_records(n_beams, nv):
    """Record building 16 beams at a time: beam counts around the group, 3 to
    31 vertices (fewer and more than the 8 lanes of a beam).  FP64 without
    moments, FP32C with them, and the staged batch, which has both, bit for
    bit as the host calls.  The FP32C gate is that of the traced parity tests,
    whose apertures have 3 to 12 vertices, so it is asked of those here."""
    import torch
    b = _with_nv(n_beams, nv, 6.0, 11 * n_beams + nv)
    g, w = S.grid(4, 12, plates=True), S.wave()
    M0 = oracle.po_diffract(b, g, w)
    h = GpuHandlerPO(g, w)
    st = h.stage(b)
    for prec, gate in ((abi.FP64, FP64_L2), (abi.FP32C, 2e-5)):
        M = h.new_mueller()
        assert h.handle_orientations_to_local_gpu(b, M, precision=prec)
        if prec == abi.FP64 or nv <= 12:
            assert _l2(M, M0) < gate
            assert _l2(M[:, :4], M0[:, :4]) < gate
        acc = torch.zeros(M.size, dtype=torch.float64, device="cuda:0")
        h.diffract_staged(st, acc.data_ptr(), precision=prec)
        torch.cuda.synchronize()
        assert np.array_equal(acc.cpu().numpy(), M.ravel())
    st.free()
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n_orient,beams", [(1, 2), (3, 40), (5, 127), (5, 300), (70, 33), (2, 1300)])
@pytest.mark.parametrize("phase_average", [0, 1])
def test_extinction_splits(n_orient, beams, phase_average):
    """Extinction with one to four warps per orientation, ragged and empty
    orientations, with and without the phase-averaged form.  Both sides sum
    the same terms; internal beams carry a phase of k (1e4 um + ...) = 1.2e5
    rad (rounding 1.5e-11): 1e-9 of the largest orientation's value."""
    b, w = S.ragged(n_orient, beams, 20.0, 5 + n_orient + beams), S.wave()
    w.ot_phase_average = phase_average
    want = oracle.po_extinction(b, w)
    h = GpuHandlerPO(S.grid(1, 2), w)
    got = h.extinction(b)
    h.close()
    assert np.max(np.abs(got - want)) <= 1e-9 * np.max(np.abs(want))


@pytest.mark.gpu
@pytest.mark.parametrize("n_points,n_az,n_orient,beams,nv", [
    (1, 1, 1, 2, 0), (64, 3, 2, 63, 0), (65, 2, 3, 65, 0), (129, 5, 2, 40, 0), (200, 1, 40, 12, 0), (130, 2, 1, 20, 9)])
def test_theta_scan_splits(n_points, n_az, n_orient, beams, nv):
    """Zenith scan at the edges of its tiles (64 and 192 points), stages (64
    beams, 256 vertices) and vertex-count cases, poles included.  Sums of
    squares of the FP64 path's terms: its gate per point."""
    b = _with_nv(beams, nv, 15.0, 3) if nv else S.ragged(n_orient, beams, 15.0, 9 + n_points)
    g, w = S.grid(n_az, 2), S.wave()
    th = np.deg2rad(np.linspace(0.0, 180.0, n_points)) if n_points > 1 else np.array([0.7])
    want = oracle.thetas_m11(b, n_az, g.az_step, th, w)
    h = GpuHandlerPO(g, w)
    got = h.diffract_thetas_gpu(b, th)
    h.close()
    assert np.max(np.abs(got / want - 1.0)) < FP64_L2


@pytest.mark.gpu
@pytest.mark.parametrize("n_az,n_zen,n_orient", [(1, 1, 1), (7, 31, 2), (9, 32, 3), (16, 70, 5)])
def test_reduced_planes_and_rows(n_az, n_zen, n_orient):
    """Plane sums by tiles of 32 directions and per-orientation rows by tiles
    of 32 zenith rows: direction and row counts around the tiles; the staged
    call adds to what the accumulator holds, the host call returns its sums."""
    import torch
    b = S.ragged(n_orient, 6, 10.0, n_az + n_zen)
    g, w = S.grid(n_az, n_zen), S.wave()
    h = GpuHandlerPO(g, w)
    M = h.new_mueller()
    assert h.handle_orientations_to_local_gpu(b, M, precision=abi.FP64)
    assert _l2(M, oracle.po_diffract(b, g, w)) < FP64_L2
    acc = torch.full((M.size,), 2.0, dtype=torch.float64, device="cuda:0")
    st = h.stage(b)
    h.diffract_staged(st, acc.data_ptr(), precision=abi.FP64)
    torch.cuda.synchronize()
    np.testing.assert_allclose(acc.cpu().numpy(), M.ravel() + 2.0, rtol=1e-15, atol=0)
    st.free()
    rows = h.orientation_rows(b, precision=abi.FP64)
    h.close()
    for o in range(n_orient):
        want = oracle.phi_average(oracle.po_diffract(b.select(o, 1), g, w), g)[0]
        assert np.linalg.norm(rows[o] - want) <= FP64_L2 * np.linalg.norm(want)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 385])
def test_proposal_network_step(n):
    """One training step over the whole set at the edges of the 32-sample CTAs
    and 128-sample images: gradients against the oracle with BF16 rounding
    (the gate of tests/test_mlp.py), and the Adam update against the same
    formula in float64 on the returned gradients (float32 rounding of a
    handful of operations: 1e-6 of the step size)."""
    from mbs_fast_b200.mlp import ProposalNet
    from oracle import mlp_oracle as MO
    rng = np.random.default_rng(n)
    q = rng.normal(size=(n, 4))
    q = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)
    t = np.sin(3 * q[:, 0]).astype(np.float32)
    net = ProposalNet(seed=4)
    p0 = net.params
    loss, g = net.loss_grad(q, t)
    loss_bf, g_bf = MO.loss_grad(p0, q, t, bf16_round=True)
    assert abs(loss - loss_bf) <= 2e-3 * max(loss_bf, 1e-3)
    assert np.linalg.norm(g - g_bf) <= 1e-2 * np.linalg.norm(g_bf) + 1e-7
    net.train(q, t, epochs=1, batch=n, lr=1e-3, seed=1)
    got = net.params
    net.close()
    # the shuffled order changes the sums over samples: gradients to 1e-5
    # of their norm, so entries well above that step by lr sign(g)
    big = np.abs(g) > 1e-2 * np.linalg.norm(g) / np.sqrt(len(g))
    step = 1e-3 * g / (np.abs(g) + 1e-8)
    assert np.max(np.abs((p0 - got - step)[big])) <= 1e-3 * 2e-3


def _in_a_whole_tile(b, w, g, M, tile, precision):
    """The grid's last `tile` rows (polar rows left out) evaluated as a grid of
    their own, padded with rows between the first ones when there are fewer:
    M must hold the same values bit for bit."""
    th, vf = g.theta[1:-1][-tile:], g.vf[:, 1:-1][:, -tile:]
    n = len(th)
    fill = tile - n
    extra = np.linspace(0.01, 0.02, fill)
    th2 = np.concatenate([extra, th])
    phi = np.arange(2) * g.az_step
    reg = np.stack([-np.sin(phi), np.cos(phi), np.zeros(2)], -1)
    g2 = type(g)(2, tile - 1, g.az_step, np.ascontiguousarray(th2),
                 np.ascontiguousarray(np.concatenate([np.repeat(reg[:, None], fill, 1), vf], 1)), None)
    h2 = GpuHandlerPO(g2, w)
    M2 = h2.new_mueller()
    assert h2.handle_orientations_to_local_gpu(b, M2, precision=precision)
    h2.close()
    if n:
        assert np.array_equal(M[:, 1:-1][:, -n:], M2[:, fill:])


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tile,rest", [
    (p, n, r) for p, n, rs in ((abi.FP64, 192, (1, 64, 65, 96, 97, 128, 129, 160, 161)),
                               (abi.FP32C, 384, (1, 64, 65, 96, 97, 128, 129, 192, 193, 256, 257)))
    for r in rs])
@pytest.mark.parametrize("whole", [0, 1])
def test_row_tails(precision, tile, rest, whole):
    """Zenith rows past the last whole tile (alone, and after a whole tile):
    against the oracle, and bit for bit against the same directions evaluated
    inside a whole tile of the main shape (FP32C sums included: the tail
    shapes stage the same beams)."""
    b, w = S.ragged(3, 70, 12.0, 17), S.wave()
    g = S.grid(2, whole * tile + rest - 1)
    h = GpuHandlerPO(g, w)
    M = h.new_mueller()
    assert h.handle_orientations_to_local_gpu(b, M, precision=precision)
    h.close()
    assert _l2(M, oracle.po_diffract(b, g, w)) < (FP64_L2 if precision == abi.FP64 else 2e-5)
    _in_a_whole_tile(b, w, g, M, tile, precision)


@pytest.mark.gpu
@pytest.mark.parametrize("rest", [50, 90, 120, 180, 250])
def test_row_tails_of_several_stages(rest):
    """FP32C tails with more beams per orientation than a stage holds: the
    shapes end their stages at the same beams, so the sums are bit for bit
    those of the main shape."""
    b, w = S.batch(2, 300, 12.0, 23), S.wave()
    g = S.grid(2, rest - 1)
    h = GpuHandlerPO(g, w)
    M = h.new_mueller()
    assert h.handle_orientations_to_local_gpu(b, M, precision=abi.FP32C)
    h.close()
    _in_a_whole_tile(b, w, g, M, 384, abi.FP32C)


@pytest.mark.gpu
def test_staged_memory_is_reused_and_given_back():
    """A staged batch freed while a diffraction that reads it is in flight on
    another stream; its memory staged again at once; a batch larger than the
    pool keeps goes back in part when it is freed, does not pile up over
    stage and free cycles, and leaves nothing behind the context (64 MiB for
    the driver's own blocks)."""
    import torch
    b, w = S.batch(40, 60, 12.0, 5), S.wave()
    g = S.grid(16, 200)
    h = GpuHandlerPO(g, w)
    n = g.n_dirs * 16
    ref = torch.zeros(n, dtype=torch.float64, device="cuda:0")
    st = h.stage(b)
    h.diffract_staged(st, ref.data_ptr(), precision=abi.FP64)
    torch.cuda.synchronize()
    st.free()
    side = torch.cuda.Stream()
    other = S.batch(40, 60, 12.0, 6)
    for _ in range(3):
        st = h.stage(b)
        acc = torch.zeros(n, dtype=torch.float64, device="cuda:0")
        torch.cuda.synchronize()
        h.diffract_staged(st, acc.data_ptr(), precision=abi.FP64, stream=side.cuda_stream, stats=False)
        st.free()
        st2 = h.stage(other)          # takes the freed memory
        torch.cuda.synchronize()
        assert torch.equal(acc, ref)
        st2.free()
    h.close()
    one = _with_nv(99, 31, 6.0, 2)
    many = one.concat([one] * 2200)   # about 750 MB of records
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    h = GpuHandlerPO(g, w)
    left = []
    for _ in range(3):
        st = h.stage(many)
        held = torch.cuda.mem_get_info()[0]
        st.free()
        left.append(torch.cuda.mem_get_info()[0])
        assert left[-1] > held             # part of it at once
    assert left[0] == left[1] == left[2]   # nothing piles up
    h.close()
    assert torch.cuda.mem_get_info()[0] > before - (64 << 20)   # the rest with the context


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32C])
@pytest.mark.parametrize("external", ["none", "first", "every third", "all"])
def test_noshadow_sums(precision, external):
    """The sums over internal beams beside the full sums: no, one, mixed and
    only external beams, near-forward and polar rows among the directions;
    the full sums as without the second set (FP32C bit for bit: the same
    additions; FP64 to the rounding of a different grouping of 150 beams,
    150 x 1.1e-16 of the largest element's scale times a margin of 10)."""
    b, w = S.batch(3, 150, 12.0, 31), S.wave()
    i = np.arange(b.n_beams)
    if external != "first":
        b.beam_flags = np.where({"none": i < 0, "every third": i % 3 == 0, "all": i >= 0}[external], 1, 0).astype(np.uint8)
    g = S.grid(3, 140, plates=True)
    M0, N0 = oracle.po_diffract(b, g, w, noshadow=True)
    h = GpuHandlerPO(g, w)
    M, N, P = h.new_mueller(), h.new_mueller(), h.new_mueller()
    assert h.handle_orientations_to_local_gpu(b, M, N, precision=precision)
    assert h.handle_orientations_to_local_gpu(b, P, precision=precision)
    h.close()
    gate = FP64_L2 if precision == abi.FP64 else 1e-4
    assert _l2(M, M0) < gate
    assert _l2(N, N0) < gate if external != "all" else not N.any()
    if precision == abi.FP32C:
        assert np.array_equal(M, P)
    else:
        assert np.max(np.abs(M - P)) <= 1.7e-13 * np.max(np.abs(P))


@pytest.mark.gpu
@pytest.mark.parametrize("n_zen", [95, 383, 500])
@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32C])
def test_row_tails_in_a_captured_graph(n_zen, precision):
    """A tail alone, no FP32C tail, and a tail beside the main launch (side
    stream forked and joined) in a captured call: its replays add what the
    direct call adds, bit for bit."""
    import torch
    b, w = S.batch(5, 40, 12.0, 8), S.wave()
    g = S.grid(6, n_zen)
    h = GpuHandlerPO(g, w)
    st = h.stage(b)
    acc = torch.zeros(g.n_dirs * 16, dtype=torch.float64, device="cuda:0")
    h.diffract_staged(st, acc.data_ptr(), precision=precision)
    torch.cuda.synchronize()
    want = acc.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        h.diffract_staged(st, acc.data_ptr(), precision=precision,
                          stream=torch.cuda.current_stream().cuda_stream, stats=False)
    for _ in range(2):
        acc.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(acc, want)
    del graph
    st.free()
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("beams", [3, 700, 2600])
def test_small_uploads_and_results_in_parts(beams):
    """Batches below and above the size that goes up as one image (with size
    instances and absorption paths too), and results of one to eight parts,
    with the boundary of the two sets inside a part; calls in turn on one
    context, so each finds the buffers as the last one left them."""
    b, w = S.batch(2, beams, 8.0, 44, raw=True, absorbing=True), S.wave(True)
    rng = np.random.default_rng(beams)
    for n_az, n_zen in ((3, 10), (7, 400), (37, 800)):
        g = S.grid(n_az, n_zen)
        h = GpuHandlerPO(g, w)
        add, add_ns = h.diffract_pinned(b, noshadow=True, precision=abi.FP64)
        M, N = rng.normal(size=add.shape), rng.normal(size=add.shape)
        want, want_ns = M + add, N + add_ns
        assert h.handle_orientations_to_local_gpu(b, M, N, precision=abi.FP64)
        assert np.array_equal(M, want) and np.array_equal(N, want_ns)
        if n_az == 3:
            assert _l2(add, oracle.po_diffract(b, g, w)) < FP64_L2
            ms = [h.new_mueller(), h.new_mueller()]
            assert h.handle_orientations_to_local_gpu_multik(b, 0, 2, [0.7, 1.6], w.wave_index, ms)
            for s, m in zip((0.7, 1.6), ms):
                assert _l2(m, oracle.po_diffract(oracle.scale_batch(b, s, w.wave_index, w.abs_coeff), g, w)) < FP64_L2
            one = b.select(1, 1)
            P = h.new_mueller()
            assert h.handle_orientations_to_local_gpu(one, P, precision=abi.FP64)
            assert _l2(P, oracle.po_diffract(one, g, w)) < FP64_L2
        h.close()


@pytest.mark.gpu
def test_theta_scan_opposite_to_a_beam():
    """Shadow beams alone, up to the direction opposite to them, where the
    rotation vanishes by cancellation: its entries are sums of four products of
    unit vectors' components (rounding of 4 eps) and are 1 + cos theta large;
    their squares, on both sides, differ by up to 16 eps / (1 + cos theta)
    beside the FP64 gate."""
    b = S.batch(1, 2, 11.0, 1).select(0, 1)
    n = int(b.vert_offsets[1])
    b = type(b)(beam_offsets=np.array([0, 1]), orient_weight=np.ones(1), vert_offsets=b.vert_offsets[:2].copy(),
                vx=b.vx[:n].copy(), vy=b.vy[:n].copy(), slope_yx=b.slope_yx[:n].copy(), slope_xy=b.slope_xy[:n].copy(),
                edge_flags=b.edge_flags[:n].copy(), beam_geom=b.beam_geom[:1].copy(), beam_flags=b.beam_flags[:1].copy())
    g, w = S.grid(5, 2), S.wave()
    th = np.deg2rad(np.array([150.0, 170.0, 175.0, 179.0, 179.5, 179.9, 179.95, 179.99]))
    want = oracle.thetas_m11(b, 5, g.az_step, th, w)
    h = GpuHandlerPO(g, w)
    got = h.diffract_thetas_gpu(b, th)
    h.close()
    assert np.all(np.abs(got / want - 1.0) < FP64_L2 + 16 * 2.3e-16 / (1.0 + np.cos(th)))


def _first_beams(b, n):
    """The batch's first n beams as two orientations, the first of one beam."""
    v = int(b.vert_offsets[n])
    return type(b)(beam_offsets=np.array([0, 1, n]), orient_weight=np.array([0.6, 0.4]),
                   vert_offsets=b.vert_offsets[:n + 1].copy(), vx=b.vx[:v].copy(), vy=b.vy[:v].copy(),
                   slope_yx=b.slope_yx[:v].copy(), slope_xy=b.slope_xy[:v].copy(), edge_flags=b.edge_flags[:v].copy(),
                   beam_geom=b.beam_geom[:n].copy(), beam_flags=b.beam_flags[:n].copy())


def _bins_for_one_chunk():
    """Azimuth bins that give each bin's CTA all beams: at least the scan's
    resident CTAs, four an SM."""
    import torch
    return 4 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.gpu
@pytest.mark.parametrize("n_points,beams,nv", [(3, 63, 0), (3, 64, 0), (3, 65, 0), (3, 128, 0), (3, 150, 0),
                                               (3, 20, 31), (3, 70, 9), (130, 65, 0), (130, 20, 31)])
def test_theta_scan_stages(n_points, beams, nv):
    """Zenith scan whose CTAs take several stages: beam counts around the 64
    and vertex counts around the 256 of a stage, one and three points per
    thread, near-forward (marked) pairs in every stage.  The gate per point."""
    b = _first_beams(_with_nv(2 * beams, nv, 15.0, 3) if nv else S.batch(3, beams, 4.0, 9 + beams), beams)
    g, w = S.grid(_bins_for_one_chunk(), 2), S.wave()
    th = np.deg2rad(np.linspace(0.0, 180.0, n_points)) if n_points > 3 else np.array([0.0, 1e-4, 0.7])
    want = oracle.thetas_m11(b, g.n_az, g.az_step, th, w)
    h = GpuHandlerPO(g, w)
    got = h.diffract_thetas_gpu(b, th)
    h.close()
    assert np.max(np.abs(got / want - 1.0)) < FP64_L2


@pytest.mark.gpu
def test_theta_scan_scratch_is_bounded():
    """A scan with many beams needs no memory beyond its batch's; many azimuth
    bins go in slabs of points (192 and the rest)."""
    import torch
    w = S.wave()
    b = S.batch(1000, 100, 12.0, 5)
    h = GpuHandlerPO(S.grid(48, 2), w)
    h.extinction(b)                        # the upload area and the batch have their sizes
    free = torch.cuda.mem_get_info()[0]
    h.diffract_thetas_gpu(b, np.linspace(0.1, 3.0, 721))
    assert torch.cuda.mem_get_info()[0] == free
    h.close()
    b, g = S.batch(1, 3, 12.0, 6), S.grid(16400, 2)
    th = np.linspace(0.2, 3.0, 200)
    want = oracle.thetas_m11(b, g.n_az, g.az_step, th, w)
    h = GpuHandlerPO(g, w)
    got = h.diffract_thetas_gpu(b, th)
    h.close()
    assert np.max(np.abs(got / want - 1.0)) < FP64_L2


@pytest.mark.gpu
def test_failed_training_leaves_the_network_alone():
    """A tensor-core wait that runs out during training (the MMAs left out): the
    call fails, the parameters are bit for bit what they were, and training
    afterwards gives what an untouched network gives (moments and step count
    included).  In a network that has trained before, and in a new one whose
    activation memory nothing has written."""
    from mbs_fast_b200.mlp import ProposalNet
    rng = np.random.default_rng(5)
    q = rng.normal(size=(300, 4))
    q = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)
    t = np.sin(3 * q[:, 0]).astype(np.float32)
    for before in (0, 2):
        a, b = ProposalNet(seed=6), ProposalNet(seed=6)
        for net in (a, b):
            if before:
                net.train(q, t, epochs=before, batch=128, lr=1e-3, seed=1)
        p0 = a.params
        a.set_watchdog(poll_limit=64, skip_mma=True)
        with pytest.raises(RuntimeError, match="timed out"):
            a.train(q, t, epochs=3, batch=128, lr=1e-3, seed=2)
        a.set_watchdog(0, False)
        assert np.array_equal(a.params, p0)
        la, lb = (net.train(q, t, epochs=2, batch=128, lr=1e-3, seed=3) for net in (a, b))
        assert la == lb and np.array_equal(a.params, b.params)
        a.close()
        b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("noalloc", [False, True])
def test_calls_beside_an_open_capture(noalloc):
    """A grid without polar rows and with a row tail: while a capture of one
    call is open, the context's other calls run, a second capture is taken, and
    all give what the plain call gives."""
    import torch
    w, phi = S.wave(), np.arange(4) * (2 * np.pi / 4)
    g = S.grid(4, 500)
    vf = np.repeat(np.stack([-np.sin(phi), np.cos(phi), np.zeros(4)], -1)[:, None], 501, 1)
    g = type(g)(4, 500, g.az_step, np.linspace(0.1, 3.0, 501), np.ascontiguousarray(vf), None)
    h = GpuHandlerPO(g, w)
    b = S.batch(3, 30, 12.0, 2)
    st = h.stage(b)
    accs = [torch.zeros(g.n_dirs * 16, dtype=torch.float64, device="cuda:0") for _ in range(3)]

    def call(acc, stream):
        if noalloc:
            h.diffract_staged_noalloc(st, acc.data_ptr(), precision=abi.FP64, stream=stream.cuda_stream)
        else:
            h.diffract_staged(st, acc.data_ptr(), precision=abi.FP64, stream=stream.cuda_stream, stats=False)

    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    call(accs[2], streams[0])
    torch.cuda.synchronize()
    graphs = [torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()]
    with torch.cuda.stream(streams[0]):
        graphs[0].capture_begin(capture_error_mode="relaxed")
    call(accs[0], streams[0])
    M = h.new_mueller()
    assert h.handle_orientations_to_local_gpu(b, M, precision=abi.FP64)
    with torch.cuda.stream(streams[1]):
        graphs[1].capture_begin(capture_error_mode="relaxed")
    call(accs[1], streams[1])
    for s, gr in zip(streams, graphs):
        with torch.cuda.stream(s):
            gr.capture_end()
    for gr in graphs:
        gr.replay()
        torch.cuda.synchronize()
    assert torch.equal(accs[0], accs[2]) and torch.equal(accs[1], accs[2])
    assert np.max(np.abs(M.ravel() - accs[2].cpu().numpy())) <= 1e-12 * np.max(np.abs(M))
    del graphs
    st.free()
    h.close()


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["weight", "jones", "vertex"])
def test_theta_scan_with_nan(what):
    """A NaN weight or Jones matrix reaches every point of the scan; a beam whose
    aperture integral is NaN (a NaN vertex) is left out (reference
    GpuDiffraction.cu:1909-1956): as the oracle, point by point."""
    b, g, w = S.batch(2, 30, 12.0, 8), S.grid(3, 2), S.wave()
    th = np.array([0.3, 1.1, 2.6])
    if what == "weight":
        b.orient_weight = np.array([0.5, np.nan])
    elif what == "jones":
        b.beam_geom = b.beam_geom.copy()
        b.beam_geom[7, abi.G_JP + 3] = np.nan
    else:
        b.vx = b.vx.copy()
        b.vx[b.vert_offsets[7]] = np.nan
    want = oracle.thetas_m11(b, 3, g.az_step, th, w)
    assert np.isnan(want).all() == (what != "vertex") == np.isnan(want).any()
    h = GpuHandlerPO(g, w)
    got = h.diffract_thetas_gpu(b, th)
    h.close()
    np.testing.assert_allclose(got, want, rtol=FP64_L2)
