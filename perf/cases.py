"""Workloads of the physical-optics diffraction library, through its public entry points.

Each case is one call (or the short sequence of calls) that a program makes on
a batch of traced beams: direct diffraction of host batches, device-resident
orientation averages, a size scan, per-orientation rows, the zenith scan, the
optical-theorem extinction and the training of the proposal network.  Particles
and grids follow the benchmark configurations (hexagonal column, aggregate of
columns, plate size scan); the beams are synthetic: polygon apertures, beam
directions, polarisation vectors and Jones matrices with the counts, sizes and
relations that traced batches have.

  listed()              the cases
  draw(rng)             one more case of the same ranges
  prepare(case, seed)   the inputs and handles a program holds before the call
  run(state)            one pass
  work(case)            bytes and operations a pass cannot do without
  exact(case, seed)     the pass's outputs in 64 bits, without this library
"""
import math

import numpy as np
import torch

from mbs_fast_b200 import abi
from mbs_fast_b200.beams import BeamBatch, GridTables
from mbs_fast_b200.handler import GpuHandlerPO
from mbs_fast_b200.mlp import N_PARAMS, ProposalNet
from mbs_fast_b200.proposal import averaged_rows

WAVELENGTH = 0.532
EPS1 = 1e9 * 2.220446049250313e-16
# Mean vertices of an aperture, for the counts of work().
MEAN_NV = 4.0


def listed():
    return [
        # One fixed orientation of a 10 x 20 um column on the 2 x 0.25 degree
        # grid: the single-particle calculation, in the default precision.
        _case("fixed_orientation", "host", "fp64", orient=1, beams=80, n_az=180, n_zen=720, size=11.0),
        # The first, small batch of an average (batches grow call by call
        # from a few orientations): the shortest call of an ordinary run.
        _case("first_batch", "host", "fp64", orient=16, beams=80, n_az=48, n_zen=180, size=11.0),
        # Orientation average of the 40 x 100 um column on the 0.1 degree
        # grid, beams resident on the device, in the fast precision.
        _case("column_fp32c", "staged", "fp32c", orient=320, beams=87, n_az=48, n_zen=1800, size=54.0),
        # The same average in plain FP64.
        _case("column_fp64", "staged", "fp64", orient=96, beams=87, n_az=48, n_zen=1800, size=54.0),
        # Host batch with the second set of sums (without external beams), on
        # a grid whose sizes divide nothing.
        _case("noshadow_sums", "host_ns", "fp32c", orient=61, beams=93, n_az=47, n_zen=357, size=30.0),
        # Aggregate of columns: more than a thousand beams per orientation.
        _case("aggregate", "staged", "fp32c", orient=12, beams=1200, n_az=48, n_zen=1800, size=60.0),
        # Plate size scan: every orientation at several sizes, staged and
        # diffracted in one launch, on the non-uniform zenith grid.
        _case("size_scan", "sizes", "fp64", orient=24, beams=60, n_az=48, n_zen=540, size=6.0, sizes=8),
        # One batch of a traced average: staged, diffracted, averaged over
        # azimuth, rows and cross-sections back on the host.
        _case("averaged_rows", "rows", "fp32c", orient=128, beams=87, n_az=48, n_zen=900, size=54.0),
        # Pilot of the learned proposal: the rows of every orientation alone.
        _case("pilot_rows", "pilot", "fp32c", orient=300, beams=87, n_az=48, n_zen=95, size=54.0),
        # Incoherent zenith scan (adaptive zenith grids are built from it).
        _case("theta_scan", "thetas", "fp64", orient=24, beams=87, n_az=48, n_zen=180, size=54.0),
        # Extinction of every orientation of a batch.
        _case("extinction", "extinction", "fp64", orient=1024, beams=87, n_az=48, n_zen=180, size=54.0),
        # Training of the proposal network on the pilot and its table.
        {"name": "proposal_fit", "kind": "mlp", "samples": 1638, "epochs": 100, "batch": 256, "cells": 128},
    ]


def _case(name, kind, precision, **kw):
    return dict({"name": name, "kind": kind, "precision": precision, "sizes": 1}, **kw)


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "host", "staged", "staged", "host_ns", "sizes", "rows", "pilot", "thetas",
                       "extinction", "mlp"])
    if kind == "mlp":
        return {"kind": kind, "samples": _log_int(rng, 300, 4000), "epochs": _log_int(rng, 10, 100),
                "batch": rng.choice([64, 100, 256, 500]), "cells": rng.choice([64, 96, 128])}
    c = {"kind": kind, "precision": rng.choice(["fp32c", "fp64"]), "sizes": 1,
         "beams": _log_int(rng, 24, 1400) if kind == "staged" else _log_int(rng, 40, 200),
         "size": math.exp(rng.uniform(math.log(5.0), math.log(80.0))), "n_az": rng.randint(24, 72),
         "n_zen": _log_int(rng, 60, 1800)}
    budget = 2.0e9 if c["precision"] == "fp32c" else 6.0e8     # beam-directions of a pass
    if kind == "pilot":
        c["n_zen"] = rng.randint(30, 200)
        budget /= 4
    elif kind == "thetas":
        c["precision"], c["n_zen"], budget = "fp64", _log_int(rng, 20, 360), 1.0e7
    elif kind == "extinction":
        c["precision"], c["n_zen"] = "fp64", 180
        c["orient"] = _log_int(rng, 8, 1500)
        return c
    elif kind == "sizes":
        c["sizes"] = rng.randint(2, 12)
        budget /= 2
    elif kind in ("host", "host_ns"):
        budget /= 4
    most = int(budget / (c["beams"] * c["n_az"] * (c["n_zen"] + 1) * c["sizes"]))
    c["orient"] = _log_int(rng, 1, max(1, min(400, most)))
    return c


# ------------------------------------------------------------------ inputs

def _wave(absorbing=False):
    w = abi.Wave()
    w.wave_index = 2 * math.pi / WAVELENGTH
    w.wavelength = WAVELENGTH
    w.compl_wave_im = -WAVELENGTH / (2 * math.pi) ** 2
    w.inv_compl_wave_im = 1.0 / WAVELENGTH
    w.eps1 = EPS1
    w.abs_coeff = -0.02 if absorbing else 0.0
    w.ot_far_reference_path = 10000.0
    return w


def _grid(n_az, n_zen, plates=False):
    """Zenith rows from 0 to 180 degrees (plates: the first 3/8 of them over
    0-10 degrees), azimuth bins over the circle, and the polarisation basis."""
    if plates:
        a = 3 * n_zen // 8
        deg = np.concatenate([np.linspace(0.0, 10.0, a, endpoint=False), np.linspace(10.0, 180.0, n_zen + 1 - a)])
    else:
        deg = np.linspace(0.0, 180.0, n_zen + 1)
    theta = np.deg2rad(deg)
    step = 2 * math.pi / n_az
    phi = np.arange(n_az) * step
    vf = np.empty((n_az, n_zen + 1, 3))
    vf[:, :, 0] = -np.sin(phi)[:, None]
    vf[:, :, 1] = np.cos(phi)[:, None]
    vf[:, :, 2] = 0.0
    vf[:, 0] = (0.0, 1.0, 0.0)       # polar rows: the incident basis, for every azimuth
    vf[:, -1] = (0.0, -1.0, 0.0)
    mid = np.concatenate([theta[:1], 0.5 * (theta[1:] + theta[:-1]), theta[-1:]])
    return GridTables(n_az, n_zen, step, theta, vf, 2 * math.pi * (np.cos(mid[:-1]) - np.cos(mid[1:])))


def _unit(a):
    return a / np.linalg.norm(a, axis=-1, keepdims=True)


def _batch(n_orient, mean_beams, size, seed, raw=False, absorbing=False):
    """A batch of n_orient orientations with about mean_beams beams each of a
    particle of radius `size` (um)."""
    rng = np.random.default_rng(seed)
    counts = np.maximum(2, np.round(mean_beams * rng.uniform(0.75, 1.25, n_orient))).astype(np.int64)
    off = np.concatenate([[0], np.cumsum(counts)])
    n = int(off[-1])
    ext = np.zeros(n, bool)
    ext[off[:-1]] = True             # each orientation's first beam: its external (shadow) beam
    # apertures: convex polygons of 3 to 8 vertices, mostly quadrangles
    nv = rng.choice([3, 4, 5, 6, 7, 8], n, p=[0.12, 0.76, 0.05, 0.045, 0.005, 0.02])
    nv[ext] = rng.choice([6, 8], int(ext.sum()))
    i = np.arange(8)[None, :]
    mask = i < nv[:, None]
    ang = (i + rng.uniform(-0.32, 0.32, (n, 8))) * (2 * np.pi / nv[:, None])
    half = nv // 2
    sym = (nv % 2 == 0) & (rng.random(n) < 0.6)          # facets cut to parallelograms and the like
    back = np.take_along_axis(ang, np.clip(i - half[:, None], 0, 7), 1) + np.pi
    ang = np.where(sym[:, None] & (i >= half[:, None]), back, ang)
    ra = size * np.clip(np.exp(rng.normal(-1.1, 0.7, n)), 0.02, 0.9)
    rb = ra * rng.uniform(0.12, 0.95, n)
    ra[ext], rb[ext] = size, size * 0.45
    x, y = ra[:, None] * np.cos(ang), rb[:, None] * np.sin(ang)
    rot = rng.uniform(0, 2 * np.pi, n)
    x, y = (np.cos(rot)[:, None] * x - np.sin(rot)[:, None] * y, np.sin(rot)[:, None] * x + np.cos(rot)[:, None] * y)
    rect = (nv == 4) & (rng.random(n) < 0.03)            # rectangles along the facet's axes
    x[rect, :4] = ra[rect, None] * np.array([1.0, -1.0, -1.0, 1.0])
    y[rect, :4] = rb[rect, None] * np.array([1.0, 1.0, -1.0, -1.0])
    cnt = nv[:, None]
    x -= np.where(mask, x, 0).sum(1, keepdims=True) / cnt
    y -= np.where(mask, y, 0).sum(1, keepdims=True) / cnt
    nxt = np.where(i + 1 < cnt, i + 1, 0) % 8
    dx, dy = np.take_along_axis(x, nxt, 1) - x, np.take_along_axis(y, nxt, 1) - y
    tol = 1e-9 * size
    okx, oky = np.abs(dx) > tol, np.abs(dy) > tol
    syx = np.where(okx, dy / np.where(okx, dx, 1), 0.0)
    sxy = np.where(oky, dx / np.where(oky, dy, 1), 0.0)
    cross = x * np.take_along_axis(y, nxt, 1) - np.take_along_axis(x, nxt, 1) * y
    area = 0.5 * np.where(mask, cross, 0).sum(1)
    # facet frame, beam direction and polarisation
    N = _unit(rng.normal(size=(n, 3)))
    bd = _unit(rng.normal(size=(n, 3)))
    flat = np.abs((bd * N).sum(1)) < 0.02
    bd[flat] = N[flat]
    N[ext], bd[ext] = (0.0, 0.0, -1.0), (0.0, 0.0, -1.0)
    up = np.where(np.abs(N[:, 2:3]) < 0.99, np.array([[0.0, 0.0, 1.0]]), np.array([[1.0, 0.0, 0.0]]))
    hor = _unit(np.cross(up, N))
    hor[ext] = (0.0, 1.0, 0.0)
    ver = np.cross(N, hor)
    pol = _unit(np.cross(bd, _unit(rng.normal(size=(n, 3)))))
    pol[ext] = (0.0, 1.0, 0.0)
    par = np.cross(pol, bd)
    cen = rng.normal(size=(n, 3)) * (0.35 * size)
    cen[ext] = 0.0
    path = rng.uniform(0.5, 4.0, n) * size
    J = rng.normal(size=(n, 4)) + 1j * rng.normal(size=(n, 4))
    J *= (np.exp(rng.normal(-1.6, 1.1, n)) / np.linalg.norm(J, axis=1))[:, None]
    J[ext] = (1.0, 0.0, 0.0, -1.0)
    path[ext] = 0.0
    sign = np.where(rng.random(n) < 0.5, -1.0, 1.0)
    k = 2 * math.pi / WAVELENGTH
    Jp = J * (sign * np.exp(1j * k * path))[:, None]
    g = np.empty((n, abi.GEOM_STRIDE))
    g[:, 0:3], g[:, 3:6], g[:, 6:9], g[:, 9:12], g[:, 12] = bd, hor, ver, cen, area
    g[:, 13:16], g[:, 16:19] = np.cross(N, pol), np.cross(N, par)
    g[:, 19:22], g[:, 22:25] = np.cross(N, np.cross(bd, pol)), np.cross(N, np.cross(bd, par))
    g[:, 25:33:2], g[:, 26:33:2] = Jp.real, Jp.imag
    g[:, 33] = path * np.where(ext, 0.0, 1.0)
    c = np.ascontiguousarray
    b = BeamBatch(beam_offsets=off, orient_weight=np.full(n_orient, 1.0 / n_orient),
                  vert_offsets=np.concatenate([[0], np.cumsum(nv)]).astype(np.int64), vx=c(x[mask]), vy=c(y[mask]),
                  slope_yx=c(syx[mask]), slope_xy=c(sxy[mask]),
                  edge_flags=c((okx * abi.EDGE_VALID_X + oky * abi.EDGE_VALID_Y)[mask].astype(np.uint8)),
                  beam_geom=g, beam_flags=np.where(ext, abi.BEAM_EXTERNAL, 0).astype(np.uint8))
    if raw:
        r = np.empty((n, abi.RAW_STRIDE))
        r[:, 0:8:2], r[:, 1:8:2], r[:, 8], r[:, 9] = J.real, J.imag, path, sign
        paths = np.where(ext, 0, rng.integers(1, 4, n)) if absorbing else np.zeros(n, np.int64)
        b.beam_raw = r
        b.abs_offsets = np.concatenate([[0], np.cumsum(paths)]).astype(np.int64)
        b.abs_paths = rng.uniform(0.2, 2.0, int(b.abs_offsets[-1])) * size
    return b


def _scales(case):
    return np.geomspace(1.0, 12.0, case["sizes"])


def _host_batch(case, seed):
    many = case["kind"] == "sizes"
    return _batch(case["orient"], case["beams"], case["size"], seed, raw=many, absorbing=many)


def _samples(case, seed):
    """Pilot points of the unit square as quaternions and standardised log targets."""
    rng = np.random.default_rng(seed)
    u, v = rng.random(case["samples"]), rng.random(case["samples"])
    q = _quaternions(u, v)
    t = np.sin(5 * u) * np.cos(7 * v) + 0.6 * np.exp(-((u - 0.3) ** 2 + (v - 0.6) ** 2) * 20)
    t = t + rng.normal(0, 0.1, len(u))
    return q, ((t - t.mean()) / t.std()).astype(np.float32)


def _quaternions(u, v):
    beta, gamma = np.arccos(1 - u), v * math.pi / 3
    cb, sb, cs, ss = np.cos(beta / 2), np.sin(beta / 2), np.cos(gamma / 2), np.sin(gamma / 2)
    return np.stack([cb * cs, sb * ss, sb * cs, cb * ss], -1).astype(np.float32)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    kind = case["kind"]
    if kind == "mlp":
        s.q, s.t = _samples(case, seed)
        c = (np.arange(case["cells"]) + 0.5) / case["cells"]
        U, V = np.meshgrid(c, c, indexing="ij")
        s.table = _quaternions(U.ravel(), V.ravel())
        s.net = ProposalNet(seed=1 + seed % 1000)
        s.initial = s.net.params
        return s
    s.batch = _host_batch(case, seed)
    s.precision = abi.FP32C if case["precision"] == "fp32c" else abi.FP64
    s.handler = GpuHandlerPO(_grid(case["n_az"], case["n_zen"], kind == "sizes"), _wave(kind == "sizes"))
    if kind in ("host", "host_ns"):
        s.M, s.Mns = s.handler.new_mueller(), s.handler.new_mueller() if kind == "host_ns" else None
    elif kind in ("staged", "sizes"):
        s.acc = torch.zeros((case["sizes"], case["n_az"], case["n_zen"] + 1, 16), dtype=torch.float64, device="cuda")
        if kind == "staged":
            s.staged = s.handler.stage(s.batch)
    elif kind == "thetas":
        s.theta = np.deg2rad(np.linspace(0.0, 180.0, case["n_zen"] + 1))
    return s


# -------------------------------------------------------------------- pass

def run(s):
    kind = s.case["kind"]
    if kind == "mlp":
        s.net.params = s.initial
        loss = s.net.train(s.q, s.t, epochs=s.case["epochs"], batch=s.case["batch"], lr=2e-3, seed=7)
        return {"loss": loss, "params": s.net.params, "table": s.net.forward(s.table)}
    h = s.handler
    if kind in ("host", "host_ns"):
        s.M.fill(0.0)
        if s.Mns is not None:
            s.Mns.fill(0.0)
        h.handle_orientations_to_local_gpu(s.batch, s.M, s.Mns, precision=s.precision)
        return {"M": s.M} if s.Mns is None else {"M": s.M, "Mns": s.Mns}
    if kind == "staged":
        s.acc.zero_()
        h.diffract_staged(s.staged, s.acc.data_ptr(), precision=s.precision,
                          stream=torch.cuda.current_stream().cuda_stream, stats=False)
        return {"M": s.acc}
    if kind == "sizes":
        s.acc.zero_()
        st = h.stage_multisize(s.batch, _scales(s.case))
        h.diffract_staged(st, s.acc.data_ptr(), precision=s.precision,
                          stream=torch.cuda.current_stream().cuda_stream)
        st.free()
        return {"M": s.acc}
    if kind == "rows":
        rows, csca, g = averaged_rows(h, s.batch, s.precision, stream=torch.cuda.current_stream().cuda_stream)
        return {"rows": rows, "csca": csca, "g": g}
    if kind == "pilot":
        return {"rows": h.orientation_rows(s.batch, precision=s.precision)}
    if kind == "thetas":
        return {"m11": h.diffract_thetas_gpu(s.batch, s.theta)}
    return {"cext": h.extinction(s.batch)}


def work(case):
    if case["kind"] == "mlp":
        per = 2 * N_PARAMS
        return {"bytes": 4 * (5 * case["samples"] + 5 * case["cells"] ** 2 + 2 * N_PARAMS),
                "flops": 3 * per * case["samples"] * case["epochs"] + per * case["cells"] ** 2}
    n = case["orient"] * case["beams"]
    rows, dirs = case["n_zen"] + 1, case["n_az"] * (case["n_zen"] + 1)
    read = n * (34 * 8 + 1 + 8) + n * MEAN_NV * 33
    per = 12 * MEAN_NV + 168
    kind = case["kind"]
    if kind == "extinction":
        return {"bytes": int(read + 8 * case["orient"]), "flops": int(n * per)}
    if kind == "thetas":
        return {"bytes": int(read + 16 * rows), "flops": int(n * dirs * per)}
    out = {"rows": rows, "pilot": case["orient"] * rows, "host_ns": 2 * dirs}.get(kind, dirs * case["sizes"]) * 128
    return {"bytes": int(read + out),
            "flops": int(case["sizes"] * dirs * (n * per + 100 * case["orient"]))}


# ----------------------------------------------------------- 64-bit results

def _beams64(b, scale=1.0, wave=None):
    """The batch's beams as float64 tensors, apertures padded to 8 vertices,
    at a size factor (Jones matrices re-phased when wave is given)."""
    d = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")
    nv = np.diff(b.vert_offsets)
    idx = b.vert_offsets[:-1, None] + np.minimum(np.arange(8)[None, :], nv[:, None] - 1)
    real = np.arange(8)[None, :] < nv[:, None]
    nxt = np.where(np.arange(8)[None, :] + 1 < nv[:, None], np.arange(8)[None, :] + 1, 0)
    B = _State()
    B.x, B.y = d(b.vx[idx] * scale), d(b.vy[idx] * scale)
    B.nxt, B.real = d(nxt), d(real)
    B.syx, B.sxy = d(b.slope_yx[idx]), d(b.slope_xy[idx])
    B.okx, B.oky = d(((b.edge_flags[idx] & 1) != 0) & real), d(((b.edge_flags[idx] & 2) != 0) & real)
    g = d(b.beam_geom)
    B.g = g
    B.hor, B.ver, B.cen = g[:, 3:6], g[:, 6:9], g[:, 9:12] * scale
    B.a0, B.b0 = (g[:, 0:3] * B.hor).sum(1), (g[:, 0:3] * B.ver).sum(1)
    B.area = g[:, 12] * scale * scale
    B.opath = g[:, 33] * scale
    B.J = torch.complex(g[:, 25:33:2], g[:, 26:33:2]).reshape(-1, 2, 2)
    if wave is not None:
        r = d(b.beam_raw)
        at = np.ones(b.n_beams)
        has = np.diff(b.abs_offsets) > 0
        if has.any():
            e = np.exp(wave.abs_coeff * b.abs_paths * scale)
            s = np.concatenate([[0.0], np.cumsum(e)])
            lo, hi = b.abs_offsets[:-1][has], b.abs_offsets[1:][has]
            at[has] = np.array([np.mean(e[p:q]) for p, q in zip(lo, hi)])
        ph = wave.wave_index * r[:, 8] * scale
        f = r[:, 9] * d(at) * torch.polar(torch.ones_like(ph), ph)
        B.J = (torch.complex(r[:, 0:8:2], r[:, 1:8:2]) * f[:, None]).reshape(-1, 2, 2)
    B.ext = d(b.beam_flags & 1) != 0
    return B


def _part(B, lo, hi):
    P = _State()
    for name, v in B.__dict__.items():
        setattr(P, name, v[lo:hi])
    return P


def _aperture(P, dirs, wave, singular=True, common=True):
    """Aperture integral [beams, directions] of the beams in P: the second-
    order small-phase value where every vertex phase is within 1e-3, else the
    edge sum with every edge in its stable form."""
    k = wave.wave_index
    A = P.a0[:, None] - P.hor @ dirs.T
    B = P.b0[:, None] - P.ver @ dirs.T
    small = torch.ones_like(A, dtype=torch.bool)
    for v in range(8):
        small &= (k * (A * P.x[:, v:v + 1] + B * P.y[:, v:v + 1])).abs() <= 1e-3
    useX = B.abs() > A.abs()
    X1, X2 = torch.where(useX, B, A), torch.where(useX, A, B)
    S = torch.zeros_like(A, dtype=torch.complex128)
    top = int(P.real.sum(1).max())
    one = torch.ones_like(A)
    for e in range(top):
        nx = P.nxt[:, e:e + 1]
        xe, ye = P.x[:, e:e + 1], P.y[:, e:e + 1]
        dx, dy = P.x.gather(1, nx) - xe, P.y.gather(1, nx) - ye
        C = torch.where(useX, P.syx[:, e:e + 1], P.sxy[:, e:e + 1]) * X1 + X2
        delta = torch.where(useX, dx, dy)
        ok = torch.where(useX, P.okx[:, e:e + 1], P.oky[:, e:e + 1])
        if not singular:
            ok = ok & (C.abs() > wave.eps1)
        z = 0.5 * k * C * delta
        S += torch.where(ok, k * delta * torch.sinc(z / math.pi), 0.0) * torch.polar(one, k * (A * xe + B * ye) + z)
    S = 1j * S / torch.where(useX, B, -A)
    F = complex(wave.compl_wave_re, wave.compl_wave_im) * S
    if bool(small.any()):
        n = P.nxt
        xj, yj = P.x.gather(1, n), P.y.gather(1, n)
        m = P.real.double()
        cr = (P.x * yj - xj * P.y) * m
        a2 = cr.sum(1)
        mx, my = ((P.x + xj) * cr).sum(1) / (3 * a2), ((P.y + yj) * cr).sum(1) / (3 * a2)
        mxx = ((P.x ** 2 + P.x * xj + xj ** 2) * cr).sum(1) / (6 * a2)
        myy = ((P.y ** 2 + P.y * yj + yj ** 2) * cr).sum(1) / (6 * a2)
        mxy = ((2 * P.x * P.y + P.x * yj + xj * P.y + 2 * xj * yj) * cr).sum(1) / (12 * a2)
        qx, qy = k * A, k * B
        re = 1 - 0.5 * (qx * qx * mxx[:, None] + 2 * qx * qy * mxy[:, None] + qy * qy * myy[:, None])
        lim = -complex(wave.inv_compl_wave_re, wave.inv_compl_wave_im) * P.area[:, None]
        F = torch.where(small, lim * torch.complex(re, qx * mx[:, None] + qy * my[:, None]), F)
    if common:
        ph = torch.where(P.ext[:, None], 0.0, -k * (P.cen @ dirs.T))
        F = F * torch.polar(torch.ones_like(ph), ph)
    return F, A, B, small


def _rotation(P, dirs, vf):
    """Rotation matrices: four [beams, directions] tensors (r00, r01, r10, r11)."""
    u = torch.linalg.cross(vf, dirs)
    vt = u / u.norm(dim=1, keepdim=True)
    w = torch.linalg.cross(vt, dirs)
    NT, NP, DT, DP = (P.g[:, i:i + 3] for i in (13, 16, 19, 22))
    return NT @ w.T + DT @ vt.T, NP @ w.T + DP @ vt.T, NT @ u.T + DT @ vf.T, NP @ u.T + DP @ vf.T


def _jones(P, dirs, vf, wave, singular=True):
    """Jones contributions (d00, d01, d10, d11), each [beams, directions]."""
    F = _aperture(P, dirs, wave, singular)[0]
    r00, r01, r10, r11 = _rotation(P, dirs, vf)
    J = P.J[:, :, :, None]
    return (F * (r00 * J[:, 0, 0] + r01 * J[:, 1, 0]), F * (r00 * J[:, 0, 1] + r01 * J[:, 1, 1]),
            F * (r10 * J[:, 0, 0] + r11 * J[:, 1, 0]), F * (r10 * J[:, 0, 1] + r11 * J[:, 1, 1]))


def _mueller(a, b, c, d, weight):
    """Mueller elements [directions, 16] of Jones sums [[a, b], [c, d]]."""
    aa, bb, cc, dd = (z.abs() ** 2 for z in (a, b, c, d))
    ab, dc, ac, db, ad, bc = a * b.conj(), d * c.conj(), a * c.conj(), d * b.conj(), a * d.conj(), b * c.conj()
    m = [(aa + cc + bb + dd) / 2, (aa + cc - bb - dd) / 2, -ab.real - dc.real, dc.imag - ab.imag,
         (aa - cc + bb - dd) / 2, (aa - cc - bb + dd) / 2, dc.real - ab.real, -ab.imag - dc.imag,
         -ac.real - db.real, db.real - ac.real, ad.real + bc.real, ad.imag - bc.imag,
         ac.imag - db.imag, db.imag + ac.imag, -ad.imag - bc.imag, ad.real - bc.real]
    return torch.stack(m, -1) * (0.25 * weight)


def _directions(grid):
    th = torch.as_tensor(grid.theta, device="cuda")
    ph = torch.arange(grid.n_az, device="cuda", dtype=torch.float64) * grid.az_step
    st, ct = torch.sin(th)[None, :], torch.cos(th)[None, :]
    d = torch.stack([st * torch.cos(ph)[:, None], st * torch.sin(ph)[:, None], -ct.expand(grid.n_az, -1)], -1)
    return d.reshape(-1, 3), torch.as_tensor(grid.vf, device="cuda").reshape(-1, 3)


def _planes(b, B, grid, wave, each=False):
    """Mueller sums over the orientations [directions, 16] with all beams and
    without external ones; each: the list of single orientations instead."""
    dirs, vf = _directions(grid)
    total = torch.zeros(dirs.shape[0], 16, dtype=torch.float64, device="cuda")
    inner = torch.zeros_like(total)
    single = []
    block = max(1, int(6e6 // dirs.shape[0]))
    for o in range(b.n_orient):
        sums, sums_in = 0, 0
        for lo in range(int(b.beam_offsets[o]), int(b.beam_offsets[o + 1]), block):
            P = _part(B, lo, min(lo + block, int(b.beam_offsets[o + 1])))
            d = torch.stack(_jones(P, dirs, vf, wave))
            keep = (~P.ext).to(d.dtype)
            sums = sums + d.sum(1)
            sums_in = sums_in + torch.einsum("cbd,b->cd", d, keep)
        m = _mueller(*sums, float(b.orient_weight[o]))
        if each:
            single.append(_azimuth_rows(m, grid))
        total += m
        inner += _mueller(*sums_in, float(b.orient_weight[o]))
    return single if each else (total, inner)


def _azimuth_rows(m, grid):
    """Azimuth average [n_zen + 1, 16]: M(p) L(2 az_p), polar rows projected."""
    M = m.reshape(grid.n_az, grid.n_zen + 1, 4, 4)
    az = -2.0 * torch.arange(grid.n_az, device=m.device, dtype=torch.float64) * grid.az_step
    c, s = torch.cos(az)[:, None, None], torch.sin(az)[:, None, None]
    R = torch.stack([M[..., 0], M[..., 1] * c - M[..., 2] * s, M[..., 1] * s + M[..., 2] * c, M[..., 3]], -1).mean(0)
    plain = M.mean(0)
    for t, sign in ((0, 1.0), (grid.n_zen, -1.0)):
        p = plain[t].clone()
        R[t] = 0.0
        half = 0.5 * (p[1, 1] + sign * p[2, 2])
        R[t, 0, 0], R[t, 1, 1], R[t, 2, 2], R[t, 3, 3], R[t, 0, 3], R[t, 3, 0] = \
            p[0, 0], half, sign * half, p[3, 3], p[0, 3], p[0, 3]
    return R.reshape(grid.n_zen + 1, 16)


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        return None                  # a BF16 training run has no 64-bit value
    b = _host_batch(case, seed)
    wave = _wave(kind == "sizes")
    grid = _grid(case["n_az"], case["n_zen"], kind == "sizes")
    shape = (case["n_az"], case["n_zen"] + 1, 16)
    if kind == "sizes":
        return {"M": torch.stack([_planes(b, _beams64(b, float(s), wave), grid, wave)[0].reshape(shape)
                                  for s in _scales(case)])}
    B = _beams64(b)
    if kind in ("host", "host_ns", "staged"):
        M, Mns = _planes(b, B, grid, wave)
        if kind == "staged":
            return {"M": M.reshape((1,) + shape)}
        return {"M": M.reshape(shape)} if kind == "host" else {"M": M.reshape(shape), "Mns": Mns.reshape(shape)}
    if kind == "rows":
        rows = _azimuth_rows(_planes(b, B, grid, wave)[0], grid)
        dc, th = torch.as_tensor(grid.dcos2pi, device="cuda"), torch.as_tensor(grid.theta, device="cuda")
        csca = (rows[:, 0] * dc).sum()
        return {"rows": rows, "csca": float(csca), "g": float((torch.cos(th) * rows[:, 0] * dc).sum() / csca)}
    if kind == "pilot":
        return {"rows": torch.stack(_planes(b, B, grid, wave, each=True))}
    if kind == "thetas":
        return {"m11": _scan(b, B, grid, wave)}
    return {"cext": _extinction(b, B, wave)}


def _scan(b, B, grid, wave):
    th = np.clip(grid.theta, 1e-6, math.pi - 1e-6)
    phi = np.arange(grid.n_az) * grid.az_step
    ones = np.ones((len(th), 1))
    dirs = np.stack([np.sin(th)[:, None] * np.cos(phi), np.sin(th)[:, None] * np.sin(phi), -np.cos(th)[:, None] * np.ones_like(phi)], -1)
    vf = np.stack([-np.sin(phi) * ones, np.cos(phi) * ones, np.zeros((len(th), grid.n_az))], -1)
    dirs, vf = (torch.as_tensor(a.reshape(-1, 3), device="cuda") for a in (dirs, vf))
    w = torch.as_tensor(np.repeat(b.orient_weight, np.diff(b.beam_offsets)), device="cuda")
    out = torch.zeros(len(th), dtype=torch.float64, device="cuda")
    block = max(1, int(6e6 // dirs.shape[0]))
    for lo in range(0, b.n_beams, block):
        P = _part(B, lo, min(lo + block, b.n_beams))
        e = sum(z.abs() ** 2 for z in _jones(P, dirs, vf, wave, singular=False))
        out += (0.5 * w[lo:lo + block, None] * e).sum(0).reshape(len(th), grid.n_az).sum(1) / (grid.n_az + 1)
    return out


def _extinction(b, B, wave):
    d = lambda *v: torch.tensor([v], dtype=torch.float64, device="cuda")
    dirs, vf, k = d(0.0, 0.0, -1.0), d(0.0, 1.0, 0.0), wave.wave_index
    F, A, Bc, small = _aperture(B, dirs, wave, common=False)
    drop = ~small & (torch.maximum(A.abs(), Bc.abs()) <= wave.eps1)
    r00, r01, r10, r11 = _rotation(B, dirs, vf)
    J = B.J[:, :, :, None]
    trace = F * (r00 * J[:, 0, 0] + r01 * J[:, 1, 0] + r10 * J[:, 0, 1] + r11 * J[:, 1, 1])
    ph = torch.where(B.ext, -k * B.opath, -k * (-B.cen[:, 2] + wave.ot_far_reference_path))
    s = 0.5 * torch.where(drop, 0.0, trace)[:, 0] * torch.polar(torch.ones_like(ph), ph)
    o = torch.as_tensor(np.repeat(np.arange(b.n_orient), np.diff(b.beam_offsets)), device="cuda")
    amp = torch.zeros(b.n_orient, dtype=torch.float64, device="cuda").index_add_(0, o, s.imag)
    return wave.wavelength * amp * torch.as_tensor(b.orient_weight, device="cuda")
