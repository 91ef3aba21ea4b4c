"""Synthetic beam batches, grids and wave constants for kernel tests that need
no traced particle: the generators of the workload cases (perf/cases.py)."""
import importlib.util
import os

_path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "perf", "cases.py")
_spec = importlib.util.spec_from_file_location("workload_cases", _path)
_cases = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(_cases)

batch = _cases._batch      # (n_orient, mean_beams, size_um, seed, raw=False, absorbing=False)
grid = _cases._grid        # (n_az, n_zen, plates=False)
wave = _cases._wave        # (absorbing=False)


def ragged(n_orient, mean_beams, size, seed, **kw):
    """A batch whose beam counts run from a single beam to twice the mean,
    with an empty orientation in the middle (n_orient > 2)."""
    b = batch(n_orient, mean_beams, size, seed, **kw)
    if n_orient > 2:
        o = n_orient // 2
        off = b.beam_offsets.copy()
        off[o] = off[o + 1]                # orientation o empty, o - 1 gets its beams
        off[n_orient - 1] = off[n_orient] - 1   # the last orientation: one beam
        b.beam_offsets = off
    return b
