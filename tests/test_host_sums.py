"""The addition of a host call's result while later parts are being copied
(mbs_fast_b200/csrc/host_sums.h), with the copies played by the test."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "host_sums.h"
// Part p of `copy` arrives in src when it is waited for; once more than `all`
// parts have, every one has; waiting for part `fail` fails.
extern "C" int run(double *src, const double *copy, size_t total, size_t n, int parts, double *M, double *Mns,
                   double *kept, int fail, int all)
{
    int have = 0;
    auto take = [&](int upto) {
        for (; have < upto; ++have) {
            const size_t a = mbs::result_part(total, parts, have), b = mbs::result_part(total, parts, have + 1);
            std::copy(copy + a, copy + b, src + a);
        }
    };
    return mbs::add_in_parts(src, total, n, parts, M, Mns, kept,
                             [&](int p) { if (p == fail) return false; if (have <= p) take(p + 1); return true; },
                             [&]() { if (have > all) take(parts); return have == parts; });
}
"""
dp = C.POINTER(C.c_double)


def _p(a):
    return a.ctypes.data_as(dp) if a is not None else None


def _kept(total):
    """NaNs on a 16-byte boundary."""
    a = np.full(total + 2, np.nan)
    return a[(a.ctypes.data % 16) // 8:][:total]


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("sums")
    (d / "sums.cpp").write_text(SOURCE)
    subprocess.run([shutil.which("g++") or "g++", "-O2", "-std=c++17", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "mbs_fast_b200", "csrc"), "-o", str(d / "sums.so"), str(d / "sums.cpp")],
                   check=True)
    f = C.CDLL(str(d / "sums.so")).run
    f.argtypes = [dp, dp, C.c_size_t, C.c_size_t, C.c_int, dp, dp, dp, C.c_int, C.c_int]
    return lambda src, copy, n, parts, M, N, kept, fail, all_: f(
        _p(src), _p(copy), len(copy), n, parts, _p(M), _p(N), _p(kept), fail, all_)


@pytest.mark.parametrize("two", [False, True])
@pytest.mark.parametrize("n,parts", [(16, 1), (112, 2), (1008, 8), (1008, 3), (4096, 8)])
def test_all_or_nothing(run, n, parts, two):
    """Every failing part, with the rest arriving at any point before it, with
    and without a place for the caller's values: the caller's arrays are as they
    were, bit for bit; without a failure they hold the plain sums."""
    rng = np.random.default_rng(n + parts)
    total = 2 * n if two else n
    copy = rng.normal(size=total)
    full = rng.normal(size=n) * 1e8, rng.normal(size=n) * 1e-8       # subtracting would not restore them
    holes = full[0] * (np.arange(n) > n // 2), full[1] * (np.arange(n) > n // 3)
    signed = np.zeros(n), np.where(np.arange(n) == n - 1, -0.0, 0.0)  # -0 is not +0
    for M0, N0 in (full, holes, signed):
        for fail in list(range(parts)) + [-1]:
            for all_ in range(parts + 1):
                if 0 <= all_ < fail:
                    continue                    # all parts have arrived: none can fail after that
                for kept in (_kept(total), None):
                    M, N = M0.copy(), N0.copy()
                    ok = run(np.full(total, np.nan), copy, n, parts, M, N if two else None, kept, fail, all_)
                    assert ok == (fail < 0)
                    want_m, want_n = (M0 + copy[:n], N0 + copy[n:] if two else N0) if ok else (M0, N0)
                    assert M.tobytes() == want_m.tobytes() and N.tobytes() == want_n.tobytes()


def test_one_array_for_both_sets(run):
    """The same array given for both sums: both are added, and taken back."""
    n = 320
    copy = np.random.default_rng(1).normal(size=2 * n)
    for M0 in (np.arange(float(n)), np.zeros(n)):
        for fail in (1, 2, 3, -1):
            M = M0.copy()
            assert run(np.full(2 * n, np.nan), copy, n, 4, M, M, _kept(2 * n), fail, 9) == (fail < 0)
            assert np.array_equal(M, M0 + copy[:n] + copy[n:] if fail < 0 else M0)
