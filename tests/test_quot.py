"""The integer-pipe binary64 division and square root of the FP64 path
(tenjin_gb300/csrc/tj_quot.h) against the language's own: the same bits, over
all bit patterns, significands at both ends of their range, quotients next to
one and to a power of two, small integers, zeros, infinities, NaN, subnormal
numbers and results. On the host every step runs with the binary32 seed moved
by up to three units in the last place; on the GPU with the hardware's seed.
The tolerance is none: IEEE division and square root are correctly rounded. The
conversions to and from binary32 against the casts, in the same way."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
N = 200000
KINDS = ["bits", "short", "low_over_high", "near_equal", "over_one", "over_two", "tiny", "integers", "special"]
ONE = np.uint64(0x3FF0000000000000)
FRAC = np.uint64(0x000FFFFFFFFFFFFF)


def _args(kind):
    rng = np.random.default_rng(KINDS.index(kind) + 3)
    p, q = (rng.integers(0, 2 ** 64, N, dtype=np.uint64) for _ in range(2))
    if kind == "short":
        p, q = p & np.uint64(0xFFF000000000000F), q & np.uint64(0xFFFFFFFF00000000)
    elif kind == "low_over_high":
        p, q = ONE + (p & np.uint64(0xFF)), ONE + FRAC - (q & np.uint64(0xFFF))
    elif kind == "near_equal":
        p = (p & FRAC) | ONE
        q = p + (q & np.uint64(7)) - np.uint64(3)
    elif kind == "over_one":
        p, q = (p & FRAC) | ONE, ONE + (q & np.uint64(0xFFF))
    elif kind == "over_two":
        p, q = (p & FRAC) | ONE, ONE + FRAC - (q & np.uint64(0x7FFFFFFF))
    elif kind == "tiny":  # zeros, subnormal and small numerators over every sign and small exponents
        p = np.where(p % np.uint64(3) == 0, np.uint64(0), p & np.uint64(0x801FFFFFFFFFFFFF))
        q = (q & FRAC) | ((q >> np.uint64(60)) << np.uint64(52))
    elif kind == "integers":
        a = (p >> np.uint64(40)).astype(np.float64)
        return a, (q >> np.uint64(40)).astype(np.float64) + 1.0
    elif kind == "special":
        v = np.array([0.0, -0.0, 1.0, -1.0, 2.0, 4.0, 0.25, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308,
                      1.7976931348623157e308, 2.225073858507201e-308, 3.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 4.0 - 2.0 ** -51])
        a, b = np.meshgrid(v, v)
        return a.ravel().copy(), b.ravel().copy()
    return p.view(np.float64), q.view(np.float64)


def _check(lib, kind, ulps):
    a, b = _args(kind)
    out = [np.empty_like(a) for _ in range(4)]
    P = ctypes.POINTER(ctypes.c_double)
    rc = lib.tjq_eval(a.ctypes.data_as(P), b.ctypes.data_as(P), len(a), ulps, *[o.ctypes.data_as(P) for o in out])
    assert rc == 0
    for name, got, want in (("a / b", out[0], out[1]), ("sqrt(a)", out[2], out[3])):
        same = (got.view(np.int64) == want.view(np.int64)) | (np.isnan(got) & np.isnan(want))
        k = int(np.argmin(same))
        assert same.all(), f"{name}: {(~same).sum()} differ, first a={a[k].hex()} b={b[k].hex()}: {got[k].hex()} for {want[k].hex()}"


def _check_convert(lib, kind):
    a, b = _args(kind)
    # the same significands over the binary32 exponents, their ends and the ties between binary32 neighbours
    e = np.uint64(890) + b.view(np.uint64) % np.uint64(270)
    c = (a.view(np.uint64) & (FRAC | np.uint64(1 << 63))) | (e << np.uint64(52))
    tie = (c & ~np.uint64(0x1FFFFFFF)) | np.uint64(0x10000000)
    a = np.concatenate([a, c.view(np.float64), tie.view(np.float64)])
    f, f0 = np.empty(len(a), np.float32), np.empty(len(a), np.float32)
    w, w0 = np.empty_like(a), np.empty_like(a)
    D, F = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_float)
    assert lib.tjq_convert(a.ctypes.data_as(D), len(a), f.ctypes.data_as(F), f0.ctypes.data_as(F), w.ctypes.data_as(D),
                           w0.ctypes.data_as(D)) == 0
    assert np.array_equal(f.view(np.int32)[~np.isnan(f0)], f0.view(np.int32)[~np.isnan(f0)]) and np.isnan(f[np.isnan(f0)]).all()
    assert np.array_equal(w.view(np.int64)[~np.isnan(w0)], w0.view(np.int64)[~np.isnan(w0)]) and np.isnan(w[np.isnan(w0)]).all()


@pytest.fixture(scope="module")
def host_lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("quot") / "libtjq_host.so")
    subprocess.run([cxx, "-O2", "-std=c++14", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "tenjin_gb300", "csrc"),
                    "-x", "c++", os.path.join(HERE, "libm", "quot_harness.cu"), "-o", out], check=True)
    return ctypes.CDLL(out)


@pytest.fixture(scope="module")
def gpu_lib(tmp_path_factory):
    from tenjin_gb300 import build
    out = str(tmp_path_factory.mktemp("quot") / "libtjq_gpu.so")
    subprocess.run([build.nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-fmad=false", "-shared",
                    "-Xcompiler", "-fPIC", "-I" + os.path.join(ROOT, "tenjin_gb300", "csrc"),
                    os.path.join(HERE, "libm", "quot_harness.cu"), "-o", out], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("ulps", [-3, 0, 3])
@pytest.mark.parametrize("kind", KINDS)
def test_host_build_gives_the_ieee_bits(host_lib, kind, ulps):
    with np.errstate(all="ignore"):
        _check(host_lib, kind, ulps)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_gpu_build_gives_the_ieee_bits(gpu_lib, kind):
    with np.errstate(all="ignore"):
        _check(gpu_lib, kind, 0)


@pytest.mark.parametrize("kind", KINDS)
def test_host_conversions_are_the_casts(host_lib, kind):
    with np.errstate(all="ignore"):
        _check_convert(host_lib, kind)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_gpu_conversions_are_the_casts(gpu_lib, kind):
    with np.errstate(all="ignore"):
        _check_convert(gpu_lib, kind)
