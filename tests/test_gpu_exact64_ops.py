"""The integer-path products, scalings, comparisons and limiters (csrc/exact64.cuh,
csrc/ed.cuh) and the EMF difference (csrc/emf_diff.cuh) as the device runs them:
the built-in operations' values.  No tolerance; products and scalings have the
same bits, and a zero's sign is left open for the rest (NaN for NaN)."""
import ctypes as C
import itertools
import os
import subprocess

import numpy as np
import pytest

from test_exact64 import CSRC, ROOT, _operands

pytestmark = pytest.mark.gpu

BITS = 17  # rows of products and scalings; then ge, max, min, minmod, minmod3, zero, range
ROWS = 24


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from mlau_gb300 import _build
    out = str(tmp_path_factory.mktemp("ops") / "libexact64ops.so")
    subprocess.run([_build.nvcc(), *_build.ARCH, "--fmad=false", "-O2", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "c", "exact64_ops_gpu.cu"), "-o", out],
                   check=True, capture_output=True)
    L = C.CDLL(out)
    for f in (L.exact64_ops, L.emf_diff_gpu):
        f.argtypes = [C.c_void_p, C.c_long, C.c_void_p]
    return L


EDGE = [s * v for s in (1.0, -1.0)
        for v in (0.0, 1.0, 1.5, float.fromhex("0x1.fffffffffffffp0"), 3.0, 1e-3, float.fromhex("0x1p-255"),
                  float.fromhex("0x1p-511"), float.fromhex("0x1.fffffffffffffp-512"),
                  float.fromhex("0x1.fffffffffffffp512"), float.fromhex("0x1p513"), 2.0 ** -1022, 5e-324,
                  float.fromhex("0x1p1023"), np.inf, np.nan)]


def _check(lib, abc):
    n = abc.shape[1]
    out = np.empty((2, ROWS, n))
    assert lib.exact64_ops(abc.ctypes.data, n, out.ctypes.data) == 0
    got, want = out
    bits = (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))
    assert bits[:BITS].all(axis=1).all(), np.argwhere(~bits[:BITS])[:4]
    same = (got == want) | (np.isnan(got) & np.isnan(want))
    same[BITS] |= (abc[0] == 0.0) & (abc[1] == 0.0)  # >= of two zeros: either, both are the maximum
    assert same.all(axis=1).all(), np.argwhere(~same)[:4]


@pytest.mark.parametrize("kind", ["near one", "runs", "all"])
def test_operations(lib, kind):
    n = (1 << 19) + 5
    a, b, c = (_operands(kind, n, s) for s in (1, 2, 3))
    b[: n // 8] = a[: n // 8]  # equal operands, and neighbours
    with np.errstate(invalid="ignore"):
        b[n // 8: n // 4] = np.nextafter(a[n // 8: n // 4], np.inf)
    _check(lib, np.ascontiguousarray(np.stack([a, b, c])))


def test_edges(lib):
    _check(lib, np.ascontiguousarray(np.array(list(itertools.product(EDGE, EDGE, EDGE[::3]))).T))


def _emf_operands(kind, n, seed):
    rng = np.random.default_rng(seed)
    mant = rng.integers(0, 1 << 23, (n, 4), dtype=np.uint32)
    ex = {"smooth": lambda: rng.integers(120, 128, (n, 4)), "window": lambda: rng.integers(100, 126, (n, 4)),
          "all": lambda: rng.integers(0, 256, (n, 4)), "low": lambda: rng.integers(0, 30, (n, 4)),
          "cancelling": lambda: np.full((n, 4), 130), "ties": lambda: rng.integers(100, 128, (n, 4))}[kind]()
    if kind == "cancelling":
        mant = (mant & np.uint32(63)) | np.uint32(1 << 22)
    if kind == "ties":  # few leading bits, long runs of ones: exact halves and carries into the exponent
        k = rng.integers(0, 24, (n, 4), dtype=np.uint32)
        mant = np.where(rng.random((n, 4)) < 0.5, np.uint32(0x7fffff) >> k << k, (np.uint32(1) << k) - 1) & 0x7fffff
    u = (rng.integers(0, 2, (n, 4), dtype=np.uint32) << 31) | (ex.astype(np.uint32) << 23) | mant.astype(np.uint32)
    u[rng.random((n, 4)) < 0.1] &= np.uint32(0x80000000)
    same = np.arange(n) % 11 == 0
    u[same, 1:] = u[same, :1]
    u[0], u[1] = 0, np.uint32(0x80000000)
    return np.ascontiguousarray(u).view(np.float32)


@pytest.mark.parametrize("kind", ["smooth", "window", "all", "low", "cancelling", "ties"])
def test_emf_difference(lib, kind):
    n = 1 << 20
    e = _emf_operands(kind, n, len(kind))
    got = np.empty(n)
    assert lib.emf_diff_gpu(e.ctypes.data, n, got.ctypes.data) == 0
    with np.errstate(all="ignore"):
        d = e.astype(np.float64)
        want = 27.0 * (d[:, 2] - d[:, 1]) - (d[:, 3] - d[:, 0])
    ok = (got == want) | (np.isnan(got) & np.isnan(want))
    assert ok.all(), (e[~ok][:3], got[~ok][:3], want[~ok][:3])
