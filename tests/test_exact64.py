"""The plain FP64 kernels' integer-path division, reciprocal and square root
(csrc/exact64.cuh) and their double type (csrc/ed.cuh).

They replace the FP64 pipe's operations in kernels whose results must equal the
reference's bit for bit, so the tolerance is none: the same bits as the host's
(CPU) and CUDA's (GPU) IEEE operations, NaN for NaN."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mlau_gb300", "csrc")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("exact64") / "libexact64.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I" + CSRC,
                    os.path.join(ROOT, "tests", "c", "exact64_check.cpp"), "-o", out], check=True)
    f = C.CDLL(out).exact64_check
    f.argtypes, f.restype = [C.c_int, C.c_int, C.c_long, C.c_long], C.c_long
    return f


@pytest.mark.parametrize("ulps", [0, 1, 2])
@pytest.mark.parametrize("kind", [0, 1, 2])
def test_host_same_bits(host, kind, ulps):
    """Operands near 1, with long runs of equal bits, and of every exponent;
    the FP32 seeds off by up to `ulps` units."""
    assert host(kind, ulps, 400000, 17 + kind) == 0


def _operands(kind, n, seed):
    rng = np.random.default_rng(seed)
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    if kind == "near one":
        e = rng.integers(1003, 1044, n, dtype=np.uint64)
    elif kind == "runs":
        k = rng.integers(0, 53, n, dtype=np.uint64)
        ones = (np.uint64(1) << k) - np.uint64(1)
        m = np.where(rng.random(n) < 0.5, m & ~ones, m | ones) & np.uint64((1 << 52) - 1)
        e = rng.integers(1022, 1025, n, dtype=np.uint64)
    else:
        e = rng.integers(0, 2048, n, dtype=np.uint64)
    s = rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63)
    x = (s | (e << np.uint64(52)) | m).view(np.float64)
    x[:6] = 0.0, -0.0, np.inf, np.nan, 1.0, 2.0
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["near one", "runs", "all"])
def test_device_same_bits(kind, tmp_path):
    from mlau_gb300 import _build
    out = str(tmp_path / "libexact64gpu.so")
    subprocess.run([_build.nvcc(), *_build.ARCH, "--fmad=false", "-O2", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "c", "exact64_gpu.cu"), "-o", out],
                   check=True, capture_output=True)
    run = C.CDLL(out).exact64_run
    run.argtypes = [C.c_void_p, C.c_void_p, C.c_long, C.c_void_p]
    n = (1 << 20) + 7
    a, b, o = _operands(kind, n, 1), _operands(kind, n, 2), np.empty((2, 8, n))
    assert run(a.ctypes.data, b.ctypes.data, n, o.ctypes.data) == 0
    got, want = o
    same = (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))
    assert same.all(axis=1).all(), np.argwhere(~same)[:4]
