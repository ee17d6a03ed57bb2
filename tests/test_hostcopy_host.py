"""The host side of the array moves (csrc/hostcopy.cu), compiled by the host
compiler against a fake CUDA runtime: no GPU."""
import ctypes as C
import os
import subprocess

import pytest

from mlau_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("hostcopy") / "libhostcopy.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc()))), "include")
    # -Bsymbolic: the fake runtime's own functions, whatever else the process loaded
    subprocess.run(["g++", "-O2", "-std=c++17", "-w", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I" + cuda,
                    "-I" + _build.INCLUDE, "-I" + _build.CSRC,
                    os.path.join(ROOT, "tests", "c", "hostcopy_check.cpp"), "-o", out], check=True)
    return C.CDLL(out)


def test_an_earlier_error_is_not_the_moves(fake):
    assert fake.pending_error_check() == 0


@pytest.mark.parametrize("to_host", [0, 1])
@pytest.mark.parametrize("back", [0, 1, 511])
def test_a_bad_array_fails_on_the_host(fake, back, to_host):
    """An array one double too long for its mapping, or with a page of it not
    accessible, is met by the CPU before anything is launched; one that just
    fits moves."""
    page = os.sysconf("SC_PAGESIZE") // 8
    n = 3 * page - back
    assert fake.bad_array_check(4, C.c_longlong(n), 0, 0, to_host) == 0
    assert fake.bad_array_check(4, C.c_longlong(n), 1, 0, to_host) == 1
    assert fake.bad_array_check(4, C.c_longlong(n), 0, 1, to_host) == 1
    assert fake.bad_array_check(1, C.c_longlong(1), 0, 0, to_host) == 0
    assert fake.bad_array_check(1, C.c_longlong(1), 1, 0, to_host) == 1


def test_large_arrays_are_copied(fake):
    """To the device above 4 MB, to the host above 256 KB."""
    for to_host, limit in ((0, 1 << 19), (1, 1 << 15)):
        for n, by in ((1, 1), (4096, 1), (limit, 1), (limit + 1, 2), (1 << 20, 2)):
            assert fake.moved_by(C.c_longlong(n), to_host) == by, (n, to_host)


def test_a_failed_download_waits_for_the_stream(fake):
    """The upload of the same call may still read the caller's arrays."""
    assert fake.failed_download_check() == 0


def test_a_download_of_nothing_waits_for_the_stream(fake):
    assert fake.empty_download_check() == 0
