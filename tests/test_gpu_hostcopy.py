"""Host arrays to the device and back, by the copy kernel and by copies: odd and
even lengths, arrays aligned to 8 bytes only, arrays above the kernel's limit
(4 MB), fresh and shared destinations, pinned memory.  The same bytes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

NAMES = ("ro", "mx", "my", "mz", "en", "bx", "by", "bz")


def _array(shape, shift, pinned=False):
    n = int(np.prod(shape))
    if pinned:
        a = torch.empty(n + 2, dtype=torch.float64, pin_memory=True).numpy()
    else:
        a = np.empty(n + 2)
    off = ((shift * 8 - a.ctypes.data) % 16) // 8  # 16-byte boundary, or 8 beyond one
    return a[off:off + n].reshape(shape)


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("shape", [(12,), (13,), (2055,), (21, 17), (1000, 520), (1100, 500), (13, 14, 15)])
@pytest.mark.parametrize("shift", [0, 1])
def test_round_trip(gpu_lib, shape, shift, pinned):
    M = gpu_lib
    rng = np.random.default_rng(len(shape) + shift)
    names = [k for k in NAMES if not (len(shape) == 1 and k == "bx")]
    st = {}
    for k in names:
        st[k] = _array(shape, shift, pinned)
        st[k][...] = rng.standard_normal(shape)
    want = {k: a.copy() for k, a in st.items()}
    h = dict(zip(("dx", "dy", "dz"), [0.1] * len(shape)))
    with M.Sim(len(shape), shape, **h) as s:
        s.upload(st)
        for k in names:
            st[k][...] = 0.0  # the upload is over
        got = s.download()
        assert all(np.array_equal(got[k], want[k]) for k in names)
        out = {k: _array(shape, shift, pinned) for k in names}
        got = s.download(out)
        assert all(np.array_equal(got[k], want[k]) for k in names)


def test_batch_refuses_a_missing_array(gpu_lib):
    M = gpu_lib
    import ctypes as C
    with M.Batch.open(1000, 2) as b:
        one = np.ones((20, 20))
        ptrs = (C.POINTER(C.c_double) * 8)(*[one.ctypes.data_as(C.POINTER(C.c_double))] * 7)
        rc = M.lib().mlau_batch_add(b._h, 20, 20, C.c_double(0.1), C.c_double(0.1), C.c_double(1.6), 0,
                                    C.c_double(0.4), C.c_double(1.0), ptrs, C.byref(C.c_int()))
        assert rc != 0
