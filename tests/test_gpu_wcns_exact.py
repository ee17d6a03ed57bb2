"""The plain FP64 WCNS4 reconstruction where its integer path hands over: five
equal values, exact zeros, differences too small for its range, jumps, and
both eigen-systems, on ragged grids.  The step must equal the CPU oracle's value
for value (no tolerance: the plain form's contract)."""
import numpy as np
import pytest

from mlau_gb300 import ics
from oracle import Port

pytestmark = pytest.mark.gpu


def _amplitude(kind, shape, rng):
    """Multiplier of a field's variation."""
    if kind == "uniform":
        return np.zeros(shape)
    if kind == "tiny":
        return np.full(shape, 1e-45)
    a = np.ones(shape)
    if kind == "half uniform":
        a[..., : shape[-1] // 2] = 0.0
    if kind == "jump":
        a[..., : shape[-1] // 2] = -7.0
    return a


def _vary(st, kind, rng):
    core = (slice(4, -4),) * st["ro"].ndim
    for k in ("ro", "mx", "my", "mz"):
        f = st[k][core]
        base = 1.0 if k == "ro" else 0.0
        g = base + _amplitude(kind, f.shape, rng) * (f - base)
        st[k] = ics.pad_periodic(np.abs(g) + 0.1 if k == "ro" and kind == "jump" else g, 4)
    return st


@pytest.mark.parametrize("mach", [0.3, 1.6])
@pytest.mark.parametrize("kind", ["uniform", "half uniform", "tiny", "jump", "smooth"])
def test_step_equals_oracle(gpu_lib, kind, mach):
    M, rng = gpu_lib, np.random.default_rng(5)
    st, m = ics.turbulence_3d(n=19, ny=13, nz=9, mach=mach, seed=2)
    st = _vary(st, kind, rng)
    ref = ics.copy_state(st)
    with M.Sim(3, st["ro"].shape, dx=m["dx"], dy=m["dy"], dz=m["dz"], odr=4, flux="mlau") as s:
        s.upload(st)
        s.step(5e-4, 2)
        got = s.download()
    for _ in range(2):
        Port.step3d(ref, 5e-4, m["dx"], m["dy"], m["dz"], odr=4, flux="mlau")
    assert all(np.array_equal(got[k], ref[k], equal_nan=True) for k in ref)

    st, m = ics.turbulence_2d(n=37, ny=21, vrms=mach, seed=3)
    st = _vary(st, kind, rng)
    ref = ics.copy_state(st)
    with M.Sim(2, st["ro"].shape, dx=m["dx"], dy=m["dy"], odr=4, flux="lhlld") as s:
        s.upload(st)
        s.step(5e-4, 2)
        got = s.download()
    for _ in range(2):
        Port.step2d(ref, 5e-4, m["dx"], m["dy"], odr=4, flux="lhlld")
    assert all(np.array_equal(got[k], ref[k], equal_nan=True) for k in ref)
