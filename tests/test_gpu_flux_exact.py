"""The plain FP64 Riemann fluxes where their integer path hands over or takes its
special branches: flow at rest, no normal or no tangential field, supersonic
flow, jumps, values outside the integer range, on ragged 2D and 3D grids.
The step must equal the CPU oracle's value for value (no tolerance)."""
import numpy as np
import pytest

from mlau_gb300 import ics
from oracle import Port

pytestmark = pytest.mark.gpu


def _state(kind, dim):
    if dim == 3:
        st, m = ics.turbulence_3d(n=14, ny=11, nz=9, mach=0.4, seed=7, odr=2)
    else:
        st, m = ics.turbulence_2d(n=43, ny=18, vrms=0.4, seed=7, odr=2)
    g, f = m["gamma"], np.zeros_like(st["ro"])
    if kind in ("rest", "hydro", "supersonic", "tiny", "jump"):
        ro = st["ro"] if dim == 3 else 1.0 + 0.3 * np.cos(np.arange(f.size)).reshape(f.shape)
        v = [0.0, 0.0, 0.0]
        b = [0.7, -0.2, 0.4]
        if kind == "hydro":
            v, b = [0.3, -0.1, 0.2], [0.0, 0.0, 0.0]
        if kind == "supersonic":
            v = [4.0, -3.5, 0.3]
        if kind == "tiny":
            v, b = [1e-200, -1e-170, 0.0], [1e-160, 1e-90, 0.0]
        if kind == "jump":
            v = [np.where(ro > np.median(ro), 2.0, -2.0), 0.1, -0.4]
        st = dict(ro=ro, mx=ro * v[0] + f, my=ro * v[1] + f, mz=ro * v[2] + f, bx=f + b[0], by=f + b[1],
                  bz=f + b[2])
        v2 = sum((st[k] / ro) ** 2 for k in ("mx", "my", "mz"))
        st["en"] = 0.6 / (g - 1) * (1 + 0.1 * np.sin(ro)) + 0.5 * (ro * v2 + sum(x * x for x in b))
        core = (slice(4, -4),) * dim
        st = {k: ics.pad_periodic(np.ascontiguousarray(a[core]), 4) for k, a in st.items()}
    return st, m


@pytest.mark.parametrize("flux", ["mlau", "lhlld", "hlld"])
@pytest.mark.parametrize("kind", ["turbulence", "rest", "hydro", "supersonic", "tiny", "jump"])
@pytest.mark.parametrize("dim", [2, 3])
def test_step_equals_oracle(gpu_lib, dim, kind, flux):
    M = gpu_lib
    st, m = _state(kind, dim)
    ref = ics.copy_state(st)
    h = [m[k] for k in ("dx", "dy", "dz")[:dim]]
    for odr in (2, 5):
        with M.Sim(dim, st["ro"].shape, **dict(zip(("dx", "dy", "dz"), h)), odr=odr, flux=flux) as s:
            s.upload(ref)
            s.step(2e-4, 2)
            got = s.download()
        for _ in range(2):
            (Port.step3d if dim == 3 else Port.step2d)(ref, 2e-4, *h, odr=odr, flux=flux)
        assert all(np.array_equal(got[k], ref[k], equal_nan=True) for k in ref), odr
