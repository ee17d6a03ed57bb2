"""The plain FP64 2D step's two sweeps in one launch: narrow grids, where the
sweeps' cell counts differ most, and both sides of the block-size rule (97280
threads).  Equal to the CPU oracle value for value (no tolerance)."""
import numpy as np
import pytest

from mlau_gb300 import ics
from oracle import Port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(4, 60), (60, 4), (5, 7), (212, 213), (213, 213)])
@pytest.mark.parametrize("odr,flux,eig", [(4, "mlau", "full"), (2, "lhlld", "full"), (1, "hlld", "full"),
                                          (3, "roe", "full"), (2, "mlau", "miyoshi")])
def test_step_equals_oracle(gpu_lib, n, odr, flux, eig):
    M = gpu_lib
    st, m = ics.turbulence_2d(n=n[0], ny=n[1], vrms=1.0, seed=3, odr=odr)
    ref = ics.copy_state(st)
    with M.Sim(2, st["ro"].shape, dx=m["dx"], dy=m["dy"], gamma=m["gamma"], odr=odr, flux=flux) as s:
        s.set_eigen(eig)
        s.upload(st)
        s.step(1e-4, 2)
        got = s.download()
    for _ in range(2):
        Port.step2d(ref, 1e-4, m["dx"], m["dy"], odr=odr, flux=flux, eig=eig)
    assert all(np.array_equal(got[k], ref[k], equal_nan=True) for k in ref)
