"""Per-kernel timing names what was launched."""
import pytest

from mlau_gb300 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrk", [1, 2, 3])
def test_1d_stages_are_reported_as_stages(gpu_lib, nrk):
    M = gpu_lib
    st, m = ics.riemann_1d(n=64, seed=0)
    with M.Sim(1, st["ro"].shape, dx=m["dx"], gamma=m["gamma"], odr=2, nrk=nrk) as s:
        s.set_bx(m["bx"])
        s.upload(st)
        s.set_timing(True)
        s.step(1e-4, 5)
        t = s.timing()
    assert set(t) == {"stage"} and t["stage"][0] == 5 * nrk == 5 * s_launches(M, st, m, nrk)
    assert t["stage"][1] > 0.0


def s_launches(M, st, m, nrk):
    with M.Sim(1, st["ro"].shape, dx=m["dx"], gamma=m["gamma"], odr=2, nrk=nrk) as s:
        return s.launches_per_step
