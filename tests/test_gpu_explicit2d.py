"""The explicit MRX operators on either side of the size where they change
between the built-in double and the integer forms (20480 padded cells below 4th
order), against the oracle: equal values."""
import pytest

import mlau_gb300 as M
from _util import equal_values, max_rel_diff
from mlau_gb300 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [152, 153])
@pytest.mark.parametrize("tables", [((0,) * 8, (0,) * 8), ics.MRX_TABLES])
@pytest.mark.parametrize("odr", (1, 2, 4, 5))
@pytest.mark.parametrize("op", ("resistive", "viscous"))
def test_either_side_equals_the_oracle(port, op, odr, tables, n):
    st, m = ics.turbulence_2d(n=n, ny=120, seed=odr, odr=odr, vrms=0.4)
    port.setbc2d(st, *tables)
    dt = 0.3 * m["dx"] / m["vfast"]
    coef = 0.06 * m["dx"] ** 2 / dt
    ref = ics.copy_state(st)
    for _ in range(2):
        getattr(port, op + "2d")(ref, coef, dt, m["dx"], m["dy"], gamma=m["gamma"], odr=odr, nrk=3,
                                 dnx=tables[0], dny=tables[1])
    with M.Sim(2, st["ro"].shape, dx=m["dx"], dy=m["dy"], odr=odr, flux="lhlld", nrk=3) as s:
        s.set_bc2d(*tables)
        s.upload(st)
        for _ in range(2):
            getattr(s, op)(coef, dt)
        got = s.download()
    assert equal_values(got, ref), max_rel_diff(got, ref)
