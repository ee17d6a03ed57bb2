"""The plain FP64 1D step, whose RK stages work in tiles of 14 (2nd order) or 12
(4th order) new cells: interiors of the smallest size, around one and two tiles,
and beyond, with each boundary, solver and stage count, at rest, supersonic
(full characteristics) and out of the integer arithmetic's range.  Equal to the
CPU oracle value for value (no tolerance)."""
import numpy as np
import pytest

from _util import equal_values
from mlau_gb300 import ics

pytestmark = pytest.mark.gpu


def _state(n, kind):
    st, m = ics.riemann_1d(n=n, seed=n)
    x = np.arange(n + 8)
    if kind == "rest":
        st["mx"], st["by"] = 0.0 * x, 0.0 * x
    if kind == "supersonic":
        boost = 5.0 + 0.1 * np.sin(x)
        st["en"] = st["en"] + boost * st["mx"] + 0.5 * st["ro"] * boost**2
        st["mx"] = st["mx"] + st["ro"] * boost
    if kind == "tiny":
        for k in ("my", "by"):
            st[k] = st[k] * np.where(x % 3, 1e-250, 1.0)
    return st, m


@pytest.mark.parametrize("kind", ["riemann", "rest", "supersonic", "tiny"])
@pytest.mark.parametrize("flux", ["mlau", "lhlld", "hlld", "roe"])
@pytest.mark.parametrize("bc", ["open", "periodic"])
def test_tile_edges(gpu_lib, port, bc, flux, kind):
    M = gpu_lib
    for i, n in enumerate((4, 5, 11, 12, 13, 14, 15, 24, 27, 29, 150)):
        st, m = _state(n, kind)
        if bc == "periodic":
            st = {k: np.take(a, (np.arange(n + 8) - 4) % n + 4) for k, a in st.items()}
        dt = port.dt1d(st, m["bx"], m["gamma"], 0.3, m["dx"])
        for odr, nrk in ((1 + i % 2, 1 + i % 3), (4 - i % 2, 3), (5 + i % 2, 2)):
            ref = ics.copy_state(st)
            for _ in range(3):
                port.step1d(ref, m["bx"], dt, m["dx"], gamma=m["gamma"], odr=odr, flux=flux, nrk=nrk, bc=bc)
            with M.Sim(1, st["ro"].shape, dx=m["dx"], gamma=m["gamma"], odr=odr, flux=flux, nrk=nrk) as s:
                s.set_bx(m["bx"])
                s.set_bc(bc)
                s.upload(st)
                s.step(dt, 3)
                got = s.download()
            assert equal_values(got, ref, keys=ref.keys()), (n, odr, nrk)


@pytest.mark.parametrize("odr", [2, 4])
@pytest.mark.parametrize("threads", [64, 128, 256])
def test_batched_tile_edges(gpu_lib, port, threads, odr):
    """The batched engine's tiles: threads - 2 (2nd order) or - 4 new cells."""
    M = gpu_lib
    no = threads - (4 if odr == 4 else 2)
    cases, kinds = [], ("riemann", "rest", "supersonic", "tiny")
    for k, n in enumerate((4, no - 1, no, no + 1, no + 3, 2 * no, 2 * no + 1, 40, no, no + 1, 9, 3 * no)):
        st, m = _state(n, kinds[(k // 2) % 4])
        bc = "open" if k % 3 else "periodic"
        if bc == "periodic":
            st = {v: np.take(a, (np.arange(n + 8) - 4) % n + 4) for v, a in st.items()}
        cases.append((st, m, ("mlau", "lhlld", "hlld", "roe")[k % 4], 1 + (k // 4) % 3, bc))
    cells = sum(c[0]["ro"].size for c in cases)
    with M.Batch.open1d(cells, len(cases), odr=odr) as b:
        b.set_tile(threads, 1)
        slots = [b.add1d(st, m["dx"], m["bx"], m["gamma"], flux, nrk, bc, 0.3, 1.0)
                 for st, m, flux, nrk, bc in cases]
        b.run(3)
        got = [b.download(s) for s in slots]
        assert all(b.info(s)[1] == 3 for s in slots)
    for (st, m, flux, nrk, bc), g in zip(cases, got):
        ref, dt = ics.copy_state(st), port.dt1d(st, m["bx"], m["gamma"], 0.3, m["dx"])
        for _ in range(3):
            port.step1d(ref, m["bx"], dt, m["dx"], gamma=m["gamma"], odr=odr, flux=flux, nrk=nrk, bc=bc)
        assert equal_values(g, ref, keys=ref.keys()), (st["ro"].size, flux, nrk, bc)
