"""The blocks a 1D request is granted are the tiles the engine cuts it into
(batch2d.cu::build_tiles: 256 threads, of whose cells 254 are new, 252 at the
orders with five-point stencils, and one tile more for an open boundary)."""
import pytest

from mlau_gb300 import serve


@pytest.mark.parametrize("bc", ["open", "periodic"])
@pytest.mark.parametrize("odr,new", [(1, 254), (2, 254), (3, 252), (4, 252), (5, 254), (6, 254)])
def test_blocks_are_the_engines_tiles(odr, new, bc):
    for n in (4, 251, 252, 253, 254, 255, 508, 509, 2048, 16384):
        r = serve.Request(0, "1d", 0, 0.0, {}, {"bc": bc}, n)
        assert serve.blocks_1d(r, odr) == len(range(0, n, new)) + (bc == "open")


def test_the_1d_lane_asks_for_them(monkeypatch):
    class Engine:
        max_grid = 152

    monkeypatch.setattr(serve.Batch, "open1d", staticmethod(lambda *a, **k: Engine()))
    monkeypatch.setattr(serve.Batch, "open", staticmethod(lambda *a, **k: Engine()))
    monkeypatch.setattr(serve, "_Lane3D", lambda *a: None)
    lane = serve.Server().lanes["1d"]
    r = serve.Request(0, "1d", 0, 0.0, {}, {"bc": "open"}, 2048)
    assert lane.blocks_of(r) == 10
