"""The server's figures of its engines against the engines."""
import pytest

from mlau_gb300 import FP32_SPLIT, FP64, Batch, serve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lane", ["1d", "2d64", "2d32"])
def test_bytes_per_cell(gpu_lib, lane):
    """A lane's pool takes what its share pays for: not more, and within 2 %."""
    cells = 1 << 20
    b = (Batch.open1d(cells, 8) if lane == "1d"
         else Batch.open(cells, 8, precision=FP64 if lane == "2d64" else FP32_SPLIT))
    with b:
        ratio = b.device_bytes / cells / serve.Server.BYTES_PER_CELL[lane]
    assert 0.98 < ratio <= 1.001, ratio
