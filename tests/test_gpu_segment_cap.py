"""Marching segments at their longest, 40 rows in the flux pass and 24 in the stage
pass, with a last segment of 3 rows: Float64, bit for bit the tile kernels."""
import numpy as np
import pytest

from test_gpu_march_general import run
from vfhelpers import hills_rect

pytestmark = pytest.mark.gpu


def test_longest_segments_equal_tiles(monkeypatch):
    # 83 strips of 1203 rows for 2432 resident warps (four blocks of four on 152 SMs): 42 rows each
    sc = hills_rect(2300, 1203)
    dt_t, tile = run(sc, 3, "tile", np.float64, monkeypatch)
    dt_m, march = run(sc, 3, "march", np.float64, monkeypatch)
    assert np.array_equal(dt_t, dt_m)
    assert np.array_equal(tile, march)
