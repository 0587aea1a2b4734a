"""The Float32 marching kernels with 64-bit offsets, which planes of 4 GB and more take,
on grids of every boundary kind, reconstruction, source and stepper: the same bits as
with 32-bit offsets."""
import numpy as np
import pytest

import volumefluxes_sm103 as vf
from test_gpu_march_general import CASES, run
from vfhelpers import hills_rect

pytestmark = pytest.mark.gpu

WALLS = {
    "wall": lambda: hills_rect(70, 45),
    "wall_two_cells": lambda: hills_rect(2, 2),
    "wall_strip_edge_fe": lambda: hills_rect(56, 33, stepper="fe"),
    "wall_long": lambda: hills_rect(901, 250),
    "wall_flat": lambda: hills_rect(64, 50, B=None, bottom_source=False),
}


@pytest.mark.parametrize("case", sorted(CASES | WALLS))
def test_far_offsets_equal_near_ones(case, monkeypatch):
    sc = (CASES | WALLS)[case]()
    dt, near = run(sc, 8, "march", np.float32, monkeypatch)
    dt_far, far = run(sc, 8, "march64", np.float32, monkeypatch)
    assert np.array_equal(dt, dt_far)
    assert np.array_equal(near, far)
