"""The marching kernels with the segment lengths their launch chooses (one row on
small grids, up to 40 and 24 on large ones, a shorter last segment) against the
tile kernels: Float64, bit for bit, ghost cells included."""
import math

import numpy as np
import pytest

import volumefluxes_sm103 as vf
from vfhelpers import hills_rect

pytestmark = pytest.mark.gpu


# segments of 1, 2 (last of 1), 4 (last of 2), 13 and 24/31 rows
@pytest.mark.parametrize("nx,ny", [(57, 3), (900, 101), (901, 250), (1500, 530), (2300, 900)])
def test_marching_segments_equal_tiles(nx, ny, monkeypatch):
    sc = hills_rect(nx, ny)
    got = {}
    for design in ("tile", "march"):
        monkeypatch.setenv("VF_KERNELS", design)
        sim = sc.build(vf.SM103Backend(np.float64))
        for _ in range(3):
            vf.perform_step(sim, math.inf)
        got[design] = (vf.current_timestep(sim), vf.current_state(sim).stack())
        sim.close()
    assert got["tile"][0] == got["march"][0]
    assert np.array_equal(got["tile"][1], got["march"][1])
