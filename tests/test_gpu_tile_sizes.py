"""The Float64 tile kernels on either side of the size where their tile changes
(8x8 up to 456 of those, 16x16 beyond): every boundary kind, interior widths of
every residue mod 4, time- and cell-dependent sources, cells whose size is no
power of two, bit for bit the oracle's run, ghost cells of TMA and plain staging
included."""
import numpy as np
import pytest

import volumefluxes_sm103 as vf
from test_gpu_next_rows import run_pair, terrain_sources
from test_gpu_parity import assert_bitwise
from test_gpu_tma import run
from vfhelpers import hills_rect

pytestmark = pytest.mark.gpu

CASES = {
    "last_8x8": lambda: hills_rect(152, 192),
    "first_16x16": lambda: hills_rect(153, 192),
    "width_mod_0_periodic": lambda: hills_rect(188, 161, bc="periodic"),
    "width_mod_1_neumann": lambda: hills_rect(189, 165, bc="neumann"),
    "width_mod_2_bh2021_nonpow2": lambda: hills_rect(190, 159, friction_law="bh2021",
                                                     extent=((0.0, 133.0), (0.0, 70.0))),
    "width_mod_3_sources_neumann": lambda: terrain_sources(191, 157, bc="neumann"),
    "sources_periodic_fe": lambda: terrain_sources(175, 177, bc="periodic", stepper="fe"),
    "no_reconstruction": lambda: hills_rect(170, 176, reconstruction="none"),
    "one_tile_row": lambda: hills_rect(3700, 3),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_tiles_match_oracle(case):
    sim, ora = run_pair(CASES[case](), 6)
    assert_bitwise(vf.current_interior_state(sim), ora.interior())


@pytest.mark.parametrize("case", sorted(CASES))
def test_tma_matches_plain_loads(case):
    a, b = run(CASES[case](), 6, tma=True), run(CASES[case](), 6, tma=False)
    for x, y, name in zip(a, b, ("dt", "w", "hu", "hv")):
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64)), name
