"""Infinite and NaN values that a face or cell must not hand on. A momentum that is
not finite in a dry cell touches no other cell and is cleared by the dry clamp
(src/numericalflux/swe/centralupwind.jl:48-77, src/timestepper/timestepper.jl:41-51):
the step equals, bit for bit, that of the same state with zero there."""
import math

import numpy as np
import pytest

import volumefluxes_sm103 as vf
from volumefluxes_sm103 import ensemble as E
from vfhelpers import hills_rect

pytestmark = pytest.mark.gpu

DESIGNS = {  # scenario, VF_KERNELS
    "lean": (lambda: hills_rect(70, 45), "march"),
    "periodic": (lambda: hills_rect(70, 45, bc="periodic"), "march"),
    "no_reconstruction_fe": (lambda: hills_rect(70, 45, reconstruction="none", stepper="fe"), "march"),
    "tile": (lambda: hills_rect(70, 45), "tile"),
}


def dry_cell(sc):
    """A cell whose 7x7 neighbourhood is dry."""
    Bc = 0.25 * (sc.B[:-1, :-1] + sc.B[1:, :-1] + sc.B[:-1, 1:] + sc.B[1:, 1:])[2:-2, 2:-2]
    wet = sc.w0 > Bc
    for i, j in np.ndindex(wet.shape):
        if 3 <= i < sc.nx - 3 and 3 <= j < sc.ny - 3 and not wet[i - 3:i + 4, j - 3:j + 4].any():
            return i, j
    raise AssertionError("no dry patch")


@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan])
@pytest.mark.parametrize("real", [np.float32, np.float64])
@pytest.mark.parametrize("design", sorted(DESIGNS))
def test_momentum_of_a_dry_cell_stays_there(design, real, value, monkeypatch):
    make, kernels = DESIGNS[design]
    monkeypatch.setenv("VF_KERNELS", kernels)
    got = []
    for v in (0.0, value):
        sc = make()
        sc.hu0[dry_cell(sc)] = sc.hv0[dry_cell(sc)] = v
        sim = sc.build(vf.SM103Backend(real))
        for _ in range(2):
            vf.perform_step(sim, math.inf)
        got.append((vf.current_timestep(sim), vf.current_state(sim).stack()))
        sim.close()
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("make", [lambda: hills_rect(70, 45), lambda: hills_rect(70, 45, bc="periodic")])
def test_momentum_of_a_dry_cell_in_a_batch(make):
    got = []
    for v in (0.0, math.nan):
        sc = make()
        sc.hu0[dry_cell(sc)] = v
        sim = sc.build(vf.SM103Backend(np.float32))
        E.simulate_batch([sim], [1e30], max_steps=2)
        got.append(vf.current_interior_state(sim))
    for a, b in zip((got[0].h, got[0].hu, got[0].hv), (got[1].h, got[1].hu, got[1].hv)):
        assert np.array_equal(a, b)
