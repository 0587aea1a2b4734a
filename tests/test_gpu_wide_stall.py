"""A batch member whose time stands still (t + dt rounds to t), on launches of its own:
the result is the state after the steps it reports, also where the last chunk of steps
is a short one of odd length."""
import math

import numpy as np
import pytest

import volumefluxes_sm103 as vf
from test_gpu_ensemble import interior
from volumefluxes_sm103 import _native as N
from volumefluxes_sm103 import ensemble as E
from vfhelpers import hills_rect

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_steps", [None, 19, 33])
@pytest.mark.parametrize("real,options", [(np.float64, None), (np.float64, E.BatchOptions(wide_cells=1)),
                                          (np.float32, E.BatchOptions(wide_cells=1))])
def test_a_wide_member_whose_time_stands_still(real, options, max_steps):
    sims = [hills_rect(70, 64 + k).build(vf.SM103Backend(real)) for k in range(3)]
    ref = hills_rect(70, 64).build(vf.SM103Backend(real))
    sims[0].t = 2.0 ** 66
    kw = {} if max_steps is None else {"max_steps": max_steps}
    res = E.simulate_batch(sims, [2.0 ** 70, 0.1, 0.1], options=options, **kw)
    assert res[0].status == N.VF_BATCH_STALLED and res[0].t == 2.0 ** 66
    assert max_steps is None or res[0].steps <= max_steps
    for _ in range(res[0].steps):
        vf.perform_step(ref, math.inf)
    assert res[0].last_dt == vf.current_timestep(ref)
    for a, b in zip(interior(sims[0]), interior(ref)):
        assert np.array_equal(a, b)
