"""A batch member whose time stands still (t + dt rounds to t), on launches of its own:
it ends with the step that left t unchanged, as a cluster member does, and so does a
Float32 one whose end time is not a Float32 number."""
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
    assert res[0].steps == 1
    vf.perform_step(ref, math.inf)
    assert res[0].last_dt == vf.current_timestep(ref)
    for a, b in zip(interior(sims[0]), interior(ref)):
        assert np.array_equal(a, b)


def test_an_end_time_between_two_float32_numbers():
    """The same steps, t and status on launches of its own as in a cluster."""
    got = []
    for options in (E.BatchOptions(wide_cells=1), E.BatchOptions(wide_cells=-1)):
        sim = hills_rect(300, 280, B=None, bottom_source=False).build(vf.SM103Backend(np.float32))
        r, = E.simulate_batch([sim], [0.7], options=options)
        got.append((r.t, r.steps, r.status))
    assert got[0] == got[1]
    assert got[0][2] == N.VF_BATCH_STALLED
