"""Float32 members that run whole-grid launches side by side take longer marching
segments than one alone; a member's bits are the same for every length: batches of
one to nine wide members of every kernel form against the plain loop, long enough
that chunks are captured as graphs and with end times of their own."""
import numpy as np
import pytest

import volumefluxes_sm103 as vf
from test_gpu_ensemble import interior
from volumefluxes_sm103 import ensemble as E
from vfhelpers import hills_rect

pytestmark = pytest.mark.gpu

KINDS = [dict(), dict(bc="periodic"), dict(bc="neumann"), dict(reconstruction="none"), dict(stepper="fe")]
SIZES = [(97, 45), (64, 3), (29, 130), (256, 257), (301, 90)]


@pytest.mark.parametrize("members", [1, 2, 9])
def test_wide_float32_members_match_the_plain_loop(members):
    def build():
        return [hills_rect(*SIZES[k % 5], **KINDS[(k + k // 5) % 5]).build(vf.SM103Backend(np.float32))
                for k in range(members)]

    batch, alone = build(), build()
    ends = [float(np.float32(0.3 * (k + 1))) for k in range(members)]
    res = E.simulate_batch(batch, ends, options=E.BatchOptions(wide_cells=1))
    for k, r in enumerate(res):
        vf.simulate_to_time(alone[k], ends[k])
        assert r.t == alone[k].t, k
        for x, y, name in zip(interior(batch[k]), interior(alone[k]), ("h", "hu", "hv")):
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (k, name)
