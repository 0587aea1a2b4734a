"""Batches whose Float64 members are stepped together: members of every boundary
kind, reconstruction and source, at the smallest and largest sizes that are packed
and just beyond them, with end times of their own, a limit on the steps that is no multiple of
the steps between two reads of the records, and a member whose time stands still.
Bit for bit the plain loop of every member."""
import math
import time

import numpy as np
import pytest

import volumefluxes_sm103 as vf
from test_gpu_ensemble import interior
from test_gpu_next_rows import terrain_sources
from volumefluxes_sm103 import _native as N
from volumefluxes_sm103 import ensemble as E
from vfhelpers import hills_rect

pytestmark = pytest.mark.gpu

MEMBERS = [  # scenario, end time [s]
    (lambda: hills_rect(64, 64), 1.5),
    (lambda: hills_rect(63, 65), 1.0),  # 4095 cells: not packed
    (lambda: hills_rect(97, 45, bc="periodic"), 0.7),
    (lambda: hills_rect(189, 65, bc="neumann"), 0.1),
    (lambda: terrain_sources(67, 70), 1.0),
    (lambda: hills_rect(65, 64, reconstruction="none"), 0.0),  # has ended before its first step
    (lambda: hills_rect(2, 2049), 0.4),
    (lambda: hills_rect(200, 150), 0.6),
    (lambda: hills_rect(256, 255, friction_law="bh2021"), 0.2),
    (lambda: hills_rect(256, 256), 0.2),  # 65536 cells: runs alone
]


def build():
    return [make().build(vf.SM103Backend()) for make, _ in MEMBERS]


def assert_same(a, b, what):
    for x, y, name in zip(interior(a), interior(b), ("h", "hu", "hv")):
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64)), (what, name)


def test_packed_members_match_the_plain_loop():
    batch, alone = build(), build()
    res = E.simulate_batch(batch, [end for _, end in MEMBERS])
    for k, (sim, ref, r) in enumerate(zip(batch, alone, res)):
        vf.simulate_to_time(ref, MEMBERS[k][1])
        assert r.t == ref.t, k
        assert_same(sim, ref, k)


def test_too_few_members_for_a_pack():
    batch, alone = build()[:3], build()[:3]
    E.simulate_batch(batch, [end for _, end in MEMBERS[:3]])
    for k in range(3):
        vf.simulate_to_time(alone[k], MEMBERS[k][1])
        assert_same(batch[k], alone[k], k)


@pytest.mark.parametrize("max_steps", [1, 8, 11])
def test_packed_members_stop_at_the_step_limit(max_steps):
    batch, alone = build(), build()
    ends = [end for _, end in MEMBERS]
    res = E.simulate_batch(batch, ends, max_steps=max_steps)
    ref = E.simulate_batch(alone, ends, max_steps=max_steps, options=E.BatchOptions(wide_cells=1))
    assert [(r.t, r.steps, r.last_dt, r.status) for r in res] == [(r.t, r.steps, r.last_dt, r.status) for r in ref]
    for k in range(len(MEMBERS)):
        assert_same(batch[k], alone[k], k)


def test_a_member_whose_time_stands_still():
    batch, alone = build(), build()
    ends = [end for _, end in MEMBERS]
    batch[0].t, ends[0] = 1e20, 1e21  # t + dt rounds to t
    res = E.simulate_batch(batch, ends)
    assert res[0].status == N.VF_BATCH_STALLED and res[0].t == 1e20
    for _ in range(res[0].steps):
        vf.perform_step(alone[0], math.inf)
    assert_same(batch[0], alone[0], 0)
    for k in range(1, len(MEMBERS)):
        vf.simulate_to_time(alone[k], ends[k])
        assert res[k].status == N.VF_BATCH_OK and res[k].t == alone[k].t, k
        assert_same(batch[k], alone[k], k)


@pytest.mark.parametrize("members", [3, len(MEMBERS)])  # launches of their own, a pack
def test_a_batch_left_alone_gets_to_its_end(members):
    batch, alone = build()[:members], build()[:members]
    ends = [20 * end for _, end in MEMBERS[:members]]
    run = E.BatchRun(batch, ends)
    left, limit = set(range(members)), time.monotonic() + 60
    while left and time.monotonic() < limit:  # collect does not feed the batch
        time.sleep(0.05)
        for i in sorted(left):
            if run._lib.vf_batch_collect(run._b, i, None, None, None, None) == N.VF_OK:
                left.remove(i)
    assert not left
    for k, r in enumerate(run.finish()):
        vf.simulate_to_time(alone[k], ends[k])
        assert r.t == alone[k].t, k
        assert_same(batch[k], alone[k], k)
