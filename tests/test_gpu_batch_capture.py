"""A batch in flight, or a server at work, beside a graph capture in the global mode
(torch's default): the capture holds, and the work gets to its end by itself."""
import time

import numpy as np
import pytest

import volumefluxes_sm103 as vf
from volumefluxes_sm103 import _native as N
from volumefluxes_sm103 import ensemble as E
from volumefluxes_sm103.serving import Request, Server
from vfhelpers import hills_rect

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members", [3, 10])  # launches of their own, a pack
def test_a_capture_beside_a_batch(members):
    torch = pytest.importorskip("torch")
    sims, alone = ([hills_rect(70, 64 + k).build(vf.SM103Backend(np.float64)) for k in range(members)] for _ in range(2))
    ends = [8.0] * members
    x = torch.ones(1024, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    run = E.BatchRun(sims, ends)
    with torch.cuda.graph(graph, capture_error_mode="global"):
        y = x
        left, limit = set(range(members)), time.monotonic() + 60
        while left and time.monotonic() < limit:  # collect does not feed the batch
            y = y + 1
            time.sleep(0.01)
            left -= {i for i in left if run._lib.vf_batch_collect(run._b, i, None, None, None, None) == N.VF_OK}
        assert not left
        assert run.n_done() == members
    graph.replay()
    torch.cuda.synchronize()
    assert float(y[0]) > 1
    for sim, ref, r in zip(sims, alone, run.finish()):
        vf.simulate_to_time(ref, 8.0)
        assert r.t == ref.t == 8.0
        a, b = vf.current_interior_state(sim), vf.current_interior_state(ref)
        assert np.array_equal(a.h, b.h) and np.array_equal(a.hu, b.hu) and np.array_equal(a.hv, b.hv)


def test_a_capture_beside_a_server():
    torch = pytest.importorskip("torch")
    requests = [Request(hills_rect(70, 64 + k), np.float64, 8.0) for k in range(3)]
    x = torch.ones(1024, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with Server(1 << 30) as srv:
        with torch.cuda.graph(graph, capture_error_mode="global"):
            y = x + 1
            left, limit = {srv.submit(r) for r in requests}, time.monotonic() + 60
            tickets = sorted(left)
            while left and time.monotonic() < limit:
                time.sleep(0.01)
                left -= set(srv.poll())
            assert not left
        graph.replay()
        torch.cuda.synchronize()
        assert float(y[0]) == 2
        for k, t in enumerate(tickets):
            res, ref = srv.result(t), hills_rect(70, 64 + k).build(vf.SM103Backend(np.float64))
            vf.simulate_to_time(ref, 8.0)
            assert res.status == N.VF_BATCH_OK and res.t == ref.t == 8.0
            assert np.array_equal(res.state.h, vf.current_interior_state(ref).h)
