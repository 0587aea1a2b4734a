"""The reverse sweep on grids that are not square and fill their blocks unevenly:
one column past a block, one row past a block, a single block column of many rows.
The gradient against the oracle on dual numbers, to the 1e-9 the other gradient
tests hold it to; the friction direction alone as well, whose sum is spread over the
pointwise kernel's blocks."""
import math
from dataclasses import replace
from types import SimpleNamespace

import numpy as np
import pytest

from oracle import vf_oracle as O
from test_gpu_adjoint import run_adjoint
from vfhelpers import hills_rect, oracle_from

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(33, 9), (70, 33), (7, 65), (64, 2), (32, 16)])
def test_gradient_on_ragged_grids(nx, ny):
    steps = 9
    sc = hills_rect(nx, ny)
    wet = sc.w0 <= 1.5  # in motion, so that friction acts from the first step
    sc = replace(sc, hu0=np.where(wet, 0.2, 0.0), hv0=np.where(wet, -0.1, 0.0))
    gauges = np.array([[0, 0], [nx - 1, ny - 1], [nx // 2, ny // 2], [nx - 2, 0], [1, ny - 1]], dtype=np.int32)
    case = SimpleNamespace(scenario=sc, B_target=sc.B + 1e-3 * np.cos(np.arange(sc.B.size)).reshape(sc.B.shape))
    dts, target, loss, gB, gCz = run_adjoint(case, gauges, steps)
    o = oracle_from(sc)
    assert list(dts) == [o.perform_step(math.inf) for _ in range(steps)]
    rng = np.random.default_rng(5)
    for v, cz in ((rng.standard_normal(sc.B.shape), 1e-3), (np.zeros_like(sc.B), 1.0)):
        lo, dlo = O.dual_gauge_loss(oracle_from(sc).o, sc.w0, sc.hu0, sc.hv0, dts, gauges, target, Bdot=v, Cz_dot=cz)
        assert lo == loss
        got = float(np.sum(gB * v)) + gCz * cz
        assert abs(got - dlo) <= 1e-9 * abs(dlo), (got, dlo)
