"""Square and cube roots as the Float64 kernels compute them (integers and
Float32 seeds) on the device: the square root against the IEEE one bit for bit,
the cube root against the oracle's correctly rounded one."""
import numpy as np
import pytest

from oracle import vf_oracle as O
from volumefluxes_sm103 import _native as N

pytestmark = pytest.mark.gpu


def roots(x):
    lib = N.load()
    x = np.ascontiguousarray(x, dtype=np.float64)
    sq, cb = np.empty_like(x), np.empty_like(x)
    assert lib.vf_selftest_roots(0, N.ptr(x), x.size, N.ptr(sq), N.ptr(cb)) == N.VF_OK, lib.vf_last_error(None)
    return sq, cb


def values(n, kind):
    rng = np.random.default_rng(11)
    if kind == "bits":      # every exponent, both signs, subnormals, infinities, NaNs
        return rng.integers(0, 2**64, n, dtype=np.uint64).view(np.float64)
    if kind == "squares":   # a few ulps around exact squares and cubes
        s = np.round(rng.uniform(2**25, 2**26, n))
        c = np.round(rng.uniform(2**16, 2**17, n))
        v = np.where(rng.integers(0, 2, n) == 0, s * s, c * c * c)
        return (v.view(np.int64) + rng.integers(-3, 4, n)).view(np.float64)
    return 9.81 * rng.uniform(1e-5, 8.0, n)  # g*h of the step


@pytest.mark.parametrize("kind", ["bits", "squares", "depths"])
def test_square_roots_are_ieee(kind):
    x = values(2_000_000, kind)
    sq, _ = roots(x)
    with np.errstate(all="ignore"):
        want = np.sqrt(x)
    same = (sq.view(np.uint64) == want.view(np.uint64)) | (np.isnan(sq) & np.isnan(want))
    assert same.all(), (x[~same][:4], sq[~same][:4], want[~same][:4])


@pytest.mark.parametrize("kind", ["bits", "squares", "depths"])
def test_cube_roots_are_correctly_rounded(kind):
    x = values(20_000, kind)
    _, cb = roots(x)
    cbrt = O.load().vfo_cbrt
    want = np.array([cbrt(float(v)) for v in x])
    same = (cb.view(np.uint64) == want.view(np.uint64)) | (np.isnan(cb) & np.isnan(want))
    assert same.all(), (x[~same][:4], cb[~same][:4], want[~same][:4])
