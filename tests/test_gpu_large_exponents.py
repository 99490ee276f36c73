"""Exponents far beyond FP32's range: bilinear lookups on a given map and
bisection with large coefficients.  exp(-x) is 0 there, so that such a voxel
adds nothing to the mean; exponents as far below 0 give no finite mean.  The
other voxels' share is held to 5e-7 relative (expf and the compensated FP32
mean), as in the lookups' and the bisection's own tests."""
import numpy as np
import pytest

from anacor_public_gb300 import build, gridding, synth, tracer
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
EXPONENTS = [1e3, 4095.0, 4097.0, 1e5, 3e7, 6.6e9, 2.4e10, 3.3e11, 1e13, 2e16, 3e18, 1e21, 1e30]


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


@pytest.fixture(scope="module")
def kept(small):
    plan = tracer.Plan(small.label, small.coords[:37], small.voxel, small.mu)
    g = gridding.GriddingMap(plan, 36, 18)
    yield g
    g.close()
    plan.close()


@pytest.mark.parametrize("x", EXPONENTS)
def test_bilinear(small, kept, x):
    m = np.full((kept.n_dirs, 37), 0.25, np.float32)   # a lookup's weights sum to 1 on each leg: 0.5 a voxel
    look = lambda: kept.interpolate(small.s1[:20], small.omega[:20], small.xray, small.omega_axis, small.F, "linear")  # noqa: E731
    m[:, 11] = x / 2
    m[:, 36] = x / 2
    kept.set_map(m)
    want = 35 * np.exp(-0.5) / 37   # exp(-1e3) is far below a float
    assert np.all(np.abs(look() - want) <= 5e-7 * want)
    m[:, 11] = -x / 2
    kept.set_map(m)
    assert not np.isfinite(look()).any()


@pytest.mark.parametrize("x", EXPONENTS)
@pytest.mark.parametrize("length", [40, 1030])   # fixed-point searches; FP64 ones
def test_bisection(x, length):
    lab = np.zeros((length, 20, 18), np.int8)
    lab[4:36, 3:17, 3:15] = 1
    lab[8:30, 5:15, 5:13] = 3
    coords = np.argwhere(lab == 3)[::97].astype(np.int64)
    vox, axis, F = np.array([0.3, 0.27, 0.35]), np.array([0.0, 1.0, 0.0]), np.eye(3).reshape(-1)
    xray, s1 = np.array([-0.8, 0.37, 0.47]), np.array([[0.6, -0.3, 0.74], [-0.2, -0.5, 0.84]])
    o = Oracle()
    for sign in (1, -1):
        mu = np.array([sign * x, 0.011, 0.03, 0.004])   # every path crosses liquor
        got = tracer.bisection(lab, coords, s1, np.zeros(2), xray, axis, F, vox, mu, 4)
        for i in range(2):
            L = o.ib(coords, s1[i], xray, vox, mu, lab, 4, lengths=True)[1].reshape(len(coords), -1, 4).sum(1)
            assert np.min(sign * (L @ mu)) > 110.0   # exp(-104) is below half the smallest float
        if sign > 0:
            assert np.all(got == 0.0)
        else:
            assert not np.isfinite(got).any()
