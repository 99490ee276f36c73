"""exp(-x) of bilinear lookups at the ends of a float: the largest exponents a
map can hold, subnormal results, infinite and undefined ones.  0 for large
exponents of either leg, no finite mean for large negative ones, NaN for
undefined ones; FP32's own last values within the spacing of the smallest
floats and 5e-7 relative."""
import numpy as np
import pytest

from anacor_public_gb300 import build, gridding, synth, tracer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


@pytest.fixture(scope="module")
def kept():
    s = synth.small_sample(n_refl=30)
    plan = tracer.Plan(s.label, s.coords[:5], s.voxel, s.mu)
    g = gridding.GriddingMap(plan, 36, 18)

    def mean(x):
        g.set_map(np.full((g.n_dirs, 5), np.float32(x) / 2, np.float32))
        return g.interpolate(s.s1, s.omega, s.xray, s.omega_axis, s.F, "linear")

    yield mean
    g.close()
    plan.close()


@pytest.mark.parametrize("x", [0.0, 0.3, 20.0, 80.0, 87.0, 88.6, 90.0, 100.0, 103.0, 110.0, 4095.0, 4158.0, 4159.5, 1e4,
                               1e9, 1e18, 1e30, 2.3e38, 2.5e38, 3.3e38])
def test_exponents(kept, x):
    want = np.exp(-np.float64(np.float32(x)))
    got = kept(x)
    # the sum of two halves is exact, each lookup's weights sum to one within a float pair
    assert np.all(np.abs(got - want) <= want * (5e-7 + x * 2.0 ** -40) + 2.0 ** -149)
    if x >= 88.8:
        assert not np.isfinite(kept(-x)).any()


@pytest.mark.parametrize("x", [np.inf, -np.inf, np.nan])
def test_undefined(kept, x):
    assert not np.isfinite(kept(x)).any()
