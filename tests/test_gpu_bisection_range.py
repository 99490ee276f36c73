"""Bisection with voxel edges and coefficients far from one, whose squares,
products or own values a float does not hold: against the oracle's FP64
evaluation, 5e-7 relative (expf and the compensated FP32 mean)."""
import numpy as np
import pytest

from anacor_public_gb300 import build, tracer
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


@pytest.mark.parametrize("scale", [1e-30, 1e-24, 1e-13, 1e-11, 1e-3, 1e3, 1e11, 1e13, 1e22, 1e40])
def test_scaled_bisection(scale):
    """Edges times scale, coefficients over it: the exponents are those of scale 1."""
    lab = np.zeros((40, 36, 44), np.int8)
    lab[4:36, 3:33, 3:41] = 1
    lab[8:30, 8:28, 9:35] = 3
    lab[30:34, 10:30, 10:30] = 2
    coords = np.argwhere(lab == 3)[::197].astype(np.int64)
    vox, mu = np.array([0.3, 0.27, 0.35]) * scale, np.array([0.02, 0.011, 0.03, 0.004]) / scale
    xray, s1 = np.array([-0.8, 0.37, 0.47]), np.array([[0.6, -0.3, 0.74], [-0.2, -0.5, 0.84], [0.1, 0.9, 0.42]])
    got = tracer.bisection(lab, coords, s1, np.zeros(3), xray, np.array([0.0, 1.0, 0.0]), np.eye(3).reshape(-1), vox,
                           mu, 4)
    o = Oracle()
    for i in range(3):
        want = o.ib(coords, s1[i], xray, vox, mu, lab, 4)
        assert abs(got[i] - want) <= 5e-7 * want, (i, got[i], want)
