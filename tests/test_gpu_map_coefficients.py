"""Map values under coefficients and voxel edges at the ends of the range:
infinite and undefined coefficients (an absent class counts with length zero,
so they give NaN for it, also for a leg without length), and edges whose
squares a float does not hold.  Against the oracle's FP64 lengths, bit for bit
(method 1: CUDA's FP64 exp within one ulp, so one float step)."""
import numpy as np
import pytest

from anacor_public_gb300 import build, gridding, tracer
from oracle import gridding_oracle as go
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
INF, NAN = np.inf, np.nan


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


@pytest.mark.parametrize("mu,edge", [((INF, 0.1, 0.1, 0.1), 0.3), ((0.1, INF, 0.1, 0.1), 0.3), ((0.1, 0.1, 0.1, NAN), 0.3),
                                     ((NAN, 0.1, 0.1, 0.1), 0.3), ((1e300, 0.1, 0.1, 0.0), 0.3), ((0.0, 0.0, 0.0, 0.0), 0.3),
                                     ((-INF, 0.1, 0.1, 0.1), 0.3), ((1e22, 2e22, 1e23, 0.0), 1e-24),
                                     ((1e-22, 2e-22, 1e-23, 0.0), 1e22)])
@pytest.mark.parametrize("method", [1, 2])
def test_map_coefficients(mu, edge, method):
    lab = np.zeros((20, 21, 22), np.int8)
    lab[3:17, 3:17, 3:17] = 1
    lab[6:12, 6:12, 6:12] = 3
    lab[7:9, 7:9, 4:7] = 2
    coords = np.array([[8, 8, 8], [2, 8, 8], [7, 9, 10], [11, 6, 7], [16, 16, 16], [1, 1, 1]], np.int64)
    vox, mu = np.array([1.0, 0.9, 1.1]) * edge, np.array(mu)
    plan = tracer.Plan(lab, coords, vox, mu)
    g = gridding.GriddingMap(plan, 19, 18, method).build()
    m = g.map()
    s1, _, _ = gridding.directions(19, 18)
    o = Oracle()
    with np.errstate(all="ignore"):
        for d in range(0, len(s1), 7):
            det = o.leg_detail(coords, s1[d], s1[d], vox, lab)
            if (det["status"][:, 1] != 0).any():
                continue
            want = go.map_value(det["L"][:, 1, :], mu, 1 if method == 1 else 0)
            if method == 1:
                ok = np.isfinite(want)   # infinite where an exponent is -infinity
                assert np.array_equal(m[d][~ok], want[~ok], equal_nan=True), d
                assert np.max(np.abs(m[d][ok] - want[ok]), initial=0.0) <= np.spacing(np.float32(1.0)), d
            else:
                assert np.array_equal(m[d], want, equal_nan=True), d
    g.close()
    plan.close()
