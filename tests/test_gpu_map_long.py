"""Map values of legs of thousands of voxels, bit for bit against the oracle's
FP64 lengths: thin volumes with one axis up to the longest that is accepted,
legs along it whose squared displacement is a whole number of more than 24
bits, in both senses."""
import math

import numpy as np
import pytest

from anacor_public_gb300 import build, gridding, tracer
from oracle import gridding_oracle as go
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


def polar(v):
    """dials_2_thetaphi of a vector whose second component is not zero, with the C library's functions."""
    r = math.sqrt(v[0] * v[0] + v[1] * v[1])
    if v[1] < 0:
        return math.atan(-v[2] / r), math.atan(-v[0] / v[1])
    t = math.atan(-v[2] / r)
    return (math.pi - t if v[2] < 0 else -math.pi - t), -math.atan(-v[0] / -v[1])


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [4100, 5003, 8191])
def test_long_legs_bit_for_bit(axis, n):
    rng = np.random.default_rng([axis, n])
    shape = [14, 14, 14]
    shape[axis] = n
    lab = np.zeros(shape, np.int8)
    inside = tuple(slice(3, k - 3) for k in shape)
    along = np.arange(n - 6)
    label = np.where(along % 1501 < 400, 2, 1)
    label[:40] = label[-40:] = 3
    lab[inside] = label.reshape([-1 if a == axis else 1 for a in range(3)])
    c = rng.integers(4, 10, (60, 3))
    c[:, axis] = np.concatenate([rng.integers(4, 40, 30), n - 1 - rng.integers(4, 40, 30)])
    coords = np.ascontiguousarray(c.astype(np.int64))
    d = rng.uniform(-3.0, 3.0, (324, 3)) / n
    d[:, axis] = np.where(np.arange(324) % 2, 1.0, -1.0)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    s1 = np.ascontiguousarray(d[:, [0, 2, 1]])   # (z, y, x) of the volume are components 0, 2, 1 of the vector
    ang = np.array([polar(v) for v in s1])
    vox, mu = np.array([0.31, 0.3, 0.27]), np.array([0.01, 0.007, 0.012, 0.0])
    plan = tracer.Plan(lab, coords, vox, mu)
    g = gridding.GriddingMap(plan, 18, 18).build(s1, ang[:, 0], ang[:, 1])
    m = g.map()
    o = Oracle()
    longest = 0
    for k in range(0, 324, 5):
        det = o.leg_detail(coords, s1[k], s1[k], vox, lab)
        assert (det["status"][:, 1] == 0).all()
        longest = max(longest, int(det["len"][:, 1].max()))
        assert np.array_equal(m[k], go.map_value(det["L"][:, 1, :], mu)), k
    assert longest > n - 60
    g.close()
    plan.close()
