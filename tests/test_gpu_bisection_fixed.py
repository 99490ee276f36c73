"""Fixed-point bisection at the edges of its range, against the oracle.

Axes up to 1023 voxels run the fixed-point searches, longer ones the FP64
searches; elongated volumes have ratios beyond the 32-bit products, and
directions close to fractions put probe points near voxel boundaries.  Both
take the oracle's decisions, so A_h differs by the FP32 exponential and the
compensated FP32 mean only: two ulp (2^-23) for expf, half an ulp each for its
argument below 1, the scaling and the sum, below 5e-7 relative."""
import numpy as np
import pytest

from anacor_public_gb300 import build, tracer
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu
EYE = np.eye(3).reshape(-1)
AXIS = np.array([0.0, 1.0, 0.0])


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


def ball(shape, room):
    """Crystal inside liquor inside loop and bubble shells, `room` voxels from the walls."""
    g = np.meshgrid(*[(np.arange(n) - (n - 1) / 2) / max((n - 1) / 2 - room, 0.5) for n in shape], indexing="ij")
    r = np.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2)
    lab = np.zeros(shape, np.int8)
    lab[r <= 1.0] = 2
    lab[r <= 0.85] = 1
    lab[(r <= 0.8) & (r > 0.65) & (g[0] > 0)] = 4
    lab[r <= 0.6] = 3
    return lab


@pytest.mark.parametrize("shape", [(40, 36, 44), (1023, 9, 12), (11, 1022, 10), (1024, 10, 9), (150, 33, 60), (5, 6, 7)])
@pytest.mark.parametrize("cls", [3, 4])
def test_bisection_matches_oracle(shape, cls):
    rng = np.random.default_rng([shape[0], shape[1], cls])
    lab = ball(shape, 1)
    coords = np.argwhere(lab == 3).astype(np.int64)
    coords = np.ascontiguousarray(coords[rng.permutation(len(coords))[:200]])
    v = rng.normal(size=(12, 3)) * np.array([shape[0], shape[2], shape[1]]) ** 0.5
    for k in range(0, 12, 2):   # ratios within 2^-20..2^-34 of a fraction
        d = int(rng.integers(2, 17))
        v[k] = [1.0, 1.0 / d, rng.integers(1, d) / d]
        v[k] = rng.permutation(v[k]) * rng.choice([-1, 1], 3) + 2.0 ** -rng.uniform(20, 34, 3)
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    xray = np.array([-0.8, 0.37, 0.47])
    vox, mu = np.array([0.3, 0.27, 0.35]), np.array([0.02, 0.011, 0.03, 0.004])
    got = tracer.bisection(lab, coords, v, np.zeros(12), xray, AXIS, EYE, vox, mu, cls)
    o = Oracle()
    for i in range(12):
        want = o.ib(coords, v[i], xray, vox, mu, lab, cls)
        assert abs(got[i] - want) <= 5e-7 * want, (i, got[i], want)
