"""The map kernel on the octant fields, bit for bit against the oracle's FP64
lengths: volumes with and without room at the walls, odd sizes, label stripes
(more class changes than the list holds), both methods, coefficients that are
zero or negative.  And bilinear lookups at voxel counts around a load of four
and around the line between a warp and a block per reflection, against the
numpy oracle (FP64): expf and the compensated FP32 mean, 5e-7 relative."""
import numpy as np
import pytest

from anacor_public_gb300 import build, gridding, synth, tracer
from oracle import gridding_oracle as go
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


def striped(shape, room):
    lab = np.zeros(shape, np.int8)
    core = tuple(slice(room, n - room) for n in shape)
    z, y, x = np.indices(tuple(n - 2 * room for n in shape))
    lab[core] = 1 + ((z + 2 * y + x) // (2 if room == 1 else 5)) % 4
    return lab


@pytest.mark.parametrize("shape,room", [((33, 41, 27), 3), ((33, 41, 27), 1), ((60, 19, 22), 2), ((30, 31, 32), 0)])
@pytest.mark.parametrize("mu", [(0.01, 0.007, 0.012, 0.0), (0.02, -0.003, 0.01, 0.001)])
@pytest.mark.parametrize("method", [1, 2])
def test_map_bit_for_bit(shape, room, mu, method):
    lab = striped(shape, room)
    coords = np.argwhere(lab > 0)[::11].astype(np.int64)
    coords = np.ascontiguousarray(coords[coords.min(1) > 0])
    vox, mu = np.array([0.31, 0.3, 0.27]), np.array(mu)
    plan = tracer.Plan(lab, coords, vox, mu)
    g = gridding.GriddingMap(plan, 19, 18, method).build()
    m = g.map()
    s1, _, _ = gridding.directions(19, 18)
    o = Oracle()
    for d in range(0, len(s1), 17):
        det = o.leg_detail(coords, s1[d], s1[d], vox, lab)
        if (det["status"][:, 1] != 0).any():
            continue
        want = go.map_value(det["L"][:, 1, :], mu, 1 if method == 1 else 0)
        if method == 1:   # CUDA's FP64 exp is within one ulp of the C library's: a float tie may fall the other way
            assert np.max(np.abs(m[d] - want)) <= np.spacing(np.float32(1.0))
            assert np.mean(m[d] != want) < 1e-3
        else:
            assert np.array_equal(m[d], want), d
    g.close()
    plan.close()


@pytest.mark.parametrize("n_vox", [1, 3, 4, 127, 1030])
@pytest.mark.parametrize("n_refl", [5, 9800])
def test_bilinear_counts(n_vox, n_refl):
    s = synth.small_sample(n_refl=8)
    plan = tracer.Plan(s.label, s.coords[:n_vox], s.voxel, s.mu)
    g = gridding.GriddingMap(plan, 40, 24).build()
    rng = np.random.default_rng(n_vox)
    omega, s1 = synth.reflections(n_refl, rng)
    got = g.interpolate(s1, omega, s.xray, s.omega_axis, s.F, method="linear")
    grid, tl, pl = go.padded(g.map(), 40, 24)
    rx, rs = tracer.rotated_vectors(s.omega_axis, omega, s.F, s.xray, s1)
    for i in list(range(3)) + [n_refl - 1]:
        want = go.interpolate(grid, tl, pl, rx[i], rs[i], 2)
        assert abs(got[i] - want) <= 5e-7 * want
    g.close()
    plan.close()
