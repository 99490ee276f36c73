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


def test_map_ties_and_launch_groups():
    """Whole-degree directions on the diagonals of a cube (exit-face ties), in
    a map of enough directions for several uploads and launches: bit for bit,
    around the lines between them too."""
    lab = np.zeros((34, 34, 34), np.int8)
    lab[3:31, 3:31, 3:31] = 3
    lab[8:20, 10:25, 6:30] = 1
    a = np.arange(4, 30, 2)
    coords = np.concatenate([np.stack([a, a, a], 1), np.stack([a, a, 34 - a], 1), np.stack([a, 34 - a, a], 1),
                             np.stack([a, a + 0 * a, 17 + 0 * a], 1)]).astype(np.int64)
    vox, mu = np.array([0.3, 0.3, 0.3]), np.array([0.01, 0.007, 0.012, 0.0])
    plan = tracer.Plan(lab, np.ascontiguousarray(coords), vox, mu)
    g = gridding.GriddingMap(plan, 240, 120, 2).build()   # 28,800 directions, 1.5 degrees
    m = g.map()
    s1, _, _ = gridding.directions(240, 120)
    o = Oracle()
    ties = [ip * 240 + it for ip in (0, 30, 60, 90) for it in range(0, 240, 30)]
    for d in ties + [4095, 4096, 4097, 20479, 20480, 28799]:
        det = o.leg_detail(coords, s1[d], s1[d], vox, lab)
        if (det["status"][:, 1] != 0).any():
            continue
        assert np.array_equal(m[d], go.map_value(det["L"][:, 1, :], mu, 0)), d
    g.close()
    plan.close()


def test_lookups_in_chunks():
    """A call with more lookups than the staging holds equals its parts."""
    s = synth.small_sample(n_refl=61)
    plan = tracer.Plan(s.label, s.coords[:40], s.voxel, s.mu)
    g = gridding.GriddingMap(plan, 36, 18, 2).build()
    s1, om = np.tile(s.s1, (960, 1)), np.tile(s.omega, 960)   # 58,560
    whole = g.interpolate(s1, om, s.xray, s.omega_axis, s.F, method="linear")
    part = g.interpolate(s.s1, s.omega, s.xray, s.omega_axis, s.F, method="linear")
    assert np.array_equal(whole, np.tile(part, 960))
    g.close()
    plan.close()
