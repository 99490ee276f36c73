"""The field march's own branches against the cooperative march, bit for bit.

Volumes whose labels keep 0, 1, 2, ... voxels of room from the walls (the leg
is marched to vacuum without wall limits from floor(qmax) + 2 on), elongated
ones (ratios above 1), ones with more class changes than the segment list
holds, labels 5..7, and directions whose ratios lie within 2^-32..2^-20 of a
fraction, so that increments fall near rounding boundaries.  Both marches
visit the same voxels and form the same FP32 terms in the same order: A_h and
the step totals are equal.
"""
import numpy as np
import pytest

from anacor_public_gb300 import build, tracer

pytestmark = pytest.mark.gpu
EYE = np.eye(3).reshape(-1)
AXIS = np.array([0.0, 1.0, 0.0])


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


def directions(n, rng):
    """Unit vectors, half of them with component ratios close to small fractions."""
    v = rng.normal(size=(n, 3))
    for k in range(0, n, 2):
        s = rng.permutation(3)
        v[k, s[0]] = rng.choice([-1.0, 1.0])
        for a in s[1:]:
            d = int(rng.integers(2, 31))
            v[k, a] = rng.choice([-1, 1]) * (rng.integers(1, d) / d + rng.choice([-1, 1]) * 2.0 ** -rng.uniform(20, 33))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def volume(shape, room, kind, rng):
    lab = np.zeros(shape, np.int8)
    core = tuple(slice(min(room, (n - 1) // 2), n - min(room, (n - 1) // 2)) for n in shape)
    inner = tuple(n.stop - n.start for n in core)
    if kind == "blocks":
        coarse = rng.integers(1, 5, tuple(-(-n // 9) for n in inner))
        lab[core] = np.kron(coarse, np.ones((9, 9, 9)))[:inner[0], :inner[1], :inner[2]]
    elif kind == "stripes":   # a change every other voxel: more than the segment list holds
        z, y, x = np.indices(inner)
        lab[core] = 1 + ((z + y + x) // 2) % 7
    else:                     # a solid block
        lab[core] = 3
    return lab


@pytest.mark.parametrize("shape", [(48, 48, 48), (90, 31, 44), (26, 120, 37)])
@pytest.mark.parametrize("room", [0, 1, 2, 3, 5])
@pytest.mark.parametrize("kind", ["blocks", "stripes", "solid"])
def test_field_march_equals_cooperative(shape, room, kind):
    rng = np.random.default_rng([room, shape[0], len(kind)])
    lab = volume(shape, room, kind, rng)
    coords = np.argwhere(lab > 0)[::5].astype(np.int64)
    coords = np.ascontiguousarray(coords[coords.min(1) > 0])   # a start on a min plane leaves through it (the reference asserts)
    s1 = directions(24, rng)
    # one sweep per incident direction; the rotation is the identity
    for xray in directions(3, rng):
        p = tracer.Plan(lab, coords, np.array([0.3, 0.25, 0.4]), np.array([0.01, 0.007, 0.012, 0.002]))
        p.set_reflections(s1, np.zeros(len(s1)), xray, AXIS, EYE)
        p.configure(4, 512, 1)
        p.run()
        want, steps = p.result(), p.count_steps()
        for variant in (8, 9, 12, 16):
            p.configure(variant, 512, 1)
            p.run()
            assert np.array_equal(p.result(), want), variant
            assert p.count_steps() == steps, variant
        p.close()
