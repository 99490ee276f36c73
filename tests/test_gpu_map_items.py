"""A map's work items follow the number of its directions and voxels: rows of a
large map (256 voxels an item) and of small ones with the same directions (down
to 32) are the same bits, with and without room at the walls, and with
full_iteration.  And few directions keep the device busy: 342 of them take at
most a fifth of the time of 4,277, a twelfth of whose work they are."""
import time

import numpy as np
import pytest

from anacor_public_gb300 import build, gridding, tracer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


def striped(shape, room, width):
    lab = np.zeros(shape, np.int8)
    core = tuple(slice(room, n - room) for n in shape)
    z, y, x = np.indices(shape)
    lab[core] = (1 + (z + 2 * y + x) // width % 4)[core]
    return lab


def plan_of(lab, n_vox, full=0):
    c = np.argwhere(lab > 0)
    c = c[c.min(1) > 0]
    c = np.ascontiguousarray(c[np.random.default_rng(n_vox).permutation(len(c))[:n_vox]].astype(np.int64))
    return tracer.Plan(lab, c, np.array([0.31, 0.3, 0.27]), np.array([0.01, 0.007, 0.012, 0.0]), full)


@pytest.mark.parametrize("n_vox,room,full", [(1, 3, 0), (31, 1, 0), (257, 3, 0), (1000, 1, 0), (600, 3, 1)])
def test_rows_do_not_depend_on_items(n_vox, room, full):
    p = plan_of(striped((40, 33, 47), room, 6), n_vox, full)
    big = gridding.GriddingMap(p, 360, 180).build()
    m = big.map()
    s1, theta, phi = gridding.directions(360, 180)
    for nt, npf in ((19, 18), (90, 45)):
        pick = np.sort(np.random.default_rng(nt).permutation(len(s1))[:nt * npf])
        small = gridding.GriddingMap(p, nt, npf).build(s1[pick], theta[pick], phi[pick])
        assert np.array_equal(small.map(), m[pick])
        small.close()
    big.close()
    p.close()


def test_few_directions_fill_the_device():
    p = plan_of(striped((200, 180, 160), 1, 2), 1500)
    took = {}
    for nt, npf in ((19, 18), (91, 47)):
        g = gridding.GriddingMap(p, nt, npf)
        times = []
        for _ in range(6):
            t = time.perf_counter()
            g.build()
            times.append(time.perf_counter() - t)
        took[nt * npf] = min(times[1:])
        g.close()
    assert took[342] <= took[4277] / 5, took
    p.close()
