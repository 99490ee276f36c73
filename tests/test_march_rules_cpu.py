"""Rules the field march rests on, checked on the CPU.

* fixed point: i * Q (Q = llrint(q * 2^32)) and the reference's FP64
  c + fl(i * q) have the same floor and C round unless the fixed-point
  fraction lies within kFieldMargin units of the boundary;
* wall room: a leg whose non-vacuum labels keep floor(qmax) + 2 voxels of room
  from the walls it moves toward examines no position outside the volume
  before it meets vacuum, whichever increments it skips.
"""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "anacor_public_gb300", "csrc", "trace_kernels.cu")


def margin():
    m = re.search(r"kFieldMargin = (\d+)u \+ (\d+)u;", open(CSRC).read())
    return int(m.group(1)) + int(m.group(2))


def c_round(v):
    return np.where(v >= 0, np.floor(np.abs(v) + 0.5), -np.floor(np.abs(v) + 0.5))


@pytest.mark.parametrize("rational", [False, True])
def test_fixed_point_agrees_outside_the_margin(rational):
    rng = np.random.default_rng(5)
    n = 400_000
    q = rng.uniform(-3.0, 3.0, n)
    if rational:   # ratios close to a fraction: many increments fall near a boundary
        k = rng.integers(1, 40, n)
        q = rng.integers(-3 * k, 3 * k + 1) / k + rng.uniform(-1, 1, n) * 2.0 ** rng.uniform(-44, -18, n)
    i = rng.integers(0, 8193, n)
    c = rng.integers(0, 8192, n)
    inside = np.abs(c + i * q) < 8192
    q, i, c = q[inside], i[inside], c[inside]
    Q = np.rint(q * 2.0 ** 32).astype(np.int64)
    v = c + (i * q)
    for off, want in ((0, np.floor(v)), (1 << 31, c_round(v))):
        keep = v >= 0 if off else np.ones(v.shape, bool)   # positions inside the volume
        e = i * Q + off
        frac = e & 0xFFFFFFFF
        near = (frac + margin()) & 0xFFFFFFFF < 2 * margin()
        ok = ~near & keep
        assert np.array_equal((e >> 32)[ok] + c[ok], want[ok].astype(np.int64))
        if rational:
            assert near.any()
        # the margin is folded into the start: the integer part changes only near a boundary
        assert np.array_equal(((e + margin()) >> 32)[~near], (e >> 32)[~near])


@pytest.mark.parametrize("qmax", [0.4, 1.0, 1.7, 4.9])
def test_free_legs_stay_inside(qmax):
    rng = np.random.default_rng(int(qmax * 10))
    for _ in range(300):
        q = rng.uniform(-qmax, qmax, 2)
        need = int(np.floor(np.max(np.abs(q)))) + 2
        dims = rng.integers(2 * need + 1, 40, 3)
        # the step axis is 0; the box of non-vacuum labels keeps `need` voxels on the walls ahead
        step = rng.choice([-1, 1])
        sign = np.array([step, -1 if q[0] < 0 else 1, -1 if q[1] < 0 else 1])
        lo = np.where(sign < 0, need, 0)
        hi = np.where(sign < 0, dims - 1, dims - 1 - need)
        c = rng.integers(lo, hi + 1)
        i = 0
        for _ in range(2000):
            p = np.array([c[0] + i * step, int(np.floor(c[1] + i * q[0])), int(np.floor(c[2] + i * q[1]))])
            # one voxel either way: the inner loop's position near a rounding boundary
            assert np.all(p[1:] - 1 >= -1) and np.all(p >= 0) and np.all(p < dims)
            near = p + np.array([0, sign[1], sign[2]])
            assert np.all(near >= 0) and np.all(near < dims)
            if not (np.all(p >= lo) and np.all(p <= hi)):
                break   # vacuum
            # any number of increments proven to keep a label inside the box, then the examined one
            k = 1
            while rng.random() < 0.4:
                n = np.array([c[0] + (i + k) * step, int(np.floor(c[1] + (i + k) * q[0])),
                              int(np.floor(c[2] + (i + k) * q[1]))])
                if not (np.all(n >= lo) and np.all(n <= hi)):
                    break
                k += 1
            i += k
        else:
            raise AssertionError("the leg met no vacuum")
