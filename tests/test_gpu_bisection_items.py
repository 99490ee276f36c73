"""Work items of the bisection with an axis beyond the fixed-point searches:
few reflections of many voxels, many of few, and counts around a warp, against
the oracle (5e-7 relative: expf and the compensated FP32 mean).  And few
reflections keep the device busy: 20 of 20,000 voxels are 12,500 items of one
voxel a lane, five waves of the resident warps, so a leg of them may take no
more than twice a leg of 500 reflections (with an item a block it took 3.5
times as long, seven warps of eight idle)."""
import numpy as np
import pytest
import torch

from anacor_public_gb300 import build, synth, tracer
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


def ellipsoid(shape):
    g = np.ogrid[:shape[0], :shape[1], :shape[2]]
    r = sum(((a - (n - 1) / 2) / (n / 2 - 3)) ** 2 for a, n in zip(g, shape))
    lab = np.zeros(shape, np.int8)
    lab[r <= 1.0], lab[r <= 0.8], lab[r <= 0.5] = 2, 1, 3
    return lab


def plan_of(lab, n_vox, n_refl):
    c = np.argwhere(lab == 3)
    c = c[np.random.default_rng(n_vox).permutation(len(c))[:n_vox]].astype(np.int64)
    s = synth.small_sample(n_refl=n_refl)
    p = tracer.Plan(lab, np.ascontiguousarray(c), s.voxel, s.mu)
    p.set_reflections(s.s1, s.omega, s.xray, s.omega_axis, s.F)
    return p, np.ascontiguousarray(c), s


@pytest.mark.parametrize("n_vox,n_refl", [(1, 1), (31, 3), (33, 40), (257, 2), (2049, 5), (300, 900)])
def test_counts(n_vox, n_refl):
    lab = ellipsoid((1030, 60, 50))
    p, c, s = plan_of(lab, n_vox, n_refl)
    p.run_bisection(4)
    got = p.result()
    o = Oracle()
    for i in {0, n_refl // 2, n_refl - 1}:
        xr, sr = o.rotate(s, i)
        want = o.ib(c, sr, xr, s.voxel, s.mu, lab, 4)
        assert abs(got[i] - want) <= 5e-7 * want, (i, got[i], want)
    p.close()


def test_few_reflections_fill_the_device():
    lab = ellipsoid((1100, 220, 210))
    per_leg = []
    for n_refl in (20, 500):
        p, c, _ = plan_of(lab, 20000, n_refl)
        stream = torch.cuda.Stream()
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            p.run_bisection(4, stream.cuda_stream)
            b.record(stream)
            b.synchronize()
            times.append(a.elapsed_time(b))
        p.result(stream.cuda_stream)
        per_leg.append(min(times[1:]) / (len(c) * n_refl))
        p.close()
    assert per_leg[0] <= 2.0 * per_leg[1], per_leg
