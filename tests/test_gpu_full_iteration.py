"""Calls with full_iteration: every leg is left to the per-lane march, which
reads labels, so a call builds no fields (14 bytes a voxel of device memory),
whatever its size, and a plan or batch set to a field variant takes no longer
than the cooperative one of the same budget (the same kernel: 1.15 times, for
the clocks; out of line in the field kernel they took 1.3 times as long).  A_h is what a plan on the octant fields gives: the same
terms summed over other work items, 2e-11 relative (the compensation's own
roundings over at most 64 terms a lane, (64^2 / 2 + 10 x 69) 2^-48 on each
side)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from anacor_public_gb300 import build, synth, tracer

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SIZE = 300


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


def sample(n, n_vox, n_refl):
    lab = np.zeros((n, n, n), np.int8)
    lab[n // 4:n - n // 4, n // 4:n - n // 4, n // 4:n - n // 4] = 1
    lab[n // 3:n // 2, n // 3:n // 2, n // 3:n // 2] = 3
    coords = np.argwhere(lab == 3)
    coords = np.ascontiguousarray(coords[::max(1, len(coords) // n_vox)][:n_vox].astype(np.int64))
    return lab, coords, synth.small_sample(n_refl=n_refl)


def call(lab, coords, s, full):
    return tracer.absorption(lab, coords, s.s1, s.omega, s.xray, s.omega_axis, s.F, s.voxel, s.mu, full_iteration=full)


def memory_kept():
    """Device memory a call adds to what the library keeps, without and then
    with fields, after a small call has set the library up."""
    import torch
    call(*sample(20, 10, 40), 1)
    free = [torch.cuda.mem_get_info()[0]]
    for full in (1, 0):
        call(*sample(SIZE, 2000, 3000), full)
        free.append(torch.cuda.mem_get_info()[0])
    print("kept", free[0] - free[1], free[1] - free[2])


def test_no_fields_for_full_iteration():
    run = subprocess.run([sys.executable, "-c", "from tests.test_gpu_full_iteration import memory_kept; memory_kept()"],
                         cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stderr[-2000:]
    full, stopped = map(int, run.stdout.split("kept")[1].split())
    assert full < 7 * SIZE ** 3, full          # the volume, and less than half of the fields
    assert stopped > 10 * SIZE ** 3, stopped   # the same call without full_iteration builds them


@pytest.mark.parametrize("n,n_vox,n_refl", [(60, 300, 700), (150, 1500, 900)])
def test_full_iteration_same_terms(n, n_vox, n_refl):
    lab, coords, s = sample(n, n_vox, n_refl)
    got = call(lab, coords, s, 1)
    p = tracer.Plan(lab, coords, s.voxel, s.mu, full_iteration=1)
    p.set_reflections(s.s1, s.omega, s.xray, s.omega_axis, s.F)
    p.configure(12, 1024, 1)
    p.run()
    want = p.result()
    p.close()
    assert np.all(np.abs(got - want) <= 2e-11 * want)


def test_field_variants_cost_nothing():
    import torch
    lab, coords, s = sample(SIZE, 5000, 2000)
    plans = [tracer.Plan(lab, coords, s.voxel, s.mu, full_iteration=f) for f in (1, 1, 0)]
    for p in plans:
        p.set_reflections(s.s1, s.omega, s.xray, s.omega_axis, s.F)
    stream = torch.cuda.Stream()

    def timed(run):
        ms = []
        for _ in range(5):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            run(stream.cuda_stream)
            b.record(stream)
            b.synchronize()
            ms.append(a.elapsed_time(b))
        return min(ms[1:])

    took, ah = {}, {}
    for variant in (4, 8, 12, 16):
        plans[0].configure(variant, 1024, 1)
        took[variant] = timed(plans[0].run)
        ah[variant] = plans[0].result(stream.cuda_stream)
    for variant in (8, 12, 16):
        assert took[variant] <= 1.15 * took[4], took
        assert np.array_equal(ah[variant], ah[4])
    plans[1].configure(4, 1024, 1)
    plans[2].configure(4, 1024, 1)
    for members, at in ((plans[:2], 4), (plans[:2], 12), (plans, 12)):
        b = tracer.Batch(members)
        b.configure(at)
        took[len(members), at] = timed(b.launch)
        b.wait(stream.cuda_stream)
        got = b.results(stream.cuda_stream)
        assert np.array_equal(got[0], ah[4]) and np.array_equal(got[1], ah[4])
        b.close()
    assert took[2, 12] <= 1.15 * took[2, 4], took
    for p in plans:
        p.close()
