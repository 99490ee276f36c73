"""Fields of a second kind built for a plan while marches on the first are in
flight on another stream: labels that reach the walls, so that the march's
limits depend on the plan's room at the walls, which stays as it is.  A_h bit
for bit what the march gave before, and on either kind what the cooperative
march gives (the same legs in the same order)."""
import numpy as np
import pytest
import torch

from anacor_public_gb300 import build, gridding, synth, tracer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


@pytest.mark.parametrize("room", [0, 1, 5])
@pytest.mark.parametrize("first,second", [(8, 12), (12, 8), (8, None), (12, 16)])
def test_second_field_beside_replays(room, first, second):
    lab = np.zeros((121, 110, 97), np.int8)
    core = tuple(slice(room, n - room) for n in lab.shape)
    z, y, x = np.indices(lab.shape)
    lab[core] = (1 + (z + y + x) // 40 % 2)[core]
    lab[50:70, 40:60, 40:60] = 3
    coords = np.argwhere(lab == 3)[::7].astype(np.int64)
    s = synth.small_sample(n_refl=900)
    plan = tracer.Plan(lab, coords, np.array([0.3, 0.3, 0.3]), s.mu)
    plan.set_reflections(s.s1, s.omega, s.xray, s.omega_axis, s.F)
    plan.configure(4, 1024, 1)
    plan.run()
    want = plan.result()
    stream = torch.cuda.Stream()
    batch = tracer.Batch([plan])
    batch.configure(first)
    batch.capture(stream.cuda_stream)
    for _ in range(20):
        batch.replay(stream.cuda_stream)
    if second is None:   # a map's creation builds the octant fields
        g = gridding.GriddingMap(plan, 20, 18)
    else:
        plan.configure(second, 1024, 1)
    batch.wait(stream.cuda_stream)
    assert np.array_equal(batch.results(stream.cuda_stream)[0], want)
    batch.replay(stream.cuda_stream)
    batch.wait(stream.cuda_stream)
    assert np.array_equal(batch.results(stream.cuda_stream)[0], want)
    batch.close()
    if second is None:
        g.close()
    else:
        plan.run()
        assert np.array_equal(plan.result(), want)
    plan.close()
