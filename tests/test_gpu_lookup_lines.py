"""Synchronous lookups on both sides of the line between one stream and two
(2,048 reflections), after one another and beside prepared ones: every part of
a large call gives its own values, bit for bit (the same kernel, a block each)."""
import numpy as np
import pytest
import torch

from anacor_public_gb300 import build, gridding, synth, tracer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


@pytest.mark.parametrize("method", ["nearest", "linear"])
@pytest.mark.parametrize("n_vox", [1, 37, 300])
def test_parts(method, n_vox):
    s = synth.small_sample(n_refl=8)
    plan = tracer.Plan(s.label, s.coords[:n_vox], s.voxel, s.mu)
    g = gridding.GriddingMap(plan, 40, 24).build()
    omega, s1 = synth.reflections(5000, np.random.default_rng(n_vox))
    look = lambda i, n: g.interpolate(s1[i:i + n], omega[i:i + n], s.xray, s.omega_axis, s.F, method=method)  # noqa: E731
    whole = look(0, 5000)
    g.prepare(s1[:300], omega[:300], s.xray, s.omega_axis, s.F, method=method)
    for i, n in ((0, 1), (7, 256), (9, 257), (0, 2047), (100, 2048), (50, 2049), (0, 1), (4999, 1), (1000, 4000)):
        assert np.array_equal(look(i, n), whole[i:i + n]), (i, n)
    out = torch.zeros(300, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    g.run(out.data_ptr())
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), whole[:300])
    g.close()
    plan.close()
