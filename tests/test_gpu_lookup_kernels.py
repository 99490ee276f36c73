"""Prepared and asynchronous bilinear lookups, whose launches hold all of a
call's rows (a synchronous call launches at most 2,048 at a time): counts on
both sides of the line from a block to a warp per reflection (64 for each SM),
and voxel counts around a load of four and around one load for each lane of a
warp and of a block.  Against the numpy oracle (FP64): expf and the compensated
FP32 mean, 5e-7 relative; and prepared and asynchronous ones bit for bit."""
import numpy as np
import pytest
import torch

from anacor_public_gb300 import build, gridding, synth, tracer
from oracle import gridding_oracle as go

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


@pytest.mark.parametrize("n_vox", [1, 3, 4, 127, 128, 133, 1030])
@pytest.mark.parametrize("beyond", [-1, 0, 5])
def test_one_launch(n_vox, beyond):
    n = 64 * torch.cuda.get_device_properties(0).multi_processor_count + beyond
    s = synth.small_sample(n_refl=8)
    plan = tracer.Plan(s.label, s.coords[:n_vox], s.voxel, s.mu)
    g = gridding.GriddingMap(plan, 40, 24).build()
    omega, s1 = synth.reflections(n, np.random.default_rng([n_vox, beyond + 1]))
    args = s1, omega, s.xray, s.omega_axis, s.F
    out = torch.full((2, n), -1.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()   # the plan's stream is another one
    g.prepare(*args, method="linear")
    g.run(out[0].data_ptr())
    g.interpolate_async(*args, d_out=out[1].data_ptr(), method="linear")
    torch.cuda.synchronize()
    got, same = out.cpu().numpy()
    assert np.array_equal(got, same)
    grid, tl, pl = go.padded(g.map(), 40, 24)
    rx, rs = tracer.rotated_vectors(s.omega_axis, omega, s.F, s.xray, s1)
    for i in list(range(0, n, 811)) + list(range(n - 9, n)):
        want = go.interpolate(grid, tl, pl, rx[i], rs[i], 2)
        assert abs(got[i] - want) <= 5e-7 * want, i
    g.close()
    plan.close()
