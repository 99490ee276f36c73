"""The fused training step at batches and ensemble sizes where its work
distribution changes (one to several 128-row tiles per CTA, one to several
64-row blocks per K split), against the FP64 statement of the network with the
same BF16 rounding points, and steps that do not depend on
what was run before."""
import numpy as np
import pytest

from anacor_public_gb300 import build, surrogate
from oracle import surrogate_oracle as so

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


@pytest.mark.parametrize("members,rows", [(1, 1024), (3, 2048), (2, 5120), (5, 4096), (9, 3072)])
def test_gradients(members, rows):
    rng = np.random.default_rng(rows + members)
    x7 = rng.uniform(-1, 1, (rows, 7)).astype(np.float32)
    t = rng.normal(size=rows).astype(np.float32)
    m = surrogate.Surrogate(members=members, seed=2, fourier_scale=0.4)
    g, y = m.gradients(x7, t)
    p = m.get_params()
    X0 = so.features(x7, m.get_fourier())
    m.close()
    hidden, (o5, ob5) = so.offsets()
    for e in {0, members - 1}:
        _, y_ref, g_ref = so.loss_and_grads(p[e], X0, t.astype(np.float64))
        # BF16 roundings (2^-9 each) of weights, activations and gradients through eight products, in the 2-norm
        assert np.allclose(y[e], y_ref, rtol=0, atol=2e-2 * np.abs(y_ref).max())
        parts = [(o, 256 * k) for (o, _), k in zip(hidden, so.IN_DIMS)] + [(ob, 256) for _, ob in hidden]
        for o, n in parts + [(o5, 256), (ob5, 1)]:
            a, b = g[e, o:o + n], g_ref[o:o + n]
            assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b) + 1e-7, (o, n)


def test_training_repeats():
    rng = np.random.default_rng(4)
    x7 = rng.uniform(-1, 1, (6000, 7)).astype(np.float32)
    t = np.sin(x7 @ np.arange(1, 8)) * 0.3 - 1.0
    out = []
    for warm in (False, True):
        m = surrogate.Surrogate(members=3, seed=5)
        if warm:   # another batch size first, and gradients: neither moves the step count or the loss
            m.gradients(x7[:1024], t[:1024].astype(np.float32))
        m.set_data(x7, t)
        loss = np.concatenate([m.train(3, batch=2048, total_steps=100), m.train(4, batch=2048, total_steps=100)])
        out.append((loss, m.get_params(), m.predict(x7[:300])[0]))
        m.close()
    assert np.allclose(out[0][0], out[1][0], rtol=1e-6) and np.all(out[0][0] > 0)
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
