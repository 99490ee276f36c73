"""The layers' BF16 GELU over every float: the approximation with its interval
and the reference decision give the reference's bits, and it decides by itself
for all but a small part of what the layers see."""
import ctypes as ct

import pytest

from anacor_public_gb300 import _lib, build

pytestmark = pytest.mark.gpu


def test_every_float_rounds_as_the_reference():
    build.build()
    L = _lib.load()
    wrong, opened = ct.c_uint64(), ct.c_uint64()
    assert L.anacor_gelu_check(ct.byref(wrong), ct.byref(opened)) == 0, _lib.last_error(L)
    assert wrong.value == 0
    # floats below about -4 (a quarter of all exponents there are) and few others
    assert opened.value < 0.26 * 2 ** 32


@pytest.mark.parametrize("members", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("rows", [1, 127, 128, 129, 1000, 4864, 9729, 19457, 40000])
def test_fused_inference_splits(members, rows):
    """Row counts around the lines where a tile's members move from one CTA to
    clusters of two, four and eight, against the layer-by-layer path: the same bits."""
    import numpy as np

    from anacor_public_gb300 import surrogate
    rng = np.random.default_rng(rows + members)
    x7 = rng.uniform(-1, 1, (rows, 7)).astype(np.float32)
    m = surrogate.Surrogate(members=members, seed=3)
    m.scale = (-1.0, 0.3)
    got = m.predict(x7, members=True)
    m.set_inference(False)
    want = m.predict(x7, members=True)
    m.close()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
