"""A map whose rebuild fails after it has been written to is no map: lookups
are refused until a build succeeds, which gives the first build's values again.
Directions that are refused before any launch leave the map as it is."""
import numpy as np
import pytest

from anacor_public_gb300 import _lib, build, gridding, synth, tracer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


@pytest.mark.parametrize("outside", [False, True])   # a label without fields: the cooperative map
def test_failed_rebuild(outside):
    s = synth.small_sample(n_refl=20)
    lab = s.label.copy()
    if outside:
        lab[1, 1, 1] = 9
    plan = tracer.Plan(lab, s.coords[:70], s.voxel, s.mu)
    g = gridding.GriddingMap(plan, 120, 60).build()   # 7,200 directions: two uploads
    first = g.map()
    look = lambda: g.interpolate(s.s1, s.omega, s.xray, s.omega_axis, s.F, "linear")  # noqa: E731
    want = look()
    s1, theta, phi = gridding.directions(120, 60)
    for bad in (np.nan, 0.0):
        d = s1.copy()
        d[7100] = bad
        with pytest.raises(_lib.AnacorError):
            g.build(d, theta, phi)
        assert np.array_equal(look(), want)
    with pytest.raises(_lib.AnacorError):   # angles of the opposite side: no face's rule takes them
        g.build(s1, -theta, phi)
    with pytest.raises(_lib.AnacorError):
        look()
    g.build()
    assert np.array_equal(g.map(), first) and np.array_equal(look(), want)
    g.close()
    plan.close()
