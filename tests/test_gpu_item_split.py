"""The cut of a launch into work items does not show in A_h: the per-voxel terms
are summed exactly (three floats a lane, an item and a reflection) while they lie
within about 2^40 of each other, so a reflection has the same bits in a full
set, in a part of one, in a batch, at every tile and voxel order, and the
bisection likewise.  The terms themselves are the same in all of them.  (Two
floats, 48 bits, left the last bits of strong absorbers to the cut: A_h of
1e-4 and below.)"""
import math

import numpy as np
import pytest

from anacor_public_gb300 import build, shard, synth, tracer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()


def plan_of(s, part=slice(None)):
    p = tracer.Plan(s.label, s.coords[:4321], s.voxel, s.mu)
    p.set_reflections(s.s1[part], s.omega[part], s.xray, s.omega_axis, s.F)
    return p


def results(p, bisection):
    p.run_bisection(4) if bisection else p.run()
    return p.result()


@pytest.fixture(scope="module", params=[1.0, 40.0, 150.0, 600.0])
def sample(request):
    s = synth.small_sample(n_refl=1501)
    s.mu = s.mu * request.param
    return s


@pytest.mark.parametrize("variant", [4, 8, 12, 16])
@pytest.mark.parametrize("bisection", [False, True])
def test_parts_of_a_set(sample, variant, bisection):
    p = plan_of(sample)
    p.configure(variant, 1024, 1)
    whole = results(p, bisection)
    p.close()
    for world in (2, 7, 200):
        for rank in (0, world // 2, world - 1):
            part = shard.reflection_slice(len(whole), rank, world)
            q = plan_of(sample, part)
            q.configure(variant, 1024, 1)
            assert np.array_equal(results(q, bisection), whole[part]), (world, rank)
            q.close()


@pytest.mark.parametrize("variant", [4, 12])
def test_tiles_orders_and_batches(sample, variant):
    p = plan_of(sample)
    p.configure(variant, 1024, 1)
    whole = results(p, False)
    for tile, order in ((128, 1), (512, 1), (2048, 1), (4000, 1), (1024, 0), (1024, 5)):
        p.configure(variant, tile, order)
        assert np.array_equal(results(p, False), whole), (tile, order)
    many = [plan_of(sample, slice(0, n)) for n in (1501, 40, 1501, 700, 1501, 1501)]
    for members in (many[:1], many):
        for q in members:
            q.configure(variant, 1024, 1)
        b = tracer.Batch(members)
        b.configure(variant)
        b.launch()
        b.wait()
        for got, q in zip(b.results(), members):
            assert np.array_equal(got, whole[:len(got)])
        b.close()
    for q in [p] + many:
        q.close()


def test_sum_is_the_rounded_sum(sample):
    """One voxel a call gives the terms; their exact sum over a set of voxels,
    rounded once and divided, is A_h of the set."""
    s = sample
    n, m = 97, 5
    terms = np.empty((n, m))
    for k in range(n):
        p = tracer.Plan(s.label, s.coords[k:k + 1], s.voxel, s.mu)
        p.set_reflections(s.s1[:m], s.omega[:m], s.xray, s.omega_axis, s.F)
        p.configure(4, 1024, 1)
        terms[k] = results(p, False)
        p.close()
    assert np.array_equal(terms, terms.astype(np.float32))
    p = tracer.Plan(s.label, s.coords[:n], s.voxel, s.mu)
    p.set_reflections(s.s1[:m], s.omega[:m], s.xray, s.omega_axis, s.F)
    p.configure(4, 1024, 1)
    got = results(p, False)
    p.close()
    assert np.array_equal(got, [math.fsum(terms[:, i]) / n for i in range(m)])
