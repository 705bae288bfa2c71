"""Geodesic batches and frames on resident warps (geodesic_math.cuh): a ray's
result does not depend on the batch it comes in, at sizes around a warp, a
block and the resident lanes (19,456 or 38,912 on 152 SMs), and a Kerr or
wormhole frame at ragged sizes is the sum of its sample ranges."""
import dataclasses

import numpy as np
import pytest

import wormhole_cases
from prender_gb300 import _abi as A
from prender_gb300 import gpu, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__ as g
    g.build_library()
    c = gpu.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("kind", ["kerr64", "kerr32", "kerr_disk", "worm"])
def test_a_ray_does_not_depend_on_its_batch(ctx, kind):
    n = 40000
    if kind == "worm":
        s = wormhole_cases.build("worm_objects", 250, 160, 1, 1, max_steps=12)
        trace = ctx.wormhole_trace
    else:
        build = scenes.kerr_accretion if kind == "kerr_disk" else scenes.kerr_lensing
        s = build(a=0.9, width=250, height=160, max_steps=40)
        s.kerr["precision"] = A.PR_KERR_FP32 if kind == "kerr32" else A.PR_KERR_FP64
        trace = ctx.kerr_trace
    ctx.upload(s)
    rays = scenes.camera_rays(s)
    assert len(rays) == n
    whole = trace(rays)
    for m in (1, 31, 32, 33, 127, 129, 19455, 19457, 38913):
        part = trace(rays[:m])
        for key in whole:  # NaN-safe: bit for bit
            assert np.array_equal(part[key].view(np.uint8), whole[key][:m].view(np.uint8)), (key, m)


@pytest.mark.parametrize("w,h", [(1, 1), (5, 3), (33, 31), (160, 130)])
@pytest.mark.parametrize("kind", ["kerr64", "kerr32", "worm"])
def test_frames_are_the_sum_of_their_sample_ranges(ctx, kind, w, h):
    if kind == "worm":
        s = wormhole_cases.build("worm_objects", w, h, 2, 1, max_steps=30)
    else:
        s = scenes.kerr_accretion(a=0.9, width=w, height=h, max_steps=300, samples=2,
                                  precision=A.PR_KERR_FP32 if kind == "kerr32" else A.PR_KERR_FP64)
    ctx.upload(s)
    whole = ctx.render(s)
    assert np.isfinite(whole).all()
    assert ctx.stats()["paths"] == 2 * w * h
    half = dataclasses.replace(s.settings, samples=1, supersamples=1, total_spp=2, tent_filter=1)
    full = dataclasses.replace(s.settings, samples=2, supersamples=1, tent_filter=1)
    whole = ctx.render(s, settings=full)
    parts = ctx.render(s, settings=half) + ctx.render(s, settings=half, sample_offset=1)
    # two FP32 roundings of fixed-point sums
    np.testing.assert_allclose(parts, whole, rtol=4 * 2.0 ** -24, atol=2.0 ** -38)


@pytest.mark.parametrize("kind", ["kerr64", "kerr32", "worm"])
def test_frames_far_along_the_streams(ctx, kind):
    """Sample ids (offset x pixels + ...) wrap past 2^64: frames whose rays
    draw nothing are the same at any offset."""
    if kind == "worm":
        s = wormhole_cases.build("worm_bg", 37, 23, 1, 1, max_steps=60)
    else:
        s = scenes.kerr_lensing(a=0.9, width=37, height=23, max_steps=300)
        s.kerr["precision"] = A.PR_KERR_FP32 if kind == "kerr32" else A.PR_KERR_FP64
    s.settings = dataclasses.replace(s.settings, samples=1, supersamples=1, tent_filter=0)
    ctx.upload(s)
    near = ctx.render(s)
    assert near.std() > 0.0
    for offset in (2 ** 60 + 1, 2 ** 64 - 2):
        assert np.array_equal(ctx.render(s, sample_offset=offset), near)
