"""Sums of a pixel's samples (sum_samples) in the plain form, Kerr and wormhole
frames: any finite radiance, bright or dim, as the per-thread form's float
sums hold it; the group sizes of the sum (powers of two up to 32 threads a
pixel, a block from 1024 samples on); frames in several passes."""
import ctypes as C
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


def _both(ctx, s):
    import torch
    ctx.upload(s)
    out = []
    for fn in (ctx.L.pr_render_dev, ctx.L.pr_render_dev_noalloc):
        cam, prm = s.camera.to_c(), s.settings.to_c()
        t = torch.full((s.camera.height, s.camera.width, 3), float("nan"), device="cuda:0")
        assert fn(ctx.h, C.byref(cam), C.byref(prm), C.c_void_p(t.data_ptr()), 0, 0) == 0, ctx.L.pr_last_error(ctx.h)
        out.append(t.cpu().numpy())
    return out


def _close(a, b, spp):
    """one float rounding per added sample on the per-thread side, four for
    the conversions and the sensor response on either; denormal sums in full steps"""
    assert a.max() > 0.0
    np.testing.assert_allclose(a, b, rtol=(spp + 8) * 2.0 ** -24, atol=spp * 2.0 ** -149)


@pytest.mark.parametrize("scale", [1.0e-30, 1.0e-10, 1.0, 3.0e6, 1.0e7, 1.0e30])
@pytest.mark.parametrize("scene", ["spheres", "glass", "phong"])
def test_any_radiance_is_summed_as_floats_hold_it(ctx, scene, scale):
    s = scenes.cornell_spheres(33, 17, 4, 2) if scene == "spheres" else \
        scenes.mesh_cornell(33, 17, 4, 2, subdiv=3, material=scene)
    for m in s.materials:
        m.emission = tuple(scale * e for e in m.emission)
    s.settings.luminance_cutoff = 0.0
    _close(*_both(ctx, s), 16)


@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (7, 3, 1), (7, 3, 2), (7, 3, 3), (5, 3, 31), (5, 3, 32), (5, 3, 33),
                                     (3, 2, 1023), (3, 2, 1024), (3, 2, 1025), (1, 1, 5000), (300, 7, 15)])
def test_group_sizes(ctx, w, h, spp):
    s = scenes.mesh_cornell(w, h, spp, 1, subdiv=2, seed=spp)
    s.settings.luminance_cutoff = 0.0
    _close(*_both(ctx, s), spp)


@pytest.mark.parametrize("most", [1, 7, 100, 101, 5000])
def test_passes_of_a_frame_make_the_same_image(ctx, monkeypatch, most):
    s = scenes.mesh_cornell(67, 23, 7, 1, subdiv=2)
    ctx.upload(s)
    whole, st = ctx.render(s), ctx.stats()
    monkeypatch.setenv("PR_PASS_SAMPLES", str(most))
    parts, sp = ctx.render(s), ctx.stats()
    assert np.array_equal(whole, parts)
    assert st["kernel_launches"] == 2 and sp["kernel_launches"] == 2 * -(-67 * 23 // max(1, most // 7))
    for k in ("paths", "segments", "nodes_visited", "tri_tests"):
        assert st[k] == sp[k], k


def _curved(kind, scale):
    if kind == "worm":
        s = wormhole_cases.build("worm_objects", 37, 23, 1, 2, max_steps=60)
        s.wormhole["texture_coef"] = tuple(scale * c for c in (1.0, 1.5))
        for m in s.materials:
            m.emission = tuple(scale * e for e in m.emission)
    else:
        s = scenes.kerr_lensing(a=0.9, width=37, height=23, max_steps=300)
        s.kerr["precision"] = A.PR_KERR_FP32 if kind == "kerr32" else A.PR_KERR_FP64
        s.kerr["texture_coef"] = scale
        for m in s.materials:
            m.emission = tuple(scale * e for e in m.emission)
        s.settings = dataclasses.replace(s.settings, samples=1, supersamples=2, tent_filter=0)
    s.settings.luminance_cutoff = 0.0
    return s


@pytest.mark.parametrize("scale", [2.0 ** -60, 2.0 ** 30])
@pytest.mark.parametrize("kind", ["kerr64", "kerr32", "worm"])
def test_curved_frames_scale_with_their_light(ctx, monkeypatch, kind, scale):
    """powers of two times the same samples: the same sums, exactly; and in passes too"""
    img = []
    for f in (1.0, scale):
        s = _curved(kind, f)
        ctx.upload(s)
        img.append(ctx.render(s))
    assert img[0].std() > 0.0
    assert np.array_equal(img[0] * np.float32(scale), img[1])
    monkeypatch.setenv("PR_PASS_SAMPLES", "333")
    assert np.array_equal(ctx.render(s), img[1])
