"""The plain form's block kernel (block_paths.cuh: paths of a block in lock
step, fixed-point pixel sums) against the one-path-per-thread kernel that
pr_render_dev_noalloc keeps: the same samples, so images agree up to float
summation order.  Sizes at the edges: one pixel, fewer samples than lanes,
warps and blocks, ragged sides, the switch between its two block sizes
(two samples per resident slot)."""
import ctypes as C

import numpy as np
import pytest

from prender_gb300 import gpu, scenes
from prender_gb300.scene import Material

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__ as g
    g.build_library()
    c = gpu.Context(0)
    yield c
    c.close()


def _both(ctx, s, offset=0, accumulate=None):
    import torch
    ctx.upload(s)
    out = []
    for fn in (ctx.L.pr_render_dev, ctx.L.pr_render_dev_noalloc):
        cam, prm = s.camera.to_c(), s.settings.to_c()
        t = torch.full((s.camera.height, s.camera.width, 3), 0.25 if accumulate else 0.0, device="cuda:0")
        rc = fn(ctx.h, C.byref(cam), C.byref(prm), C.c_void_p(t.data_ptr()), offset, 1 if accumulate else 0)
        assert rc == 0, ctx.L.pr_last_error(ctx.h)
        st = ctx.stats()
        out.append((t.cpu().numpy(), st["paths"], st["segments"]))
    return out


def _agree(a, b, spp):
    # one rounding per added sample on either side, and the fixed point's 2^-41 per sample
    assert a[1] == b[1] and a[2] == b[2]
    np.testing.assert_allclose(a[0], b[0], rtol=4.0 * spp * 2.0 ** -24, atol=spp * 2.0 ** -40)


SIZES = [(1, 1, 1, 1), (1, 1, 3, 1), (7, 5, 1, 1), (33, 3, 2, 1), (64, 48, 1, 2), (129, 65, 4, 2), (341, 342, 1, 2),
         (342, 342, 1, 2), (500, 333, 3, 1)]


@pytest.mark.parametrize("w,h,n,ss", SIZES)
@pytest.mark.parametrize("scene", ["spheres", "diffuse", "glass", "media"])
def test_block_form_equals_the_per_thread_form(ctx, scene, w, h, n, ss):
    if scene == "spheres":
        s = scenes.cornell_spheres(w, h, n, ss, seed=w)
    elif scene == "media":
        s = scenes.media_cornell(w, h, n, ss, seed=w)
    else:
        s = scenes.mesh_cornell(w, h, n, ss, subdiv=4, material=scene, seed=w)
    _agree(*_both(ctx, s, offset=5 * n, accumulate=w == 33), n * ss * ss + 1)


@pytest.mark.parametrize("scene", ["phong", "ward", "lights", "textured"])
def test_block_form_equals_the_per_thread_form_full_shading(ctx, scene):
    if scene in ("phong", "ward"):
        s = scenes.mesh_cornell(97, 61, 2, 2, subdiv=4, material=scene)
    else:
        s = scenes.mesh_cornell(97, 61, 2, 2, subdiv=4)
        if scene == "lights":
            s.add_spot_light((20, 70, 120), 2.0, (30, 30, 30), (0.2, -1, -0.3), (30, 10), falloff=1.0,
                             attenuation=(1.0, 0.0, 0.0))
            s.add_infinity_light((0.1, -1.0, -0.2), (0.5, 0.5, 0.5))
        else:
            m = Material.diffuse((0.6, 0.6, 0.6))
            m.texture = np.random.default_rng(1).integers(0, 256, (16, 16, 3)).astype(np.uint8)
            s.add_uvplane((2, 1.0, 40), (0, 0, 16), (16, 0, 0), m)
    _agree(*_both(ctx, s), 9)


@pytest.mark.parametrize("w,h", [(1, 1), (9, 5), (33, 3), (129, 65)])
def test_adjoint_of_two_sample_ranges_adds_up(ctx, w, h):
    """Ragged tiles and few samples in the adjoint's passes: the gradients of
    samples 0..3 are those of 0..1 and 2..3 together.  Each gradient is a sum
    of at most w h 4 weighted terms in FP32 per warp and FP64 above."""
    import dataclasses
    s = scenes.diff_cornell(w, h, samples=4, supersamples=1, subdiv=3, seed=2)
    ctx.upload(s)
    dl = np.random.default_rng(w).uniform(0.5, 1.5, (h, w, 3)).astype(np.float32)  # one sign: no cancellation
    whole = ctx.render_adjoint(dl)
    half = dataclasses.replace(s.settings, samples=2, total_spp=4)
    parts = [ctx.render_adjoint(dl, settings=half, sample_offset=k) for k in (0, 2)]
    for key in ("color", "emission"):
        both = parts[0][key] + parts[1][key]
        np.testing.assert_allclose(both, whole[key], rtol=1e-5, atol=1e-6 * np.abs(whole[key]).max() + 1e-30)


@pytest.mark.parametrize("offset", [2 ** 60 + 1, 2 ** 63, 2 ** 64 - 2])
@pytest.mark.parametrize("scene", ["spheres", "diffuse"])
def test_block_form_equals_the_per_thread_form_far_along_the_streams(ctx, scene, offset):
    """sample ids (offset x 33 x 17 + ...) wrap past 2^64: the streams go by
    them, the pixels do not"""
    if scene == "spheres":
        s = scenes.cornell_spheres(33, 17, 1, 1)
    else:
        s = scenes.mesh_cornell(33, 17, 1, 1, subdiv=3)
    _agree(*_both(ctx, s, offset=offset), 1)
