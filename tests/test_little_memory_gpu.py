"""Frames on a device with little memory left (PR_DEVICE_MEMORY_MB bounds what
the library holds): the scratch falls back to smaller pools and passes, the
results stay, and the context keeps to the small sizes instead of freeing and
allocating its pool anew in every frame."""
import dataclasses

import numpy as np
import pytest

from prender_gb300 import _abi as A
from prender_gb300 import gpu, scenes

pytestmark = pytest.mark.gpu


def _context():
    import __graft_entry__ as g
    g.build_library()
    return gpu.Context(0)


def _scene(kind):
    if kind == "plain":
        return scenes.mesh_cornell(512, 384, 4, 2, subdiv=3)
    if kind == "kerr32":
        return scenes.kerr_accretion(a=0.9, width=1024, height=512, max_steps=60, precision=A.PR_KERR_FP32)
    if kind == "wavefront":
        s = scenes.mesh_cornell(1024, 500, 16, 1, subdiv=3, material="glass")
    elif kind == "subsurface":
        s = scenes.media_batch(n=2, seed=3, sizes=[1024], samples=8, supersamples=1, subdiv=3)[1]
        assert (s.camera.width, s.camera.height) == (1024, 1024)
    else:
        return scenes.diff_cornell(256, 256, samples=4, supersamples=2, subdiv=3, seed=1)
    s.settings.mode = A.PR_MODE_WAVEFRONT
    return s


# MiB: the usual scratch needs more, the small one less
LIMITS = {"plain": 120, "kerr32": 100, "wavefront": 1450, "subsurface": 4600, "adjoint": 150}


@pytest.mark.parametrize("kind", list(LIMITS))
def test_results_on_a_device_with_little_memory(monkeypatch, kind):
    import torch
    s = _scene(kind)
    dl = np.random.default_rng(2).uniform(0.5, 1.5, (s.camera.height, s.camera.width, 3)).astype(np.float32)

    def run(c):
        return c.render_adjoint(dl) if kind == "adjoint" else c.render(s)

    c = _context()
    c.upload(s)
    free = torch.cuda.mem_get_info()[0]
    whole = run(c)
    usual = free - torch.cuda.mem_get_info()[0]
    c.close()
    assert usual > LIMITS[kind] << 20  # the case needs the fallback
    c = _context()
    c.upload(s)
    monkeypatch.setenv("PR_DEVICE_MEMORY_MB", str(LIMITS[kind]))
    first = run(c)
    monkeypatch.delenv("PR_DEVICE_MEMORY_MB")
    free = torch.cuda.mem_get_info()[0]
    second = run(c)  # the small scratch, kept
    assert torch.cuda.mem_get_info()[0] == free
    c.upload(s)
    third = run(c)  # the usual sizes again
    assert free - torch.cuda.mem_get_info()[0] > 64 << 20
    for got in (first, second, third):
        if kind == "adjoint":  # FP64 sums over the warps in any order
            for k in ("color", "emission"):
                np.testing.assert_allclose(got[k], whole[k], rtol=1e-9, atol=1e-9 * np.abs(whole[k]).max())
        else:
            assert np.array_equal(got, whole)
    c.close()


def test_batch_on_a_device_with_little_memory(monkeypatch):
    import torch
    ss = [scenes.mesh_cornell(256, 192, 4, 2, subdiv=3, seed=k) for k in range(3)]
    imgs = []
    for limit in (None, 150):
        c = _context()
        objs = [c.scene_object(s) for s in ss]
        outs = [torch.empty((192, 256, 3), device="cuda:0") for _ in ss]
        if limit:
            monkeypatch.setenv("PR_DEVICE_MEMORY_MB", str(limit))
        c.render_batch(list(zip(objs, outs)))
        imgs.append([o.cpu().numpy() for o in outs])
        for o in objs:
            o.release()
        c.close()
    assert all(np.array_equal(a, b) for a, b in zip(*imgs))


def test_a_bound_too_small_for_the_small_sizes_is_an_error(monkeypatch):
    s = _scene("plain")
    c = _context()
    c.upload(s)
    monkeypatch.setenv("PR_DEVICE_MEMORY_MB", "8")
    with pytest.raises(gpu.PrenderError):
        c.render(s)
    monkeypatch.delenv("PR_DEVICE_MEMORY_MB")
    c.upload(s)
    assert np.isfinite(c.render(s)).all()
    c.close()
