"""The wavefront form's pool, grids and traversal schedule do not show in the
image: frames around the pool's size rule (one slot group, one rounding step,
all samples at once, half of them), compared bit for bit with a pool of 2^12
slots and the host-driven loop, and more launch shapes in turn than the
context keeps graphs for.  The glass scene starts every path in the glass
(its waiting branches outnumber the slots), the spheres leave steps without
triangles, the mesh gives some rays of a warp many."""
import numpy as np
import pytest

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


def _scene(name, w, h, n):
    if name == "spheres":
        s = scenes.cornell_spheres(w, h, n, 1, seed=w)
    else:
        s = scenes.mesh_cornell(w, h, n, 1, subdiv=4, material=name, seed=w)
    if name == "glass":  # inside the displaced ball: every camera ray splits
        s.camera.position = (50.0, 24.0, 70.0)
    s.settings.mode = A.PR_MODE_WAVEFRONT
    return s


SIZES = [(1, 1, 1), (64, 2, 1), (91, 90, 1), (91, 91, 1), (724, 724, 1), (725, 725, 1), (1024, 1023, 1), (1025, 1025, 1)]


@pytest.mark.parametrize("w,h,n", SIZES)
@pytest.mark.parametrize("scene", ["spheres", "diffuse", "glass"])
def test_image_is_that_of_a_small_pool(ctx, monkeypatch, scene, w, h, n):
    s = _scene(scene, w, h, n)
    ctx.upload(s)
    a = ctx.render(s)
    st = ctx.stats()
    monkeypatch.setenv("PR_WF_SLOTS", str(1 << (12 if w < 200 else 17)))
    monkeypatch.setenv("PR_WF_HOST_LOOP", "1")
    b = ctx.render(s)
    t = ctx.stats()
    assert np.array_equal(a, b)
    for k in ("paths", "segments", "nodes_visited", "tri_tests"):
        assert st[k] == t[k], k


def test_more_launch_shapes_than_graphs(ctx):
    s = _scene("diffuse", 50, 40, 1)
    ctx.upload(s)
    first = None
    for rep in range(2):
        for n in (1, 5, 9, 13, 17, 21, 25, 29, 33, 37):
            s.settings.samples = n
            img = ctx.render(s)
            if n == 1 and rep == 0:
                first = img
            if n == 1:
                assert np.array_equal(img, first)
