"""Exact first hits where the FP32 bounds of the triangle test and the
pending list (device_common.cuh) could go wrong, bit for bit against the
oracle: more coincident and near-coincident triangles than the list holds
(ties keep the first in order of visit), rays through vertices and edges,
in a triangle's plane, from a triangle's own surface, scenes far from the
origin and at small and large scale, directions of any length."""
import numpy as np
import pytest

from oracle import oracle as O
from prender_gb300 import gpu, scenes
from prender_gb300.scene import Material, Scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__ as g
    g.build_library()
    c = gpu.Context(0)
    yield c
    c.close()


def _stacks(shift, scale):
    """20 copies of one quad, a stack of quads one float apart and an
    icosphere, with rays aimed at their vertices, edges and insides"""
    quad = np.array([[0, 0, 0], [4, 0, 0], [4, 4, 0], [0, 4, 0]], np.float64)
    v, f = [], []
    for k in range(40):
        q = quad.copy()
        if k >= 20:
            q[:, 2] = 1.0 + (k - 20) * 2.0 ** -23
        f += [[4 * k, 4 * k + 1, 4 * k + 2], [4 * k, 4 * k + 2, 4 * k + 3]]
        v.append(q)
    v = np.concatenate(v)
    s = Scene()
    s.add_mesh((v * scale + shift).astype(np.float32), np.array(f, np.int32), Material.diffuse((0.5, 0.5, 0.5)))
    iv, jf = scenes.displaced_icosphere(3, (2, 2, -6), 3.0, amp=0.05, seed=3)
    s.add_mesh((np.asarray(iv, np.float64) * scale + shift).astype(np.float32), jf, Material.diffuse((0.4, 0.5, 0.6)))
    s.add_uvplane(tuple(np.array([-1, -1, -2.0]) * scale + shift), (6 * scale, 0, 0), (0, 6 * scale, 0),
                  Material.diffuse((0, 0, 0), (4, 4, 4)))
    m0, m1 = np.asarray(s.meshes[0].vertices, np.float64), np.asarray(s.meshes[1].vertices, np.float64)
    f0, f1 = np.asarray(s.meshes[0].faces), np.asarray(s.meshes[1].faces)
    rng = np.random.default_rng(5)
    targets = [m0, m1]
    for m, f in ((m0, f0), (m1, f1)):
        t = m[f]
        targets += [0.5 * (t[:, 0] + t[:, 1]), t.mean(1), (t * rng.dirichlet((1, 1, 1), len(t))[..., None]).sum(1)]
    p = np.concatenate(targets)
    org = (rng.normal(size=p.shape) * 8.0 + (2, 2, 0)) * scale + shift
    aimed = np.concatenate([org, p - org], 1)                                 # t = 1 there, any length
    unit = aimed.copy()
    unit[:, 3:] /= np.linalg.norm(unit[:, 3:], axis=1, keepdims=True)
    away = np.concatenate([p, unit[:, 3:]], 1)                                # from the surface itself
    down = np.concatenate([p + np.array([0, 0, 3.0 * scale]), np.tile([0, 0, -1.0], (len(p), 1))], 1)
    flat = np.concatenate([p - np.array([9.0 * scale, 0, 0]), np.tile([1.0, 0, 0], (len(p), 1))], 1)  # in the plane
    return s, np.ascontiguousarray(np.concatenate([aimed, unit, away, down, flat, aimed * ([1] * 3 + [1e-3] * 3),
                                                   aimed * ([1] * 3 + [1e4] * 3)]))


@pytest.mark.parametrize("shift,scale", [(0.0, 1.0), (1000.0, 1.0), (0.0, 1.0e-3), (-3.0e4, 50.0), (0.0, 1.0e5)])
def test_ties_edges_and_scales(ctx, shift, scale):
    s, rays = _stacks(shift, scale)
    ctx.upload(s)
    h, o = ctx.first_hit(rays), O.OracleScene(s).first_hit(rays)
    assert (o["entity"] >= 0).any() and (o["entity"] < 0).any()
    for k in ("entity", "prim", "t"):
        assert np.array_equal(h[k], o[k]), k
