"""The renderer's sphere queries rule spheres out by FP32 error bounds before
the FP64 test of the rest (trace_fast.cuh).  pr_trace_fast against the FP64
test of every sphere in numpy: walls of radius 1e5 and their like (anchored
bounds), tiny and nested spheres, hemispheres, and origins on, just off,
inside and outside of the surfaces."""
import numpy as np
import pytest

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


def _scene(name):
    if name == "walls":
        return scenes.cornell_spheres(width=16, height=12)
    s, m = Scene(), Material.diffuse((0.5, 0.5, 0.5))
    rng = np.random.default_rng(3)
    if name == "nested":  # concentric shells and a needle's-eye gap between two large ones
        for r in (1e-3, 0.5, 0.500001, 7.0, 300.0, 4.0e4):
            s.add_sphere((1.0, 2.0, 3.0), r, m)
        s.add_sphere((1.0, 1.0e6 + 60.0, 3.0), 1.0e6, m)
    elif name == "hemispheres":
        for k in range(6):
            (s.add_hemisphere if k % 2 else s.add_sphere)(tuple(rng.uniform(-5, 5, 3)), float(rng.uniform(0.5, 4)), m)
        s.add_hemisphere((0.0, -2.0e4, 0.0), 2.0e4, m)
    else:  # "many": the entity limit, radii over six decades
        for _ in range(48):
            s.add_sphere(tuple(rng.uniform(-50, 50, 3)), float(10.0 ** rng.uniform(-3, 3)), m)
    return s


def _rays(s, n, seed):
    """a quarter anywhere, the rest from points on, 1e-5 and 1e-3 (relative and
    absolute) off the spheres' surfaces; FP32 values"""
    rng = np.random.default_rng(seed)
    c = np.array([e.p for e in s.entities])
    r = np.array([e.radius for e in s.entities])
    k = rng.integers(0, len(r), n)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    big = r[k] > 1e3  # of the large ones, the side that faces the others
    u[big] = c[~(r > 1e3)].mean(0) - c[k[big]] + rng.normal(scale=20.0, size=(big.sum(), 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    off = rng.choice([0.0, 1e-5, -1e-5, 1e-3, -1e-3], n)
    o = c[k] + u * (r[k] * (1.0 + np.where(big, 0.0, off)) + off)[:, None]
    anywhere = rng.random(n) < 0.25
    o[anywhere] = rng.uniform(-60, 110, (anywhere.sum(), 3))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d], 1).astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("name", ["walls", "nested", "hemispheres", "many"])
def test_sphere_queries_equal_the_fp64_test_of_every_sphere(ctx, name):
    s = _scene(name)
    ctx.upload(s)
    rays = _rays(s, 200000, seed=11)
    got = ctx.trace_fast(rays)
    o, d = rays[:, :3], rays[:, 3:]
    best = np.full(len(rays), np.inf)
    ent = np.full(len(rays), -1)
    unsure = np.zeros(len(rays), bool)
    for i, e in enumerate(s.entities):
        p = np.asarray(e.p) - o
        b = (p * d).sum(1)
        pp = (p * p).sum(1)
        D4 = b * b - pp + e.radius ** 2
        with np.errstate(invalid="ignore"):
            q = np.sqrt(D4)
        t1, t2 = b - q, b + q
        hit = (D4 >= 0) & ~((t1 < 1e-6) & (t2 < 1e-6))
        t = np.where(t1 > 1e-6, t1, t2)
        if getattr(e, "hemisphere", 0):
            hit &= ~(o[:, 1] + t * d[:, 1] - e.p[1] < 0)
        # decisions within the FP64 rounding of either evaluation order
        err = 1e-15 * (b * b + pp + e.radius ** 2)
        with np.errstate(invalid="ignore", divide="ignore"):
            terr = np.where(D4 > err, err / np.maximum(q, 1e-300), np.sqrt(np.maximum(D4, 0) + err))
        unsure |= (np.abs(D4) <= err) | (np.abs(t1 - 1e-6) <= terr) | (np.abs(t2 - 1e-6) <= terr)
        closer = hit & (t < best)
        unsure |= hit & (ent >= 0) & (np.abs(t - best) <= 1e-6 * np.abs(t))  # FP32 order of near ties
        best = np.where(closer, t, best)
        ent = np.where(closer, i, ent)
    sure = ~unsure
    assert sure.mean() > 0.9
    assert np.array_equal(got["entity"][sure], ent[sure])
