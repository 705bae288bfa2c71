"""Metropolis chains on the block kernel (mlt.cu over block_paths.cuh): which
slot runs a chain, and when, is up to the scheduler, so two renders of one
seed differ only by the order of the float splats, and every bootstrap path
and proposal is counted once.  Sizes at the edges: one chain, chains around
the switch between the two block shapes and around a block's slots, more
chains than slots, and iterations around a launch's 64."""
import numpy as np
import pytest

from prender_gb300 import _abi as A
from prender_gb300 import gpu, scenes
from prender_gb300.scene import Material, RenderSettings, Scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__ as g
    g.build_library()
    c = gpu.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("chains,mutations", [(1, 1), (1, 129), (2, 64), (31, 65), (913, 3), (19455, 2), (19456, 2),
                                              (65536, 1), (233473, 1)])
def test_chains_do_not_depend_on_their_slots(ctx, chains, mutations):
    w, h = 32, 24
    s = scenes.cornell_spheres(w, h, 1, 1, seed=chains)
    st = s.settings
    st.mode, st.nee, st.pre_sample = A.PR_MODE_MLT, 1, 3.0
    st.mutation, st.mlt_chains = (chains * mutations + 0.5) / (w * h), chains
    ctx.upload(s)
    a = ctx.render(s)
    n = ctx.stats()
    assert n["paths"] == 3 * w * h + chains * mutations
    assert n["kernel_launches"] == 3 + -(-mutations // 64)
    b = ctx.render(s)
    assert np.isfinite(a).all() and a.mean() > 0.0
    # sums of at most k non-negative floats in any order
    k = 2 * chains * mutations
    np.testing.assert_allclose(a, b, rtol=2.0 * k * 2.0 ** -24, atol=0.0)


@pytest.mark.parametrize("chains,mutations", [(1, 129), (913, 3), (19455, 2), (19456, 2), (65536, 1), (4096, 65),
                                              (233473, 1)])
def test_every_splat_counts_once(ctx, chains, mutations):
    """Every path sees a background of radiance 1, so every proposal is taken
    and splats once, with one weight or (a large step) twice that: a pixel is
    a whole number of them, the same in every run, and their sum is that of
    all proposals.  A pixel's n float splats are off by at most n^2 2^-24 of
    one (n up to some 1500 here: 0.14); a lost or doubled one is off by 1."""
    w, h = 32, 24
    s = Scene()
    s.camera = scenes.cornell_spheres(w, h, 1, 1).camera
    s.background = (1.0, 1.0, 1.0)
    p, d = np.array(s.camera.position), np.array(s.camera.dir)
    s.add_sphere(tuple(p - 50.0 * d), 0.5, Material.diffuse((0.5, 0.5, 0.5)))  # behind the camera
    st = s.settings = RenderSettings(samples=1, supersamples=1, mode=A.PR_MODE_MLT, seed=chains, pre_sample=3.0,
                                     mutation=(chains * mutations + 0.5) / (w * h), mlt_chains=chains)
    assert st.nee == 0
    ctx.upload(s)
    n = chains * mutations
    counts = []
    for _ in range(2):
        img = ctx.render(s).astype(np.float64)
        k = img * 1.5 * n / (w * h)  # a splat: (1 + large) / (1 / b + 1/2), b = 1
        assert np.abs(k - np.rint(k)).max() < 0.25
        counts += [np.rint(k[..., c]) for c in range(3)]  # each channel has its own order of additions
    assert all(np.array_equal(k, counts[0]) for k in counts)
    large = counts[0].sum() - n  # of n proposals, each with probability 1/2
    assert abs(large - n / 2) <= 6.0 * np.sqrt(n / 4) + 1
