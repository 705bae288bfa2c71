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
