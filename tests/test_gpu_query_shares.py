"""Ray queries dealt out to the warps in shares: the same hits and answers however many rays
come in one call, at the sizes where shares and chunks have their edges."""
from __future__ import annotations

import numpy as np
import pytest

import gammaray_gb300 as g
from gammaray_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bvh", [2, 4, 8])
def test_shares_answer_every_query(gpu, bvh):
    w = scenes.displaced_sphere(8, 8, tris=3000)
    st = g.Stage(w.prims, lib=gpu, bvh_width=bvh)
    rng = np.random.default_rng(3)
    most = 400_003  # several chunks of 32 a warp, the last one partial
    o = rng.standard_normal((most, 3))
    o *= 2.5 / np.linalg.norm(o, axis=1, keepdims=True)
    d = rng.standard_normal((most, 3)) - o
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    pairs = np.concatenate([o, rng.standard_normal((most, 3)) * 1.2], 1).astype(np.float32)
    pairs[5::97, 3:] = pairs[5::97, :3]  # coincident points: answered without a ray
    hits, vis = st.intersect(rays), st.visibility(pairs)
    naive = st.intersect_naive(rays[:2000])
    same = (hits["prim"][:2000] == naive["prim"]) & (hits["component"][:2000] == naive["component"])
    assert (same | (hits["t"][:2000] == naive["t"])).all() and not vis[5::97].any()
    for n in (1, 2, 31, 33, 257, 5471, 20_000, 175_105):
        np.testing.assert_array_equal(st.intersect(rays[:n]), hits[:n])
        np.testing.assert_array_equal(st.visibility(pairs[:n]), vis[:n])


def test_sphere_hits_have_no_barycentrics(gpu):
    """u and v of a sphere hit are 0, whatever triangle the same warp met before."""
    w = scenes.displaced_sphere(8, 8, tris=3000)
    ball = g.Sphere(w.prims[0].material, g.Mat.translation((1.3, 0.2, 0.1)), 0.5)
    st = g.Stage([w.prims[0], ball], lib=gpu)
    rng = np.random.default_rng(4)
    o = rng.standard_normal((20_000, 3)) * 2.0
    d = rng.standard_normal((20_000, 3)) - o
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    for hits in (st.intersect(rays), st.intersect_naive(rays)):
        sphere = hits["prim"] == 1
        assert sphere.sum() > 500 and (hits["prim"] == 0).sum() > 500
        assert not hits["u"][sphere].any() and not hits["v"][sphere].any()
