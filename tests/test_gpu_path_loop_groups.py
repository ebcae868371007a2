"""The path loop's last rays, traced by groups of lanes: the same films as the launches per
bounce where stacks outgrow their shared part (groups give such rays back), leaves hold more
primitives than a group has lanes, and the scene is just large enough for groups.  A render
that counts its traversal steps never takes the path loop."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import gammaray_gb300 as g
from gammaray_gb300 import _abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bvh,leaf", [(2, 1), (4, 2), (4, 16), (8, 3), (8, 16)])
@pytest.mark.parametrize("tris", [1023, 1024, 6000])
def test_groups_equal_launches_per_bounce(gpu, tris, bvh, leaf):
    # Large triangles all through each other: deep stacks and many ties of boxes.
    rng = np.random.default_rng(tris)
    v = rng.uniform(-1, 1, (3 * tris, 3)).astype(np.float32)
    t = np.arange(3 * tris, dtype=np.uint32).reshape(-1, 3)
    mat = g.Material.disney().build()
    st = g.Stage([g.Mesh(mat, None, v, t)], lib=gpu, environment=(0.6, 0.7, 0.8), bvh_width=bvh, leaf_size=leaf, seed=3)
    cam = scenes.displaced_sphere(61, 47, tris=200).camera.desc()
    films, rays = [], []
    for flags in (0, _abi.RENDER_COUNT_TRAVERSAL):
        p = st.params(g.PathTracerIntegrator(max_depth=0), 2, 0)
        p.flags = flags
        film = g.Film(61, 47, lib=gpu)
        gpu.call("gr_render", st.handle, C.byref(cam), C.byref(p), film.handle)
        films.append(film.read())
        rays.append(st.last_stats().extension_rays)
    assert rays[0] == rays[1] > 2 * 61 * 47 * 1.2
    for a, b in zip(*films):
        np.testing.assert_array_equal(a, b)
