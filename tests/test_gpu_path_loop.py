"""The path loop (few paths carried to their end in one launch) against the launches per
bounce: the same films bit for bit and the same rays, around the sizes where it can go
wrong.  A render that counts its traversal steps never takes the path loop."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import gammaray_gb300 as g
from gammaray_gb300 import _abi, batch, scenes

pytestmark = pytest.mark.gpu


def render(gpu, stage, camera, integ, width, height, spp, flags):
    p = stage.params(integ, spp, 0)
    p.flags = flags
    film = g.Film(width, height, lib=gpu)
    cam = camera.desc()
    gpu.call("gr_render", stage.handle, C.byref(cam), C.byref(p), film.handle)
    return film.read(), stage.last_stats()


CASES = [  # width, height, spp, max_depth, BVH width, scene
    (1, 1, 1, 0, 4, "cornell"),      # one lane of one warp
    (33, 3, 1, 5, 2, "cornell"),     # a partial warp, the narrowest tree
    (97, 61, 3, 0, 8, "mesh"),       # unbounded depth, the widest tree
    (512, 512, 1, 8, 4, "cornell"),  # the most paths a loop starts with
    (512, 513, 1, 8, 4, "cornell"),  # one row more: queues first, the loop at their end
    (400, 300, 5, 0, 4, "mesh"),
    (64, 64, 2, 1, 4, "mesh"),       # one bounce
    (64, 64, 2, 257, 4, "cornell"),  # deeper than the loop takes
]


@pytest.mark.parametrize("width,height,spp,depth,bvh,scene", CASES)
def test_path_loop_equals_launches_per_bounce(gpu, width, height, spp, depth, bvh, scene):
    w = scenes.cornell_spheres(width, height) if scene == "cornell" else scenes.displaced_sphere(width, height, tris=3000)
    st = g.Stage(w.prims, lib=gpu, environment=w.environment, bvh_width=bvh, seed=7)
    integ = g.PathTracerIntegrator(max_depth=depth)
    (acc, wt), s = render(gpu, st, w.camera, integ, width, height, spp, 0)
    (acc_q, wt_q), s_q = render(gpu, st, w.camera, integ, width, height, spp, _abi.RENDER_COUNT_TRAVERSAL)
    np.testing.assert_array_equal(acc, acc_q)
    np.testing.assert_array_equal(wt, wt_q)
    assert s.extension_rays == s_q.extension_rays and s.samples == s_q.samples
    if depth != 257:
        assert s.kernel_launches < s_q.kernel_launches or depth == 1


@pytest.mark.parametrize("capacity", [1024, 1 << 14, 1 << 20])
@pytest.mark.parametrize("depth", [3, 0, 257])  # 257: deeper than the loop takes
def test_batch_equals_plain_renders(gpu, capacity, depth):
    # A pool smaller than one image (its units start in pieces), a few images, and one that
    # holds everything (the loop takes the queue's end).
    jobs, refs = [], []
    for k, (width, height, spp) in enumerate([(61, 47, 3), (33, 8, 5), (128, 96, 2)]):
        w = scenes.cornell_spheres(width, height) if k else scenes.displaced_sphere(width, height, tris=3000)
        st = g.Stage(w.prims, lib=gpu, environment=w.environment, seed=k)
        integ = g.PathTracerIntegrator(max_depth=depth)
        jobs.append(batch.Job(st, w.camera, integ, g.Film(width, height, lib=gpu), spp))
        film = g.Film(width, height, lib=gpu)
        g.Stage(w.prims, lib=gpu, environment=w.environment, seed=k).render(w.camera, integ, film, spp)
        refs.append(film)
    batch.render_batch(jobs, gpu, capacity)
    for j, ref in zip(jobs, refs):
        for a, b in zip(j.film.read(), ref.read()):
            np.testing.assert_array_equal(a, b)
