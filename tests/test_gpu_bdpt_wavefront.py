"""BDPT's launches per bounce and their hand-over to the path loop: renders large enough to
start with queues, against the same render in groups small enough for the path loop alone
(bit for bit) and, path by path, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import gammaray_gb300 as g
from gammaray_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bvh", [2, 4, 8])
@pytest.mark.parametrize("mis,scene", [(0, "cornell"), (1, "cornell"), (0, "mesh"), (1, "mesh")])
def test_queues_equal_the_path_loop(gpu, monkeypatch, mis, scene, bvh):
    size, spp = 256, 6
    w = scenes.cornell_spheres(size, size) if scene == "cornell" else scenes.displaced_sphere(size, size, tris=3000)
    integ = g.BdptIntegrator(max_depth=7, mis=mis)
    films, rays, launches = [], [], []
    # 786,432 walks at once (the path loop takes 262,144), then pass by pass
    for paths in (None, str(size * size)):
        if paths is None:
            monkeypatch.delenv("GR_BDPT_PATHS_IN_FLIGHT", raising=False)
        else:
            monkeypatch.setenv("GR_BDPT_PATHS_IN_FLIGHT", paths)
        st = g.Stage(w.prims, lib=gpu, environment=w.environment, seed=5, bvh_width=bvh)
        film = g.Film(size, size, lib=gpu)
        st.render(w.camera, integ, film, spp)
        films.append(film.read())
        s = st.last_stats()
        rays.append((s.extension_rays, s.shadow_rays))
        launches.append(s.kernel_launches)
    for a, b in zip(*films):
        np.testing.assert_array_equal(a, b)
    assert rays[0] == rays[1]
    assert launches[0] >= launches[1] // spp + 2  # a bounce's two launches at least


@pytest.mark.parametrize("mis,lt", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("width,height", [(400, 331), (640, 420)])  # 264,800 and 537,600 walks
def test_queues_per_path(gpu, oracle, width, height, mis, lt):
    w = scenes.cornell_spheres(width, height)
    integ = g.BdptIntegrator(max_depth=6, mis=mis, light_tracing=lt)
    a = g.Stage(w.prims, lib=gpu, environment=(0.3, 0.2, 0.1), seed=11).samples(w.camera, integ, width, height, 2)
    b = g.Stage(w.prims, lib=oracle, environment=(0.3, 0.2, 0.1), seed=11).samples(w.camera, integ, width, height, 2)
    np.testing.assert_array_equal(a[..., :2], b[..., :2])
    close = np.isclose(a[..., 2:], b[..., 2:], rtol=1e-4, atol=1e-5).all(axis=-1)
    assert close.mean() >= 0.99, f"{close.mean():.4f} of paths agree"
