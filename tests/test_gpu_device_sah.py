"""The SAH tree of large scenes built on the device: the host build's tree, so the same hits,
films, node counts and stack bound, with large and small nodes, nodes of coincident
centroids, degenerate extents and costs that no split improves.  A mesh with more vertices
than its triangles can name keeps the host's build, so unused vertices appended to a scene
give its other route."""
from __future__ import annotations

import numpy as np
import pytest

import gammaray_gb300 as g
from gammaray_gb300 import scenes
from test_gpu_parity import random_rays

pytestmark = pytest.mark.gpu

MIN = 4096  # components from which the device builds the tree


def soup(kind: str):
    rng = np.random.default_rng(9)
    if kind == "sphere":
        m = scenes.displaced_sphere(8, 8, tris=50_000).prims[0]
        return m.vertices, m.triangles
    if kind == "random":
        n = 40_000
        v = rng.uniform(-1, 1, (n, 1, 3)) + rng.normal(0, 0.02, (n, 3, 3))
    elif kind == "uneven":  # most of them in one corner, a few far away
        n = 30_000
        v = rng.exponential(0.02, (n, 1, 3)) ** 2 * 400 + rng.normal(0, 1e-4, (n, 3, 3))
    elif kind == "copies":  # 20,000 of one triangle among others, on a lattice
        n = 30_000
        c = np.round(rng.uniform(-4, 4, (n, 1, 3))) / 4
        c[5000:25_000] = (0.25, 0.0, -0.5)
        v = c + np.array([[0, 0, 0], [0.2, 0, 0.01], [0, 0.2, 0]])
    elif kind == "flat":  # one plane, one row
        n = 20_000
        c = np.stack([rng.uniform(-1, 1, n), np.zeros(n), np.zeros(n)], 1)[:, None]
        v = c + np.array([[0, 0, 0], [1e-3, 0, 0], [0, 1e-3, 0]])
    elif kind == "large":  # triangles all through each other: no split is worth its cost
        n = 17_000
        v = rng.uniform(-1, 1, (n, 3, 3))
    elif kind == "nan":  # left to the host
        n = 9000
        v = rng.uniform(-1, 1, (n, 1, 3)) + rng.normal(0, 0.02, (n, 3, 3))
        v[4321, 1, 2] = np.nan
    else:  # the smallest and the one below it
        n = MIN + int(kind)
        v = rng.uniform(-1, 1, (n, 1, 3)) + rng.normal(0, 0.05, (n, 3, 3))
    return v.reshape(-1, 3).astype(np.float32), np.arange(3 * len(v), dtype=np.uint32).reshape(-1, 3)


CASES = [("sphere", 4, 2), ("sphere", 2, 1), ("sphere", 8, 4), ("random", 4, 2), ("uneven", 4, 2), ("copies", 4, 2),
         ("copies", 8, 3), ("flat", 4, 2), ("large", 4, 2), ("nan", 4, 2), ("-1", 4, 2), ("0", 4, 2), ("1", 4, 1)]


@pytest.mark.parametrize("kind,bvh,leaf", CASES)
def test_device_sah_equals_host_sah(gpu, kind, bvh, leaf):
    v, t = soup(kind)
    w = scenes.displaced_sphere(48, 36, tris=200)
    mat = w.prims[0].material
    got = []
    for extra in (0, 3 * len(t)):
        verts = np.concatenate([v, np.full((extra, 3), 5.0, np.float32)])
        st = g.Stage([g.Mesh(mat, None, verts, t)], lib=gpu, environment=w.environment, seed=2, bvh_width=bvh,
                     leaf_size=leaf)
        i = st.info()
        film = g.Film(48, 36, lib=gpu)
        st.render(w.camera, w.integrator, film, 2)
        got.append((st.intersect(random_rays(20_000, 3, target=(0, 0, 0))), *film.read(),
                    (i.num_components, i.num_binary_nodes, i.num_wide_nodes, i.stack_depth, i.device_bytes)))
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
