"""The SAH tree built on the device against the host's (a mesh with more vertices than its
triangles can name keeps the host's build) for scenes of several prims, in either order,
with lights, spheres, shading normals and uvs, and on both sides of the scene size from
which a block builds larger subtrees."""
from __future__ import annotations

import numpy as np
import pytest

import gammaray_gb300 as g
from gammaray_gb300 import scenes
from test_gpu_parity import random_rays

pytestmark = pytest.mark.gpu

MANY = 150_000  # components from which a block's subtrees have up to 1024 components
NO_INDEX = 0xFFFFFFFF


def equal(gpu, make, components, **kw):
    """The scene make(extra vertices) on both routes."""
    w = scenes.displaced_sphere(48, 36, tris=200)
    got = []
    for extra in (0, 3 * components + 1):
        st = g.Stage(make(extra), lib=gpu, environment=w.environment, seed=2, **kw)
        i = st.info()
        assert i.num_components == components
        film = g.Film(48, 36, lib=gpu)
        st.render(w.camera, w.integrator, film, 3)
        rng = np.random.default_rng(1)
        lights = [st.sample_light(rng.random((64, 6)).astype(np.float32))] if i.num_lights else []
        got.append([st.intersect(random_rays(30_000, 3, target=(0, 0, 0))), *film.read(),
                    (i.num_binary_nodes, i.num_wide_nodes, i.stack_depth, i.device_bytes), *lights])
    assert (got[0][0]["prim"] >= 0).sum() > 1000
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("bvh,leaf", [(4, 2), (2, 1), (8, 4)])
@pytest.mark.parametrize("order", [1, -1])
def test_several_prims(gpu, bvh, leaf, order):
    m = scenes.displaced_sphere(8, 8, tris=5000).prims[0]
    rng = np.random.default_rng(6)
    n = rng.normal(size=m.vertices.shape).astype(np.float32)
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    tn = m.triangles.copy()
    tn[::7] = NO_INDEX  # geometric normals
    quad = np.array([[-1, 0, -1], [1, 0, -1], [1, 0, 1], [-1, 0, 1]], np.float32)
    two = np.array([[0, 1, 2], [0, 2, 3]], np.uint32)
    uv = rng.random((4, 2)).astype(np.float32)
    light, base = g.Material.diffuse_light((3.0, 2.0, 1.0)), g.Material.disney().build()

    def make(extra):
        v = np.concatenate([m.vertices, np.full((extra, 3), 9.0, np.float32)])
        prims = [g.Mesh(light, None, quad + np.float32([0, 30, 0]), two[:, ::-1].copy()),
                 g.Sphere(base, g.Mat.translation((-1.4, 0.2, 0.1)), 0.3),
                 g.Mesh(base, None, quad * 3 + np.float32([0, -1.5, 0]), two, uvs=uv, tri_uvs=two),
                 g.Mesh(base, None, v, m.triangles, normals=n, tri_normals=tn),
                 g.Sphere(light, g.Mat.translation((1.3, 0.9, 0.2)), 0.25)]
        return prims[::order]

    equal(gpu, make, len(m.triangles) + 6, bvh_width=bvh, leaf_size=leaf)


@pytest.mark.parametrize("kind", ["random", "uneven", "copies", "large"])
@pytest.mark.parametrize("components", [MANY - 1, MANY, MANY + 7001])
def test_both_sizes_of_subtrees(gpu, kind, components):
    rng = np.random.default_rng(components)
    c = rng.uniform(-1, 1, (components, 1, 3))
    corner = rng.normal(0, 0.01, (components, 3, 3))
    if kind == "uneven":  # most of them in one corner
        c = rng.exponential(0.02, c.shape) ** 2 * 400
    elif kind == "copies":  # many centroids coincide
        c = np.round(c * 8) / 8
        corner = np.array([[0, 0, 0], [0.02, 0, 0.001], [0, 0.02, 0]])
    elif kind == "large":  # no split of a few is worth its cost
        c, corner = 0 * c, rng.uniform(-1, 1, corner.shape)
    v = (c + corner).reshape(-1, 3).astype(np.float32)
    t = np.arange(3 * components, dtype=np.uint32).reshape(-1, 3)
    mat = g.Material.disney().build()

    def make(extra):
        return [g.Mesh(mat, None, np.concatenate([v, np.full((extra, 3), 5.0, np.float32)]), t)]

    equal(gpu, make, components)
