"""Records and boxes made on the device (large device-built scenes of few prims): the same
scene as with the host's records, and the same answers to indices out of range.  A mesh
with more vertices than its triangles can name keeps the host's records, so unused vertices
appended to a scene give its other route."""
from __future__ import annotations

import numpy as np
import pytest

import gammaray_gb300 as g
from gammaray_gb300 import scenes
from test_gpu_parity import check_hits, random_rays

pytestmark = pytest.mark.gpu

SPHERES = [((-1.4, 0.2, 0.1), 0.3), ((1.3, -0.4, 0.2), 0.25)]


def build_prims(tris, extra):
    """A mesh of `tris` triangles with normals (one row geometric), a mesh with uvs, a light
    mesh and two spheres; `extra` appends vertices that no triangle names."""
    w = scenes.displaced_sphere(8, 8, tris=4000)
    m = w.prims[0]
    light = g.Material.diffuse_light((3.0, 2.0, 1.0))
    base = g.Material.disney().build()
    n = np.random.default_rng(6).normal(size=(len(m.vertices), 3)).astype(np.float32)
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    t = m.triangles[:tris]
    tn = t.copy()
    tn[tris // 2] = 0xFFFFFFFF
    v = np.concatenate([m.vertices, np.full((extra, 3), 9.0, np.float32)])
    quad = np.array([[-2, -2, -2], [2, -2, -2], [2, 2, -2], [-2, 2, -2]], np.float32)
    two = np.array([[0, 1, 2], [0, 2, 3]], np.uint32)
    uv = np.random.default_rng(7).random((4, 2)).astype(np.float32)
    prims = [g.Mesh(base, None, v, t, normals=n, tri_normals=tn),
             g.Mesh(base, None, quad, two, uvs=uv, tri_uvs=two),
             g.Mesh(light, None, quad + np.float32([0, 0, 5]), two[:, ::-1].copy())]
    prims += [g.Sphere(base, g.Mat.translation(c), r) for c, r in SPHERES]
    return w, prims


@pytest.mark.parametrize("components,bvh,leaf", [(2047, 4, 2), (2048, 4, 2), (2049, 2, 1), (3001, 8, 4)])
def test_device_records_equal_host_records(gpu, components, bvh, leaf):
    got = []
    for extra in (0, 20_000):
        w, prims = build_prims(components - 6, extra)
        st = g.Stage(prims, lib=gpu, environment=w.environment, seed=8, bvh_width=bvh, leaf_size=leaf,
                     device_build=True)
        info = st.info()
        assert info.num_components == components
        film = g.Film(40, 32, lib=gpu)
        st.render(w.camera, w.integrator, film, 3)
        rays = random_rays(20_000, 5, target=(0, 0, 0))
        got.append((st.intersect(rays), film.read(), info.num_wide_nodes, info.stack_depth, info.device_bytes))
    hits = got[0][0]
    assert (hits["prim"] >= 0).sum() > 5000
    np.testing.assert_array_equal(hits, got[1][0])
    for a, b in zip(got[0][1], got[1][1]):
        np.testing.assert_array_equal(a, b)
    assert got[0][2:] == got[1][2:]
    check_hits(hits[:4000], st.intersect_naive(rays[:4000]))


@pytest.mark.parametrize("what,text", [("vertex", "vertex index"), ("normal", "normal index"), ("uv", "uv index")])
def test_device_records_refuse_bad_indices(gpu, what, text):
    w, prims = build_prims(3000, 0)
    if what == "vertex":
        prims[0].triangles = prims[0].triangles.copy()
        prims[0].triangles[2999, 2] = len(prims[0].vertices)
    elif what == "normal":
        prims[0].tri_normals[7, 1] = len(prims[0].normals)
    else:
        prims[1].tri_uvs = np.array([[0, 1, 2], [0, 2, 4]], np.uint32)
    with pytest.raises(Exception, match=text + " out of range"):
        g.Stage(prims, lib=gpu, device_build=True)
