"""BDPT connections laid out as items (all paths of one strategy next to each other): per
path against the oracle at the path lengths and light counts where the layout has edges."""
from __future__ import annotations

import numpy as np
import pytest

import gammaray_gb300 as g
from gammaray_gb300 import scenes

pytestmark = pytest.mark.gpu

CASES = [  # width, height, max_depth, mis, light tracing, lights
    (1, 1, 16, 0, 0, True),    # one path
    (37, 11, 1, 0, 0, True),   # a single strategy
    (37, 11, 2, 1, 1, True),
    (29, 23, 16, 1, 1, True),  # the longest walks
    (29, 23, 16, 0, 1, True),  # light tracing with uniform weights
    (24, 24, 16, 0, 0, False), # no lights: no light walks
]


@pytest.mark.parametrize("width,height,depth,mis,lt,lights", CASES)
def test_bdpt_items_per_path(gpu, oracle, width, height, depth, mis, lt, lights):
    w = scenes.cornell_spheres(width, height)
    prims = w.prims if lights else [p for p in w.prims if not p.material.has_light()]
    env = (0.3, 0.2, 0.1)
    integ = g.BdptIntegrator(max_depth=depth, mis=mis, light_tracing=lt)
    a = g.Stage(prims, lib=gpu, environment=env, seed=11).samples(w.camera, integ, width, height, 2)
    b = g.Stage(prims, lib=oracle, environment=env, seed=11).samples(w.camera, integ, width, height, 2)
    np.testing.assert_array_equal(a[..., :2], b[..., :2])
    close = np.isclose(a[..., 2:], b[..., 2:], rtol=1e-4, atol=1e-5).all(axis=-1)
    assert close.mean() >= 0.99, f"{close.mean():.4f} of paths agree"
