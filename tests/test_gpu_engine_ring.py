"""The batch engine's ring of path slots, full: a unit starts only when every slot of it is
free.  Images of nearly half the ring, more passes of them than the ring holds, among
images of odd sizes, equal plain renders bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import gammaray_gb300 as g
from gammaray_gb300 import batch, scenes

pytestmark = pytest.mark.gpu

CAPACITY = 1 << 16  # a ring of 2^23 slots: the power of two from 2 x CAPACITY + 2^22 on
SIZES = [(61, 47, 5), (2039, 2011, 3), (333, 217, 4), (2011, 2039, 2)]


@pytest.mark.parametrize("depth", [1, 3])
def test_units_wait_for_their_slots(gpu, depth):
    jobs, want = [], []
    for k, (width, height, spp) in enumerate(SIZES):
        w = scenes.cornell_spheres(width, height)
        integ = g.PathTracerIntegrator(max_depth=depth)
        st = g.Stage(w.prims, lib=gpu, environment=w.environment, seed=k)
        film = g.Film(width, height, lib=gpu)
        st.render(w.camera, integ, film, spp)
        want.append(film.read())
        jobs.append(batch.Job(st, w.camera, integ, g.Film(width, height, lib=gpu), spp))
    assert sum(a * b * n for a, b, n in SIZES) > 2 << 23 and 2039 * 2011 > 31 << 17  # of at most 32 << 17
    batch.render_batch(jobs, gpu, CAPACITY)
    for j, ref in zip(jobs, want):
        for a, b in zip(j.film.read(), ref):
            np.testing.assert_array_equal(a, b)
