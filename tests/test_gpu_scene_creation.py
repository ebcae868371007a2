"""Making a scene waits for its own device work only, whichever route makes its tree: a
program that renders on other streams meanwhile is not held up, nor is the creation."""
from __future__ import annotations

import numpy as np
import pytest

import gammaray_gb300 as g
from gammaray_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tris,device_build", [(3000, False), (5000, False), (160_000, False), (5000, True)])
def test_creation_does_not_wait_for_the_device(gpu, tris, device_build):
    import torch

    w = scenes.displaced_sphere(16, 16, tris=tris)

    def create():
        return g.Stage(w.prims, lib=gpu, environment=w.environment, device_build=device_build)

    first = create()  # (its kernels are loaded now)
    torch.cuda.synchronize()
    side, ended = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(side):
        torch.cuda._sleep(1_000_000_000)  # one waiting thread for half a second or so
        ended.record()
    second = create()
    assert not ended.query(), "the creation waited for another stream's work"
    films = []
    for st in (first, second):
        film = g.Film(16, 16, lib=gpu)
        st.render(w.camera, w.integrator, film, 2)
        films.append(film.read())
    for a, b in zip(*films):
        np.testing.assert_array_equal(a, b)
