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


def test_scratch_is_bounded_and_given_back(gpu):
    import torch

    from gammaray_gb300 import batch

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    w = scenes.displaced_sphere(16, 16, tris=400_000)  # about 140 MB of scratch
    for _ in range(2):  # (the first turn loads kernels and sets the allocator up)
        batch.release(gpu)
        before = free()
        for _ in range(3):
            g.Stage(w.prims, lib=gpu).close()
        kept = before - free()
        assert 64 << 20 < kept <= (512 + 64) << 20, kept
        batch.release(gpu)
    assert before - free() < 16 << 20


def test_scenes_made_by_several_threads(gpu):
    from concurrent.futures import ThreadPoolExecutor

    from test_gpu_parity import random_rays

    rays = random_rays(5000, 3, target=(0, 0, 0))
    work = [(scenes.displaced_sphere(16, 16, tris=t, seed=t), dev)
            for t in (3000, 5000, 20_000, 60_000) for dev in (False, True)]

    def hits(job):
        w, dev = job
        st = g.Stage(w.prims, lib=gpu, environment=w.environment, device_build=dev)
        return st.intersect(rays)

    want = [hits(j) for j in work]
    with ThreadPoolExecutor(4) as pool:
        for got in [list(pool.map(hits, work)) for _ in range(3)]:
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
