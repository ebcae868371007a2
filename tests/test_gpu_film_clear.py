"""A film is cleared before anything is added to it, also when the default stream, on which
films are cleared, is busy and the render runs on a stream of its own."""
from __future__ import annotations

import numpy as np
import pytest

import gammaray_gb300 as g
from gammaray_gb300 import batch, scenes, serve

pytestmark = pytest.mark.gpu

SIZES = [(61, 47, 3), (128, 96, 2)]


def busy_default_stream():
    """Half a second or so of one waiting thread on the default stream."""
    import torch

    torch.cuda._sleep(1_000_000_000)
    assert not torch.cuda.current_stream().query()


def jobs_of(gpu):
    jobs = []
    for k, (width, height, spp) in enumerate(SIZES):
        w = scenes.cornell_spheres(width, height)
        st = g.Stage(w.prims, lib=gpu, environment=w.environment, seed=k)
        jobs.append((st, w.camera, g.PathTracerIntegrator(max_depth=5), width, height, spp))
    return jobs


def plain(gpu, jobs):
    out = []
    for st, camera, integ, width, height, spp in jobs:
        film = g.Film(width, height, lib=gpu)
        st.render(camera, integ, film, spp)
        out.append(film.read())
    return out


@pytest.mark.parametrize("how", ["render", "batch", "serve", "progressive"])
def test_a_clear_comes_first(gpu, how):
    jobs = jobs_of(gpu)
    want = plain(gpu, jobs)
    films = [g.Film(j[3], j[4], lib=gpu) for j in jobs]
    srv = serve.Server(gpu, path_capacity=1 << 16) if how in ("serve", "progressive") else None
    got = []
    for turn in range(2):  # the second turn finds everything set up and its films used
        if turn:
            busy_default_stream()
        if how == "render":
            for j, f in zip(jobs, films):
                f.clear()
                j[0]._pass = 0  # the passes of the plain render, again
                j[0].render(j[1], j[2], f, j[5])
            got = [f.read() for f in films]
        elif how == "batch":
            for f in films:
                f.clear()
            batch.render_batch([batch.Job(j[0], j[1], j[2], f, j[5]) for j, f in zip(jobs, films)], gpu, 1 << 16)
            got = [f.read() for f in films]
        else:
            # (a progressive request's two half-films, summed, end at its passes: the target is never met)
            ids = [srv.submit(*j, target_rel_mse=1e-30 if how == "progressive" else 0.0) for j in jobs]
            srv.run_until_done(ids)
            got = [srv.take(i) for i in ids]
    for a, b in zip(got, want):
        for x, y in zip(a, b):
            if how == "progressive":  # even and odd passes are summed apart: below 100 roundings of 2^-24
                np.testing.assert_allclose(x, y, rtol=0, atol=1e-5 * np.abs(y).max())
            else:
                np.testing.assert_array_equal(x, y)
