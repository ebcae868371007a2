"""The order in which camera paths enter the queue (csrc/path_order.cuh), compiled for the
host from the same source: every sample of a group is one queue entry, once."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from gammaray_gb300 import build

PROGRAM = r"""
#include "path_order.cuh"
#include <cstdio>
#include <vector>

int main() {
    unsigned long long bad = 0, checks = 0;
    for (uint32_t w : {1u, 2u, 3u, 4u, 5u, 7u, 8u, 31u, 33u, 64u, 333u})
        for (uint32_t h : {1u, 2u, 7u, 8u, 9u, 15u, 32u, 50u, 217u})
            for (uint32_t passes : {1u, 2u, 3u, 9u, 64u}) {
                const gr::PathOrder o = gr::make_path_order(w, h, passes);
                std::vector<unsigned char> seen(static_cast<size_t>(w) * h * passes, 0);
                for (uint32_t q = 0; q < w * h * passes; ++q, ++checks) {
                    const gr::PathSample s = gr::path_sample(o, q);
                    if (s.row >= h || s.col >= w || s.pass >= passes ||
                        s.slot != s.pass * w * h + s.row * w + s.col || seen[s.slot]++)
                        ++bad;
                }
            }
    // The largest group: the first and the last entries.
    const gr::PathOrder o = gr::make_path_order(32768, 32768, 1);
    for (uint32_t k = 0; k < 1000000u; ++k, ++checks) {
        const gr::PathSample s = gr::path_sample(o, (1u << 30) - 1u - k);
        if (s.row >= 32768u || s.col >= 32768u || s.slot != s.row * 32768u + s.col) ++bad;
    }
    std::printf("%llu %llu\n", checks, bad);
    return bad ? 1 : 0;
}
"""


def test_every_sample_is_one_queue_entry(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    here = os.path.dirname(os.path.abspath(build.__file__))
    src = tmp_path / "order.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "order"
    cmd = [gxx, "-O2", "-std=c++17", "-I" + os.path.join(build._cuda_home(), "include"),
           "-I" + os.path.join(here, "csrc"), "-I" + os.path.join(here, "..", "include"), str(src), "-o", str(exe)]
    subprocess.run(cmd, check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    checks, bad = (int(x) for x in out.stdout.split())
    assert checks > 10_000_000 and bad == 0 and out.returncode == 0
