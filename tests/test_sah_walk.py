"""The walk of the device SAH build's partition (csrc/sah_walk.cuh), compiled for the host
from the same source: every non-match ends where the reference's swap partition
(geom/util.rs) leaves it, in a number of loads that does not grow with the scene."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from gammaray_gb300 import build

PROGRAM = r"""
#include "sah_walk.cuh"
#include <cmath>
#include <cstdio>
#include <random>
#include <utility>
#include <vector>

template <class I>
struct Counted {
    const I* p;
    mutable unsigned long long loads;
    I operator[](unsigned long long i) const { ++loads; return p[i]; }
};

static unsigned long long bad = 0, walks = 0, most = 0;

template <class I>
static void check(const std::vector<char>& match) {
    const uint32_t n = static_cast<uint32_t>(match.size());
    std::vector<uint32_t> order(n), place(n);
    for (uint32_t i = 0; i < n; ++i) order[i] = i;
    uint32_t k = 0;
    for (uint32_t i = 0; i < n; ++i)
        if (match[order[i]]) std::swap(order[i], order[k++]);
    for (uint32_t i = 0; i < n; ++i) place[order[i]] = i;
    uint32_t p1 = 0;
    while (p1 < n && match[p1]) ++p1;
    std::vector<I> moved;
    uint32_t runs = 0;  // runs of matches after p1
    for (uint32_t i = p1; i < n; ++i)
        if (match[i]) {
            moved.push_back(static_cast<I>(i));
            runs += match[i - 1] ? 0 : 1;
        }
    const uint32_t R = k - p1;
    // At most sqrt(2 R) + 1 runs are met, each for the doublings of its steps and as many
    // halvings.
    const double met = std::fmin(runs, std::sqrt(2.0 * R) + 1.0);
    const double limit = 2.0 * met * (std::log2(R + 1.0) + 2.0) + 2.0;
    for (uint32_t i = p1; i < n; ++i) {
        if (match[i]) continue;
        Counted<I> T{moved.data(), 0};
        const uint32_t to = k + gr::sah_back(T, i - p1, R, p1) - R;
        ++walks;
        if (to != place[i] || T.loads > limit) ++bad;
        if (T.loads > most) most = T.loads;
    }
}

int main() {
    std::mt19937 rng(5);
    for (uint32_t n : {1u, 2u, 3u, 5u, 33u, 255u, 1000u, 102422u, 400000u}) {
        for (uint32_t first : {1u, 2u, 3u, 7u, 22u}) {  // non-matches first, all others match
            std::vector<char> m(n, 1);
            for (uint32_t i = 0; i < first && i < n; ++i) m[i] = 0;
            check<uint32_t>(m);
            if (n <= 1024) check<uint16_t>(m);
            if (n > 100) {  // and after some matches
                for (uint32_t i = 0; i < first; ++i) std::swap(m[i], m[i + n / 3]);
                check<uint32_t>(m);
            }
        }
        for (double p : {0.0001, 0.001, 0.01, 0.3, 0.5, 0.9, 0.999}) {
            std::vector<char> m(n);
            std::bernoulli_distribution out(p);
            for (auto& x : m) x = out(rng) ? 0 : 1;
            check<uint32_t>(m);
            if (n <= 1024) check<uint16_t>(m);
        }
        for (uint32_t run : {1u, 2u, 10u, 1000u}) {  // single non-matches between runs
            std::vector<char> m(n, 1), grow(n, 1);
            for (uint32_t i = 0; i < n; i += run + 1) m[i] = 0;
            for (uint32_t i = 0, g = 1; i < n; i += run * g++ + 1) grow[i] = 0;  // runs of run, 2 run, ...
            check<uint32_t>(m);
            check<uint32_t>(grow);
        }
    }
    std::printf("%llu %llu %llu\n", walks, most, bad);
    return bad ? 1 : 0;
}
"""


def test_walks_end_where_the_swap_partition_does(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    here = os.path.dirname(os.path.abspath(build.__file__))
    src = tmp_path / "walk.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "walk"
    cmd = [gxx, "-O2", "-std=c++17", "-I" + os.path.join(build._cuda_home(), "include"),
           "-I" + os.path.join(here, "csrc"), "-I" + os.path.join(here, "..", "include"), str(src), "-o", str(exe)]
    subprocess.run(cmd, check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    walks, most, bad = (int(x) for x in out.stdout.split())
    assert walks > 1_000_000 and bad == 0 and out.returncode == 0, (walks, most, bad)
