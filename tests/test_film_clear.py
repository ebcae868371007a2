"""Clearing a film (csrc/film_clear.hpp) with another device current than the film's, compiled
for the host against a stand-in for the CUDA runtime that refuses, as CUDA does, to record
an event of one device on a stream of another."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from gammaray_gb300 import build

PROGRAM = r"""
#include "film_clear.hpp"
#include <cstdio>
#include <cstring>

static int current = 0, recorded = 0, sets = 0;
struct CUevent_st { int device; };

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current = d; ++sets; return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    if (e->device != current) return cudaErrorInvalidResourceHandle;
    ++recorded;
    return cudaSuccess;
}
}

int main() {
    CUevent_st event{1};
    int bad = 0;
    for (int now = 0; now < 3; ++now)
        for (int with_splat = 0; with_splat < 2; ++with_splat) {
            unsigned char pixels[16], splat[16];
            std::memset(pixels, 7, sizeof(pixels));
            std::memset(splat, 7, sizeof(splat));
            current = now;
            recorded = sets = 0;
            const cudaError_t e = gr::clear_film(1, pixels, with_splat ? splat : nullptr, 16, &event);
            bad += e != cudaSuccess || recorded != 1 || current != now || sets != (now == 1 ? 0 : 2);
            for (int k = 0; k < 16; ++k) bad += pixels[k] != 0 || splat[k] != (with_splat ? 0 : 7);
        }
    std::printf("%d\n", bad);
    return bad ? 1 : 0;
}
"""


def test_a_film_is_cleared_whatever_device_is_current(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    here = os.path.dirname(os.path.abspath(build.__file__))
    src = tmp_path / "clear.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "clear"
    subprocess.run([gxx, "-O1", "-std=c++17", "-I" + os.path.join(build._cuda_home(), "include"),
                    "-I" + os.path.join(here, "csrc"), str(src), "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
