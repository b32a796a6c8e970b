"""What an engine asks of its device, and sets on it, concerns the current one, not
the first that the process met: the launch shapes of the built step kernels under
a stand-in for the runtime with two devices."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

# two devices of 10 and 20 multiprocessors; the shared memory limit of one kernel
FAKE = r"""
static int current, limit[2];
void set_current(int d) { current = d; }
int limit_of(int d) { return limit[d]; }
int cudaGetDevice(int* d) { *d = current; return 0; }
int cudaDeviceGetAttribute(int* v, int attribute, int d) { *v = attribute == 16 ? 10 * (d + 1) : 0; return 0; }
int cudaFuncSetAttribute(const void* f, int attribute, int v) { limit[current] = attribute == 8 ? v : 0; return 0; }
"""

ASK = r"""
#include <stdio.h>
#include <string.h>
#include "gdem_step.cuh"
extern "C" void set_current(int);
extern "C" int limit_of(int);
int main() {
    for (int d : {0, 1, 0}) {
        set_current(d);
        printf("%d ", gdem::sm_count());
    }
    gdem::View<gdem::Mixed> v;
    memset((void*)&v, 0, sizeof(v));
    v.n = 1000;
    v.wall_cap = 32;
    v.kernel_variant = 2;  // staged
    for (int d : {0, 1}) {
        set_current(d);
        const gdem::StepLaunch L = gdem::step_launch(v, 0);
        printf("%d ", limit_of(d) >= (int)L.smem && L.smem > 48 * 1024);
    }
    return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
def test_launch_shapes_are_those_of_the_current_device(tmp_path):
    from gpudem_gb300 import _build
    _build.build_engine()
    (tmp_path / "fake.c").write_text(FAKE)
    (tmp_path / "ask.cu").write_text(ASK)
    subprocess.run(["gcc", "-c", "-fPIC", "fake.c", "-o", "fake.o"], cwd=tmp_path, check=True)
    subprocess.run([NVCC, *_build.ARCH, "-std=c++17", "-cudart", "shared", "-I" + _build.CSRC,
                    "-I" + os.path.join(ROOT, "include"), "ask.cu", "fake.o",
                    os.path.join(_build.OUT, "gdem_step_mixed.o"), "-o", "ask"], cwd=tmp_path, check=True)
    out = subprocess.run([str(tmp_path / "ask")], check=True, capture_output=True, text=True).stdout.split()
    assert out[:3] == ["10", "20", "10"]   # multiprocessors
    assert out[3:] == ["1", "1"]           # the staged kernel's limit, set on each device
