"""The step graphs are built by the first call that steps, whatever its length,
so that no later call pays for them: instantiations counted in a child process
by a library loaded before the CUDA runtime."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

COUNTER = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
static int built;
int graphs_built(void) { return built; }
int cudaGraphInstantiate(void** exec, void* graph, unsigned long long flags) {
    static int (*real)(void**, void*, unsigned long long);
    if (!real) *(void**)&real = dlsym(dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD), "cudaGraphInstantiate");
    built++;
    return real(exec, graph, flags);
}
"""

CHILD = r"""
import ctypes, sys
from dataclasses import replace
sys.path.insert(0, sys.argv[1])
from gpudem_gb300 import engine, scenes
count = ctypes.CDLL(sys.argv[2]).graphs_built
sc = scenes.config2_tilted_box(n=500, r0=2e-3)
for precision in ("fp64", "mixed"):
    for tree in (False, True):
        E = engine.Engine(sc, precision=precision, model="hertz_mindlin", bvh_every_step=tree)
        E.step(0)
        at = count()
        E.step(1)
        first = count()
        for c in (20, 1, 2, 3, 9):
            E.step(c)
        E.import_particles(sc)                 # the same grid
        E.step(17)
        E.sync()
        same = count()
        E.import_particles(replace(sc, r=sc.r * 0.9))
        E.step(40)
        other = count()
        E.step(1)
        E.sync()
        print(precision, tree, first - at, same - first, other - same, count() - other)
        E.close()
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs a C compiler")
def test_the_first_call_builds_every_graph(tmp_path):
    src, lib = tmp_path / "counter.c", tmp_path / "counter.so"
    src.write_text(COUNTER)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(lib), str(src), "-ldl"], check=True)
    out = subprocess.run([sys.executable, "-c", CHILD, ROOT, str(lib)], check=True, capture_output=True, text=True,
                         env=dict(os.environ, LD_PRELOAD=str(lib)), timeout=300).stdout
    rows = [ln.split() for ln in out.splitlines() if ln.startswith(("fp64", "mixed"))]
    assert len(rows) == 4, out
    for r in rows:
        # built by the first step; nothing by any later call; both again for
        # another grid, and nothing after that
        assert [int(x) for x in r[2:]] == [2, 0, 2, 0], out
