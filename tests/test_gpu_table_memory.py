"""A small group's step where the device has no memory for its cell table: the
library linked once more with a cudaMalloc that refuses large blocks."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

from gpusteer_gb300 import build as b

REPO = Path(__file__).resolve().parents[1]

SHIM = """
#include <cuda_runtime.h>
extern "C" cudaError_t __real_cudaMalloc(void**, size_t);
static size_t most = ~size_t(0);
static unsigned refused = 0;
extern "C" void shim_most(size_t bytes) { most = bytes; refused = 0; }
extern "C" unsigned shim_refused() { return refused; }
extern "C" cudaError_t __wrap_cudaMalloc(void** p, size_t bytes) {
    if (bytes <= most) return __real_cudaMalloc(p, bytes);
    ++refused;
    return cudaErrorMemoryAllocation;
}
"""

CHILD = """
import ctypes as C, sys
from pathlib import Path
from gpusteer_gb300 import build
build.LIB = Path(sys.argv[1])
import numpy as np
import gpusteer_gb300 as gs, oracle_lib as ol
from gpusteer_gb300 import scenario as sc
lib = gs.load()
assert Path(lib._name) == build.LIB
lib.shim_most.argtypes = [C.c_size_t]

def step(g, want, p, steps, walls=None):
    bins = gs.KNNBinData(p.world_cells, p.world_size, 1)
    w = gs.WallGroup(walls, bins=bins, knw=p.knw) if walls is not None else None
    gs.step(g, bins, w, p, steps)
    ol.run(want, p, steps, walls=w.download() if w else None)
    got = g.download()
    for f in ("position", "direction", "up", "speed"):
        np.testing.assert_array_equal(getattr(got, f), getattr(want, f), err_msg=f)

p, q = sc.boids_params(k=7, world=160.0), sc.boids_params(k=7, world=160.0, cell=5.0)
s = sc.boids_sphere(3000, radius=30.0, seed=1)
g = gs.AgentGroup(p.k, s.n); g.upload(s)
want = s.copy()
lib.shim_most(8 << 20)
step(g, want, p, 2)             # no table: 64,000 cells
assert lib.shim_refused() == 1
step(g, want, p, 3)             # nor asked for again
assert lib.shim_refused() == 1
lib.shim_most(1 << 30)
step(g, want, q, 3)             # another grid: a table
lib.shim_most(8 << 20)
step(g, want, p, 1)             # its table is given up, none to be had
assert lib.shim_refused() == 1
g.upload(s); want = s.copy()
step(g, want, p, 2)
pc = sc.chokepoint_params(k=16)
sw = sc.chokepoint_agents(1500, seed=1)
gc = gs.AgentGroup(pc.k, sw.n); gc.upload(sw)
step(gc, sw.copy(), pc, 3, sc.chokepoint_walls(10.0))
print("steps without a table")
"""


def link(tmp_path):
    src, lib = tmp_path / "shim.cu", tmp_path / "libgpusteer_shim.so"
    src.write_text(SHIM)
    objs = [str(b.BUILD / (Path(s).stem + ".o")) for s in b.SOURCES]
    b.build()
    r = subprocess.run([b.nvcc(), *b.ARCH, "-shared", "--cudart", "static", "-Xcompiler", "-fPIC",
                        "-Xlinker", "--wrap=cudaMalloc", "-o", str(lib), str(src), *objs],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return lib


@pytest.mark.gpu
def test_steps_where_no_table_can_be_allocated(tmp_path):
    r = subprocess.run([sys.executable, "-c", CHILD, str(link(tmp_path))], capture_output=True,
                       text=True, timeout=600, cwd=REPO,
                       env={**__import__("os").environ, "PYTHONPATH": f"{REPO}:{REPO / 'tests'}"})
    assert r.returncode == 0, r.stderr[-3000:]
    assert "steps without a table" in r.stdout
