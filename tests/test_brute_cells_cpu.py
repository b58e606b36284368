"""Brute force over cells, on the host: a cell's number as the kernels compile it
grows with the coordinate whatever the automatic grid is, so the box from the
cell of q - D to that of q + D holds every candidate within the k-th distance
D."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from gpusteer_gb300 import build as b

PROBE = """
#include "gs_db.cuh"
using namespace gs;
extern "C" void cells(const float* x, unsigned n, float mid, float ws, unsigned wc, unsigned* out) {
    const AutoGrid a{Grid{{ws, ws, ws}, {wc, wc, wc}}, {mid, mid, mid}};
    for (unsigned i = 0; i < n; ++i) {
        unsigned y, z;
        auto_coords(a, v3(x[i], 0.f, 0.f), out[i], y, z);
    }
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    d = tmp_path_factory.mktemp("cells")
    (d / "probe.cu").write_text(PROBE)
    r = subprocess.run([b.nvcc(), *b.ARCH, *b.NVCC_FLAGS, "-shared", "--cudart", "static", "-I",
                        str(b.CSRC), "-o", str(d / "probe.so"), str(d / "probe.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(str(d / "probe.so"))
    lib.cells.argtypes = [C.POINTER(C.c_float), C.c_uint, C.c_float, C.c_float, C.c_uint,
                          C.POINTER(C.c_uint)]
    return lib


def cell(lib, x, grid):
    x = np.ascontiguousarray(x, np.float32)
    out = np.empty(x.shape, np.uint32)
    lib.cells(x.ctypes.data_as(C.POINTER(C.c_float)), x.size, *grid,
              out.ctypes.data_as(C.POINTER(C.c_uint)))
    return out


def positions(name, rng, n=700):
    u = rng.uniform(-256, 256, n)
    return {"uniform": u, "offset": u * 0.01 + 1e6, "outliers": np.where(rng.random(n) < 0.02, u * 1e30, u),
            "clusters": rng.integers(-4, 4, n) * 1e4 + rng.normal(0, 1, n), "point": np.full(n, -2.5),
            "heavy": rng.standard_cauchy(n), "denormal": u * 1e-41,
            "widest": u / 256 * 3.4e38}[name].astype(np.float32)


NAMES = ["uniform", "offset", "outliers", "clusters", "point", "heavy", "denormal", "widest"]
# centre, width and cells of an axis
GRIDS = [(0.0, 512.0, 32), (3.25, 1e-30, 7), (1e6, 5.12, 50), (-17.0, 8.5e37, 1024), (0.3, 900.1, 1),
         (256.0, 33.3, 101)]


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("name", NAMES)
def test_cells_grow_with_the_coordinate(probe, name, grid):
    rng = np.random.default_rng(grid[2])
    big = np.finfo(np.float32).max
    edge = np.float32(grid[0]) + np.float32(grid[1]) * (np.arange(grid[2] + 1, dtype=np.float32) / grid[2] - 0.5)
    x = positions(name, rng)
    at = np.concatenate([x, edge, np.nextafter(edge, np.float32(np.inf)),
                         np.nextafter(edge, np.float32(-np.inf)), rng.normal(0, 1e3, 3000),
                         rng.normal(0, 1, 1000) * 1e30, [0.0, -0.0, big, -big, np.inf, -np.inf]])
    s = cell(probe, np.sort(at.astype(np.float32)), grid)
    assert s.max() < grid[2]
    assert (np.diff(s.astype(np.int64)) >= 0).all()


def ru(x):
    """The next float32 at or above the float64 x."""
    y = np.asarray(x, np.float64).astype(np.float32)
    return np.where(y.astype(np.float64) < x, np.nextafter(y, np.float32(np.inf)), y).astype(np.float32)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("k", [1, 16])
def test_the_box_of_the_kth_distance_holds_the_list(probe, name, grid, k):
    """Every candidate at a float32 distance of at most the k-th from a query
    lies, on each axis, between the cells of q - D and q + D as the kernel
    widens and rounds them."""
    n = 700
    pos = np.stack([positions(name, np.random.default_rng(a), n) for a in range(3)], 1)
    with np.errstate(over="ignore", invalid="ignore"):
        d = pos[:, None, :] - pos[None, :, :]
        dist = np.sqrt((d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2])
        np.fill_diagonal(dist, np.inf)
        D = np.sort(dist, axis=1)[:, k - 1]
        within = (dist <= D[:, None]) & np.isfinite(D)[:, None]
        assert within.any() or name == "widest"
        reach = ru(ru(D.astype(np.float64) * np.float64(np.float32(1.00001))).astype(np.float64)
                   + np.float64(np.float32(1e-18))).astype(np.float64)
        for a in range(3):
            q = pos[:, a].astype(np.float64)
            s = cell(probe, pos[:, a], grid)
            low, high = cell(probe, -ru(-(q - reach)), grid), cell(probe, ru(q + reach), grid)
            inside = (s[None, :] >= low[:, None]) & (s[None, :] <= high[:, None])
            assert (inside | ~within).all(), (name, a)
