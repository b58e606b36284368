"""findKNearestNeighbors (binned) against the oracle, indices and distances
bit for bit, where its forms and lane groups turn over: list lengths about 8,
16, 32 and 64, radius 1 to 5 (more rows of cells than the row table holds),
flat and 3D grids, ties, crowded boxes, and queries on either side of the
thread-per-query dispatch."""
from __future__ import annotations

import numpy as np
import pytest

import gpusteer_gb300 as gs
import oracle_lib as ol
from gpusteer_gb300 import scenario as sc

pytestmark = pytest.mark.gpu


def check(s, ws, wc, r, k, other=None):
    bins = gs.KNNBinData(wc, ws, r)
    g = gs.AgentGroup(k, s.n)
    g.upload(s)
    gs.updateKNNDatabase(g, bins)
    o, os_ = g, s
    if other is not None:
        o, os_ = gs.AgentGroup(k, other.n), other
        o.upload(other)
        gs.updateKNNDatabase(o, bins)
    knn = gs.KNNData(s.n, k)
    gs.findKNearestNeighbors(g, knn, bins, o, r)
    idx, dist = knn.download(g)
    wi, wd = ol.knn_binned(s.position, os_.position, other is None, ws, wc, r, k)
    np.testing.assert_array_equal(idx, wi)
    np.testing.assert_array_equal(dist, wd)


@pytest.mark.parametrize("k", [1, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("r", [1, 2, 5])
def test_list_lengths_and_radii(k, r):
    check(sc.boids_sphere(1501, radius=11.0, seed=k), (64.0,) * 3, (16,) * 3, r, k)


@pytest.mark.parametrize("n", [1, 2, 9])
def test_fewer_candidates_than_entries(n):
    check(sc.boids_sphere(n, radius=2.0, seed=n), (64.0,) * 3, (16,) * 3, 1, 16)


@pytest.mark.parametrize("k", [7, 16])
@pytest.mark.parametrize("n", [98304, 98305])
def test_either_side_of_the_dispatch(n, k):
    check(sc.boids_cube(n, size=200.0, seed=k), (232.0,) * 3, (58,) * 3, 1, k)


@pytest.mark.parametrize("n", [98400, 300])
def test_flat_crowds_and_lattices(n):
    """Exact ties (the index decides) in boxes past every register scan."""
    side = int(np.ceil(n ** 0.5))
    x, z = np.meshgrid(np.arange(side), np.arange(side), indexing="ij")
    s = sc.chokepoint_agents(n, seed=1)
    s.position[:, 0] = (x.reshape(-1)[:n] - side // 2) * 0.5
    s.position[:, 2] = (z.reshape(-1)[:n] - side // 2) * 0.5
    s.position[::7, :3] = s.position[0, :3]
    ws, wc = (float(side), 10.0, float(side)), (max(1, side // 4), 1, max(1, side // 4))
    check(s, ws, wc, 1, 16)
    check(s, ws, wc, 1, 16, other=sc.chokepoint_agents(177, x_range=(-9, 9), z_range=(-9, 9), seed=2))
