"""The fused step of small groups (a group of lanes per agent) against the
oracle, bit for bit, at the sizes where its lane groups, chunks and dispatch
turn over.  Capacity 0 (automatic) is what takes it; a fixed capacity keeps
the thread-per-agent kernels."""
from __future__ import annotations

import numpy as np
import pytest

import gpusteer_gb300 as gs
import oracle_lib as ol
from gpusteer_gb300 import scenario as sc

pytestmark = pytest.mark.gpu
FIELDS = ("position", "direction", "side", "up", "speed", "applied")


def check(s, p, steps, gap=None, capacity=0):
    bins = gs.KNNBinData(p.world_cells, p.world_size, p.search_radius)
    walls = gs.WallGroup(sc.chokepoint_walls(gap), bins=bins, knw=p.knw) if gap else None
    g = gs.AgentGroup(p.k, s.n)
    g.upload(s)
    gs.set_knn_capacity(g, capacity)
    gs.step(g, bins, walls, p, steps)
    got, want = g.download(), s.copy()
    ol.run(want, p, steps, walls=walls.download() if walls else None)
    moving = want.speed != 0  # a speed of 0 keeps the side vector (reference: uninitialised)
    for f in FIELDS:
        a, b = getattr(got, f), getattr(want, f)
        if f == "side":
            a, b = a[moving], b[moving]
        np.testing.assert_array_equal(a, b, err_msg=f"n={s.n} k={p.k} {f}")


@pytest.mark.parametrize("k", [1, 7, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("n", [1, 2, 3, 15, 130, 2049])
def test_flock_lane_groups(n, k):
    s = sc.boids_sphere(n, radius=2.0 + 0.9 * n ** (1 / 3), seed=n + k)
    check(s, sc.boids_params(k=k, world=64.0), 3)


@pytest.mark.parametrize("n", [16384, 16385])
def test_flock_either_side_of_the_dispatch(n):
    check(sc.boids_sphere(n, radius=60.0, seed=3), sc.boids_params(k=16, world=160.0), 2)


@pytest.mark.parametrize("n,k", [(1, 16), (33, 7), (1001, 16), (5003, 24), (20000, 16), (20001, 16)])
@pytest.mark.parametrize("close", [0, 1])
def test_crowd_lane_groups(n, k, close):
    p = sc.chokepoint_params(k=k).replace(avoid_close=close)
    check(sc.chokepoint_agents(n, seed=n), p, 3, gap=10.0)


@pytest.mark.parametrize("k", [7, 16, 20])
@pytest.mark.parametrize("radius", [1, 2])
def test_lattice_ties_and_wider_boxes(k, radius):
    """Equal distances everywhere (the index decides), duplicates, and boxes
    of 27 and 125 cells with several chunks per lane group."""
    g3 = np.stack(np.meshgrid(*(np.arange(9),) * 3, indexing="ij"), -1).reshape(-1, 3)
    pts = np.concatenate([g3, g3[::4]]).astype(np.float32) - 4.0
    s = sc.boids_sphere(pts.shape[0], seed=k)
    s.position[:, :3] = pts
    check(s, sc.boids_params(k=k, world=64.0, cell=2.0).replace(search_radius=radius), 2)


def test_flat_world_without_walls_and_radius_two():
    p = sc.chokepoint_params().replace(order=(sc.B_AVOID_NEIGHBORS, sc.B_SEPARATION, sc.B_SEEK))
    s = sc.chokepoint_agents(3001, seed=9)
    for r in (1, 2):
        check(s, p.replace(search_radius=r), 2)
    check(s, sc.chokepoint_params().replace(search_radius=2), 2, gap=10.0)
