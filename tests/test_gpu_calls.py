"""The per-function behaviour calls against the oracle's whole step, bit for
bit, where their forms turn over (a group of lanes per agent, or one thread
taking the list in chunks): list lengths about the chunk and lane-group sizes,
and group sizes on either side of the dispatches."""
from __future__ import annotations

import numpy as np
import pytest

import gpusteer_gb300 as gs
import oracle_lib as ol
from gpusteer_gb300 import scenario as sc

pytestmark = pytest.mark.gpu
FIELDS = ("position", "direction", "side", "up", "speed")


def same(g, s, p, steps, walls=None):
    got, want = g.download(), s.copy()
    ol.run(want, p, steps, walls=walls)
    moving = want.speed != 0
    for f in FIELDS:
        a, b = getattr(got, f), getattr(want, f)
        if f == "side":
            a, b = a[moving], b[moving]
        np.testing.assert_array_equal(a, b, err_msg=f"n={s.n} k={p.k} {f}")


def crowd_frames(s, p, frames):
    bins = gs.KNNBinData(p.world_cells, p.world_size, 1)
    walls = gs.WallGroup(sc.chokepoint_walls(10.0), bins=bins, knw=p.knw)
    g = gs.AgentGroup(p.k, s.n)
    g.upload(s)
    gs.updateKNNDatabase(walls, bins)
    knn, knw = gs.KNNData(s.n, p.k), gs.KNNData(s.n, p.knw)
    for _ in range(frames):
        gs.wrapWorld(g, p.world_size, p.wrap_mode)
        gs.updateKNNDatabase(g, bins)
        gs.findKNearestNeighbors(g, knn, bins, g, 1)
        gs.findKNearestNeighbors(g, knw, bins, walls, 1)
        gs.steerToAvoidWalls(g, knw, walls, p.min_time_to_wall, p.w_walls, p.mask_walls)
        gs.steerToAvoidNeighbors(g, knn, g, p.min_time_to_collision, p.min_separation_distance,
                                 p.avoid_close, p.w_avoid, p.mask_avoid)
        gs.steerForSeparation(g, knn, g, p.sep_min, p.sep_max, p.sep_cos, p.w_sep, p.mask_sep)
        gs.steerForSeek(g, p.seek_target, p.w_seek, p.mask_seek)
        gs.updateGroup(g, p.dt)
    same(g, s, p, frames, walls=walls.download())


@pytest.mark.parametrize("close", [0, 1])
@pytest.mark.parametrize("n,k,knw", [(1, 7, 1), (37, 1, 3), (501, 8, 3), (2000, 9, 8), (3001, 17, 3),
                                     (1500, 32, 3), (20001, 16, 3)])
def test_crowd_calls(n, k, knw, close):
    p = sc.chokepoint_params(k=k, knw=knw).replace(avoid_close=close)
    s = sc.chokepoint_agents(n, seed=n + k)
    crowd_frames(s, p, 2)


@pytest.mark.parametrize("n", [65536, 65537])
def test_crowd_calls_either_side_of_the_avoidance_dispatch(n):
    p = sc.chokepoint_params(k=16).replace(avoid_close=1)
    crowd_frames(sc.chokepoint_agents(n, x_range=(-120, 120), z_range=(-120, 120), seed=4), p, 1)


@pytest.mark.parametrize("n,k", [(2, 1), (900, 7), (2049, 8), (3000, 9), (20000, 16), (20001, 7),
                                 (20001, 16), (21000, 20)])
def test_boids_calls(n, k):
    p = sc.boids_params(k=k, world=128.0)
    s = sc.boids_sphere(n, radius=2.5 * n ** (1 / 3) + 1, seed=n)
    bins = gs.KNNBinData(p.world_cells, p.world_size, 1)
    g = gs.AgentGroup(k, n)
    g.upload(s)
    knn = gs.KNNData(n, k)
    for _ in range(2):
        gs.wrapWorld(g, p.world_size, p.wrap_mode)
        gs.updateKNNDatabase(g, bins)
        gs.findKNearestNeighbors(g, knn, bins, g, 1)
        gs.steerForSeparation(g, knn, g, p.sep_min, p.sep_max, p.sep_cos, p.w_sep, p.mask_sep)
        gs.steerForCohesion(g, knn, g, p.coh_min, p.coh_max, p.coh_cos, p.w_coh, p.mask_coh)
        gs.steerForAlignment(g, knn, g, p.ali_min, p.ali_max, p.ali_cos, p.w_ali, p.mask_ali)
        gs.updateGroup(g, p.dt)
    same(g, s, p, 2)
