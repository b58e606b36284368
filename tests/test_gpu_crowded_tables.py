"""Small groups' cell tables where cells hold more than a row: results against
the oracle, bit for bit, about the edges of rows and at the most further rows a
table can need, and a step's cost, which follows an agent's own box."""
from __future__ import annotations

import numpy as np
import pytest

import gpusteer_gb300 as gs
import oracle_lib as ol
from gpusteer_gb300 import scenario as sc
from gpusteer_gb300.groups import cell_avg_velocity, cell_density

pytestmark = pytest.mark.gpu
FIELDS = ("position", "direction", "side", "up", "speed", "applied")


def same(got, want, what):
    moving = want.speed != 0
    for f in FIELDS:
        a, b = getattr(got, f), getattr(want, f)
        if f == "side":
            a, b = a[moving], b[moving]
        np.testing.assert_array_equal(a, b, err_msg=f"{what} {f}")


def clumps(n, per, span, size, seed):
    """n boids in balls of `per` scattered over a cube of side `span`."""
    s = sc.boids_cube(n, size=10.0, seed=seed)
    rng = np.random.default_rng(seed)
    at = np.repeat(rng.uniform(-span / 2, span / 2, ((n + per - 1) // per, 3)), per, 0)[:n]
    s.position[:, :3] = (at + rng.uniform(-size / 2, size / 2, (n, 3))).astype(np.float32)
    return s


def stepped(s, p, steps, walls=None):
    g = gs.AgentGroup(p.k, s.n)
    g.upload(s)
    bins = gs.KNNBinData(p.world_cells, p.world_size, 1)
    gs.step(g, bins, walls, p, steps)
    return g, bins


@pytest.mark.parametrize("n,per,size", [(300, 16, 1.0), (300, 17, 1.0), (400, 32, 1.0), (400, 33, 1.0),
                                        (500, 49, 1.0), (3000, 100, 2.5), (16384, 60, 3.0)])
@pytest.mark.parametrize("k", [7, 16, 32])
def test_clumps(n, per, size, k):
    p = sc.boids_params(k=k, world=128.0)
    s = clumps(n, per, 100.0, size, n + per)
    g, _ = stepped(s, p, 3)
    want = s.copy()
    ol.run(want, p, 3)
    same(g.download(), want, f"n={n} per={per} k={k}")


def test_every_agent_in_one_cell():
    """The most further rows: all of the largest group's agents in one cell of
    a grid of few, and of many."""
    for n, cell in ((16384, 64.0), (4001, 4.0)):
        p = sc.boids_params(k=7, world=128.0, cell=cell)
        s = sc.boids_cube(n, size=3.0, seed=n)
        s.position[:, :3] += np.float32(2.0)
        g, _ = stepped(s, p, 1)
        want = s.copy()
        ol.run(want, p, 1)
        same(g.download(), want, f"n={n}")


@pytest.mark.parametrize("n,width", [(65, 1.5), (2500, 6.0), (20000, 40.0)])
def test_crowded_flat_world(n, width):
    p = sc.chokepoint_params(k=16)
    s = sc.chokepoint_agents(n, x_range=(0.1, width), z_range=(14.0, 14.0 + width), seed=n)
    bins = gs.KNNBinData(p.world_cells, p.world_size, 1)
    walls = gs.WallGroup(sc.chokepoint_walls(10.0), bins=bins, knw=p.knw)
    g, _ = stepped(s, p, 2, walls)
    want = s.copy()
    ol.run(want, p, 2, walls=walls.download())
    same(g.download(), want, f"n={n} width={width}")


def test_diagnostics_of_crowded_cells():
    p = sc.boids_params(k=9, world=64.0)
    s = clumps(2500, 70, 50.0, 3.0, 8)
    g, bins = stepped(s, p, 1)
    frame, want = s.copy(), s.copy()
    ol.oracle().orc_wrap_world(ol.C.byref(ol.group_struct(frame)), ol.f3(p.world_size), p.wrap_mode)
    ol.run(want, p, 1)
    np.testing.assert_array_equal(cell_density(g, bins),
                                  ol.cell_density(frame.position, p.world_size, p.world_cells))
    np.testing.assert_array_equal(
        cell_avg_velocity(g, bins),
        ol.cell_avg_velocity(frame.position, want.direction, want.speed, p.world_size, p.world_cells))


def step_us(s, p, capacity):
    import torch

    g = gs.AgentGroup(p.k, s.n)
    bins = gs.KNNBinData(p.world_cells, p.world_size, 1)
    gs.set_knn_capacity(g, capacity)
    stream = torch.cuda.ExternalStream(g.stream)
    times = []
    for _ in range(7):
        g.upload(s)
        gs.step(g, bins, None, p, 1)
        g.upload(s)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        gs.step(g, bins, None, p, 8)
        b.record(stream)
        b.synchronize()
        times.append(a.elapsed_time(b) * 1e3)
    return sorted(times)[3]


def test_a_crowded_step_costs_its_own_box():
    """16,384 boids in clumps of 60, some 270 clumps apart: a step of the
    automatic form takes no longer than the sorting step at a fixed capacity,
    whose agents read their own box alone (half its time is expected; reading
    every clump's excess took five times as long)."""
    p = sc.boids_params(k=16, world=256.0, cell=4.0)
    s = clumps(16384, 60, 240.0, 3.0, 60)
    assert step_us(s, p, 0) < step_us(s, p, 256)


@pytest.mark.parametrize("odd", [1, 2])
def test_a_crowd_too_dense_for_the_table(odd):
    """Boxes of about 1,000 candidates: the step sorts instead, whether the
    group starts there, comes from a sparse grid's table or goes back to it,
    and steering left by per-function calls is taken along."""
    p_coarse = sc.boids_params(k=9, world=96.0, cell=16.0)
    p_fine = sc.boids_params(k=9, world=96.0, cell=3.0)
    s = sc.boids_cube(8192, size=96.0, seed=2)
    for order in ((p_coarse, p_fine), (p_fine, p_coarse)):
        want = s.copy()
        g = gs.AgentGroup(9, s.n)
        g.upload(s)
        gs.steerForSeek(g, (3.0, 4.0, 5.0), 0.5, 0)
        ol.oracle().orc_steer_seek(ol.C.byref(ol.group_struct(want)), ol.f3((3.0, 4.0, 5.0)),
                                   ol.C.c_float(0.5), 0)
        for p in order + order:
            gs.step(g, gs.KNNBinData(p.world_cells, p.world_size, 1), None, p, odd)
            ol.run(want, p, odd)
            same(g.download(), want, f"{p.world_cells} odd={odd}")
