"""Small groups' cell tables and the flock kernels' shared-angle branch against
the oracle, bit for bit: rows that overflow, steps taken after the table has
been given up and taken again, and what is read from a group between steps."""
from __future__ import annotations

import numpy as np
import pytest

import gpusteer_gb300 as gs
import oracle_lib as ol
from gpusteer_gb300 import scenario as sc
from gpusteer_gb300.state import AgentState

pytestmark = pytest.mark.gpu
FIELDS = ("position", "direction", "side", "up", "speed", "applied")


def same(got, want, what):
    moving = want.speed != 0  # a speed of 0 keeps the side vector (reference: uninitialised)
    for f in FIELDS:
        a, b = getattr(got, f), getattr(want, f)
        if f == "side":
            a, b = a[moving], b[moving]
        np.testing.assert_array_equal(a, b, err_msg=f"{what} {f}")


def group_of(s, p, capacity=0):
    g = gs.AgentGroup(p.k, s.n)
    g.upload(s)
    gs.set_knn_capacity(g, capacity)
    return g


@pytest.mark.parametrize("change", [{}, dict(ali_cos=0.2), dict(ali_max=6.0), dict(sep_cos=0.3),
                                    dict(sep_max=9.0, sep_min=0.0), dict(sep_min=8.0)])
@pytest.mark.parametrize("n,k", [(33, 1), (700, 8), (3001, 16), (2049, 32), (78001, 16)])
def test_flock_kernel_with_and_without_a_shared_angle(n, k, change):
    """A fixed capacity: the thread-per-agent kernels, either side of 77,824
    agents; one angle for all three behaviours, or not, and separation of
    none, some and all of the list."""
    p = sc.boids_params(k=k, world=256.0).replace(**change)
    s = sc.boids_sphere(n, radius=2.0 + 0.8 * n ** (1 / 3), seed=n + k)
    g = group_of(s, p, 32)
    gs.step(g, gs.KNNBinData(p.world_cells, p.world_size, p.search_radius), None, p, 2)
    want = s.copy()
    ol.run(want, p, 2)
    same(g.download(), want, f"n={n} k={k}")


@pytest.mark.parametrize("change", [{}, dict(coh_cos=0.1)])
@pytest.mark.parametrize("capacity", [64, 128, 256])
@pytest.mark.parametrize("n,k", [(65, 3), (2049, 7), (1501, 16), (3001, 32)])
def test_flock_kernel_at_larger_capacities(n, k, capacity, change):
    """Dense enough that some agents' boxes hold more than the capacity."""
    p = sc.boids_params(k=k, world=128.0).replace(**change)
    s = sc.boids_sphere(n, radius=1.0 + 0.5 * n ** (1 / 3), seed=n + capacity)
    g = group_of(s, p, capacity)
    gs.step(g, gs.KNNBinData(p.world_cells, p.world_size, p.search_radius), None, p, 2)
    want = s.copy()
    ol.run(want, p, 2)
    same(g.download(), want, f"n={n} k={k} capacity={capacity}")


def clump(n, inside, seed):
    """`inside` of n boids within one cell, so that its row overflows."""
    s = sc.boids_sphere(n, radius=12.0, seed=seed)
    rng = np.random.default_rng(seed)
    s.position[:inside, :3] = rng.uniform(1.0, 2.5, (inside, 3)).astype(np.float32)
    return s


@pytest.mark.parametrize("inside", [15, 16, 17, 33, 200, 1500])
@pytest.mark.parametrize("k", [7, 16])
@pytest.mark.parametrize("steps", [1, 2, 5])
def test_table_rows_that_overflow(inside, k, steps):
    p = sc.boids_params(k=k, world=64.0)
    s = clump(2000, inside, inside + k)
    g = group_of(s, p)
    bins = gs.KNNBinData(p.world_cells, p.world_size, p.search_radius)
    gs.step(g, bins, None, p, steps)
    want = s.copy()
    ol.run(want, p, steps)
    same(g.download(), want, f"inside={inside} k={k} steps={steps}")


@pytest.mark.parametrize("inside", [31, 33, 400])
def test_table_rows_of_a_flat_world_that_overflow(inside):
    p = sc.chokepoint_params(k=16)
    s = sc.chokepoint_agents(3000, seed=inside)
    rng = np.random.default_rng(inside)
    s.position[:inside, 0] = rng.uniform(0.1, 1.9, inside).astype(np.float32)
    s.position[:inside, 2] = rng.uniform(-3.9, -2.1, inside).astype(np.float32)
    bins = gs.KNNBinData(p.world_cells, p.world_size, p.search_radius)
    walls = gs.WallGroup(sc.chokepoint_walls(10.0), bins=bins, knw=p.knw)
    g = group_of(s, p)
    gs.step(g, bins, walls, p, 3)
    want = s.copy()
    ol.run(want, p, 3, walls=walls.download())
    same(g.download(), want, f"inside={inside}")


@pytest.mark.parametrize("first,then", [
    (dict(), dict(capacity=32)), (dict(capacity=64), dict(capacity=0)),
    (dict(), dict(world=96.0)), (dict(), dict(radius=2)), (dict(), dict(wrap=sc.WRAP_REFERENCE)),
    (dict(), dict(upload=True)), (dict(), dict(world=4096.0)), (dict(world=4096.0), dict(world=64.0)),
])
@pytest.mark.parametrize("odd", [1, 2])
def test_a_table_given_up_and_taken_again(first, then, odd):
    """Steps of one group under a table, then under something that has to
    leave it or file it anew, then under the first again."""
    s = sc.boids_sphere(1501, radius=10.0, seed=5)
    want = s.copy()
    g = group_of(s, sc.boids_params(k=9))
    for opt in (first, then, first):
        p = sc.boids_params(k=9, world=opt.get("world", 64.0))
        p = p.replace(search_radius=opt.get("radius", 1))
        if "wrap" in opt:
            p = p.replace(wrap_mode=opt["wrap"])
        if opt.get("upload"):
            s = sc.boids_sphere(1501, radius=14.0, seed=6)
            g.upload(s)
            want = s.copy()
        gs.set_knn_capacity(g, opt.get("capacity", 0))
        gs.step(g, gs.KNNBinData(p.world_cells, p.world_size, p.search_radius), None, p, odd)
        ol.run(want, p, odd)
        same(g.download(), want, f"{opt} odd={odd}")


@pytest.mark.parametrize("counts,k", [((20001,), 9), ((1, 3), 16), ((63,) * 7, 9),
                                      ((401, 1, 800), 24), ((5000,) * 3, 7)])
@pytest.mark.parametrize("close", [0, 1])
def test_small_batches(counts, k, close):
    """Batches keep the sorting steps: the lane groups' kernels over scenes."""
    p = sc.chokepoint_params(k=k).replace(avoid_close=close)
    states = [sc.chokepoint_agents(n, seed=i) for i, n in enumerate(counts)]
    b = gs.Batch(list(counts), p.k, p.world_cells, p.world_size, p.search_radius)
    for i in range(len(counts)):
        b.set_walls(i, sc.chokepoint_walls(10.0))
    b.upload(AgentState.concat(states))
    b.step(p, 2)
    got = b.download()
    walls = ol.split_walls(*sc.walls_from_rows(sc.chokepoint_walls(10.0)), p.world_size,
                           p.world_cells)
    at = 0
    for one in states:
        want = one.copy()
        ol.run(want, p, 2, walls=walls)
        same(got.subset(slice(at, at + one.n)), want, f"scene at {at}")
        at += one.n


@pytest.mark.parametrize("inside,steps", [(0, 1), (17, 2), (300, 3)])
def test_diagnostics_of_a_table_frame(inside, steps):
    """Agents per cell of the last frame's table and the mean of the velocities
    after it, summed in agent order whatever the row and overflow order."""
    from gpusteer_gb300.groups import cell_avg_velocity, cell_density

    p = sc.boids_params(k=9, world=64.0)
    s = clump(2000, inside, 3)
    bins = gs.KNNBinData(p.world_cells, p.world_size, p.search_radius)
    g = group_of(s, p)
    gs.step(g, bins, None, p, steps)
    frame, want = s.copy(), s.copy()
    if steps > 1:
        ol.run(frame, p, steps - 1)
    ol.oracle().orc_wrap_world(ol.C.byref(ol.group_struct(frame)), ol.f3(p.world_size),
                               p.wrap_mode)
    ol.run(want, p, steps)
    np.testing.assert_array_equal(cell_density(g, bins),
                                  ol.cell_density(frame.position, p.world_size, p.world_cells))
    np.testing.assert_array_equal(
        cell_avg_velocity(g, bins),
        ol.cell_avg_velocity(frame.position, want.direction, want.speed, p.world_size,
                             p.world_cells))


@pytest.mark.parametrize("capacity", [32, 64, 128])
@pytest.mark.parametrize("n,k,width", [(33, 16, 5.0), (34, 16, 5.0), (900, 7, 60.0), (3001, 16, 70.0),
                                       (2500, 32, 40.0)])
@pytest.mark.parametrize("radius", [1, 2])
def test_flat_rows_end_to_end(n, k, width, capacity, radius):
    """The flat worlds' three-row scan at a fixed capacity: boxes below, at
    and above it, and radius 2, which sparse boxes leave to the other scan."""
    p = sc.chokepoint_params(k=k).replace(search_radius=radius)
    s = sc.chokepoint_agents(n, x_range=(-width / 2, width / 2), z_range=(14.0, 14.0 + width),
                             seed=n + k)
    bins = gs.KNNBinData(p.world_cells, p.world_size, p.search_radius)
    walls = gs.WallGroup(sc.chokepoint_walls(10.0), bins=bins, knw=p.knw)
    g = group_of(s, p, capacity)
    gs.step(g, bins, walls, p, 3)
    want = s.copy()
    ol.run(want, p, 3, walls=walls.download())
    same(g.download(), want, f"n={n} k={k} capacity={capacity} radius={radius}")


@pytest.mark.parametrize("inside", [32, 33, 34])
def test_a_flat_box_at_its_capacity(inside):
    """Capacity 32 holds an agent's box of 32 others, itself left out:
    clumps of one agent fewer, as many and one more than fit."""
    p = sc.chokepoint_params(k=16)
    s = sc.chokepoint_agents(inside, x_range=(0.1, 1.9), z_range=(20.1, 21.9), seed=4)
    bins = gs.KNNBinData(p.world_cells, p.world_size, p.search_radius)
    walls = gs.WallGroup(sc.chokepoint_walls(10.0), bins=bins, knw=p.knw)
    g = group_of(s, p, 32)
    gs.step(g, bins, walls, p, 1)
    want = s.copy()
    ol.run(want, p, 1, walls=walls.download())
    same(g.download(), want, f"inside={inside}")
