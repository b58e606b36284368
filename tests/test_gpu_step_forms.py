"""Which form a step ran in, the launches it made, and what the benchmark's lines
say of them."""
from __future__ import annotations

import ctypes as C
import json
import subprocess
import sys
from pathlib import Path

import pytest

import gpusteer_gb300 as gs
from gpusteer_gb300 import scenario as sc
from gpusteer_gb300._lib import call

pytestmark = pytest.mark.gpu
REPO = Path(__file__).resolve().parents[1]


def flock(n, k=7, radius=1, capacity=0, steps=3, profile=False):
    p = sc.boids_params(k=k, world=128.0).replace(search_radius=radius)
    g = gs.AgentGroup(k, n)
    g.upload(sc.boids_cube(n, size=120.0, seed=1))
    gs.set_knn_capacity(g, capacity)
    assert gs.last_step(g) == ("none", 0)
    return run(g, p, None, steps, profile)


def crowd(n, k=16, capacity=0, persistent=False, steps=3, profile=False):
    p = sc.chokepoint_params(k=k)
    g = gs.AgentGroup(k, n)
    g.upload(sc.chokepoint_agents(n, seed=1))
    gs.set_knn_capacity(g, capacity)
    gs.set_persistent(g, persistent)
    return run(g, p, sc.chokepoint_walls(10.0), steps, profile)


def run(g, p, walls, steps, profile):
    bins = gs.KNNBinData(p.world_cells, p.world_size, p.search_radius)
    w = gs.WallGroup(walls, bins=bins, knw=p.knw) if walls is not None else None
    if profile:
        call("gs_group_set_profiling", g.handle, 1)
    gs.step(g, bins, w, p, steps)
    if not profile:
        return gs.last_step(g)
    ms, launches = (C.c_float * 4)(), (C.c_uint * 4)()
    call("gs_group_phase_times", g.handle, ms, launches, 4)
    return gs.last_step(g), list(ms), list(launches)


@pytest.mark.parametrize("got,want", [
    (lambda: flock(4096), ("table", 1)), (lambda: crowd(10000), ("table", 2)),
    (lambda: flock(4096, radius=2), ("lanes", 3)), (lambda: flock(4096, capacity=32), ("threads", 3)),
    (lambda: flock(20001, k=16), ("threads", 5)),  # 20 candidates a box: capacity 128
    (lambda: flock(4096, capacity=128), ("threads", 5)),
    (lambda: crowd(10000, capacity=64), ("threads", 4)), (lambda: crowd(10000, capacity=256), ("threads", 5)),
    (lambda: crowd(10000, capacity=256, persistent=True), ("persistent", 1))])
def test_form_and_launches(got, want):
    assert got() == want


def test_profiling_does_not_change_the_form():
    step, ms, launches = flock(4096, steps=4, profile=True)
    assert step == ("table", 1)
    assert launches == [0, 0, 4, 0] and ms[2] > 0
    step, ms, launches = crowd(3000, steps=4, profile=True)
    assert step == ("table", 2)
    assert launches == [0, 0, 4, 4] and ms[2] > 0 and ms[3] > 0


def line(*args):
    r = subprocess.run([sys.executable, str(REPO / "bench.py"), "--no-cpu", "--warmup", "3", *args],
                       capture_output=True, text=True, timeout=900, cwd=REPO)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads([ln for ln in r.stdout.splitlines() if ln.startswith("{")][0])


@pytest.mark.parametrize("workload,form,launches,kernel", [
    ("boids", "table", 1, "k_table_step"), ("chokepoint", "table", 2, "k_table_walls+k_table_rest")])
def test_bench_line_of_a_small_group(workload, form, launches, kernel):
    d = line("--workload", workload, "--steps", "20")
    assert d["form"] == form and d["gpu_launches"] == 20 * launches
    assert d["roofline"]["kernel"] == kernel
    assert d["phases_ms"]["scan"] is None and d["phases_ms"]["permute"] is None
    assert (d["phases_ms"]["fused_rest"] is None) == (launches == 1)


def test_bench_line_of_brute_force_counts_its_calls():
    d = line("--workload", "brute", "--steps", "3")
    assert d["gpu_launches"] == 3 * d["calls_per_step"] * d["launches_per_call"]
    assert d["launches_per_call"] == 2
    assert d["ms_per_step"] == pytest.approx(d["ms_per_call"] * d["calls_per_step"])
    assert d["value"] == pytest.approx(65536 / (d["ms_per_call"] / 1e3))


@pytest.mark.parametrize("which", ["flock 30000", "flock 65536", "crowd 40000"])
def test_a_step_takes_no_longer_than_its_phases(which):
    """Kernels that start early must not crowd the SMs: a step's launches, one
    after another, against the sum of its phases timed apart (each with its
    launch's latency). Steps of these groups took 7 to 15 % longer than in
    plain order."""
    import torch

    name, n = which.split()
    n, k = int(n), 16
    if name == "flock":
        p = sc.boids_params(k=k, world=256.0, cell=8.0)
        s = sc.boids_cube(n, size=min(250.0, 4.0 * n ** (1 / 3)), seed=n)
        walls = None
    else:
        p = sc.chokepoint_params(k=k)
        s = sc.chokepoint_agents(n, x_range=(-200, 200), z_range=(14, 250), seed=n)
        walls = sc.chokepoint_walls(10.0)
    bins = gs.KNNBinData(p.world_cells, p.world_size, 1)
    w = gs.WallGroup(walls, bins=bins, knw=p.knw) if walls is not None else None
    g = gs.AgentGroup(k, n)
    g.upload(s)
    gs.step(g, bins, w, p, 20)
    stream = torch.cuda.ExternalStream(g.stream)
    times = []
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        gs.step(g, bins, w, p, 20)
        b.record(stream)
        b.synchronize()
        times.append(a.elapsed_time(b) / 20)
    call("gs_group_set_profiling", g.handle, 1)
    gs.step(g, bins, w, p, 20)
    ms, launches = (C.c_float * 4)(), (C.c_uint * 4)()
    call("gs_group_phase_times", g.handle, ms, launches, 4)
    phases = sum(m / c for m, c in zip(ms, launches) if c)
    assert sorted(times)[2] < phases, (times, list(ms), list(launches))
