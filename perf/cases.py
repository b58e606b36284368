"""The work that programs have this library do, as timed cases.

A case is one call pattern ("kind") at one size; the listed cases are the
library's own configurations (the 4,096-boid and 1,048,576-boid flocks, the
10,000-agent choke point, the 256 batched scenes, the 65,536-agent brute force
and fit) and the plugins' call sequences at the sizes of the tests, odd ones
among them.  draw() gives further sizes of the same kinds.

  flock         the fused step of a plain 3D flock (separation, cohesion, alignment)
  crowd         the fused step of one 2D choke point (walls, avoidance, separation, seek)
  scenes        many choke points of uneven agent counts in one batch
  host          a frame with host state in and out (SyncDevice, step, SyncHost)
  boids_calls   a boids plugin's frame, one call per function, binned KNN
  brute_calls   the same frame on brute-force KNN
  crowd_calls   a choke-point plugin's frame, one call per function
  groups        MultiGroup frames: several groups that see each other
  knn           rebuild the database, then the binned lists of a large set
  brute         brute-force lists, of a group against itself or another
  fit           a differentiable rollout, forward and backward

A pass that moves agents starts from the prepared state, which it first writes
into the group's device arrays as a program that restarts an episode does, so
that every pass does the same work.
"""
import ctypes
import math
import random

import numpy as np
import torch

import gpusteer_gb300 as gs
from gpusteer_gb300.scenario import StepParams
from gpusteer_gb300.state import AgentState

NAMES = ("position", "direction", "steering", "side", "up", "speed", "max_speed", "max_force",
         "radius", "mass", "applied")
WIDTH = {"position": 4, "direction": 4, "steering": 4, "side": 3, "up": 3}
MOVED = ("position", "direction", "side", "up", "speed")  # what a step changes
WALLS, AVOID, SEPARATION, ALIGNMENT, COHESION, SEEK = 1, 2, 3, 4, 5, 6  # behaviour codes
BIT = {SEEK: 4, SEPARATION: 16, ALIGNMENT: 32, COHESION: 64, WALLS: 256, AVOID: 512}
CLOSE_BIT, PUSHED_BIT = 1024, 4096  # avoid-close-neighbours, pushed out of a wall
GAPS = (7.5, 10.0, 12.5, 15.0, 17.5, 20.0, 22.5, 25.0, 27.5, 30.0, 32.5)


def listed():
    return [
        # the smallest simulation: the 4,096-boid flock, k = 7, where a step is launches and latency
        {"name": "flock 4096", "kind": "flock", "n": 4096, "k": 7, "cells": 40, "ball": 50.0, "steps": 16},
        # the large flock: 1,048,576 boids, k = 16, in a 512^3 world
        {"name": "flock 1M", "kind": "flock", "n": 1048576, "k": 16, "cells": 128, "ball": 0.0, "steps": 8},
        # one crowd of 10,000 through a gap, k = 16, with walls
        {"name": "crowd 10000", "kind": "crowd", "n": 10000, "k": 16, "gap": 10.0, "steps": 8},
        # training and sweeps: 256 crowds of 1,000 to 20,000 agents advanced together
        {"name": "scenes 256", "kind": "scenes", "scenes": 256, "low": 1000, "high": 20000, "k": 16, "steps": 4},
        # a host program that keeps its agents in host memory and steps them once a frame
        {"name": "host 100003", "kind": "host", "n": 100003, "k": 16, "cells": 59, "steps": 1},
        # a boids plugin (wrap, rebuild, KNN, three behaviours, update) on an odd count
        {"name": "boids plugin 30011", "kind": "boids_calls", "n": 30011, "k": 7, "cells": 39, "frames": 4},
        # the brute-force boids plugin at the smallest flock's size
        {"name": "brute plugin 4096", "kind": "brute_calls", "n": 4096, "k": 7, "cells": 40, "frames": 4},
        # a choke-point plugin: two KNN calls, four behaviours, update
        {"name": "crowd plugin 10000", "kind": "crowd_calls", "n": 10000, "k": 16, "gap": 10.0, "frames": 4},
        # three groups that avoid, separate from and push each other
        {"name": "groups 3", "kind": "groups", "n": 2500, "groups": 3, "k": 8, "cells": 24, "frames": 4},
        # an offline pass over a large set: database and 32 neighbours each
        {"name": "knn 262147", "kind": "knn", "n": 262147, "k": 32, "cells": 51, "radius": 1},
        # exact neighbours without a grid, 65,536 against themselves
        {"name": "brute 65536", "kind": "brute", "n": 65536, "other": 0, "k": 16, "world": 512.0},
        # fitting steering weights: 65,536 boids, checkpoints every 8 steps, loss on the positions
        {"name": "fit 65536", "kind": "fit", "n": 65536, "k": 16, "cells": 64, "cube": 200.0, "steps": 12, "every": 8},
    ]


def draw(rng: random.Random):
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("flock", "flock", "crowd", "scenes", "host", "boids_calls", "brute_calls",
                       "crowd_calls", "groups", "knn", "brute", "fit"))
    c = {"kind": kind}
    if kind in ("flock", "host", "boids_calls", "brute_calls", "fit"):
        top = {"flock": 1000000, "host": 250000, "boids_calls": 250000, "brute_calls": 30000, "fit": 65000}
        c["n"] = between(1000, top[kind])
        c["k"] = rng.choice((5, 7, 8, 12, 16)) if kind != "flock" else rng.choice((5, 7, 12, 16, 24))
        # two cells of 4^3 for each agent, the flock's density
        c["cells"] = max(8, int(round((2.0 * c["n"]) ** (1.0 / 3.0))))
        if kind == "flock":
            c["ball"], c["steps"] = 0.0, rng.choice((4, 8, 16))
            if c["n"] > 100000:
                c["steps"] = 4
        elif kind == "host":
            c["steps"] = rng.choice((1, 1, 2))
        elif kind == "fit":
            c["cells"] = max(8, int(round((2.0 * c["n"]) ** (1.0 / 3.0) * 1.28)))
            c["cube"], c["steps"], c["every"] = 4.0 * c["cells"] / 1.28, rng.choice((3, 5, 8, 11)), rng.choice((4, 8))
        else:
            c["frames"] = rng.choice((2, 3, 4))
    elif kind in ("crowd", "crowd_calls"):
        c.update(n=between(1000, 20000), k=rng.choice((8, 12, 16, 20)), gap=rng.choice(GAPS))
        c["steps" if kind == "crowd" else "frames"] = rng.choice((3, 5, 8)) if kind == "crowd" else rng.choice((2, 4))
    elif kind == "scenes":
        low = between(100, 2000)
        c.update(scenes=between(8, 250), low=low, high=low * rng.randint(2, 9), k=rng.choice((8, 16)), steps=rng.choice((2, 4)))
    elif kind == "groups":
        c.update(n=between(300, 8000), groups=rng.randint(2, 5), k=rng.choice((5, 8, 16)), cells=24, frames=rng.choice((2, 4)))
    elif kind == "knn":
        c.update(n=between(1000, 260000), k=rng.choice((3, 8, 13, 16, 32)), radius=rng.choice((1, 1, 2)))
        # a box of 27 cells holds about the neighbours asked for, at least the flock's 13
        c["cells"] = max(8, int(round((c["n"] / max(0.5, c["k"] / 16.0)) ** (1.0 / 3.0))))
    else:
        c.update(n=between(500, 65000), other=rng.choice((0, 0, between(500, 65000))), k=rng.choice((1, 7, 16, 31, 40)), world=512.0)
    return c


# ---- inputs ---------------------------------------------------------------------------

_stream = None


def _the_stream():
    """The stream that a program's groups and its own tensor work share."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _headings(g, n, flat):
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    if flat:
        d[:, 1] = 0
    return d / d.norm(dim=1, keepdim=True).clamp_min(1e-9)


def _agents(position, heading, speed, max_speed, max_force, radius=0.5):
    """A device state: position, unit heading, a frame about +y, no steering."""
    n = position.shape[0]
    side = torch.linalg.cross(heading, torch.tensor([0.0, 1.0, 0.0], device="cuda", dtype=torch.float64).expand(n, 3))
    side = side / side.norm(dim=1, keepdim=True).clamp_min(1e-9)
    s = {"position": position, "direction": heading, "side": side, "up": torch.linalg.cross(side, heading), "speed": speed}
    s = {k: v.to(torch.float32) for k, v in s.items()}
    for k in ("position", "direction"):
        s[k] = torch.nn.functional.pad(s[k], (0, 1))
    s["steering"] = torch.zeros(n, 4, device="cuda")
    for k, v in (("max_speed", max_speed), ("max_force", max_force), ("radius", radius), ("mass", 1.0)):
        s[k] = torch.full((n,), v, device="cuda")
    s["applied"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    return {k: s[k].contiguous() for k in NAMES}


def _boids(n, seed, cube, ball, radius=0.5, salt=0, slowest=0.0):
    g = _gen(seed, salt)
    if ball > 0:
        r = torch.rand(n, 1, generator=g, device="cuda", dtype=torch.float64) ** (1.0 / 3.0)
        pos = _headings(g, n, False) * r * ball
    else:
        pos = (torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64) - 0.5) * cube
    speed = slowest + torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (9.0 - slowest)
    return _agents(pos, _headings(g, n, False), speed, 9.0, 27.0, radius)


def _people(n, seed):
    g = _gen(seed)
    u = torch.rand(n, 2, generator=g, device="cuda", dtype=torch.float64)
    pos = torch.zeros(n, 3, device="cuda", dtype=torch.float64)
    pos[:, 0], pos[:, 2] = u[:, 0] * 100.0 - 50.0, u[:, 1] * 100.0 + 13.5
    speed = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 3.0  # on their way
    return _agents(pos, _headings(g, n, True), speed, 3.0, 3.0)


def _counts(case):
    """Uneven agent counts between low and high, the same for every seed."""
    span = case["high"] - case["low"] + 1
    return [case["low"] + int(span * ((0.6180339887498949 * (i + 1)) % 1.0)) for i in range(case["scenes"])]


def _walls(gap):
    """The choke point's map: a funnel on each side of a channel of half-width gap."""
    fx, fz, wz = 1232.5, 293.5, 13.5
    return np.array([[-fx, 0, fz, -gap, 0, wz, 0, 0, 1], [-fx, 0, -fz, -gap, 0, -wz, 0, 0, -1],
                     [-gap, 0, -wz, -gap, 0, wz, 1, 0, 0], [gap, 0, wz, fx, 0, fz, 0, 0, 1],
                     [gap, 0, -wz, fx, 0, -fz, 0, 0, -1], [gap, 0, wz, gap, 0, -wz, -1, 0, 0]], np.float32)


def _flock_params(case):
    w, c = 4.0 * case["cells"], case["cells"]
    return StepParams(world_size=(w, w, w), world_cells=(c, c, c), search_radius=1, k=case["k"],
                      sep_min=0.5, sep_max=2.0, w_sep=5.0, ali_min=0.5, ali_max=7.0, w_ali=8.0,
                      coh_min=0.5, coh_max=7.0, w_coh=4.0, order=(SEPARATION, COHESION, ALIGNMENT), dt=1.0 / 60.0)


def _crowd_params(case):
    return StepParams(world_size=(512.0, 10.0, 512.0), world_cells=(256, 1, 256), search_radius=1, wrap_mode=0,
                      k=case["k"], knw=3, clear_applied=1, min_time_to_wall=10.0, w_walls=1.0,
                      min_time_to_collision=2.0, min_separation_distance=0.5, avoid_close=0, w_avoid=1.0,
                      sep_min=0.5, sep_max=1.2, sep_cos=-0.8660254037844386, w_sep=10.0, mask_sep=PUSHED_BIT,
                      seek_target=(0.0, 0.0, -93.5), w_seek=1.5, mask_seek=4480,
                      order=(WALLS, AVOID, SEPARATION, SEEK), dt=1.0 / 30.0)


GROUP = dict(wrap_mode=1, min_time_to_collision=2.0, min_separation_distance=0.5, avoid_close=1, w_avoid=1.0,
             mask_avoid=0, sep_min=0.5, sep_max=2.0, sep_cos=-0.984807753012208, w_sep=5.0, mask_sep=4096,
             ali_min=0.5, ali_max=7.0, ali_cos=-0.984807753012208, w_ali=8.0, mask_ali=272,
             coh_min=0.5, coh_max=7.0, coh_cos=-0.984807753012208, w_coh=4.0, mask_coh=272,
             path_prediction_time=5.0, w_path=1.0, mask_path=16, w_seek=1.5, mask_seek=4480, mask_antipen=4096,
             dt=1.0 / 30.0)


def _group_sizes(case):
    return [max(1, case["n"] * (10 - 3 * (i % 3)) // 10 - i) for i in range(case["groups"])]


def _group_ball(case):
    """Groups of 2,500 share a ball of radius 16; others are as dense."""
    return 16.0 * (case["n"] / 2500.0) ** (1.0 / 3.0)


def _world(case):
    return 4.0 * case["cells"]


# ---- the program's handles ----------------------------------------------------------------

class _Device:
    """An array of the library's, for torch to look at; it keeps the array's owner."""

    def __init__(self, owner, address, shape, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (address, False), "shape": shape, "typestr": kind, "version": 3, "strides": None}


def _at(owner, address, shape, kind="<f4"):
    return torch.as_tensor(_Device(owner, address, shape, kind), device="cuda")


def _views(owner, group, n):
    at = gs.AgentGroup.device_arrays(group)
    return {k: _at(owner, at[k], (n, WIDTH[k]) if k in WIDTH else (n,), "<i4" if k == "applied" else "<f4") for k in NAMES}


def _host_state(first, pinned=False):
    n = first["speed"].shape[0]
    out = gs.pinned_state(n) if pinned else AgentState.zeros(n)
    for k in NAMES:
        v = first[k].cpu().numpy()
        getattr(out, k)[...] = v.view(np.uint32) if k == "applied" else v
    return out


class _Held(np.ndarray):
    """A page-locked array that keeps the state it belongs to."""


def _held(state, k):
    a = getattr(state, k).view(_Held)
    a.owner = state
    return a


class _Episode:
    """A group and the state that its episodes start from."""

    def __init__(self, owner, group, first):
        owner.upload(_host_state(first))
        self.group, self.first = group, first
        self.now = _views(owner, group, first["speed"].shape[0])
        self.pairs = ([self.now[k] if k != "applied" else self.now[k].view(torch.float32) for k in NAMES],
                      [first[k] if k != "applied" else first[k].view(torch.float32) for k in NAMES])

    def restart(self):
        gs.AgentGroup.device_arrays(self.group)  # the program is about to write through its pointers
        with torch.cuda.stream(_the_stream()):
            torch._foreach_copy_(*self.pairs)

    def moved(self):
        gs.AgentGroup.device_arrays(self.group)  # brings the arrays up to date
        return {k: self.now[k] for k in MOVED}


def _new_group(first, k):
    n = first["speed"].shape[0]
    g = gs.AgentGroup(k, n, stream=_the_stream().cuda_stream)
    return _Episode(g, g, first)


def _knn_views(knn, n, k):
    idx, dist = ctypes.POINTER(ctypes.c_uint)(), ctypes.POINTER(ctypes.c_float)()
    if gs.load().gs_knn_device_arrays(knn.handle, ctypes.byref(idx), ctypes.byref(dist)):
        raise RuntimeError("gs_knn_device_arrays failed")
    return {"index": _at(knn, ctypes.cast(idx, ctypes.c_void_p).value, (k, n), "<i4"), "distance": _at(knn, ctypes.cast(dist, ctypes.c_void_p).value, (k, n))}


def _first(case, seed):
    kind = case["kind"]
    if kind in ("crowd", "crowd_calls"):
        return _people(case["n"], seed)
    if kind == "scenes":
        return _people(sum(_counts(case)), seed)
    if kind == "brute":
        return _boids(case["n"], seed, case["world"], 0.0)
    # a fit starts with everyone moving: headings have no derivative at rest
    return _boids(case["n"], seed, case.get("cube", _world(case)), case.get("ball", 0.0), slowest=1.0 if kind == "fit" else 0.0)


def prepare(case, seed):
    kind, s = case["kind"], {"kind": case["kind"], "case": case}
    if kind in ("flock", "host", "boids_calls", "brute_calls", "knn", "fit"):
        c, w = case["cells"], _world(case)
        s["bins"] = gs.KNNBinData((c, c, c), (w, w, w), case.get("radius", 1))
        if kind != "knn":
            s["params"] = _flock_params(case)
    elif kind in ("crowd", "crowd_calls", "scenes"):
        s["params"] = p = _crowd_params(case)
        if kind != "scenes":
            s["bins"] = gs.KNNBinData(p.world_cells, p.world_size, 1)
            s["walls"] = gs.WallGroup(_walls(case["gap"]), bins=s["bins"], knw=p.knw)
    if kind == "host":
        s["host_in"] = _host_state(_first(case, seed), pinned=True)
        s["host_out"] = out = gs.pinned_state(case["n"])
        s["held"] = {k: _held(out, k) for k in MOVED}
        s["group"] = gs.AgentGroup(case["k"], case["n"], stream=_the_stream().cuda_stream)
    elif kind == "scenes":
        p = s["params"]
        b = gs.Batch(_counts(case), p.k, p.world_cells, p.world_size, 1, stream=_the_stream().cuda_stream)
        for i in range(case["scenes"]):
            b.set_walls(i, _walls(GAPS[i % len(GAPS)]))
        s["batch"], s["episode"] = b, _Episode(b, b.group, _first(case, seed))
    elif kind == "groups":
        w, c = _world(case), case["cells"]
        sizes = _group_sizes(case)
        s["bins"] = gs.KNNBinData((c, c, c), (w, w, w), 1)
        s["params"] = gs.MultiGroupParams(world_size=(w, w, w), **GROUP)
        s["episodes"] = [_new_group(_boids(m, seed, w, _group_ball(case), 0.9, i), case["k"]) for i, m in enumerate(sizes)]
        s["knn"] = [[gs.KNNData(m, case["k"]) for _ in sizes] for m in sizes]
    else:
        s["episode"] = _new_group(_first(case, seed), case["k"])
    if kind in ("boids_calls", "brute_calls", "crowd_calls", "knn", "brute"):
        s["knn"] = gs.KNNData(case["n"], case["k"])
    if kind in ("knn", "brute"):
        s["lists"] = _knn_views(s["knn"], case["n"], case["k"])
    if kind == "brute" and case["other"]:
        s["other"] = _new_group(_boids(case["other"], seed, case["world"], 0.0, salt=1), case["k"])
    if kind == "crowd_calls":
        s["wall_knn"] = gs.KNNData(case["n"], s["params"].knw)
        gs.updateKNNDatabase(s["walls"], s["bins"])
    if kind == "fit":
        n, e = case["n"], s["episode"]
        s["rollout"] = gs.Rollout(e.group, s["bins"], case["steps"], case["every"])
        s["target"] = _target(case, seed, e.first)
        s["grad"] = [torch.zeros(n, 4, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    return s


def _target(case, seed, first):
    """Where the fit wants its boids: near where straight flight takes them."""
    t = case["steps"] / 60.0
    ahead = first["position"] + first["direction"] * first["speed"][:, None] * t
    noise = torch.randn(ahead.shape[0], 4, generator=_gen(seed, 7), device="cuda") * 0.05
    noise[:, 3] = 0
    return (ahead + noise).contiguous()


# ---- a pass -------------------------------------------------------------------------------

def run(s):
    kind, case, p = s["kind"], s["case"], s.get("params")
    if kind == "flock":
        s["episode"].restart()
        gs.step(s["episode"].group, s["bins"], None, p, case["steps"])
        return s["episode"].moved()
    if kind == "crowd":
        s["episode"].restart()
        gs.step(s["episode"].group, s["bins"], s["walls"], p, case["steps"])
        return s["episode"].moved()
    if kind == "scenes":
        s["episode"].restart()
        s["batch"].step(p, case["steps"])
        return s["episode"].moved()
    if kind == "host":
        gs.step_host(s["group"], s["bins"], None, p, case["steps"], s["host_in"], s["host_out"])
        return s["held"]
    if kind == "boids_calls" or kind == "brute_calls":
        return _boids_frames(s["episode"], s["knn"], s["bins"], p, case["frames"], kind == "brute_calls")
    if kind == "crowd_calls":
        return _crowd_frames(s["episode"], s["knn"], s["wall_knn"], s["bins"], s["walls"], p, case["frames"])
    if kind == "groups":
        for e in s["episodes"]:
            e.restart()
        gs.multigroup_step([e.group for e in s["episodes"]], s["bins"], s["knn"], p, case["frames"])
        return [dict(e.moved(), applied=e.now["applied"]) for e in s["episodes"]]
    if kind == "knn":
        g = s["episode"].group
        gs.updateKNNDatabase(g, s["bins"])
        gs.findKNearestNeighbors(g, s["knn"], s["bins"], g, case["radius"])
        return s["lists"]
    if kind == "brute":
        g = s["episode"].group
        gs.findKNearestNeighborsBruteForce(g, s["knn"], s["other"].group if "other" in s else g)
        return s["lists"]
    e, r = s["episode"], s["rollout"]
    e.restart()
    r.forward(p)
    final = e.moved()["position"]
    with torch.cuda.stream(_the_stream()):
        adjoint = (final - s["target"]) * (2.0 / (3.0 * case["n"]))
        end = final.clone()
    gw = r.backward(adjoint.data_ptr(), None, s["grad"][0].data_ptr(), s["grad"][1].data_ptr())
    return {"weights": gw, "position": s["grad"][0], "velocity": s["grad"][1], "final": end}


def _boids_frames(e, knn, bins, p, frames, brute):
    g = e.group
    e.restart()
    for _ in range(frames):
        gs.wrapWorld(g, p.world_size, p.wrap_mode)
        if brute:
            gs.findKNearestNeighborsBruteForce(g, knn, g)
        else:
            gs.updateKNNDatabase(g, bins)
            gs.findKNearestNeighbors(g, knn, bins, g, 1)
        gs.steerForSeparation(g, knn, g, p.sep_min, p.sep_max, p.sep_cos, p.w_sep, p.mask_sep)
        gs.steerForCohesion(g, knn, g, p.coh_min, p.coh_max, p.coh_cos, p.w_coh, p.mask_coh)
        gs.steerForAlignment(g, knn, g, p.ali_min, p.ali_max, p.ali_cos, p.w_ali, p.mask_ali)
        gs.updateGroup(g, p.dt)
    return e.moved()


def _crowd_frames(e, knn, wall_knn, bins, walls, p, frames):
    g = e.group
    e.restart()
    for _ in range(frames):
        gs.wrapWorld(g, p.world_size, p.wrap_mode)
        gs.updateKNNDatabase(g, bins)
        gs.findKNearestNeighbors(g, knn, bins, g, 1)
        gs.findKNearestNeighbors(g, wall_knn, bins, walls, 1)
        gs.steerToAvoidWalls(g, wall_knn, walls, p.min_time_to_wall, p.w_walls, p.mask_walls)
        gs.steerToAvoidNeighbors(g, knn, g, p.min_time_to_collision, p.min_separation_distance, p.avoid_close,
                                 p.w_avoid, p.mask_avoid)
        gs.steerForSeparation(g, knn, g, p.sep_min, p.sep_max, p.sep_cos, p.w_sep, p.mask_sep)
        gs.steerForSeek(g, p.seek_target, p.w_seek, p.mask_seek)
        gs.updateGroup(g, p.dt)
    return e.moved()


# ---- what a pass cannot do without -----------------------------------------------------------

def work(case):
    """A step reads each agent's state (92 B) and writes what it changes
    (60 B); per neighbour, about 40 operations.  Lists are 8 B an entry."""
    kind, k = case["kind"], case["k"]
    if kind == "scenes":
        n, times = sum(_counts(case)), case["steps"]
    elif kind == "groups":
        n, times = sum(_group_sizes(case)) * case["groups"], case["frames"]
    else:
        n, times = case["n"], case.get("steps", case.get("frames", 1))
    if kind in ("knn", "brute"):
        m = n + (case.get("other") or 0)
        return {"bytes": 16.0 * m + 8.0 * k * n, "flops": 8.0 * n * 4 * k}
    per = 3 if kind == "fit" else 1  # the backward pass runs each step again, then its adjoint
    lists = 16.0 * k * n * times if kind.endswith("_calls") or kind in ("groups", "fit") else 0.0
    return {"bytes": 152.0 * n * times * per + lists, "flops": 40.0 * n * k * times * per}


# ---- the same in 64 bits ----------------------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind == "groups":
        return _groups64(case, seed)
    first = _first(case, seed)
    if kind in ("knn", "brute"):
        q = first["position"][:, :3].double()
        if kind == "knn":
            c, w = case["cells"], _world(case)
            _, dist = _binned64(q, q, (w, w, w), (c, c, c), case["radius"], case["k"], True)
        else:
            o = _boids(case["other"], seed, case["world"], 0.0, salt=1)["position"][:, :3].double() if case["other"] else q
            _, dist = _nearest64(q, o, case["k"], not case["other"])
        dist = torch.where(dist.isinf(), torch.full_like(dist, float(np.finfo(np.float32).max)), dist)
        return {"index": None, "distance": dist.t().contiguous()}
    s = {k: first[k].double() for k in NAMES if k != "applied"}
    for k in ("position", "direction"):
        s[k] = s[k][:, :3]
    if kind == "fit":
        return _fit64(case, seed, s)
    if kind in ("crowd", "crowd_calls", "scenes"):
        p = _crowd_params(case)
        if kind == "scenes":
            scene = torch.repeat_interleave(torch.arange(case["scenes"], device="cuda"),
                                            torch.tensor(_counts(case), device="cuda"))
            maps = [_split64(_walls(GAPS[i % len(GAPS)]), p) for i in range(case["scenes"])]
        else:
            scene, maps = torch.zeros(case["n"], dtype=torch.long, device="cuda"), [_split64(_walls(case["gap"]), p)]
        segments = torch.cat(maps)
        of = torch.repeat_interleave(torch.arange(len(maps), device="cuda"), torch.tensor([m.shape[0] for m in maps], device="cuda"))
        for _ in range(case.get("steps", case.get("frames"))):
            s = _crowd_step64(s, p, scene, segments, of)
    else:
        p = _flock_params(case)
        for _ in range(case.get("steps", case.get("frames"))):
            s = _flock_step64(s, p, brute=kind == "brute_calls")
    return _told64(s)


def _told64(s):
    s = {k: s[k] for k in MOVED}
    for k in ("position", "direction"):
        s[k] = torch.nn.functional.pad(s[k], (0, 1))
    return s


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(v):
    n = v.norm(dim=-1, keepdim=True)
    return torch.where(n > 0, v / torch.where(n > 0, n, torch.ones_like(n)), v)


def _cells64(pos, size, cells):
    size = torch.tensor(size, device="cuda", dtype=torch.float64)
    n = torch.tensor(cells, device="cuda")
    return torch.minimum(torch.floor((pos + 0.5 * size) / size * n).clamp_min(0).long(), n - 1)


def _binned64(query, cand, size, cells, radius, k, same, q_of=None, c_of=None):
    """The k nearest candidates in the box of cells around each query's cell
    (of the same scene): indices, -1 where there are fewer, and distances."""
    nx, ny, nz = cells
    every = nx * ny * nz
    cc = _cells64(cand, size, cells)
    label = cc[:, 0] + nx * (cc[:, 2] + nz * cc[:, 1])
    if c_of is not None:
        label = label + every * c_of
    total = every * (1 if c_of is None else int(max(int(c_of.max()) + 1, int(q_of.max()) + 1)))
    order = torch.argsort(label, stable=True)
    start = torch.zeros(total + 1, dtype=torch.long, device="cuda")
    start[1:] = torch.cumsum(torch.bincount(label, minlength=total), 0)
    qc = _cells64(query, size, cells)
    idx, dist = [], []
    for at in range(0, query.shape[0], 32768):
        q, c = query[at:at + 32768], qc[at:at + 32768]
        base = 0 if q_of is None else every * q_of[at:at + 32768]
        rows = []
        for dy in range(-radius, radius + 1):
            for dz in range(-radius, radius + 1):
                y, z = c[:, 1] + dy, c[:, 2] + dz
                ok = (y >= 0) & (y < ny) & (z >= 0) & (z < nz)
                row = base + nx * (z.clamp(0, nz - 1) + nz * y.clamp(0, ny - 1))
                s0 = start[row + (c[:, 0] - radius).clamp_min(0)]
                s1 = start[row + (c[:, 0] + radius).clamp_max(nx - 1) + 1]
                rows.append((s0, torch.where(ok, s1 - s0, torch.zeros_like(s0))))
        slots, real = [], []
        for s0, length in rows:
            t = torch.arange(max(1, int(length.max())), device="cuda")
            slots.append(s0[:, None] + t)
            real.append(t < length[:, None])
        slots, real = torch.cat(slots, 1), torch.cat(real, 1)
        who = order[slots.clamp_max(order.shape[0] - 1)]
        if same:
            real = real & (who != torch.arange(at, at + q.shape[0], device="cuda")[:, None])
        d = torch.where(real, (cand[who] - q[:, None]).norm(dim=-1), torch.full(who.shape, math.inf, device="cuda", dtype=torch.float64))
        if d.shape[1] < k:
            d = torch.nn.functional.pad(d, (0, k - d.shape[1]), value=math.inf)
            who = torch.nn.functional.pad(who, (0, k - who.shape[1]))
        d, j = torch.topk(d, k, dim=1, largest=False, sorted=True)
        idx.append(torch.where(d.isinf(), torch.full_like(j, -1), torch.gather(who, 1, j)))
        dist.append(d)
    return torch.cat(idx), torch.cat(dist)


def _nearest64(query, cand, k, same):
    """The k nearest of all candidates."""
    idx, dist = [], []
    step = max(64, (1 << 26) // max(1, cand.shape[0]))
    for at in range(0, query.shape[0], step):
        d = sum((query[at:at + step, a, None] - cand[None, :, a]) ** 2 for a in range(3)).sqrt()
        if same:
            i = torch.arange(d.shape[0], device="cuda")
            d[i, at + i] = math.inf
        if d.shape[1] < k:
            d = torch.nn.functional.pad(d, (0, k - d.shape[1]), value=math.inf)
        d, j = torch.topk(d, k, dim=1, largest=False, sorted=True)
        idx.append(torch.where(d.isinf(), torch.full_like(j, -1), j))
        dist.append(d)
    return torch.cat(idx), torch.cat(dist)


def _wrap64(pos, size, mode):
    half = 0.5 * torch.tensor(size, device="cuda", dtype=torch.float64)
    out = torch.where(pos < -half, half, torch.where(pos > half, -half, pos))
    if mode == 0:  # z wraps below zero only, to 100 beyond the far edge
        z = torch.where(pos[:, 2] < 0, half[2] + 100.0, pos[:, 2])
        out = torch.cat([out[:, :2], z[:, None]], 1)
    return out


def _members64(heading, offset, d, real, lo, hi, cos):
    ahead = _dot(heading[:, None], offset / torch.where(d > 0, d, torch.ones_like(d))[..., None])
    return real & ((d < lo) | (~(d > hi) & (ahead > cos)))


def _flocking64(code, s, o, idx, lo, hi, cos, w, steer, applied, mask):
    """Separation, alignment or cohesion of group s with the listed of o."""
    real = idx >= 0
    j = idx.clamp_min(0)
    at = o["position"][j]
    offset = at - s["position"][:, None]
    d2 = _dot(offset, offset)
    inside = _members64(s["direction"], offset, torch.where(d2 > 0, d2, torch.ones_like(d2)).sqrt() * (d2 > 0), real, lo, hi, cos)
    if code == SEPARATION:
        each = -offset / torch.where(inside & (d2 > 0), d2, torch.ones_like(d2))[..., None]
    else:
        each = at if code == COHESION else o["direction"][j]
    count = inside.sum(1, keepdim=True)
    mean = torch.where(inside[..., None], each, torch.zeros_like(each)).sum(1) / count.clamp_min(1)
    own = {SEPARATION: torch.zeros_like(mean), ALIGNMENT: s["direction"], COHESION: s["position"]}[code]
    r = torch.where(count > 0, _unit(mean - own), torch.zeros_like(mean)) * w
    return _apply64(r, BIT[code], steer, applied, mask)


def _apply64(r, bit, steer, applied, mask):
    on = (applied & mask) == 0
    set_bit = on & (r != 0).any(1)
    return steer + torch.where(on[:, None], r, torch.zeros_like(r)), torch.where(set_bit, applied | bit, applied)


def _truncate64(v, most):
    n = v.norm(dim=-1, keepdim=True)
    return torch.where(n > most[:, None], v * (most[:, None] / torch.where(n > 0, n, torch.ones_like(n))), v)


def _integrate64(s, steer, dt):
    acc = _truncate64(steer, s["max_force"]) / s["mass"][:, None]
    vel = _truncate64(s["direction"] * s["speed"][:, None] + acc * dt, s["max_speed"])
    speed = vel.norm(dim=-1)
    go = (speed > 0)[:, None]
    heading = torch.where(go, vel / torch.where(go, speed[:, None], torch.ones_like(vel)), s["direction"])
    side = torch.where(go, _unit(torch.linalg.cross(heading, s["up"])), s["side"])
    up = torch.where(go, torch.linalg.cross(side, heading), s["up"])
    return dict(s, position=s["position"] + vel * dt, direction=heading, speed=speed, side=side, up=up)


def _flock_step64(s, p, brute=False):
    s = dict(s, position=_wrap64(s["position"], p.world_size, p.wrap_mode))
    if brute:
        idx, _ = _nearest64(s["position"], s["position"], p.k, True)
    else:
        idx, _ = _binned64(s["position"], s["position"], p.world_size, p.world_cells, 1, p.k, True)
    return _integrate64(s, _flock_steer64(s, idx, p, (p.w_sep, p.w_ali, p.w_coh)), p.dt)


def _flock_steer64(s, idx, p, w):
    steer, applied = torch.zeros_like(s["position"]), torch.zeros(idx.shape[0], dtype=torch.long, device="cuda")
    for code, lo, hi, cos, weight in ((SEPARATION, p.sep_min, p.sep_max, p.sep_cos, w[0]),
                                      (COHESION, p.coh_min, p.coh_max, p.coh_cos, w[2]),
                                      (ALIGNMENT, p.ali_min, p.ali_max, p.ali_cos, w[1])):
        steer, applied = _flocking64(code, s, s, idx, lo, hi, cos, weight, steer, applied, 0)
    return steer


def _fit64(case, seed, s):
    p, target = _flock_params(case), _target(case, seed, _first(case, seed))[:, :3].double()
    w = torch.tensor([p.w_sep, p.w_ali, p.w_coh], device="cuda", dtype=torch.float64, requires_grad=True)
    pos = s["position"].clone().requires_grad_(True)
    vel = (s["direction"] * s["speed"][:, None]).requires_grad_(True)
    P, V = pos, vel
    for _ in range(case["steps"]):
        P = P + (_wrap64(P.detach(), p.world_size, p.wrap_mode) - P.detach())
        idx, _ = _binned64(P.detach(), P.detach(), p.world_size, p.world_cells, 1, p.k, True)
        speed = V.norm(dim=-1)
        t = dict(s, position=P, direction=V / speed.clamp_min(1e-30)[:, None], speed=speed)
        acc = _truncate64(_flock_steer64(t, idx, p, w), s["max_force"]) / s["mass"][:, None]
        V = _truncate64(V + acc * p.dt, s["max_speed"])
        P = P + V * p.dt
    # the loss's derivative as the program forms it: 2 / (3 n) of the difference
    gw, gp, gv = torch.autograd.grad(P, (w, pos, vel), (P.detach() - target) * (2.0 / (3.0 * case["n"])))
    pad = torch.nn.functional.pad
    return {"weights": gw, "position": pad(gp, (0, 1)), "velocity": pad(gv, (0, 1)), "final": pad(P.detach(), (0, 1))}


def _split64(rows, p):
    """Wall segments (start, end, normal) cut where they cross into a cell."""
    rows = rows.astype(np.float64)
    size, cells, out = p.world_size, p.world_cells, []
    for r in rows:
        a, b = r[0:3], r[3:6]
        cuts = [0.0, 1.0]
        for axis, other in ((0, 2), (2, 0)):
            if a[axis] == b[axis]:
                continue
            t = (np.arange(cells[axis] + 1) * (size[axis] / cells[axis]) - 0.5 * size[axis] - a[axis]) / (b[axis] - a[axis])
            at = a[other] + t * (b[other] - a[other])
            cuts += [x for x, y in zip(t, at) if 0.0 < x < 1.0 and abs(y) <= 0.5 * size[other]]
        length, cuts = np.linalg.norm(b - a), sorted(cuts)
        keep = [0.0]
        for t in cuts[1:-1]:
            if (t - keep[-1]) * length > 1e-3 and (1.0 - t) * length > 1e-3:
                keep.append(t)
        keep.append(1.0)
        out += [np.concatenate([a + (b - a) * t, a + (b - a) * u, r[6:9]]) for t, u in zip(keep, keep[1:])]
    return torch.tensor(np.array(out), device="cuda", dtype=torch.float64)


def _cross64(sa, ea, sb, eb):
    """Where segment a meets segment b in the x-z plane (broadcast), and whether."""
    x, z = 0, 2
    d = (eb[..., z] - sb[..., z]) * (ea[..., x] - sa[..., x]) - (eb[..., x] - sb[..., x]) * (ea[..., z] - sa[..., z])
    na = (eb[..., x] - sb[..., x]) * (sa[..., z] - sb[..., z]) - (eb[..., z] - sb[..., z]) * (sa[..., x] - sb[..., x])
    nb = (ea[..., x] - sa[..., x]) * (sa[..., z] - sb[..., z]) - (ea[..., z] - sa[..., z]) * (sa[..., x] - sb[..., x])
    line = d.abs() < 0.001
    safe = torch.where(line, torch.ones_like(d), d)
    ua, ub = na / safe, nb / safe
    at = sa + ua[..., None] * (ea - sa)
    at = torch.stack([at[..., 0], torch.zeros_like(ua), at[..., 2]], -1)
    same = line & (na.abs() < 0.001) & (nb.abs() < 0.001)
    hit = ~line & (ua >= 0) & (ua <= 1) & (ub >= 0) & (ub <= 1)
    return torch.where(same[..., None], sa.expand_as(at), at), hit | same


def _avoid_walls64(s, p, idx, seg):
    n = idx.shape[0]
    vel = s["direction"] * s["speed"][:, None]
    reach = 4.0 * s["radius"][:, None]
    feel = [s["position"] + vel * p.min_time_to_wall, s["position"] + (s["side"] + s["direction"]) * reach,
            s["position"] + (s["direction"] - s["side"]) * reach]
    inf = torch.full((n,), math.inf, device="cuda", dtype=torch.float64)
    near, touch, found = inf.clone(), torch.zeros(n, dtype=torch.bool, device="cuda"), torch.zeros(n, dtype=torch.bool, device="cuda")
    normal, push = torch.zeros(n, 3, device="cuda", dtype=torch.float64), torch.zeros(n, device="cuda", dtype=torch.float64)
    for r in range(idx.shape[1]):
        real = idx[:, r] >= 0
        w = seg[idx[:, r].clamp_min(0)]
        ls, le, ln = w[:, 0:3], w[:, 3:6], w[:, 6:9]
        at, hit = _cross64(s["position"], s["position"] - ln * s["radius"][:, None], ls, le)
        hit = hit & real
        touch = touch | hit
        normal = torch.where(hit[:, None], ln, normal)
        near = torch.where(hit, (s["position"] - at).norm(dim=-1), near)
        for f in feel:
            at, hit = _cross64(s["position"], f, ls, le)
            d = (s["position"] - at).norm(dim=-1)
            hit = hit & real & (d < near)
            near, found = torch.where(hit, d, near), found | hit
            push = torch.where(hit, (f - at).norm(dim=-1), push)
            normal = torch.where(hit[:, None], ln, normal)
    t = touch[:, None]
    pos = torch.where(t, s["position"] + normal * (s["radius"] - near)[:, None].nan_to_num(0, 0, 0), s["position"])
    turned = _unit(s["direction"] - normal * _dot(s["direction"], normal)[:, None])
    steer = torch.where(t | ~found[:, None], torch.zeros_like(normal), normal * push[:, None]) * p.w_walls
    applied = torch.where(touch, PUSHED_BIT, torch.where(found, BIT[WALLS], 0)).long()
    return dict(s, position=pos, direction=torch.where(t, turned, s["direction"])), steer, applied


def _avoid64(s, o, idx, min_time, w, mask, steer, applied):
    n = idx.shape[0]
    vel = s["direction"] * s["speed"][:, None]
    first = torch.full((n,), min_time, device="cuda", dtype=torch.float64)
    threat = torch.full((n,), -1, dtype=torch.long, device="cuda")
    at = torch.zeros_like(vel)
    for r in range(idx.shape[1]):
        j = idx[:, r].clamp_min(0)
        ov = o["direction"][j] * o["speed"][j][:, None]
        rel = ov - vel
        fast = rel.norm(dim=-1)
        time = torch.where(fast > 0, _dot(rel, s["position"] - o["position"][j]) / torch.where(fast > 0, fast, torch.ones_like(fast)) ** 2, torch.zeros_like(fast))
        ok = (idx[:, r] >= 0) & (time >= 0) & (time < first)
        there = o["position"][j] + ov * time[:, None]
        at = torch.where(ok[:, None], there, at)
        ok = ok & ((s["position"] + vel * time[:, None] - there).norm(dim=-1) < s["radius"] + o["radius"][j])
        first, threat = torch.where(ok, time, first), torch.where(ok, idx[:, r], threat)
    j = threat.clamp_min(0)
    along = _dot(s["direction"], o["direction"][j])
    look = torch.where((along < -0.707)[:, None], at, o["position"][j]) - s["position"]
    turn = torch.where(_dot(look, s["side"]) > 0, -1.0, 1.0).double()
    slow = s["speed"] <= o["speed"][j]
    across = torch.where(slow, torch.where(_dot(s["side"], o["direction"][j] * o["speed"][j][:, None]) > 0, -1.0, 1.0).double(), torch.zeros_like(turn))
    turn = torch.where(along.abs() > 0.707, turn, across)
    r = torch.where((threat >= 0)[:, None], _unit(s["side"] * turn[:, None]) * w, torch.zeros_like(vel))
    return _apply64(r, BIT[AVOID], steer, applied, mask | CLOSE_BIT)


def _crowd_step64(s, p, scene, segments, of):
    s = dict(s, position=_wrap64(s["position"], p.world_size, p.wrap_mode))
    idx, _ = _binned64(s["position"], s["position"], p.world_size, p.world_cells, 1, p.k, True, scene, scene)
    lines, _ = _binned64(s["position"], 0.5 * (segments[:, 0:3] + segments[:, 3:6]), p.world_size, p.world_cells, 1, p.knw, False, scene, of)
    s, steer, applied = _avoid_walls64(s, p, lines, segments)
    steer, applied = _avoid64(s, s, idx, p.min_time_to_collision, p.w_avoid, p.mask_avoid, steer, applied)
    steer, applied = _flocking64(SEPARATION, s, s, idx, p.sep_min, p.sep_max, p.sep_cos, p.w_sep, steer, applied, p.mask_sep)
    goal = torch.tensor(p.seek_target, device="cuda", dtype=torch.float64)
    steer, applied = _apply64(_unit(goal - s["position"] - s["direction"]) * p.w_seek, BIT[SEEK], steer, applied, p.mask_seek)
    return _integrate64(s, steer, p.dt)


def _avoid_close64(s, o, idx, dist, min_sep, w, mask, steer, applied):
    r = torch.zeros_like(steer)
    found = torch.zeros(idx.shape[0], dtype=torch.bool, device="cuda")
    for c in range(idx.shape[1]):
        j = idx[:, c].clamp_min(0)
        hit = ~found & (idx[:, c] >= 0) & (dist[:, c] < min_sep + s["radius"] + o["radius"][j])
        away = s["position"] - o["position"][j]
        away = away - s["direction"] * _dot(away, s["direction"])[:, None]
        r = torch.where(hit[:, None], away, r)
        found = found | hit
    return _apply64(_unit(r) * w, CLOSE_BIT, steer, applied, mask)


def _groups64(case, seed):
    w, c, k, G = _world(case), case["cells"], case["k"], GROUP
    size, cells = (w, w, w), (c, c, c)
    S = []
    for i, m in enumerate(_group_sizes(case)):
        first = _boids(m, seed, w, _group_ball(case), 0.9, i)
        s = {n: first[n].double() for n in NAMES if n != "applied"}
        S.append(dict(s, position=s["position"][:, :3], direction=s["direction"][:, :3]))
    bits = [torch.zeros(s["speed"].shape[0], dtype=torch.long, device="cuda") for s in S]
    for _ in range(case["frames"]):
        for i, s in enumerate(S):
            S[i] = dict(s, position=_wrap64(s["position"], size, G["wrap_mode"]))
            bits[i] = torch.zeros_like(bits[i])
        lists = [[_binned64(a["position"], b["position"], size, cells, 1, k, a is b) for b in S] for a in S]
        for i in range(len(S)):
            s, steer, applied = S[i], torch.zeros_like(S[i]["position"]), bits[i]
            for j, o in enumerate(S):
                if j != i:
                    steer, applied = _avoid_close64(s, o, *lists[i][j], G["min_separation_distance"], G["w_avoid"], G["mask_avoid"], steer, applied)
                    steer, applied = _avoid64(s, o, lists[i][j][0], G["min_time_to_collision"], G["w_avoid"], G["mask_avoid"], steer, applied)
            for j, o in enumerate(S):
                steer, applied = _flocking64(SEPARATION, s, o, lists[i][j][0], G["sep_min"], G["sep_max"], G["sep_cos"], G["w_sep"], steer, applied, G["mask_sep"])
            for code, key in ((ALIGNMENT, "ali"), (COHESION, "coh")):
                steer, applied = _flocking64(code, s, s, lists[i][i][0], G[key + "_min"], G[key + "_max"], G[key + "_cos"], G["w_" + key], steer, applied, G["mask_" + key])
            s = _integrate64(s, steer, G["dt"])
            applied = torch.zeros_like(applied)
            for j in range(len(S)):
                o, ob = (s, applied) if j == i else (S[j], bits[j])
                near, d = lists[i][j][0][:, 0], lists[i][j][1][:, 0]
                b = near.clamp_min(0)
                over = s["radius"] + o["radius"][b] - d
                hit = ((applied & G["mask_antipen"]) == 0) & (near >= 0) & ~(over < 0)
                move = torch.where((ob[b] & G["mask_antipen"]) != 0, over, 0.5 * over)
                pos = s["position"] + _unit(s["position"] - o["position"][b]) * torch.where(hit, move, torch.zeros_like(move))[:, None]
                s, applied = dict(s, position=pos), torch.where(hit, applied | 8192, applied)
            S[i], bits[i] = s, applied
    return [dict(_told64(s), applied=None) for s in S]
