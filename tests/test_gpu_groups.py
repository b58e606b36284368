"""gs_multigroup_step against the same frames through the per-function calls,
bit for bit: one to seven groups of uneven sizes (one empty), list lengths
about the lane-group sizes and past them, avoid-close on and off, masks that
see the bits of earlier calls."""
from __future__ import annotations

import numpy as np
import pytest

import gpusteer_gb300 as gs
from gpusteer_gb300 import scenario as sc

pytestmark = pytest.mark.gpu
FIELDS = ("position", "direction", "steering", "side", "up", "speed", "applied")


@pytest.mark.parametrize("sizes,k,close,masks", [
    ((1500,), 8, 1, 0), ((700, 333), 1, 0, 0), ((900, 1, 450), 9, 1, 1), ((400, 0, 300), 16, 1, 0),
    ((300,) * 7, 17, 0, 1), ((500, 200), 40, 1, 0)])
def test_frames_equal_the_calls(sizes, k, close, masks):
    p = sc.boids_params(k=k, world=96.0, cell=4.0)
    G, frames = len(sizes), 3
    states = []
    for i, n in enumerate(sizes):
        s = sc.boids_sphere(max(n, 1), radius=12.0, seed=60 + i)
        s = s.subset(np.arange(n))
        s.radius[:] = np.float32(0.9)
        states.append(s)
    m = dict(world_size=p.world_size, wrap_mode=sc.WRAP_REFERENCE, min_time_to_collision=2.0,
             min_separation_distance=0.5, avoid_close=close, w_avoid=1.0,
             mask_avoid=16 if masks else 0, sep_min=p.sep_min, sep_max=p.sep_max, sep_cos=p.sep_cos,
             w_sep=p.w_sep, mask_sep=512 if masks else 0, ali_min=p.ali_min, ali_max=p.ali_max,
             ali_cos=p.ali_cos, w_ali=p.w_ali, mask_ali=272, coh_min=p.coh_min, coh_max=p.coh_max,
             coh_cos=p.coh_cos, w_coh=p.w_coh, mask_coh=272, path_prediction_time=5.0, w_path=1.0,
             mask_path=16, w_seek=1.5, mask_seek=4480, mask_antipen=8192 if masks else 4096,
             dt=1.0 / 30.0)
    bins = gs.KNNBinData(p.world_cells, p.world_size, 1)
    pts = [(0.0, 0.0, 0.0), (30.0, 5.0, -20.0), (-10.0, 20.0, 30.0)]
    path = gs.Path(pts, 6.0)
    paths = [path if i % 2 == 0 else None for i in range(G)]

    def make():
        groups = []
        for s in states:
            g = gs.AgentGroup(k, max(1, s.n))
            g.upload(s)
            groups.append(g)
        return groups, [[gs.KNNData(max(0, s.n), k) if s.n else gs.KNNData(0, k) for _ in range(G)]
                        for s in states]

    fused, kf = make()
    gs.multigroup_step(fused, bins, kf, gs.MultiGroupParams(**m), frames, paths=paths)
    groups, kp = make()
    for _ in range(frames):
        for g in groups:
            gs.wrapWorld(g, p.world_size, sc.WRAP_REFERENCE)
            st = g.download()
            st.applied[:] = 0
            g.upload(st)
            gs.updateKNNDatabase(g, bins)
        for i, g in enumerate(groups):
            if not states[i].n:
                continue
            for j, o in enumerate(groups):
                gs.findKNearestNeighbors(g, kp[i][j], bins, o, 1)
            for j, o in enumerate(groups):
                if j != i:
                    gs.steerToAvoidNeighbors(g, kp[i][j], o, m["min_time_to_collision"],
                                             m["min_separation_distance"], close, m["w_avoid"],
                                             m["mask_avoid"])
            for j, o in enumerate(groups):
                gs.steerForSeparation(g, kp[i][j], o, m["sep_min"], m["sep_max"], m["sep_cos"],
                                      m["w_sep"], m["mask_sep"])
            gs.steerForAlignment(g, kp[i][i], g, m["ali_min"], m["ali_max"], m["ali_cos"],
                                 m["w_ali"], m["mask_ali"])
            gs.steerForCohesion(g, kp[i][i], g, m["coh_min"], m["coh_max"], m["coh_cos"],
                                m["w_coh"], m["mask_coh"])
            if paths[i] is not None:
                gs.steerToFollowPath(g, path, m["path_prediction_time"], m["w_path"], m["mask_path"])
                gs.steerForSeek(g, pts[1], m["w_seek"], m["mask_seek"])
            gs.updateGroup(g, m["dt"])
            for j, o in enumerate(groups):
                gs.antiPenetrationAgents(g, kp[i][j], o, m["mask_antipen"])
    for i in range(G):
        a, b = fused[i].download(), groups[i].download()
        for f in FIELDS:
            np.testing.assert_array_equal(getattr(a, f), getattr(b, f), err_msg=f"group {i} {f}")
