"""steerToAvoidNeighbors and steerToAvoidWalls on either side of their dispatches,
against the oracle's whole step, bit for bit, and no dearer on one side of a
former edge than on the other."""
from __future__ import annotations

import pytest

import gpusteer_gb300 as gs
from gpusteer_gb300 import scenario as sc
from test_gpu_calls import crowd_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(56250, 7), (56251, 7), (28125, 16), (28126, 16), (14062, 32), (14063, 32),
                                 (77824, 7), (77825, 7), (77825, 16)])
@pytest.mark.parametrize("close", [0, 1])
def test_either_side(n, k, close):
    p = sc.chokepoint_params(k=k).replace(avoid_close=close)
    side = 0.9 * n ** 0.5
    s = sc.chokepoint_agents(n, x_range=(-side / 2, side / 2), z_range=(14.0, 14.0 + side), seed=n + k)
    crowd_frames(s, p, 2)


def call_us(n, k):
    import torch

    p = sc.chokepoint_params(k=k)
    side = n ** 0.5
    bins = gs.KNNBinData((256, 1, 256), (768.0, 10.0, 768.0), 1)
    g = gs.AgentGroup(k, n)
    g.upload(sc.chokepoint_agents(n, x_range=(-side / 2, side / 2), z_range=(-side / 2, side / 2), seed=1))
    gs.updateKNNDatabase(g, bins)
    knn = gs.KNNData(n, k)
    gs.findKNearestNeighbors(g, knn, bins, g, 1)
    stream = torch.cuda.ExternalStream(g.stream)
    times = []
    for _ in range(9):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(20):
            gs.steerToAvoidNeighbors(g, knn, g, p.min_time_to_collision, p.min_separation_distance, 0,
                                     p.w_avoid, 0)
        b.record(stream)
        b.synchronize()
        times.append(a.elapsed_time(b) * 50)
    return sorted(times)[4]


@pytest.mark.parametrize("k", [16, 32])
def test_no_cliff_at_65536(k):
    """One agent more took 0.4 (k = 32) to 0.65 (k = 16) of the time."""
    assert call_us(65536, k) < 1.25 * call_us(65537, k)
