"""Brute force where the candidates are no uniform cube about the origin: lists
against the oracle's full scan, and a call's time against the cube's."""
from __future__ import annotations

import numpy as np
import pytest

import gpusteer_gb300 as gs
import oracle_lib as ol
from gpusteer_gb300.state import AgentState

pytestmark = pytest.mark.gpu


def shape(name, n, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(-256, 256, (n, 3))
    if name == "outlier":
        p[n // 2] = (1e6, 5.0, -3e5)
    elif name == "far":
        p[:n // 100] *= 1000
    elif name == "nan":
        p[n // 3, 1] = np.nan
    elif name == "inf":
        p[n // 3, 0], p[n // 4, 2] = np.inf, -np.inf
    elif name == "offset":
        p = p * 0.01 + 1000.0
    elif name == "clusters":
        c = rng.uniform(-5000, 5000, (10, 3))
        p = c[rng.integers(0, 10, n)] + rng.normal(0, 10, (n, 3))
    elif name == "heavy":
        p = rng.standard_cauchy((n, 3)) * 10
    elif name == "many nan":
        p[rng.random(n) < 0.3] = np.nan
    elif name == "lattice":
        p = np.round(p / 32) * 32
    return p.astype(np.float32)


def group(p, k):
    s = AgentState.zeros(p.shape[0])
    s.position[:, :3] = p
    s.radius[:] = s.mass[:] = s.max_speed[:] = s.max_force[:] = 1.0
    g = gs.AgentGroup(k, s.n)
    g.upload(s)
    return g, s.position


SHAPES = ["outlier", "far", "nan", "inf", "offset", "clusters", "heavy", "many nan", "lattice"]


@pytest.mark.parametrize("name", SHAPES)
@pytest.mark.parametrize("n,k", [(1025, 7), (6001, 16), (3000, 33)])
def test_lists(name, n, k):
    g, pos = group(shape(name, n, n + k), k)
    o, opos = group(shape(name, n // 2, n), k)
    for b, bpos, same in ((g, pos, True), (o, opos, False)):
        knn = gs.KNNData(n, k)
        gs.findKNearestNeighborsBruteForce(g, knn, b)
        idx, dist = knn.download(g)
        wi, wd = ol.knn_brute(pos, bpos, same, k)
        np.testing.assert_array_equal(idx, wi)
        np.testing.assert_array_equal(dist, wd)


def pairs_per_query(name, n, k):
    g, _ = group(shape(name, n, 1), k)
    gs.findKNearestNeighborsBruteForce(g, gs.KNNData(n, k), g)
    return gs.bruteforce_pairs(g) / n


@pytest.mark.parametrize("name", ["outlier", "far", "nan", "inf", "offset"])
def test_a_few_far_or_broken_positions_cost_little(name):
    """65,536 agents: with a grid over the extent each of these met nearly every
    pair, 65,000 a query."""
    assert pairs_per_query(name, 65536, 16) < 5 * pairs_per_query("cube", 65536, 16)
