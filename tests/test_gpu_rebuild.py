"""The database rebuild in one cluster, and brute force over the cells of an
automatic grid, against the oracle's lists: sizes about the cluster's threads,
its dispatch and brute force's, grids whose cell counts leave a remainder,
extents of one, two and three axes, positions that are not finite, queries far
from every candidate, one point many times."""
from __future__ import annotations

import numpy as np
import pytest

import gpusteer_gb300 as gs
import oracle_lib as ol
from gpusteer_gb300 import scenario as sc
from gpusteer_gb300.state import AgentState

pytestmark = pytest.mark.gpu


def state(p):
    s = AgentState.zeros(p.shape[0])
    s.position[:, :3] = p
    s.radius[:] = s.mass[:] = s.max_speed[:] = s.max_force[:] = 1.0
    return s


def group(s, k):
    g = gs.AgentGroup(k, s.n)
    g.upload(s)
    return g


@pytest.mark.parametrize("n", [1, 31, 1024, 16385, 32768, 32769])
@pytest.mark.parametrize("wc", [(1, 1, 1), (7, 3, 5), (41, 41, 41), (130, 1, 131), (64, 32, 65)])
def test_rebuild_twice(n, wc):
    rng = np.random.default_rng(n + wc[0])
    ws = (60.0, 60.0, 60.0)
    bins = gs.KNNBinData(wc, ws, 1)
    s = state(rng.uniform(-31, 31, (n, 3)).astype(np.float32))
    g = group(s, 4)
    for _ in range(2):  # the second finds the counts the first has cleared
        gs.updateKNNDatabase(g, bins)
    from gpusteer_gb300.groups import cell_density
    np.testing.assert_array_equal(cell_density(g, bins), ol.cell_density(s.position, ws, wc))
    if n <= 1024 or wc[0] > 40:
        knn = gs.KNNData(n, 4)
        gs.findKNearestNeighbors(g, knn, bins, g, 1)
        wi, wd = ol.knn_binned(s.position, s.position, True, ws, wc, 1, 4)
        got = knn.download(g)
        np.testing.assert_array_equal(got[0], wi)
        np.testing.assert_array_equal(got[1], wd)


def brute(P, Q, k, same):
    a = group(state(P), k)
    b = a if same else group(state(Q), k)
    knn = gs.KNNData(P.shape[0], k)
    gs.findKNearestNeighborsBruteForce(a, knn, b)
    got = knn.download(a)
    pa, pb = state(P).position, state(Q).position
    want = ol.knn_brute(pa, pb, same, k)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("k", [1, 7, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("n", [127, 128, 1000, 4097])
def test_brute_sizes(n, k):
    P = np.random.default_rng(n + k).uniform(-50, 50, (n, 3)).astype(np.float32)
    brute(P, P, k, True)


@pytest.mark.parametrize("shape", ["line", "plane", "point", "clusters", "far", "tiny", "huge", "nan", "inf", "few"])
@pytest.mark.parametrize("k", [8, 16, 40])
def test_brute_shapes(shape, k):
    rng = np.random.default_rng(k)
    P = rng.normal(0, 10, (900, 3)).astype(np.float32)
    Q, same = P, True
    if shape == "line":
        P[:, 1:] = 0
    elif shape == "plane":
        P[:, 1] = 3
    elif shape == "point":
        P[:] = (1.5, -2.0, 0.25)
    elif shape == "clusters":  # most cells empty: the box grows
        P = (rng.integers(-3, 3, (900, 3)) * 40 + rng.normal(0, 0.01, (900, 3))).astype(np.float32)
        Q = P
    elif shape == "far":  # queries outside every cell, and about one in ten
        Q, same = P[:500] * 0.1, False
        P = P + np.float32([1000, 0, 0])
        P[::10] = Q[:90]
    elif shape == "tiny":
        P *= np.float32(1e-30)
        Q = P
    elif shape == "huge":
        P *= np.float32(1e17)
        Q = P
    elif shape == "nan":
        P[::50] = np.nan
        P[7, 1] = np.nan
    elif shape == "inf":
        P[::50, 0] = np.inf
        P[3] = -np.inf
    elif shape == "few":
        Q, same = P[:k + 1], False
    brute(P, Q, k, same)
