"""Lanes per vertex of the generic engine (4, 8 or 16 by the average degree):
degrees around the limits, vertices with far more and far fewer arcs than
lanes, and vertex counts around a warp's and a CTA's worth of slots; flow and
both cut sets against the oracle."""
import numpy as np
import pytest

from cugip_b200.graph_cut import SINK, SOURCE, GenericGraph
from oracle import oracle

pytestmark = pytest.mark.gpu


def check(n, a, b, f, w, s, t):
    f0, s0, t0, _ = oracle.maxflow_edges(n, a, b, f, w, s, t)
    with GenericGraph(n, a, b, f, w) as g:
        g.set_tweights(s, t)
        assert g.max_flow() == f0
        assert np.array_equal(g.fill_segments(mask=1, which=SOURCE), s0)
        assert np.array_equal(g.fill_segments(mask=1, which=SINK), t0)


@pytest.mark.parametrize("n", [31, 257, 1025, 9500])
@pytest.mark.parametrize("degree", [1, 5, 6, 11, 12, 40])
def test_average_degrees(n, degree):
    rng = np.random.default_rng(100 * n + degree)
    m = (n * degree + 1) // 2
    a, b = rng.integers(0, n, m), rng.integers(0, n, m)
    f, w = rng.integers(0, 40, m), rng.integers(0, 40, m)
    s = rng.integers(0, 60, n) * (rng.random(n) < 0.3)
    t = rng.integers(0, 60, n) * (rng.random(n) < 0.3)
    check(n, a, b, f, w, s, t)


@pytest.mark.parametrize("leaves", [3, 16, 33, 700])
def test_hubs(leaves):
    """Two hubs joined by an edge, each with its leaves: excess enters at one
    side's leaves and leaves at the other's, far more arcs than lanes."""
    rng = np.random.default_rng(leaves)
    n = 2 + 2 * leaves
    left, right = np.arange(2, 2 + leaves), np.arange(2 + leaves, n)
    a = np.concatenate([left, np.zeros(leaves, int) + 1, [0]])
    b = np.concatenate([np.zeros(leaves, int), right, [1]])
    f = np.concatenate([rng.integers(1, 9, 2 * leaves), [3 * leaves]])
    s, t = np.zeros(n, int), np.zeros(n, int)
    s[left] = rng.integers(1, 12, leaves)
    t[right] = rng.integers(1, 12, leaves)
    check(n, a, b, f, f, s, t)
