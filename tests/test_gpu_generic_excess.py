"""Excess of the generic engine while neighbours push into a vertex that is
pushing itself: small dense graphs, so that nearly every active vertex receives
flow in the pulse in which its lanes share out its own.  Nothing is lost or
made: flow delivered plus excess left equals what the source sent, and flow and
cut set are the oracle's."""
import numpy as np
import pytest

from cugip_b200 import _lib
from cugip_b200.graph_cut import SOURCE, GenericGraph, Policy
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pulses", [1, 0])
@pytest.mark.parametrize("n,degree", [(40, 4), (40, 8), (120, 20), (700, 60)])  # 4, 8 and 16 lanes
def test_excess_is_conserved(n, degree, pulses):
    rng = np.random.default_rng(n + degree)
    m = n * degree // 2
    a, b = rng.integers(0, n, m), rng.integers(0, n, m)
    f, w = rng.integers(0, 30, m), rng.integers(0, 30, m)
    s = rng.integers(0, 400, n)
    t = np.zeros(n, int)
    t[rng.integers(0, n, 4)] = 5000
    f0, s0, _, _ = oracle.maxflow_edges(n, a, b, f, w, s, t)
    for _ in range(20):
        with GenericGraph(n, a, b, f, w) as g:
            g.set_tweights(s, t)
            assert g.max_flow(Policy(sweeps_per_relabel=pulses)) == f0
            excess = np.empty(n, np.int32)
            _lib.check(g._lib.cgc_graph_get_state(g._h, None, excess.ctypes.data))
            assert (excess >= 0).all()
            assert f0 + int(excess.sum()) == int(s.sum())
            assert np.array_equal(g.fill_segments(mask=1, which=SOURCE), s0)
