"""Cycles of a persistent solve that has more than 16 active tiles per SM end
after 4 sweep pairs, except where the limit on sweeps may be met in them."""
import numpy as np
import pytest

from cugip_b200.graph_cut import SINK, SOURCE, Batch, Policy
from oracle import oracle
from tests import graphs
from tests.gpu_helpers import solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [3, 5, 8])
def test_dense_cycles_match_the_oracle(pairs):
    X, Y, Z = 118, 117, 111  # 3150 tiles
    capS, capT, fwd, bwd = graphs.random_grid(X, Y, Z, 5)
    f0, s0, t0, _ = oracle.maxflow_grid(X, Y, Z, capS, capT, fwd, bwd)
    flow, smin, treach, _ = solve(X, Y, Z, capS, capT, fwd, bwd, Policy(sweeps_per_relabel=pairs))
    assert flow == f0
    assert np.array_equal(smin, s0)
    assert np.array_equal(treach, t0)


@pytest.mark.parametrize("max_sweeps", [1, 17, 0])
def test_full_cycle_at_the_limit_on_sweeps(max_sweeps):
    """2800 chains of 12 tiles: excess moves a tile per sweep, so the flow
    arrives in the first cycle if it has 8 sweep pairs and not if it has 4."""
    n, chains = 96, 2800
    capS, capT = np.zeros(n, np.int32), np.zeros(n, np.int32)
    capS[0], capT[-1] = 5, 9
    link = np.full(n, 6, np.int32)
    link[-1] = 0
    b = Batch([(n, 1, 1)] * chains)
    try:
        for i in range(chains):
            b.set_tweights(i, capS, capT)
            b.set_nweights(i, 0, link, link)
        assert b.max_flow(Policy(sweeps_per_relabel=8, max_sweeps=max_sweeps)) == [5] * chains
        for i in (0, chains - 1):
            assert not b.fill_segments(i, 1, 0, SOURCE).any()
            assert b.fill_segments(i, 1, 0, SINK).all()
    finally:
        b.close()
