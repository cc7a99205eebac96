"""Tile visits of the persistent solve where the dispatch between 512-thread and
128-thread visits changes (sweeps of at most / more than one tile per SM), and
where groups run several rounds: flow and both cut sets against the oracle."""
import numpy as np
import pytest

from cugip_b200.graph_cut import Policy
from oracle import oracle  # the checker
from tests import graphs
from tests.gpu_helpers import solve

pytestmark = pytest.mark.gpu

# tiles in all, so about half of them in a sweep: 1, 288 (just under an SM's worth per sweep), 336 (just over),
# 1200 (several rounds per group), and ragged and thin shapes around them
SHAPES = [(8, 8, 8), (48, 48, 64), (56, 48, 64), (80, 80, 96), (47, 41, 63), (129, 3, 66), (300, 17, 2)]
POLICIES = [None, Policy(ctas_per_sm=3, local_pulses=3, region_relabels=-1), Policy(ctas_per_sm=4, local_pulses=5),
            Policy(exclusive=1, region_relabels=3, sweeps_per_relabel=2)]


@pytest.mark.parametrize("policy", range(len(POLICIES)))
@pytest.mark.parametrize("dims", SHAPES)
def test_visits_match_the_oracle(dims, policy):
    X, Y, Z = dims
    capS, capT, fwd, bwd = graphs.random_grid(X, Y, Z, 11 * X + Y)
    f0, s0, t0, _ = oracle.maxflow_grid(X, Y, Z, capS, capT, fwd, bwd)
    flow, smin, treach, _ = solve(X, Y, Z, capS, capT, fwd, bwd, POLICIES[policy])
    assert flow == f0
    assert np.array_equal(smin, s0)
    assert np.array_equal(treach, t0)
