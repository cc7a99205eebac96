"""Tile visits of the persistent solve where the dispatch changes: sweeps of at
most / more than one tile per SM (512-thread and 128-thread visits), relabel
rounds of at most / more than one tile per group (128-thread and warp visits),
several rounds per group, and heights on both sides of the
16-bit relaxations' range.  Flow and both cut sets against the oracle."""
import numpy as np
import pytest

from cugip_b200.graph_cut import SINK, SOURCE, Batch, Policy
from oracle import oracle
from tests import graphs
from tests.gpu_helpers import solve

pytestmark = pytest.mark.gpu

# tiles in all, so about half of them in a sweep: 1, 288 (just under an SM's worth per sweep), 336 (just over),
# 1200 (several rounds per group), and ragged and thin shapes around them
SHAPES = [(8, 8, 8), (48, 48, 64), (56, 48, 64), (80, 80, 96), (47, 41, 63), (129, 3, 66), (300, 17, 2)]
POLICIES = [None, Policy(local_pulses=3, region_relabels=-1), Policy(local_pulses=5, relabel=1),
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


@pytest.mark.parametrize("chains", [1, 160])
def test_heights_beyond_16_bits(chains):
    """Chains of 15 400 voxels: distances to the sink pass the 16-bit range (in
    one tile per round and in more tiles than SMs), and a unit of flow crosses
    all of it.  A link of capacity 3 is the minimum cut."""
    n = 15400
    capS, capT = np.zeros(n, np.int32), np.zeros(n, np.int32)
    capS[-1], capT[0] = 7, 5
    fwd, bwd = np.full(n, 2, np.int32), np.full(n, 9, np.int32)
    fwd[-1] = bwd[-1] = 0
    bwd[n - 40] = 3
    z = np.zeros(n, np.int32)
    f0, s0, t0, _ = oracle.maxflow_grid(n, 1, 1, capS, capT, [fwd, z, z], [bwd, z, z])
    assert f0 == 3
    b = Batch([(n, 1, 1)] * chains)
    try:
        for i in range(chains):
            b.set_tweights(i, capS, capT)
            b.set_nweights(i, 0, fwd, bwd)
        assert b.max_flow(Policy(sweeps_per_relabel=1000)) == [f0] * chains
        for i in {0, chains - 1}:
            assert np.array_equal(b.fill_segments(i, 1, 0, SOURCE), s0)
            assert np.array_equal(b.fill_segments(i, 1, 0, SINK), t0)
    finally:
        b.close()
