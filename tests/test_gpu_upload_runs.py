"""The fused upload (runs of four tiles along x) over its four variants: plane
rows of four voxels aligned or not, symmetric or directed n-links; extents at
the edges of quads, tiles and runs; capacities around the limit of the short
overflow check.  Flow and both cut sets against the oracle."""
import numpy as np
import pytest

from cugip_b200 import _lib
from cugip_b200.graph_cut import SINK, SOURCE, Batch, GridGraph
from oracle import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


def on_device(a, shift):
    """a on the device, `shift` elements off a 16-byte boundary."""
    import torch
    t = torch.zeros(a.size + 8, dtype=torch.int32, device="cuda")
    v = t[shift:shift + a.size]
    v.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return v


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("asym", [False, True])
@pytest.mark.parametrize("dims", [(4, 1, 1), (31, 9, 8), (32, 8, 8), (33, 8, 9), (36, 16, 7), (64, 24, 17), (65, 7, 16),
                                  (100, 18, 24)])
def test_bound_planes_match_the_oracle(dims, asym, shift):
    X, Y, Z = dims
    capS, capT, fwd, bwd = graphs.random_grid(X, Y, Z, 3 * X + Z, asym=asym)
    f0, s0, t0, _ = oracle.maxflow_grid(X, Y, Z, capS, capT, fwd, bwd)
    d = [on_device(a, shift) for a in (capS, capT, *fwd, *(bwd if asym else []))]
    B = Batch([dims, (5, 6, 7)])  # a second instance, so that runs come from the table
    c2 = graphs.random_grid(5, 6, 7, 1)
    d2 = [on_device(a, 0) for a in (c2[0], c2[1], *c2[2], *c2[3])]
    f2 = oracle.maxflow_grid(5, 6, 7, *c2)[0]
    try:
        B.bind_inputs(0, d[0].data_ptr(), d[1].data_ptr(), [t.data_ptr() for t in d[2:5]],
                      [t.data_ptr() for t in d[5:8]] if asym else None)
        B.bind_inputs(1, d2[0].data_ptr(), d2[1].data_ptr(), [t.data_ptr() for t in d2[2:5]],
                      [t.data_ptr() for t in d2[5:8]])
        B.enqueue()
        assert B.wait() == [f0, f2]
        assert np.array_equal(B.fill_segments(0, 1, 0, SOURCE), s0)
        assert np.array_equal(B.fill_segments(0, 1, 0, SINK), t0)
    finally:
        B.close()


@pytest.mark.parametrize("big", [2**28 - 1, 2**28, 2**29])
def test_large_capacities(big):
    """Values on both sides of 2^28, where the full overflow check takes over:
    exact where it fits, CGC_ERR_OVERFLOW and CGC_ERR_ARG where it does not."""
    X, Y, Z = 40, 9, 10
    n = X * Y * Z
    capS, capT, fwd, bwd = graphs.random_grid(X, Y, Z, 5)
    rng = np.random.default_rng(6)
    i = rng.integers(0, n, 40)
    capS[i[:20]] = big
    capT[i[20:]] = big
    fwd[0][:30] = big  # the first row's x links, except past its end
    f0, s0, t0, _ = oracle.maxflow_grid(X, Y, Z, capS, capT, fwd, bwd)
    g = GridGraph(X, Y, Z)
    try:
        def solve():
            g.set_tweights(capS, capT)
            for ax in range(3):
                g.set_nweights(ax, fwd[ax], bwd[ax])
            return g.max_flow()
        assert solve() == f0
        assert np.array_equal(g.fill_segments(mask=1, which=SOURCE), s0)
        bwd[1][7], fwd[1][7] = 2**31 - 1, 1  # a link pair beyond int32
        with pytest.raises(_lib.CgcError) as e:
            solve()
        assert e.value.code == 6
        bwd[1][7], fwd[1][7], capT[3] = 1, 1, -1
        with pytest.raises(_lib.CgcError) as e:
            solve()
        assert e.value.code == 1
    finally:
        g.close()
