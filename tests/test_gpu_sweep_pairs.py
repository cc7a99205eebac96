"""Sweep pairs per relabel while more than 16 tiles per SM are active: at most 4,
or, with a negative number, exactly as many as the caller asks for.  Batches of
chains in which excess moves a tile per sweep tell the cycles apart."""
import pytest

from cugip_b200._lib import CgcError
from cugip_b200.graph_cut import Batch, Policy

pytestmark = pytest.mark.gpu


class Chains:
    """A batch of 2400 equal chains of some tiles, excess in the first and the
    sink behind the last; solve() returns the statistics."""
    count = 2400

    def __init__(self, tiles):
        import torch
        n = 8 * tiles
        self.caps = torch.zeros((3, n), dtype=torch.int32, device="cuda")
        self.caps[0, 0], self.caps[1, -1], self.caps[2, :-1] = 5, 9, 6
        torch.cuda.synchronize()
        self.batch = Batch([(n, 1, 1)] * self.count)
        p = [c.data_ptr() for c in self.caps]
        for i in range(self.count):
            self.batch.bind_inputs(i, p[0], p[1], [p[2], None, None])

    def solve(self, policy):
        self.batch.enqueue(policy)
        assert self.batch.wait() == [5] * self.count
        return self.batch.stats()

    def __enter__(self):
        return self

    def __exit__(self, *a):
        self.batch.close()


@pytest.mark.parametrize("exclusive", [0, 1])
def test_pairs_of_dense_cycles(exclusive):
    with Chains(12) as c:
        # 12 sweeps bring the flow to the sink: one cycle of 8 pairs, two of 4, three
        # of 2; a last relabel finds nothing active
        for pairs, cycles in ((-8, 1), (-16, 1), (-4, 2), (-2, 3), (2, 3), (4, 2), (8, 2), (16, 2), (0, 2)):
            st = c.solve(Policy(sweeps_per_relabel=pairs, exclusive=exclusive))
            assert st["global_relabels"] == cycles + 1, (pairs, st)


def test_negative_pairs_elsewhere():
    """Fewer tiles, the host-driven schedule and generic graphs: n pairs as with n."""
    from cugip_b200.graph_cut import GenericGraph
    from oracle import oracle
    from tests import graphs
    from tests.gpu_helpers import solve
    X, Y, Z = 40, 33, 21
    c = graphs.random_grid(X, Y, Z, 3)
    f0 = oracle.maxflow_grid(X, Y, Z, *c)[0]
    e = graphs.grid_edges(X, Y, Z, c[2], c[3])
    for persistent in (1, -1):
        stats = [solve(X, Y, Z, *c, Policy(sweeps_per_relabel=k, persistent=persistent)) for k in (3, -3)]
        assert [s[0] for s in stats] == [f0, f0]
        assert stats[0][3]["sweeps"] == stats[1][3]["sweeps"]
        assert stats[0][3]["global_relabels"] == stats[1][3]["global_relabels"]
    with GenericGraph(X * Y * Z, *e) as g:
        g.set_tweights(c[0], c[1])
        assert g.max_flow(Policy(sweeps_per_relabel=-3)) == f0


@pytest.mark.parametrize("max_sweeps", [1, 16, 17, 32])
@pytest.mark.parametrize("pairs", [0, 8, 16])
def test_limit_on_sweeps_allows_what_full_cycles_would(pairs, max_sweeps):
    """A limit is checked before each cycle, so cycles of n pairs run it up to the
    next multiple of 2n sweeps; shortened cycles must not stop a solve earlier,
    and must still stop one that needs much more."""
    full = 2 * (pairs or 8)
    allowed = -(-max_sweeps // full) * full
    with Chains(allowed) as c:  # a tile per sweep: the last allowed sweep delivers the flow
        c.solve(Policy(sweeps_per_relabel=pairs, max_sweeps=max_sweeps))
    with Chains(allowed + 2 * full) as c:
        c.batch.enqueue(Policy(sweeps_per_relabel=pairs, max_sweeps=max_sweeps))
        with pytest.raises(CgcError) as e:
            c.batch.wait()
        assert e.value.code == 5  # CGC_ERR_NOT_CONVERGED
