"""Batches with outputs bound for some instances only, made from memory that
earlier batches used for full tables of outputs: only the bound outputs are
written."""
import numpy as np
import pytest

from cugip_b200.graph_cut import Batch
from oracle import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [2, 9, 700])
def test_only_bound_outputs_are_written(count):
    import torch
    dims = (9, 5, 4)
    n = dims[0] * dims[1] * dims[2]
    c = graphs.random_grid(*dims, count)
    f0, s0, t0, _ = oracle.maxflow_grid(*dims, *c)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()
    caps = [d(a) for a in (c[0], c[1], *c[2], *c[3])]
    p = [t.data_ptr() for t in caps]

    def solve(bound):
        sides = torch.full((count, 2, n), 7, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        b = Batch([dims] * count)
        try:
            for i in range(count):
                b.bind_inputs(i, p[0], p[1], p[2:5], p[5:8])
            for i, (src, snk) in bound.items():
                b.bind_outputs(i, sides[i, 0].data_ptr() if src else None, sides[i, 1].data_ptr() if snk else None)
            for _ in range(2):
                b.enqueue()
                assert b.wait() == [f0] * count
        finally:
            b.close()
        want = np.full((count, 2, n), 7, np.uint8)
        for i, (src, snk) in bound.items():
            if src:
                want[i, 0] = s0
            if snk:
                want[i, 1] = t0
        assert np.array_equal(sides.cpu().numpy(), want)
        return sides

    keep = []  # the earlier tables' targets stay allocated
    for _ in range(4):
        keep.append(solve({i: (True, True) for i in range(count)}))
        before = [k.clone() for k in keep]
        keep.append(solve({0: (False, True)}))
        keep.append(solve({count - 1: (True, False), 0: (True, True)}))
        assert all(torch.equal(a, b) for a, b in zip(before, keep))
