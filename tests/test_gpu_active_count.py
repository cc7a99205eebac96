"""The number of active tiles decides a cycle's length and whether the learned
scheduler's stage runs, so every CTA has to see the same number although the
first sweep activates further tiles at once.  Batches of chains at and around
both limits: the solves end (no barrier times out), give the known flow and
cut sets, and repeat their numbers of sweeps and relabels."""
import numpy as np
import pytest

from cugip_b200 import scheduler
from cugip_b200.graph_cut import Batch, Policy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exclusive", [0, 1])
@pytest.mark.parametrize("learned", [0, 1])
@pytest.mark.parametrize("per_sm", [8, 16])  # the stage's limit and the cycle length's
@pytest.mark.parametrize("off", [-1, 0, 1])
def test_decisions_at_the_limits(per_sm, off, learned, exclusive):
    import torch
    if learned:
        scheduler.load_weights()
    n = 24  # a chain of three tiles: excess in the first, the sink behind the last
    count = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + off
    caps = torch.zeros((3, n), dtype=torch.int32, device="cuda")
    caps[0, 0], caps[1, -1], caps[2, :-1] = 5, 9, 6
    sides = torch.full((4, n), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    b = Batch([(n, 1, 1)] * count)
    try:
        for i in range(count):
            b.bind_inputs(i, caps[0].data_ptr(), caps[1].data_ptr(), [caps[2].data_ptr(), None, None])
        b.bind_outputs(0, sides[0].data_ptr(), sides[1].data_ptr())
        b.bind_outputs(count - 1, sides[2].data_ptr(), sides[3].data_ptr())
        seen = set()
        for _ in range(8):
            b.enqueue(Policy(wait_limit_us=2_000_000, learned=learned, exclusive=exclusive))
            assert b.wait() == [5] * count
            assert np.array_equal(sides.cpu().numpy(), np.repeat([[0], [1], [0], [1]], n, 1))
            st = b.stats()
            seen.add((st["sweeps"], st["global_relabels"]))
        assert len(seen) == 1, seen
    finally:
        b.close()
