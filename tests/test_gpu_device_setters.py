"""Device setters on memory that is not the grid's device's own: pinned host
memory and planes at odd byte addresses go through copy commands at every size,
ordinary device planes of up to 2^18 voxels through one kernel per call (also as
views into an allocation and at its end)."""
import numpy as np
import pytest

from cugip_b200 import _lib
from cugip_b200.graph_cut import SINK, SOURCE, GridGraph
from oracle import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


def planes_of(kind, arrays, keep):
    """Addresses of copies of the arrays in the given kind of memory."""
    import torch
    if kind == "pinned":
        ts = [torch.from_numpy(a).pin_memory() for a in arrays]
    elif kind == "odd":
        ts = []
        for a in arrays:
            buf = torch.zeros(4 * a.size + 1, dtype=torch.uint8, device="cuda")
            buf[1:] = torch.from_numpy(a.view(np.uint8)).cuda()
            ts.append(buf)
        keep.extend(ts)
        return [t.data_ptr() + 1 for t in ts]
    elif kind == "views":  # back to back in one allocation, the last at its end
        whole = torch.from_numpy(np.concatenate(arrays)).cuda()
        keep.append(whole)
        return [whole.data_ptr() + 4 * arrays[0].size * i for i in range(len(arrays))]
    else:
        ts = [torch.from_numpy(a).cuda() for a in arrays]
    keep.extend(ts)
    return [t.data_ptr() for t in ts]


@pytest.mark.parametrize("dims", [(5, 4, 3), (64, 64, 64), (65, 64, 64)])
@pytest.mark.parametrize("kind", ["device", "views", "pinned", "odd"])
def test_memory_of_the_planes(dims, kind):
    import torch
    lib = _lib.load()
    capS, capT, fwd, bwd = graphs.random_grid(*dims, 31)
    f0, s0, t0, _ = oracle.maxflow_grid(*dims, capS, capT, fwd, bwd)
    keep = []
    arrays = [np.ascontiguousarray(a, dtype=np.int32) for a in (capS, capT, *fwd, *bwd)]
    at = planes_of(kind, arrays, keep)
    torch.cuda.synchronize()
    with GridGraph(*dims) as g:
        before = lib.cgc_launch_count()
        g.set_tweights_device(at[0], at[1])
        for ax in range(3):
            g.set_nweights_device(ax, at[2 + ax], at[5 + ax])
        kernels = lib.cgc_launch_count() - before
        small = dims[0] * dims[1] * dims[2] <= 1 << 18
        assert kernels == (4 if small and kind in ("device", "views") else 0)
        assert g.max_flow() == f0
        assert np.array_equal(g.fill_segments(mask=1, which=SOURCE), s0)
        assert np.array_equal(g.fill_segments(mask=1, which=SINK), t0)
