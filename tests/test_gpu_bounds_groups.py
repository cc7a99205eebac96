"""The bounds-checked build (libcgc_bounds.so) on sizes at which the solve visits
tiles by groups and by warps, hands out more entries than groups and uploads
batches by runs, and warp relabels beyond 16-bit heights in both builds; every
solve must be exact, and the checked build must report no index out of range."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BOUNDS_LIB = os.path.join(ROOT, "cugip_b200", "libcgc_bounds.so")

CHILD = r"""
import numpy as np
from cugip_b200 import _lib, scheduler
from cugip_b200.graph_cut import SINK, SOURCE, Batch, Policy
from oracle import oracle
from tests import graphs
from tests.gpu_helpers import solve
from tests.test_gpu_bounds_groups import solve_snakes
assert _lib.LIB_PATH.endswith("libcgc_bounds.so"), _lib.LIB_PATH
scheduler.load_weights()
policies = [None, Policy(relabel=1), Policy(persistent=-1), Policy(exclusive=1), Policy(learned=3),
            Policy(local_pulses=2, region_relabels=4, sweeps_per_relabel=-3, stall_sweeps=2)]
# 3150 tiles (more than four per SM, the sweeps' lists too), 980 flat ones, and 350: sweeps of group visits only
for (X, Y, Z), seed in [((118, 117, 111), 5), ((217, 273, 1), 6), ((53, 40, 76), 7)]:
    capS, capT, fwd, bwd = graphs.random_grid(X, Y, Z, seed)
    f0, s0, t0, _ = oracle.maxflow_grid(X, Y, Z, capS, capT, fwd, bwd)
    for pol in policies:
        flow, smin, treach, _ = solve(X, Y, Z, capS, capT, fwd, bwd, pol)
        assert flow == f0 and np.array_equal(smin, s0) and np.array_equal(treach, t0), ((X, Y, Z), pol)
dims = [(33, 17, 9), (8, 8, 8), (70, 65, 40), (1, 1, 1), (9, 64, 3), (41, 40, 39)]
cases = [graphs.random_grid(*d, 20 + i) for i, d in enumerate(dims)]
want = [oracle.maxflow_grid(*d, *c) for d, c in zip(dims, cases)]
for pol in policies:
    b = Batch(dims)
    for i, c in enumerate(cases):
        b.set_tweights(i, c[0], c[1])
        for ax in range(3):
            b.set_nweights(i, ax, c[2][ax], c[3][ax])
    assert b.max_flow(pol) == [w[0] for w in want], pol
    for i, w in enumerate(want):
        assert np.array_equal(b.fill_segments(i, 1, 0, SOURCE), w[1]), (pol, i)
        assert np.array_equal(b.fill_segments(i, 1, 0, SINK), w[2]), (pol, i)
    b.close()
solve_snakes(2)
print("bounds ok")
"""


def test_bounds_checked_build_at_group_and_warp_sizes():
    if not os.path.exists(BOUNDS_LIB):
        pytest.skip("libcgc_bounds.so is not built (cugip_b200/build.py --bounds-check)")
    env = dict(os.environ, CGC_LIBRARY=BOUNDS_LIB, PYTHONPATH=ROOT)
    out = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True,
                         timeout=900)
    assert out.returncode == 0, out.stdout[-3000:] + out.stderr[-3000:]
    assert "bounds ok" in out.stdout


def solve_snakes(relabel):
    """650 paths side by side, each through all voxels of a column of 32 tiles: 16384
    steps, so that the tiles at a path's far end have heights beyond 16 bits, in
    more tiles at a time than there are tile groups.  Five units enter each path
    at its far end, the sink is at the other."""
    from cugip_b200.graph_cut import SINK, SOURCE, GridGraph, Policy
    X, Y, Z = 256, 8 * 26, 8 * 25
    pos = np.arange(64).reshape(8, 8)  # order of a column's rows (z, y) at even x; reversed at odd x
    pos[1::2] = pos[1::2, ::-1]
    pos = np.tile(pos, (Z // 8, Y // 8))
    x = np.arange(X)
    at = 64 * x + np.where(x % 2 == 0, pos[..., None], 63 - pos[..., None])  # position on the path, [z, y, x]
    capS, capT = np.where(at == 64 * X - 1, 5, 0), np.where(at == 0, 9, 0)
    fwd = []
    for axis in (2, 1, 0):  # x, y, z: linked where the path goes on, inside a column
        nxt = np.roll(at, -1, axis)
        link = np.abs(nxt - at) == 1
        edge = [slice(None)] * 3
        if axis == 2:
            edge[2] = -1
        else:
            edge[axis] = slice(7, None, 8)
        link[tuple(edge)] = False
        fwd.append(np.where(link, 6, 0))
    with GridGraph(X, Y, Z) as g:
        g.set_tweights(capS, capT)
        for ax in range(3):
            g.set_nweights(ax, fwd[ax])
        assert g.max_flow(Policy(relabel=relabel)) == 5 * 650
        assert np.array_equal(g.labels().reshape(at.shape), at + 1)
        assert not g.fill_segments(mask=1, which=SOURCE).any()
        assert g.fill_segments(mask=1, which=SINK).all()


@pytest.mark.parametrize("relabel", [1, 2])
def test_warp_relabels_beyond_16_bits(relabel):
    solve_snakes(relabel)
