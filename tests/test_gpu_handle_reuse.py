"""Handles whose device memory was used by earlier handles: grids, batches and
generic graphs made, solved and dropped in turn by several threads on streams
of their own, some dropped with a solve still queued; every answer against the
oracle."""
import threading

import numpy as np
import pytest

from cugip_b200.graph_cut import SINK, SOURCE, Batch, GenericGraph, GridGraph
from oracle import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


def test_threads_and_streams_share_freed_memory():
    import torch
    dims = [(17, 9, 12), (40, 33, 21), (64, 64, 5), (8, 8, 8)]
    cases = []
    for k, d in enumerate(dims):
        c = graphs.random_grid(*d, 70 + k)
        cases.append((d, c, oracle.maxflow_grid(*d, *c)))
    n, m = 900, 4000
    rng = np.random.default_rng(3)
    edges = [rng.integers(0, n, m), rng.integers(0, n, m), rng.integers(0, 30, m), rng.integers(0, 30, m)]
    term = [rng.integers(0, 50, n), rng.integers(0, 50, n)]
    f_edges = oracle.maxflow_edges(n, *edges, *term)[0]
    errors = []

    def upload(g, c):
        g.set_tweights(c[0], c[1])
        for ax in range(3):
            g.set_nweights(ax, c[2][ax], c[3][ax])

    def work(seed):
        try:
            stream = torch.cuda.Stream()
            for i in range(12):
                d, c, (f0, s0, t0, _) = cases[(seed + i) % len(cases)]
                if i % 4 == 3:
                    g = GridGraph(*d, stream=stream.cuda_stream)
                    upload(g, c)
                    g.max_flow_async()
                    g.close()  # dropped with the solve queued
                    with GenericGraph(n, *edges, stream=stream.cuda_stream) as q:
                        q.set_tweights(*term)
                        assert q.max_flow() == f_edges
                elif i % 4 == 2:
                    b = Batch([d, dims[i % 3]], stream=stream.cuda_stream)
                    c2 = cases[i % 3][1]
                    for j, cc in enumerate((c, c2)):
                        b.set_tweights(j, cc[0], cc[1])
                        for ax in range(3):
                            b.set_nweights(j, ax, cc[2][ax], cc[3][ax])
                    assert b.max_flow() == [f0, cases[i % 3][2][0]]
                    assert np.array_equal(b.fill_segments(0, 1, 0, SOURCE), s0)
                    b.close()
                else:
                    with GridGraph(*d, stream=stream.cuda_stream) as g:
                        upload(g, c)
                        assert g.max_flow() == f0
                        assert np.array_equal(g.fill_segments(mask=1, which=SOURCE), s0)
                        assert np.array_equal(g.fill_segments(mask=1, which=SINK), t0)
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
