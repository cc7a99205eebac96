"""Handles dropped while another thread captures a stream: the capture goes on,
and the memory of a handle whose solve is still queued is not handed out before
that solve has ended (the next handles' answers equal the oracle's)."""
import threading

import numpy as np
import pytest

from cugip_b200.graph_cut import SINK, SOURCE, Batch, GenericGraph, GridGraph
from oracle import oracle
from tests import graphs

pytestmark = pytest.mark.gpu


def upload(g, c):
    g.set_tweights(c[0], c[1])
    for ax in range(3):
        g.set_nweights(ax, c[2][ax], c[3][ax])


def in_thread(f):
    errors = []

    def run():
        try:
            f()
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(repr(e))
    t = threading.Thread(target=run)
    t.start()
    t.join()
    assert not errors, errors


class Captured:
    """A thread-local capture of a torch stream, open while the body runs."""

    def __enter__(self):
        import torch
        self.x = torch.zeros(64, device="cuda")
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        self.ctx = torch.cuda.graph(self.graph, capture_error_mode="thread_local")
        self.ctx.__enter__()
        self.x += 1
        return self

    def __exit__(self, *a):
        import torch
        self.x += 1
        self.ctx.__exit__(*a)
        self.graph.replay()
        torch.cuda.synchronize()
        assert (self.x == 2).all()


def test_idle_handles_beside_a_capture():
    dims = (24, 17, 9)
    c = graphs.random_grid(*dims, 5)
    f0 = oracle.maxflow_grid(*dims, *c)[0]
    g, b = GridGraph(*dims), Batch([dims, dims])
    q = GenericGraph(3, [0, 1], [1, 2], [4, 3], [0, 0])
    upload(g, c)
    for i in range(2):
        b.set_tweights(i, c[0], c[1])
        for ax in range(3):
            b.set_nweights(i, ax, c[2][ax], c[3][ax])
    q.set_tweights([9, 0, 0], [0, 0, 9])
    assert g.max_flow() == f0 and b.max_flow() == [f0, f0] and q.max_flow() == 3
    with Captured():
        in_thread(lambda: [h.close() for h in (g, b, q)])


@pytest.mark.parametrize("through", ["async", "enqueue", "replay"])
def test_queued_solves_beside_a_capture(through):
    """A solve waits behind 50 ms of other work on its stream, its handle is
    dropped, and the next handles are made and solved on another stream."""
    import torch
    dims = (56, 48, 40)
    c = graphs.random_grid(*dims, 6)
    small = (40, 33, 21)
    cs = graphs.random_grid(*small, 7)
    f0, s0, t0, _ = oracle.maxflow_grid(*small, *cs)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()
    planes = [d(c[0]), d(c[1]), [d(a) for a in c[2]], [d(a) for a in c[3]]]
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def drop_and_go_on():
        for _ in range(3):
            if through == "async":
                h = GridGraph(*dims, stream=busy.cuda_stream)
                upload(h, c)
            else:
                h = Batch([dims], stream=busy.cuda_stream)
                h.bind_inputs(0, planes[0].data_ptr(), planes[1].data_ptr(), [p.data_ptr() for p in planes[2]],
                              [p.data_ptr() for p in planes[3]])
                if through == "replay":
                    h.graph_create()
            with torch.cuda.stream(busy):
                torch.cuda._sleep(100_000_000)
            if through == "async":
                h.max_flow_async()
            elif through == "enqueue":
                h.enqueue()
            else:
                h.graph_launch()
            h.close()
            for _ in range(3):
                with GridGraph(*small, stream=other.cuda_stream) as g:
                    upload(g, cs)
                    assert g.max_flow() == f0
                    assert np.array_equal(g.fill_segments(mask=1, which=SOURCE), s0)
                    assert np.array_equal(g.fill_segments(mask=1, which=SINK), t0)

    with Captured():
        in_thread(drop_and_go_on)


def test_solve_in_a_callers_graph_beside_a_capture():
    """The same with the solve captured into a graph of the caller's, which no
    event of the handle follows."""
    import torch
    dims, small = (56, 48, 40), (40, 33, 21)
    c, cs = graphs.random_grid(*dims, 6), graphs.random_grid(*small, 7)
    f0, s0, _, _ = oracle.maxflow_grid(*small, *cs)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()
    planes = [d(c[0]), d(c[1]), [d(a) for a in c[2]], [d(a) for a in c[3]]]
    flow = torch.zeros(1, dtype=torch.int64, device="cuda")
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    h = Batch([dims], stream=busy.cuda_stream)
    h.bind_inputs(0, planes[0].data_ptr(), planes[1].data_ptr(), [p.data_ptr() for p in planes[2]],
                  [p.data_ptr() for p in planes[3]])
    own = torch.cuda.CUDAGraph()
    with torch.cuda.graph(own, stream=busy):
        h.enqueue(None, flow.data_ptr())

    def drop_and_go_on():
        with torch.cuda.stream(busy):
            torch.cuda._sleep(100_000_000)
            own.replay()
        h.close()
        assert busy.query()  # nothing tells when the handle's memory is free but the end of all work
        for _ in range(3):
            with GridGraph(*small, stream=other.cuda_stream) as g:
                upload(g, cs)
                assert g.max_flow() == f0
                assert np.array_equal(g.fill_segments(mask=1, which=SOURCE), s0)

    with Captured():
        in_thread(drop_and_go_on)
    assert int(flow.item()) == oracle.maxflow_grid(*dims, *c)[0]
