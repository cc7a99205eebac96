"""A generic graph of more than 2^24 vertices, its edges among the last ones."""
import numpy as np
import pytest

from cugip_b200.graph_cut import SINK, SOURCE, GenericGraph

pytestmark = pytest.mark.gpu


def test_edges_beyond_2_to_24_vertices():
    chain = 3000
    n = (1 << 24) + 2 * chain
    a = np.arange(n - chain, n - 1)
    f = np.full(chain - 1, 9)
    f[700] = 4
    s, t = np.zeros(n, np.int32), np.zeros(n, np.int32)
    s[n - chain], t[n - 1] = 8, 7
    s[5], t[6] = 3, 3  # vertices without edges
    with GenericGraph(n, a, a + 1, f, np.zeros(chain - 1, int)) as g:
        g.set_tweights(s, t)
        assert g.max_flow() == 4
        source, sink = g.fill_segments(mask=1, which=SOURCE), g.fill_segments(mask=1, which=SINK)
    at = n - chain + 701  # the first vertex behind the bottleneck
    assert source[5] == 1 and source[n - chain:at].all() and source.sum() == 702
    assert sink[6] == 1 and sink[at:].all() and sink.sum() == 1 + n - at
