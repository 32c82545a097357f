"""Graphs at the edges of what gwf_ed_index takes: the filter of the walks' strings is built for them,
or left out, and the graph is usable either way."""
import pytest

pytestmark = pytest.mark.gpu


def test_graph_without_vertices(G):
    g = G.Graph.from_arrays([], [])
    g.index()
    d, st = g.ed_batch([], [])
    assert len(d) == 0 and len(st) == 0
    with pytest.raises(G.GwfError) as e:  # indexed, but there is no vertex to target
        g.ed_batch([b"ACGT"], [0], v1=0)
    assert e.value.code == G.GWF_E_BAD_INPUT
    d, st = g.ed_batch([b"ACGT"], [0])
    assert st[0] == G.GWF_E_BAD_INPUT and d[0] == -1
