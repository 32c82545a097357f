"""Graphs at the edges of what gwf_ed_index takes: the filter of the walks' strings is built for them,
or left out, and the graph is usable either way."""
import time

import numpy as np
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


def test_long_vertex_is_indexed_like_short_ones(G):
    """The filter's work is split by bases, not by vertices: 16 Mbp in one vertex take about the time of
    the same bases in vertices of 1,024 (the bound is loose; with a warp per vertex it was 8 times)."""
    n = 1 << 24
    text = np.random.default_rng(2).choice(np.frombuffer(b"ACGT", np.uint8), n).tobytes()

    def best(seqs, arcs):
        g = G.Graph.from_arrays(seqs, arcs)
        t = []
        for _ in range(3):
            t0 = time.perf_counter()
            g.index()
            t.append(time.perf_counter() - t0)
        g.close()
        return min(t)

    short = best([text[i:i + 1024] for i in range(0, n, 1024)], [(i, i + 1, 0) for i in range(n // 1024 - 1)])
    assert best([text], []) < 3 * short
