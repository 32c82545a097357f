"""Arena classes of the serving loop under budgets that hold some of them: the block form's classes
are judged by their own size, and the sorted form takes the reads whose block arenas do not fit.
Every answer is the batch path's (tolerance 0)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _serve(G, g, reads, v0, **kw):
    srv = G.Server(g, **kw)
    try:
        rid, k = srv.submit(reads, v0)
        d, st = srv.wait(rid, k, timeout_s=120)
        return d, st, srv.stats()
    finally:
        srv.close()


@pytest.mark.parametrize("nw", [1, 8])
def test_block_classes_need_only_their_own_arena(G, nw):
    """A 512 KiB budget holds the block form's first two classes of a 1 kbp read (0.04 and 0.13 MB)
    but not the sorted form's second (0.76 MB): reads unlike the graph, which outgrow the first
    class, are answered in the second."""
    g = G.load_workload("config1", n=4)["graph"]
    g.index()
    rng = np.random.default_rng(11)
    reads = [bytes(rng.choice(list(b"ACGT"), size=1000).astype(np.uint8)) for _ in range(3)]
    v0 = np.zeros(3, np.int32)
    d, st, stats = _serve(G, g, reads, v0, arena_budget_bytes=512 << 10, warps_per_read=nw)
    solo, _ = g.ed_batch(reads, v0)
    assert (st == 0).all() and np.array_equal(d, solo)
    assert stats["retries"] >= 3 and stats["arena_used"] == 0


def test_sorted_form_where_the_block_arena_does_not_fit(G):
    """On a chain of 4-base vertices a 20 kbp read's block arena takes 52 MB, its sorted one 36."""
    rng = np.random.default_rng(12)
    text = bytes(rng.choice(list(b"ACGT"), size=22000).astype(np.uint8))
    g = G.Graph.from_arrays([text[i:i + 4] for i in range(0, 22000, 4)], [(i, i + 1, 0) for i in range(5499)])
    g.index()
    reads = [text[k:k + 300] + b"T" + text[k + 300:k + 700] + text[k + 702:k + 20001] for k in (0, 400)]
    v0 = [0, 100]
    d, st, stats = _serve(G, g, reads, np.array(v0, np.int32), arena_budget_bytes=44 << 20)
    solo, _ = g.ed_batch(reads, v0)
    assert (st == 0).all() and np.array_equal(d, solo)
    assert stats["retries"] == 0


@pytest.mark.parametrize("lower", [False, True])
def test_unlike_reads_and_missing_filters_cost_one_retry_at_most(G, lower):
    """Both strands of reads on a dense graph: the reverse complements leave the first arena class before
    a step is made, and the class after it holds them. With one lower-case base the graph has no filter
    that could tell them apart; they still go straight to the class that holds them."""
    sg = G.SynthGraph(60_000, 50, 0.7, 4, 0, 0, 0, seed=41)
    text = sg.gfa
    if lower:
        i = text.index(b"\tA") + 1
        text = text[:i] + b"a" + text[i + 1:]
    g = G.Graph.from_gfa_text(text)
    g.index()
    s2v = g.vertex_of_segment()
    r = sg.reads(16, 2, 300, 2500, 300, 2500, 0.01, 0.1, seed=5)
    v0 = np.array([s2v[int(o)] for o in r["origin_seg"]], dtype=np.int32)
    reads = (r["cat"], r["offs"], r["lens"])
    d, st, stats = _serve(G, g, reads, v0, flags=G.GWF_F_BOTH_STRANDS, arena_budget_bytes=2 << 30)
    solo, st2, _ = g.ed_strand(reads, v0)
    assert np.array_equal(d, solo) and np.array_equal(st, st2) and (st == 0).all()
    assert stats["retries"] <= 16
    d, st, stats = _serve(G, g, reads, v0, arena_budget_bytes=2 << 30)
    assert (st == 0).all() and np.array_equal(d, g.ed_batch(reads, v0)[0])
    assert stats["retries"] == 0
