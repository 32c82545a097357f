"""Which kernels a batch call of the block form launches, by its launch count: the helper kernel, the
one-warp and several-warp kernels, the retry of reads unlike the graph, and the sorted form that
takes over at last. Distances are int32: tolerance 0."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _unlike(G, n, ql, seed):
    """n random reads of ql bases, unlike the graph: their bound is near one edit in seven bases."""
    rng = np.random.default_rng(seed)
    cat = rng.choice(np.frombuffer(b"ACGT", np.uint8), size=n * ql + 16)
    return cat, np.arange(n, dtype=np.int64) * ql, np.full(n, ql, np.int32)


@pytest.mark.parametrize("n", [500, 700, 1184])
def test_unlike_reads_stay_in_the_block_form(G, O, n):
    """More deferred reads than half the warp slots (8 warps on each of 148 SMs) get one warp each in
    the retry launch, which defers none of them again."""
    g = G.load_workload("config1", n=4)["graph"]
    g.index()
    cat, offs, lens = _unlike(G, n, 600, n)
    b = G.ResidentBatch(g, cat, offs, lens, np.zeros(n, np.int32), mode=G.MODE_PERSISTENT)
    b.run(ctas_per_sm=1)
    d, st = b.results()
    assert (st == 0).all()
    assert b.launches() == 3  # packing, the batch, its deferred reads
    b.run(ctas_per_sm=1, use_graph=1)
    assert np.array_equal(b.results()[0], d) and b.launches() == 3
    for use_graph in (0, 1):  # a forced count is not left for the retry, in the replay neither
        b.run(ctas_per_sm=1, warps_per_read=1, use_graph=use_graph)
        assert np.array_equal(b.results()[0], d) and b.launches() == 2
    b.close()
    og = O.OracleGraph.from_graph(g)
    pick = np.arange(0, n, 50)
    ref, _, _ = og.ed_batch(cat, offs[pick], lens[pick], np.zeros(len(pick), np.int32), stats=False)
    assert np.array_equal(d[pick], ref)


def test_tuned_counts_leave_the_split_by_length(G, tmp_path):
    """A table with eight warps for every bucket: GWF_MODE_AUTO still gives groups of warps to the longest
    reads only (two kernels side by side), as an untuned run does."""
    w = G.load_workload("config3", n=1500)
    w["graph"].index()
    b = G.ResidentBatch(w["graph"], w["cat"], w["offs"], w["lens"], w["v0"], mode=G.MODE_AUTO)
    path = tmp_path / "tune.json"
    path.write_text('{"buckets": [' + ",".join(
        '\n {"bucket": %d, "ql_max": 0, "form": "persistent", "ctas_per_sm": 4, "reads_per_s": 1.0, '
        '"warps_per_read": 8}' % k for k in range(5)) + "]}")
    b.run()
    d, launches = b.results()[0], b.launches()
    assert launches == 3  # packing, one warp per read, several warps per read
    try:
        G.tune_load(str(path))
        b.run()
        assert b.launches() == launches and np.array_equal(b.results()[0], d)
    finally:
        G.tune_clear()
        b.close()


def test_launches_of_a_replayed_graph(G):
    """The launch count of a replay is that of the kernels in it: packing and both batch kernels."""
    w = G.load_workload("config3", n=1500)
    w["graph"].index()
    b = G.ResidentBatch(w["graph"], w["cat"], w["offs"], w["lens"], w["v0"], mode=G.MODE_PERSISTENT)
    for use_graph, nw, want in ((0, 0, 3), (1, 0, 3), (1, 0, 3), (1, 1, 2), (1, 8, 2)):
        b.run(use_graph=use_graph, warps_per_read=nw)
        assert b.launches() == want
    b.close()
