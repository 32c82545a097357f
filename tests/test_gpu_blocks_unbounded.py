"""The block form where no bound prunes it: graphs without a filter (a byte other than A/C/G/T, too many
walks), reads unlike the graph, the caller's lag pruning with a large lag. The oracle gives every
distance (tolerance 0); launch counts show that arenas are large enough at the first try."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dense(G, n, site=50, lower=False, seed=31):
    """A seeded graph of n bases with a variant every `site` bases; lower: one lower-case base, so that it
    has no filter and every compare takes bytes."""
    sg = G.SynthGraph(n, site, 0.7, 4, 0, 0, 0, seed=seed)
    text = sg.gfa
    if lower:
        i = text.index(b"\tA") + 1
        text = text[:i] + b"a" + text[i + 1:]
    g = G.Graph.from_gfa_text(text)
    g.index()
    s2v = g.vertex_of_segment()
    return sg, g, s2v


def _reads(sg, s2v, *a, **kw):
    r = sg.reads(*a, **kw)
    return r["cat"], r["offs"], r["lens"], np.array([s2v[int(o)] for o in r["origin_seg"]], dtype=np.int32)


def _revcomp(cat, offs, lens):
    t = np.arange(256, dtype=np.uint8)
    for x, y in (b"AT", b"CG", b"GC", b"TA"):
        t[x] = y
    out = cat.copy()
    for o, n in zip(offs, lens):
        out[o:o + n] = t[cat[o:o + n][::-1]]
    return out


@pytest.mark.parametrize("site", [12, 50, 500])
def test_graphs_without_a_filter(G, O, site):
    """Reads of 0.6 to 6 kbp at 2 to 10%: the first arena holds them, with one warp and with eight."""
    sg, g, s2v = _dense(G, 60_000, site, lower=True)
    cat, offs, lens, v0 = _reads(sg, s2v, 24, 2, 600, 6000, 600, 6000, 0.02, 0.10, seed=site)
    ref, _, _ = O.OracleGraph.from_graph(g).ed_batch(cat, offs, lens, v0, stats=False)
    b = G.ResidentBatch(g, cat, offs, lens, v0, mode=G.MODE_PERSISTENT)
    for nw in (1, 8):
        b.run(warps_per_read=nw)
        d, st = b.results()
        assert (st == 0).all() and np.array_equal(d, ref)
        assert b.launches() == 2  # packing and the batch
    b.run()
    assert np.array_equal(b.results()[0], ref)
    b.close()


@pytest.mark.parametrize("site", [12, 50])
def test_reads_unlike_a_dense_graph(G, O, site):
    """Reverse complements, left to the retry launch: its arena holds them, the sorted form is not
    reached."""
    sg, g, s2v = _dense(G, 60_000, site)
    cat, offs, lens, v0 = _reads(sg, s2v, 12, 2, 700, 3000, 700, 3000, 0.02, 0.10, seed=site)
    cat = _revcomp(cat, offs, lens)
    ref, _, _ = O.OracleGraph.from_graph(g).ed_batch(cat, offs, lens, v0, stats=False)
    b = G.ResidentBatch(g, cat, offs, lens, v0, mode=G.MODE_PERSISTENT)
    b.run()
    d, st = b.results()
    assert (st == 0).all() and np.array_equal(d, ref)
    assert b.launches() <= 4  # packing, one warp and several warps per read, the retry
    b.run(warps_per_read=1)
    assert np.array_equal(b.results()[0], ref) and b.launches() <= 3
    b.close()


def test_large_lag_gets_warps_by_rule(G):
    """A lag of 2,000 on a dense graph prunes little: few long reads get groups of warps as they do
    without it (the time of eight warps each, with a factor to spare; with one it was several times)."""
    sg, g, s2v = _dense(G, 200_000, 20)
    cat, offs, lens, v0 = _reads(sg, s2v, 60, 0, 6000, 0, 6000, 6000, 0.08, 0.08, seed=3)

    def best(nw):
        t = []
        for _ in range(4):
            t0 = time.perf_counter()
            d, st = g.ed_batch((cat, offs, lens), v0, mode=G.MODE_PERSISTENT, flags=G.GWF_F_MAX_LAG, max_lag=2000,
                               warps_per_read=nw)
            t.append(time.perf_counter() - t0)
            assert (st == 0).all()
        return min(t), d

    (t8, d8), (t0, d0) = best(8), best(0)
    assert np.array_equal(d0, d8) and t0 < 1.6 * t8


def test_reads_without_a_filter_get_warps_by_rule(G):
    """Reads of 1.4 kbp, few enough for a group each, on a dense graph without a filter: they get one (the
    time of eight warps each, with a factor to spare; with one warp it was more than twice that)."""
    sg, g, s2v = _dense(G, 200_000, 20, lower=True)
    cat, offs, lens, v0 = _reads(sg, s2v, 200, 0, 1400, 0, 1400, 1400, 0.05, 0.05, seed=3)
    b = G.ResidentBatch(g, cat, offs, lens, v0, mode=G.MODE_PERSISTENT)
    ms, d = {}, {}
    for nw in (8, 0):
        ms[nw] = min(b.run(warps_per_read=nw) for _ in range(4))
        d[nw] = b.results()[0]
    b.close()
    assert np.array_equal(d[0], d[8]) and ms[0] < 1.6 * ms[8]


@pytest.mark.parametrize("ql", [400, 430, 500, 599, 600])
@pytest.mark.parametrize("n", [3, 592, 593])
def test_short_reads_on_a_sparse_graph(G, O, ql, n):
    """Both sides of the lines between the sorted form and the block form for short reads: below and above
    one unit of size (430 bases here), 600 bases, and a group of eight warps for each read or not. A fifth
    of the reads are reverse complements; with and without a large lag."""
    sg, g, s2v = _dense(G, 100_000, 500, seed=33)
    cat, offs, lens, v0 = _reads(sg, s2v, n, 0, ql, 0, ql, ql, 0.0, 0.10, seed=ql)
    un = _revcomp(cat, offs[::5], lens[::5])
    og = O.OracleGraph.from_graph(g)
    pick = np.unique(np.concatenate([np.arange(0, n, 40), np.arange(min(n, 3))]))
    ref, _, _ = og.ed_batch(un, offs[pick], lens[pick], v0[pick], stats=False)
    d, st = g.ed_batch((un, offs, lens), v0)
    assert (st == 0).all() and np.array_equal(d[pick], ref)
    d1, _ = g.ed_batch((un, offs, lens), v0, warps_per_read=1)
    assert np.array_equal(d, d1)
    lag, st = g.ed_batch((un, offs, lens), v0, flags=G.GWF_F_MAX_LAG, max_lag=300)
    want = [og.ed(bytes(un[offs[i]:offs[i] + lens[i]]), int(v0[i]), max_lag=300)[0] for i in pick[:4]]
    assert (st == 0).all() and list(lag[pick[:4]]) == want


@pytest.mark.parametrize("ql", [40, 150, 305, 340])
@pytest.mark.parametrize("n", [4736, 4737])
def test_many_short_reads_on_a_dense_graph(G, O, ql, n):
    """Both sides of the line between the block form and the sorted form for many short reads on a dense
    graph: the warp slots of the device, and 320 bases."""
    sg, g, s2v = _dense(G, 100_000, 50, seed=35)
    cat, offs, lens, v0 = _reads(sg, s2v, n, 0, ql, 0, ql, ql, 0.0, 0.10, seed=ql)
    d, st = g.ed_batch((cat, offs, lens), v0)
    d1, st1 = g.ed_batch((cat, offs, lens), v0, warps_per_read=1)
    assert (st == 0).all() and np.array_equal(d, d1) and np.array_equal(st, st1)
    pick = np.arange(0, n, 100)
    ref, _, _ = O.OracleGraph.from_graph(g).ed_batch(cat, offs[pick], lens[pick], v0[pick], stats=False)
    assert np.array_equal(d[pick], ref)
