"""Block wavefronts with exact pruning (the persistent form's kernel for reads without a target
vertex) against the oracle: read lengths around the shortest pruned one, clean and noisy reads,
both start rules, reads with N, vertices of many arcs, walks that end in dead ends, cycles, and
reads unlike the graph, which outgrow their first arena. Distances are int32: tolerance 0."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(G, O, seqs, arcs, reads, v0, flags=0, nw=(1, 2, 8)):
    g = G.Graph.from_arrays(seqs, arcs)
    g.index()
    d, st = g.ed_batch(reads, v0, mode=G.MODE_PERSISTENT, flags=flags)
    for k in nw:
        d2, st2 = g.ed_batch(reads, v0, mode=G.MODE_PERSISTENT, flags=flags, warps_per_read=k)
        assert np.array_equal(d2, d) and np.array_equal(st2, st)
    og = O.OracleGraph(seqs, arcs)
    ref, skip = [], []
    for q, v in zip(reads, v0):
        e, s = og.ed(q, v, -1, exact_start=bool(flags & G.GWF_F_EXACT_START), entry_key=True)
        ref.append(e)
        skip.append(bool(s.flags & O.F_NONTERM))
    keep = ~np.array(skip)
    assert (st == 0).all()
    assert np.array_equal(d[keep], np.array(ref)[keep])
    return d


def _rand_seq(rng, n):
    return bytes(rng.choice(b"ACGT") for _ in range(n))


def _walk(rng, seqs, out, v, n):
    t = bytearray()
    while len(t) < n:
        t += seqs[v]
        if not out[v]:
            break
        v = rng.choice(out[v])
    return bytes(t[:n])


def _mutate(rng, q, e):
    t = bytearray()
    for c in q:
        r = rng.random()
        if r < e / 3:
            t.append(rng.choice(b"ACGT"))
        elif r < 2 * e / 3:
            t += bytes([c, rng.choice(b"ACGT")])
        elif r >= e:
            t.append(c)
    return bytes(t)


def _graph(rng, n_sites, seg, hub=0):
    """A chain of segments with a bubble between each two (hub alleles at the third site), ending
    in a dead end, with one arc back to the second segment."""
    seqs, arcs = [_rand_seq(rng, seg)], []
    for s in range(n_sites):
        prev, k = len(seqs) - 1, hub if s == 2 and hub else 2
        alleles = [_rand_seq(rng, rng.choice([1, 1, 2, 7])) for _ in range(k)]
        first = len(seqs)
        seqs += alleles + [_rand_seq(rng, rng.randint(max(1, seg // 2), seg))]
        join = len(seqs) - 1
        for a in range(k):
            arcs += [(prev, first + a, 0), (first + a, join, 0)]
        if s % 3 == 0:
            arcs.append((prev, join, 0))
    arcs.append((len(seqs) - 1, 3, 0))
    out = [[] for _ in seqs]
    for v, w, _ in arcs:
        out[v].append(w)
    return seqs, arcs, out


@pytest.mark.parametrize("ql", [31, 599, 600, 601, 615, 616, 1100])
@pytest.mark.parametrize("exact", [0, 1])
def test_lengths_and_errors(G, O, ql, exact):
    rng = random.Random(ql * 2 + exact)
    for seg, hub in ((40, 0), (300, 20)):
        seqs, arcs, out = _graph(rng, 30, seg, hub)
        reads, v0 = [], []
        for e in (0.0, 0.01, 0.05, 0.1, 0.2):
            for _ in range(3):
                v = rng.choice([0, 0, 3])
                q = _mutate(rng, _walk(rng, seqs, out, v, ql), e)[:ql] or b"A"
                reads.append(q), v0.append(v)
        b = bytearray(reads[-1])
        b[len(b) // 2] = ord("N")
        reads.append(bytes(b)), v0.append(v0[-1])
        _check(G, O, seqs, arcs, reads, v0, flags=G.GWF_F_EXACT_START if exact else 0)


def test_dead_ends_and_unlike_reads(G, O):
    """Reads that run past the graph's end, and random reads (no bound helps them), the longest of
    which need a larger arena than the first."""
    rng = random.Random(5)
    seqs, arcs, out = _graph(rng, 12, 60)
    v, w, _ = arcs.pop()  # no way back: every walk ends
    out[v].remove(w)
    reads = [_walk(rng, seqs, out, 0, 2000) + _rand_seq(rng, n) for n in (0, 3, 200, 700)]
    reads += [_rand_seq(rng, n) for n in (600, 900, 2500)]
    _check(G, O, seqs, arcs, reads, [0] * len(reads))


def test_long_and_short_reads_side_by_side(G, O):
    """A batch whose longest reads get several warps and run beside the rest, launched and
    replayed as a graph, on new reads of the same resident shape."""
    w = G.load_workload("config3", n=400)
    long_ = G.load_workload("config3", n=6000)
    pick = np.argsort(long_["lens"])[-3:]
    reads = [bytes(w["cat"][o:o + l]) for o, l in zip(w["offs"], w["lens"])]
    reads += [bytes(long_["cat"][long_["offs"][i]:long_["offs"][i] + long_["lens"][i]]) for i in pick]
    v0 = np.concatenate([w["v0"], long_["v0"][pick]])
    g = w["graph"]
    g.index()
    cat, offs, lens = G.pack_reads(reads)
    og = O.OracleGraph.from_graph(g)
    ref, _, _ = og.ed_batch(cat, offs, lens, v0, stats=False)
    rb = G.ResidentBatch(g, cat, offs, lens, v0, mode=G.MODE_PERSISTENT)
    for graph in (0, 1, 1):
        rb.run(use_graph=graph)
        d, st = rb.results()
        assert (st == 0).all() and np.array_equal(d, ref)
    rb.close()


def test_long_reads_on_a_dense_graph(G, O):
    """Bound, refined windows and the queue of diagonals: 4 kbp reads, a variant every 50 bases."""
    sg = G.SynthGraph(60_000, 50, 0.7, 20, 10_000, 200, 800, seed=9)
    g = G.Graph.from_gfa_text(sg.gfa)
    g.index()
    r = sg.reads(24, 0, 4000, 0, 4000, 4000, 0.02, 0.12, seed=10)
    s2v = g.vertex_of_segment()
    v0 = np.array([s2v[int(o)] for o in r["origin_seg"]], dtype=np.int32)
    og = O.OracleGraph.from_graph(g)
    ref, _, _ = og.ed_batch(r["cat"], r["offs"], r["lens"], v0, stats=False)
    for kw in ({}, {"use_graph": 1}):
        d, st = g.ed_batch((r["cat"], r["offs"], r["lens"]), v0, mode=G.MODE_PERSISTENT, **kw)
        assert (st == 0).all()
        assert np.array_equal(d, ref)
    # score steps: distance + 1, as every form reports them
    rb = G.ResidentBatch(g, r["cat"], r["offs"], r["lens"], v0, mode=G.MODE_PERSISTENT)
    rb.run()
    assert np.array_equal(rb.steps(), ref + 1)
    rb.close()


@pytest.mark.parametrize("lag", [3, 60, 400])
def test_lag_pruning_in_registers_and_in_lists(G, O, lag):
    """The caller's lag pruning on a dense graph: a small lag keeps to a few blocks, a large one goes
    through the lists, with one warp and with several."""
    sg = G.SynthGraph(30_000, 50, 0.7, 20, 10_000, 200, 800, seed=19)
    g = G.Graph.from_gfa_text(sg.gfa)
    g.index()
    r = sg.reads(8, 2, 700, 2000, 700, 2000, 0.02, 0.12, seed=20)
    s2v = g.vertex_of_segment()
    v0 = np.array([s2v[int(o)] for o in r["origin_seg"]], dtype=np.int32)
    og = O.OracleGraph.from_graph(g)
    ref = [og.ed(bytes(r["cat"][o:o + n]), int(v), max_lag=lag)[0] for o, n, v in zip(r["offs"], r["lens"], v0)]
    for nw in (0, 1, 8):
        d, st = g.ed_batch((r["cat"], r["offs"], r["lens"]), v0, mode=G.MODE_PERSISTENT, flags=G.GWF_F_MAX_LAG,
                           max_lag=lag, warps_per_read=nw)
        assert (st == 0).all() and list(d) == ref
