"""Pruned reads of the block form on graphs beyond the benchmark's: arcs with overlaps, every length of
the filter's strings, graphs with too many walks for a filter, captured launches on new reads. Every
distance is the oracle's (tolerance 0)."""
import random

import numpy as np
import pytest

from randgraph import rand_graph, walk_read, walk_text

pytestmark = pytest.mark.gpu


def _check(G, O, seqs, arcs, reads, v0, g=None, nw=(0, 1, 8)):
    if g is None:
        g = G.Graph.from_arrays(seqs, arcs)
        g.index()
    og = O.OracleGraph(seqs, arcs)
    ref = [og.ed(q, int(v), -1, entry_key=True) for q, v in zip(reads, v0)]
    keep = np.array([not s.flags & O.F_NONTERM for _, s in ref])
    ref = np.array([e for e, _ in ref])
    for k in nw:
        d, st = g.ed_batch(reads, v0, mode=G.MODE_PERSISTENT, warps_per_read=k)
        assert (st == 0).all() and np.array_equal(d[keep], ref[keep]), k
    return keep.sum()


@pytest.mark.parametrize("seed", range(6))
def test_overlaps(G, O, seed):
    """Cyclic graphs whose arcs into a vertex share an offset of up to all but one of its bases: strings
    of the filter enter a vertex there, and so do the reads."""
    rng = random.Random(900 + seed)
    while True:
        seqs, arcs = rand_graph(rng, 60, rng.choice([20, 60, 200]), True, "ACGT", "uniform")
        starts = [v for v in range(60) if len(walk_text(random.Random(v), seqs, arcs, v, 1300)) == 1300]
        if len(starts) >= 3:
            break
    reads, v0 = [], []
    for n in (600, 614, 700, 1300):
        for e in (0.0, 0.02, 0.1):
            v = rng.choice(starts)
            q = walk_read(rng, seqs, arcs, v, n, e)
            if len(q) < 600:
                q += bytes(rng.choice(b"ACGT") for _ in range(600 - len(q)))
            reads.append(q), v0.append(v)
    assert _check(G, O, seqs, arcs, reads, v0) >= 6


@pytest.mark.parametrize("bases", [100_000, 400_000, 1_200_000])
def test_string_lengths_of_the_filter(G, O, bases):
    """14, 15 and 16 bases, by the graph's size."""
    sg = G.SynthGraph(bases, 200, 0.7, 10, 50_000, 300, 900, seed=bases)
    g = G.Graph.from_gfa_text(sg.gfa)
    g.index()
    s2v = g.vertex_of_segment()
    r = sg.reads(40, 2, 600, 3000, 600, 3000, 0.0, 0.12, seed=3)
    v0 = np.array([s2v[int(o)] for o in r["origin_seg"]], dtype=np.int32)
    reads = (r["cat"], r["offs"], r["lens"])
    ref, _, _ = O.OracleGraph.from_graph(g).ed_batch(*reads, v0, stats=False)
    for nw in (0, 1, 8):
        d, st = g.ed_batch(reads, v0, warps_per_read=nw)
        assert (st == 0).all() and np.array_equal(d, ref)


def test_too_many_walks_for_a_filter(G, O):
    """Sites of two 1-base vertices: 2^14 walks of 14 bases from each base."""
    rng = random.Random(77)
    seqs, arcs = [], []
    for site in range(900):
        seqs += [bytes([b]) for b in rng.sample(list(b"ACGT"), 2)]
        if site:
            arcs += [(2 * site - 2 + a, 2 * site + b, 0) for a in (0, 1) for b in (0, 1)]
    reads, v0 = [], []
    for n, e in ((600, 0.0), (600, 0.1), (800, 0.03)):
        v = rng.randrange(0, 100)
        reads.append(walk_read(rng, seqs, arcs, v, n, e)), v0.append(v)
    reads.append(bytes(rng.choice(b"ACGT") for _ in range(650))), v0.append(0)
    assert _check(G, O, seqs, arcs, reads, v0) >= 3


def test_captured_launch_on_new_reads(G, O):
    """use_graph through the batch call: batches whose longest reads run beside the others, other reads of
    the same lengths in the next call, then fewer of them."""
    w = G.load_workload("config3", n=900)
    g = w["graph"]
    g.index()
    og = O.OracleGraph.from_graph(g)
    order = np.argsort(w["lens"], kind="stable")
    halves = [order[0::2], order[1::2], order[0::6]]
    for idx in halves + halves:
        reads = (w["cat"], np.ascontiguousarray(w["offs"][idx]), np.ascontiguousarray(w["lens"][idx]))
        v0 = np.ascontiguousarray(w["v0"][idx])
        d, st = g.ed_batch(reads, v0, mode=G.MODE_PERSISTENT, use_graph=1)
        ref, _, _ = og.ed_batch(*reads, v0, stats=False)
        assert (st == 0).all() and np.array_equal(d, ref)
