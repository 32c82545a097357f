"""The sorted wavefronts at the sizes they still serve: alignments to a target vertex and graphs whose
arcs into one vertex carry different overlaps. One warp per read (k_align_persistent), groups of 2, 4
and 8 (k_align_classes, gwf_group.cuh), the rule, replayed graphs, lag pruning, reads that outgrow
their arenas, serving. Every distance is the oracle's (tolerance 0)."""
import random

import numpy as np
import pytest

from randgraph import walk_text

pytestmark = pytest.mark.gpu


def _rand_seq(rng, n):
    return bytes(rng.choice(b"ACGT") for _ in range(n))


def _chain(rng, n_sites, seg, mixed):
    """A chain of segments with a two-allele bubble between each two. mixed: the second allele's arc
    enters the next segment at its third base."""
    seqs, arcs = [_rand_seq(rng, seg)], []
    for _ in range(n_sites):
        prev, a = len(seqs) - 1, len(seqs)
        seqs += [_rand_seq(rng, rng.choice([1, 1, 3])), _rand_seq(rng, rng.choice([1, 2, 8])),
                 _rand_seq(rng, rng.randint(max(4, seg // 2), seg))]
        arcs += [(prev, a, 0), (prev, a + 1, 0), (a, a + 2, 0), (a + 1, a + 2, 2 if mixed else 0)]
    return seqs, arcs


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


def _case(rng, mixed, junk=False):
    """Reads of 0.2 to 3 kbp from the chain, the start vertices of all and the target of the batch: the
    reads run to the target's end, or near it, or (mixed) anywhere."""
    seqs, arcs = _chain(rng, 60, 60, mixed)
    v1 = -1 if mixed else 3 * 45
    reads, v0 = [], []
    for k in range(14):
        v = 3 * rng.randrange(0, 44)
        text = walk_text(rng, seqs, arcs, v, rng.randint(200, 3000))
        if not mixed:  # a walk to the target's end
            text, u = seqs[v], v
            while u != v1:
                a = u + 1 + rng.randrange(2)
                u += 3
                text += seqs[a] + seqs[u]
        reads.append(_mutate(rng, text, rng.choice([0.0, 0.02, 0.1])) or b"A")
        v0.append(v)
    if junk:
        reads += [_rand_seq(rng, n) for n in (300, 900, 1500)]
        v0 += [3 * 40, 0, 0]
    return seqs, arcs, reads, v0, v1


def _oracle(O, seqs, arcs, reads, v0, v1, lag=0):
    og = O.OracleGraph(seqs, arcs)
    ref, keep = [], []
    for q, v in zip(reads, v0):
        e, s = og.ed(q, v, v1, max_lag=lag, entry_key=True)
        ref.append(e)
        keep.append(not s.flags & O.F_NONTERM)
    return np.array(ref), np.array(keep)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("junk", [False, True])
@pytest.mark.parametrize("seed", [1, 2])
def test_shapes_equal_the_oracle(G, O, mixed, junk, seed):
    rng = random.Random(100 * seed + 2 * mixed + junk)
    seqs, arcs, reads, v0, v1 = _case(rng, mixed, junk)
    g = G.Graph.from_arrays(seqs, arcs)
    g.index()
    ref, keep = _oracle(O, seqs, arcs, reads, v0, v1)
    assert keep.sum() >= 10
    for nw in (0, 1, 2, 4, 8):
        for use_graph in (0, 1, 1):
            d, st = g.ed_batch(reads, v0, v1=v1, mode=G.MODE_PERSISTENT, warps_per_read=nw, use_graph=use_graph)
            assert (st == 0).all() and np.array_equal(d[keep], ref[keep]), (nw, use_graph)
    cat, offs, lens = G.pack_reads(reads)
    b = G.ResidentBatch(g, cat, offs, lens, np.array(v0, np.int32), v1=v1, mode=G.MODE_PERSISTENT)
    for nw, use_graph in ((1, 0), (8, 1), (0, 1)):
        b.run(warps_per_read=nw, use_graph=use_graph)
        d, st = b.results()
        hit = keep & (ref >= 0)
        assert (st == 0).all() and np.array_equal(d[keep], ref[keep])
        assert np.array_equal(b.steps()[hit], ref[hit] + 1)
    b.close()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("lag", [4, 30, 400])
def test_lag_pruning_equals_the_oracle(G, O, mixed, lag):
    rng = random.Random(lag * 2 + mixed)
    seqs, arcs, reads, v0, v1 = _case(rng, mixed)
    g = G.Graph.from_arrays(seqs, arcs)
    g.index()
    ref, keep = _oracle(O, seqs, arcs, reads, v0, v1, lag)
    for nw in (0, 1, 2, 8):
        d, st = g.ed_batch(reads, v0, v1=v1, mode=G.MODE_PERSISTENT, warps_per_read=nw, flags=G.GWF_F_MAX_LAG, max_lag=lag)
        assert (st == 0).all() and np.array_equal(d[keep], ref[keep]), nw


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("nw", [1, 2, 8])
def test_serving_equals_the_oracle(G, O, mixed, nw):
    rng = random.Random(nw * 2 + mixed)
    seqs, arcs, reads, v0, v1 = _case(rng, mixed, junk=True)
    g = G.Graph.from_arrays(seqs, arcs)
    g.index()
    ref, keep = _oracle(O, seqs, arcs, reads, v0, v1)
    srv = G.Server(g, warps_per_read=nw, arena_budget_bytes=1 << 30)
    try:
        rid, n = srv.submit(reads, np.array(v0, np.int32), v1)
        d, st = srv.wait(rid, n, timeout_s=120)
    finally:
        srv.close()
    assert (st == 0).all() and np.array_equal(d[keep], ref[keep])
