"""The work that users of this library have it do, as measurable cases.

Every case aligns seeded synthetic reads (the library's own generator) against one of the two
graphs of the benchmark configurations, through the public Python binding:

  graph "100k"  100 kbp backbone, a variant site every 500 bp (benchmark configurations 1 to 3)
  graph "5M"    5 Mbp backbone, a variant every 50 bp, a structural variant every 50 kbp
                (configurations 4 and 5)

A program indexes its graph once and keeps it (and its server), so both are kept here for the life
of the process. Reads are host data, as a program has them after parsing its FASTA file; a case's
pass takes them through the whole call, except in the resident form, whose reads are uploaded when
the batch is made.

Case fields: call (entry point), graph, n (reads), kind (read length distribution: "fixed" len_a,
"lognormal" median len_a and sigma len_b, "uniform" len_a..len_b; clipped to len_min..len_max),
err_min/err_max (range of the reads' error rates), n_reads_pct (percentage of the reads that carry
a few N, which takes the byte-compare path).
"""
import importlib.util
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GRAPHS = {
    "100k": (100_000, 500, 0.7, 10, 0, 0, 0, 1),
    "5M": (5_000_000, 50, 0.7, 20, 50_000, 1000, 5000, 4),
}
GRAPH_BYTES = {"100k": 125_000, "5M": 12_000_000}  # bases, vertex table and arcs, each once
KINDS = {"fixed": 0, "lognormal": 1, "uniform": 2}
PATH_NV, PATH_OPS = 64, 256
LAG = 20
_graphs, _servers = {}, {}


def _pkg():
    """The package's directory name is no identifier: it is loaded by path."""
    if "gwfa_b200" in sys.modules:
        return sys.modules["gwfa_b200"]
    d = os.path.join(ROOT, "gwfa-cuda-version_b200")
    spec = importlib.util.spec_from_file_location("gwfa_b200", os.path.join(d, "__init__.py"),
                                                  submodule_search_locations=[d])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["gwfa_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


def _case(name, call, graph, n, kind, len_a, len_b, len_min, len_max, err_min, err_max, n_reads_pct=0):
    return {"name": name, "call": call, "graph": graph, "n": n, "kind": kind, "len_a": len_a, "len_b": len_b,
            "len_min": len_min, "len_max": len_max, "err_min": err_min, "err_max": err_max,
            "n_reads_pct": n_reads_pct}


def listed():
    return [
        # one clean read at a time: the drop-in gwf_ed call, all launch and host latency
        _case("one_1k", "ed", "100k", 1, "fixed", 1000, 0, 1000, 1000, 0.01, 0.01),
        # one long noisy read on the dense graph: the time of a single alignment
        _case("one_20k", "ed", "5M", 1, "fixed", 20000, 0, 20000, 20000, 0.10, 0.10),
        # short ragged reads, a tenth of them with N
        _case("short_ragged", "batch", "100k", 5003, "uniform", 150, 400, 150, 400, 0.0, 0.10, 10),
        # configuration 1: a small batch of clean 1 kbp reads
        _case("batch_1k_clean", "batch", "100k", 1000, "fixed", 1000, 0, 1000, 1000, 0.01, 0.01),
        # configuration 2's size: many 1 kbp reads at 5 to 10%, host to host
        _case("batch_1k_many", "batch", "100k", 100000, "fixed", 1000, 0, 1000, 1000, 0.05, 0.10),
        # an ordinary batch of mixed lengths that does not fill the device evenly
        _case("batch_mixed_mid", "batch", "100k", 3001, "lognormal", 2000, 0.6, 500, 10000, 0.01, 0.10),
        # configuration 3's reads kept on the device and aligned again (the benchmark's form)
        _case("resident_mixed", "resident", "100k", 50000, "lognormal", 2000, 0.6, 500, 10000, 0.01, 0.10),
        # configuration 4: 10 kbp reads at 5% on the dense graph
        _case("batch_10k_dense", "batch", "5M", 4000, "fixed", 10000, 0, 10000, 10000, 0.05, 0.05),
        # configuration 5: one request of the serving loop
        _case("serve_128", "serve", "5M", 128, "uniform", 500, 20000, 500, 20000, 0.01, 0.10),
        # both strands of reads whose orientation is not known
        _case("strands_1k", "strand", "100k", 2000, "fixed", 1000, 0, 1000, 1000, 0.01, 0.10),
        # paths and CIGARs
        _case("path_cigar_1k", "path", "100k", 10000, "fixed", 1000, 0, 1000, 1000, 0.05, 0.10),
        # opt-in lag pruning of long reads
        _case("lag_10k_dense", "lag", "5M", 2000, "fixed", 10000, 0, 10000, 10000, 0.05, 0.05),
    ]


def draw(rng):
    call = rng.choice(["ed", "batch", "batch", "batch", "batch", "resident", "resident", "serve", "strand",
                       "path", "lag"])
    graph = rng.choice(["100k", "100k", "5M"]) if call not in ("strand", "path") else "100k"

    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    top_len = 1000 if call == "strand" else 3000 if call == "path" else 10000 if graph == "100k" else 20000
    mean = log(150, top_len)
    kind = "fixed" if call == "ed" else rng.choice(["fixed", "lognormal", "uniform"])
    lo, hi = (mean, mean) if kind == "fixed" else (max(100, mean // 4), min(top_len, mean * 4))
    if kind == "uniform":
        a, b = lo, hi
    else:
        a, b = mean, 0.6 if kind == "lognormal" else 0
    err_max = round(rng.uniform(0.01, 0.10), 3)
    err_min = round(rng.uniform(0.0, err_max), 3)
    # as many reads as keep the pass below the largest listed one: the work of a read grows with
    # the square of its length, and with its error rate
    long_reads = float(hi) ** 2 * max(err_max, 0.02) / 0.05
    most = (1e12 if graph == "100k" else 4e11) / long_reads
    cap = {"ed": 1, "batch": 100000, "resident": 100000, "serve": 256, "strand": 2000, "path": 10000,
           "lag": 20000}[call]
    n = 1 if call == "ed" else log(2, max(3, int(min(most, cap))))
    pct = rng.choice([0, 0, 0, 5, 20]) if call in ("batch", "resident", "serve") else 0
    c = _case("", call, graph, n, kind, a, b, lo, hi, err_min, err_max, pct)
    del c["name"]
    return c


def _graph(key):
    if key not in _graphs:
        G = _pkg()
        p = GRAPHS[key]
        sg = G.SynthGraph(*p[:7], seed=p[7])
        g = G.Graph.from_gfa_text(sg.gfa)
        g.index()
        seg = np.full(int(g.srcs().max()) // 2 + 1, -1, dtype=np.int32)
        for s, v in g.vertex_of_segment().items():
            seg[s] = v
        _graphs[key] = (sg, g, seg)
    return _graphs[key]


def prepare(case, seed):
    G = _pkg()
    sg, g, seg = _graph(case["graph"])
    r = sg.reads(case["n"], KINDS[case["kind"]], case["len_a"], case["len_b"], case["len_min"], case["len_max"],
                 case["err_min"], case["err_max"], seed=seed + 1)
    cat, offs, lens = r["cat"], r["offs"], r["lens"]
    if case["n_reads_pct"]:
        rng = np.random.default_rng(seed)
        hit = np.nonzero(rng.random(case["n"]) * 100 < case["n_reads_pct"])[0]
        for _ in range(3):
            cat[offs[hit] + (rng.random(len(hit)) * lens[hit]).astype(np.int64)] = ord("N")
    s = {"call": case["call"], "g": g, "reads": (cat, offs, lens), "v0": seg[r["origin_seg"]]}
    if case["call"] == "ed":
        s["read"] = cat[:lens[0]].tobytes()
    elif case["call"] == "resident":
        s["batch"] = G.ResidentBatch(g, cat, offs, lens, s["v0"], mode=G.MODE_PERSISTENT)
    elif case["call"] == "serve":
        if case["graph"] not in _servers:
            _servers[case["graph"]] = G.Server(g, arena_budget_bytes=16 << 30)
        s["server"] = _servers[case["graph"]]
    return s


def _filled(rows, counts):
    """An (n, width) output with zeros past each row's count: the library leaves those as they were."""
    return np.where(np.arange(rows.shape[1])[None, :] < counts[:, None], rows, 0)


def run(state):
    G = _pkg()
    call, g, v0 = state["call"], state["g"], state["v0"]
    if call == "ed":
        return g.ed(state["read"], v0=int(v0[0]))
    if call == "batch":
        return g.ed_batch(state["reads"], v0)
    if call == "resident":
        state["batch"].run(use_graph=1)
        return state["batch"].results()
    if call == "serve":
        rid, n = state["server"].submit(state["reads"], v0)
        return state["server"].wait(rid, n, timeout_s=120)
    if call == "strand":
        return g.ed_strand(state["reads"], v0)
    if call == "lag":
        return g.ed_batch(state["reads"], v0, flags=G.GWF_F_MAX_LAG, max_lag=LAG)
    if call == "path":
        dist, status, end_off, path_n, path_v, path_arc, cigar_n, cigar = g.ed_path(
            state["reads"], v0, max_nv=PATH_NV, max_ops=PATH_OPS, as_arrays=True)
        return {"dist": dist, "status": status, "end_off": end_off, "path_n": path_n,
                "path_v": _filled(path_v, path_n), "path_arc": _filled(path_arc, path_n), "cigar_n": cigar_n,
                "cigar": _filled(cigar, cigar_n)}
    raise ValueError(call)


def work(case):
    if case["kind"] == "uniform":
        mean = (case["len_a"] + case["len_b"]) / 2
    else:
        mean = case["len_a"] * float(np.exp(case["len_b"] ** 2 / 2))
    mean = min(max(mean, case["len_min"]), case["len_max"])
    n = case["n"]
    bases = n * mean
    # each read, its offset, length and start vertex once; the graph once; each result once
    out = 8.0 * n
    if case["call"] == "strand":
        out += 4.0 * n
    elif case["call"] == "path":
        # end offset, counts, vertices and arcs of a path, runs of a CIGAR (about two per edit)
        edits = mean * (case["err_min"] + case["err_max"]) / 2
        out += n * (12.0 + 8.0 * (1 + mean / 250) + 4.0 * (1 + 2 * edits))
    # every base is compared at least once
    return {"bytes": bases + 16.0 * n + GRAPH_BYTES[case["graph"]] + out, "flops": bases}
