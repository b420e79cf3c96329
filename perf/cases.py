"""Workloads whose speed this repository follows, through its public entry points.

A case is one pass of a user's program: molecules and query patterns are matched and the per-pair results are
fetched.  `form` says which entry points the program uses:

  batched   match_batched on device graphs (the whole path in one call)
  graph     the same with graph=True (CUDA-graph replay on graphs that stay resident)
  stages    the stage-per-launch calls in the order of the reference's driver
  bonds     the stage calls with the bond-label join (joinWildcardCandidates) on the driver's mapping
  serve     requests to a Server whose molecule database is resident

`upload` says what a pass copies to the device first: nothing, the query patterns (a resident molecule set asked
new questions), or both batches.  Host batches are in pinned memory and results go to pinned buffers that the program keeps, through the C calls
that take them, as the benchmark does.  Molecules and patterns come from the seeded generators with the sizes that
the benchmark and the tests use.
"""
import ctypes

import numpy as np
import torch

import sigmo_b200 as sb

# Molecule sets: (generator kind, smallest, largest, median of the lognormal kind).
MOLECULES = {
    "drug": (0, 10, 60, 22.0),  # the headline set: drug-like molecules
    "lead": (0, 10, 40, 22.0),  # the serving database: small drug-like molecules
    "tail": (1, 6, 120, 22.0),  # heavy-tailed sizes with macrocycles and fused rings
    "rings": (2, 10, 64, 22.0),  # fused aromatic rings and carbon chains
}
# Query sets: (generator kind, smallest, largest, skewed from, skewed to).
QUERIES = {
    "mixed": (0, 3, 30, 6, 15),  # the headline set
    "fragment": (0, 3, 5, 0, 0),  # the smallest patterns: functional groups
    "short": (0, 4, 12, 0, 0),  # the small configuration
    "wide": (0, 3, 40, 0, 0),  # uniform sizes, a quarter of them over 30 vertices
    "automorphic": (3, 4, 14, 0, 0),  # rings, chains and stars: many embeddings per pair
}
# Rough shares of pairs that the mapping admits and vertices per graph, for work().
ADMITTED = {"fragment": 0.5, "mixed": 0.11, "short": 0.12, "wide": 0.06, "automorphic": 0.8}
ATOMS = {"drug": 35, "lead": 25, "tail": 24, "rings": 37}
QUERY_ATOMS = {"fragment": 4, "mixed": 12, "short": 8, "wide": 21, "automorphic": 9}


def _case(name, form, molecules, count, queries, patterns, upload="none", find_first=False, profile="ref-ptx", iterations=6,
          requests=1):
    return {"name": name, "form": form, "molecules": molecules, "count": count, "queries": queries, "patterns": patterns,
            "upload": upload, "find_first": find_first, "profile": profile, "iterations": iterations, "requests": requests}


def listed():
    return [
        # one pattern looked up in a handful of molecules a user just loaded: latency alone
        _case("one_pattern", "batched", "lead", 257, "fragment", 1, upload="both", find_first=True),
        # the small configuration (1,000 x 20, find-all) on resident graphs, one call
        _case("small_batched", "batched", "lead", 1000, "short", 20),
        # the same as the reference's driver calls it, stage by stage: launches and synchronisations count
        _case("small_stages", "stages", "lead", 1000, "short", 20),
        # the reference's driver at scale: the bitset of every iteration is materialised
        _case("stages_20k", "stages", "drug", 20011, "mixed", 150),
        # the headline: 100,000 x 600 find-all on resident graphs, repeated (graph replay)
        _case("drug_100k", "graph", "drug", 100000, "mixed", 600),
        # screening end to end: both batches uploaded, match flags only
        _case("screen_100k", "batched", "drug", 100000, "mixed", 600, upload="both", find_first=True),
        # injective embeddings, new patterns against resident molecules
        _case("exact_30k", "batched", "drug", 30003, "mixed", 300, upload="queries", profile="exact"),
        # uneven molecules (up to 120 atoms) and long patterns (up to 40 vertices)
        _case("uneven_60k", "batched", "tail", 60013, "wide", 500),
        # symmetric patterns in ring systems: most of the time is the join
        _case("symmetry_10k", "batched", "rings", 10007, "automorphic", 100),
        # bond labels checked: the opt-in join of the reference on the driver's mapping
        _case("bonds_2k", "bonds", "lead", 2003, "short", 40),
        # one pattern against a resident database, alone, with the list of molecules it hits: request latency
        _case("serve_one", "serve", "lead", 200000, "mixed", 1, find_first=True),
        # eight requests of up to 64 patterns that arrive together, hits counted per pattern: continuous batching
        _case("serve_burst", "serve", "lead", 200000, "mixed", 160, find_first=True, requests=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """A case of the listed ones' ranges: sizes spread over their logarithm, bounded by the listed case of the form."""
    form = rng.choice(["batched", "batched", "batched", "graph", "stages", "bonds", "serve"])
    molecules = rng.choice(["drug", "lead", "tail", "rings"] if form in ("batched", "graph") else ["drug", "lead"])
    queries = "automorphic" if molecules == "rings" else rng.choice(["mixed", "short", "wide", "fragment"])
    count, patterns = {
        "batched": (100000, 600), "graph": (100000, 600), "stages": (20011, 150), "bonds": (2003, 40), "serve": (200000, 160),
    }[form]
    if molecules == "tail":
        count, patterns = 60013, 500
    elif molecules == "rings":
        count, patterns = 10007, 100
    requests = rng.randint(1, 8) if form == "serve" else 1
    return {"form": form, "molecules": molecules, "count": _log_int(rng, 257, count), "queries": queries,
            "patterns": max(requests, _log_int(rng, 1, patterns)),
            "upload": rng.choice(["none", "queries", "both"]) if form in ("batched", "stages") else "none",
            "find_first": form == "serve" or rng.random() < 0.5,
            "profile": "exact" if form in ("batched", "graph") and rng.random() < 0.3 else "ref-ptx",
            "iterations": rng.choice([1, 2, 3, 4, 5, 6, 6, 6]), "requests": requests}


class _State:
    pass


class _PinnedGraphs:
    """A host batch in pinned memory, as the calls that take a HostGraphs read it."""

    def __init__(self, graphs):
        self.num_graphs = graphs.num_graphs
        self._arrays = [torch.from_numpy(np.array(a)).pin_memory() for a in (
            graphs.graph_offsets.view(np.int32), graphs.row_offsets.view(np.int32), graphs.column_indices.view(np.int32),
            graphs.node_labels, graphs.edge_labels)]
        self._raw = sb._lib.HostGraphsC(graphs.num_graphs, graphs.total_nodes, graphs.total_edges,
                                        *(a.data_ptr() for a in self._arrays))


def _capacity(case):
    """Entries of the result buffers: every pair of a small case, 0.4 of the pairs (the mapping admits about 0.1) of a large one."""
    pairs = case["count"] * case["patterns"]
    return min(pairs, max(4_000_000, 2 * pairs // 5))


def _buffer(n, dtype):
    return torch.zeros(n, dtype=dtype, pin_memory=True)


def prepare(case, seed):
    kind, lo, hi, median = MOLECULES[case["molecules"]]
    qkind, qlo, qhi, skew_lo, skew_hi = QUERIES[case["queries"]]
    s = _State()
    s.case = case
    data = sb.generate_molecules(case["count"], lo, hi, seed=2 * seed + 1, kind=kind, median=median)
    query = sb.generate_queries(case["patterns"], qlo, qhi, seed=2 * seed + 2, kind=qkind, skew_lo=skew_lo, skew_hi=skew_hi)
    if case["form"] == "serve":
        # the requests share the patterns out in ragged parts (1 to 64 patterns each in the listed cases)
        n, r = case["patterns"], case["requests"]
        cuts = [max(i, n * i * (i + 1) // (r * (r + 1))) for i in range(r + 1)]
        s.requests = [query.slice(a, b - a) for a, b in zip(cuts, cuts[1:])]
        s.server = sb.Server(data, profile=case["profile"], iterations=case["iterations"], find_first=case["find_first"],
                             memory_budget=8 << 30)
        if r == 1:  # a request alone also fetches its hits
            s.pair_query, s.pair_molecule = (_buffer(_capacity(case), torch.int32) for _ in range(2))
            s.pair_count = _buffer(_capacity(case), torch.int64)
        return s
    s.data, s.query = _PinnedGraphs(data), _PinnedGraphs(query)
    s.queue = sb.Queue(0, case["profile"])
    s.gmcr = sb.GMCR(s.queue)
    s.query_graph = sb.createDeviceCSRGraph(s.queue, s.query) if case["upload"] == "none" else None
    s.data_graph = sb.createDeviceCSRGraph(s.queue, s.data) if case["upload"] != "both" else None
    s.offsets = _buffer(case["count"] + 1, torch.int32)
    s.indices = _buffer(_capacity(case), torch.int32)
    s.counts = _buffer(_capacity(case), torch.int64)
    s.queue.wait()
    return s


def _serve(s):
    pairs = len(s.requests) == 1
    tickets = [s.server.submit(q, pairs=pairs) for q in s.requests]
    out = {}
    for i, (t, q) in enumerate(zip(tickets, s.requests)):
        s.server.wait(t)
        matched, total = s.server.query_totals(t, q.num_graphs)
        out["matched%d" % i], out["total%d" % i] = matched.view(np.int64), total.view(np.int64)
        if pairs:
            found = ctypes.c_uint64()
            sb.check(sb.lib().sigmo_server_pairs(s.server._h, t, s.pair_query.data_ptr(), s.pair_molecule.data_ptr(),
                                                 s.pair_count.data_ptr(), s.pair_count.numel(), ctypes.byref(found)))
            out.update(pairs=found.value, query=s.pair_query, molecule=s.pair_molecule, count=s.pair_count)
        s.server.release(t)
    return out


def _stages(s, query, data):
    case, queue = s.case, s.queue
    candidates = sb.Candidates(queue, query.total_nodes, data.total_nodes)
    signature = sb.Signature(queue, data.total_nodes, query.total_nodes)
    signature.generateDataSignatures(data)
    signature.generateQuerySignatures(query)
    sb.filterCandidates(queue, query, data, signature, candidates)
    for r in range(1, case["iterations"] + 1):
        signature.refineDataSignatures(data, r)
        signature.refineQuerySignatures(query, r)
        sb.refineCandidates(queue, query, data, signature, candidates)
    s.gmcr.generateGMCR(query, data, candidates)
    total = np.zeros(1, np.uint64)
    join = sb.joinWildcardCandidates if case["form"] == "bonds" else sb.joinCandidates
    join(queue, query, data, candidates, s.gmcr, total, case["find_first"])
    return int(total[0])


def run(s):
    case = s.case
    if case["form"] == "serve":
        return _serve(s)
    query = s.query_graph or sb.createDeviceCSRGraph(s.queue, s.query)
    data = s.data_graph or sb.createDeviceCSRGraph(s.queue, s.data)
    if case["form"] in ("stages", "bonds"):
        total = _stages(s, query, data)
    else:
        total = sb.match_batched(s.queue, query, data, case["iterations"], case["find_first"], None, s.gmcr,
                                 graph=case["form"] == "graph")["total_matches"]
    lib = sb.lib()
    sb.check(lib.sigmo_gmcr_download(s.gmcr._h, s.offsets.data_ptr(), s.offsets.numel(), s.indices.data_ptr(),
                                     s.indices.numel()))
    sb.check(lib.sigmo_match_download_counts(s.gmcr._h, s.counts.data_ptr(), s.counts.numel()))
    return {"total": total, "offsets": s.offsets, "indices": s.indices, "counts": s.counts}


def work(case):
    """Bytes that a pass cannot do without: both graph batches read once (labels, CSR) and the mapping with its counts
    written once.  The path is integer work on bit sets, so there are no floating-point operations."""
    nodes = case["count"] * ATOMS[case["molecules"]] + case["patterns"] * QUERY_ATOMS[case["queries"]]
    graphs = nodes * (1 + 4 + 2 * (4 + 1)) + 4 * (case["count"] + case["patterns"])
    pairs = case["count"] * case["patterns"] * ADMITTED[case["queries"]]
    return {"bytes": float(graphs + pairs * (4 + 8) + 4 * case["count"]), "flops": 0.0}


def exact(case, seed):
    """Every output is a whole number (match counts and indices): there is no rounding to compare with 64 bits."""
    return None
