"""The join's forms at the sizes where they take over from one another: queries
of 10 / 11 / 16 / 17 and up to 64 vertices, molecules of 64 / 65 / 128 / 129 and
up to 256 atoms, levels with no, one, two and more earlier neighbours, fewer
pairs than lanes and more, molecules below vertex 256 (the literal search) and
above, in the batched and the stage-per-launch form, against the oracle (whole
numbers: equal)."""
import numpy as np
import pytest

import oracle
import sigmo_b200 as sb

pytestmark = pytest.mark.gpu

PROF = {"ref-ptx": oracle.REF_PTX, "exact": oracle.EXACT}


def _graph(n, edges, labels=None):
    lab = labels or [8] * n
    return (f"n#{n} l#1 " + " ".join(f"{i} {lab[i]}" for i in range(n)) + f" e#{len(edges)} " +
            " ".join(f"{u} {v} 1" for u, v in edges))


def _complete(n):
    return _graph(n, [(i, j) for i in range(n) for j in range(i + 1, n)])


def _check(q, d, R, prof, ff):
    ref = oracle.run_pipeline(q, d, R, PROF[prof], ff)
    assert len(ref["indices"]) > 0
    queue = sb.Queue(0, profile=prof)
    qg, dg = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, d)
    gm = sb.GMCR(queue)
    res = sb.match_batched(queue, qg, dg, R, ff, None, gm)
    off, idx = gm.getGMCR()
    assert np.array_equal(off, ref["offsets"]) and np.array_equal(idx, ref["indices"])
    assert np.array_equal(gm.getPairCounts(), ref["per_pair"]) and res["total_matches"] == ref["total"]
    cand = sb.Candidates(queue, qg.total_nodes, dg.total_nodes)
    sig = sb.Signature(queue, dg.total_nodes, qg.total_nodes)
    sig.generateDataSignatures(dg)
    sig.generateQuerySignatures(qg)
    sb.filterCandidates(queue, qg, dg, sig, cand)
    for r in range(1, R + 1):
        sig.refineDataSignatures(dg, r)
        sig.refineQuerySignatures(qg, r)
        sb.refineCandidates(queue, qg, dg, sig, cand)
    g2 = sb.GMCR(queue)
    g2.generateGMCR(qg, dg, cand)
    total = np.zeros(1, np.uint64)
    _, per = sb.joinCandidates(queue, qg, dg, cand, g2, total, ff, per_pair=True)
    assert np.array_equal(per, ref["per_pair"]) and int(total[0]) == ref["total"]
    return ref


MODES = [("ref-ptx", False), ("ref-ptx", True), ("exact", False), ("exact", True)]


@pytest.mark.parametrize("prof,ff", MODES)
@pytest.mark.parametrize("qlo,qhi,dlo,dhi,count", [
    (2, 10, 10, 64, 40),     # one word, short queries, fewer pairs than lanes
    (9, 18, 20, 64, 400),    # short / long / wide queries side by side
    (2, 12, 60, 70, 300),    # molecules around one word
    (14, 40, 60, 130, 200),  # two words and the first of four
    (30, 64, 120, 256, 60),  # the longest queries, four words
])
def test_sizes(qlo, qhi, dlo, dhi, count, prof, ff):
    d = sb.generate_molecules(count, dlo, dhi, seed=3101 + dhi, kind=1, median=(dlo + dhi) / 2)
    # queries cut from molecules of the same kind; sizes spread over the range
    q = sb.generate_queries(24, qlo, qhi, seed=3102 + qhi)
    small = sb.generate_queries(4, 2, 4, seed=3103)
    _check(q.concat(small), d, 3, prof, ff)


@pytest.mark.parametrize("prof,ff", MODES)
def test_levels_with_any_number_of_earlier_neighbours(prof, ff):
    path = lambda n: _graph(n, [(i, i + 1) for i in range(n - 1)])  # noqa: E731
    queries = [
        _complete(3), _complete(4), _complete(5),                 # one to four earlier neighbours
        _graph(4, [(0, 1), (2, 3)]),                              # a level with none
        _graph(5, [(0, 1), (1, 2), (2, 0), (3, 4)]),
        _graph(6, [(0, 1), (1, 2), (2, 3), (3, 0), (0, 4), (2, 5)]),
        _graph(12, [(i, i + 1) for i in range(11)] + [(0, 11), (3, 8)]),  # a long query with two bridged rings
        path(2), path(7),
    ]
    graphs = [_complete(n) for n in (3, 4, 5, 6, 7)]
    graphs += [_graph(8, [(i, (i + 1) % 8) for i in range(8)] + [(0, 4)]),
               _graph(16, [(i, (i + 1) % 16) for i in range(16)] + [(3, 8), (1, 12)]),
               _graph(9, [(0, i) for i in range(1, 9)])]
    graphs = graphs * 40  # starts below vertex 256 and well above
    q, d = sb.io.parse("\n".join(queries) + "\n"), sb.io.parse("\n".join(graphs) + "\n")
    ref = _check(q, d, 2, prof, ff)
    assert ref["total"] > 0


@pytest.mark.parametrize("prof,ff", MODES)
@pytest.mark.parametrize("qlo,qhi,dlo,dhi,count", [(2, 6, 3, 64, 150), (10, 40, 20, 130, 200), (20, 48, 120, 256, 60)])
def test_bond_label_join_sizes(qlo, qhi, dlo, dhi, count, prof, ff):
    d = sb.generate_molecules(count, dlo, dhi, seed=3201 + dhi, kind=1, median=(dlo + dhi) / 2)
    q = sb.generate_queries(16, qlo, qhi, seed=3202 + qhi).concat(sb.generate_queries(4, 2, 4, seed=3203))
    queue = sb.Queue(0, profile=prof)
    qg, dg = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, d)
    cand = sb.Candidates(queue, qg.total_nodes, dg.total_nodes)
    sig = sb.Signature(queue, dg.total_nodes, qg.total_nodes)
    sb.filterCandidates(queue, qg, dg, sig, cand)  # labels only: many candidates per vertex
    sig.generateDataSignatures(dg)
    sig.generateQuerySignatures(qg)
    sig.refineDataSignatures(dg, 1)
    sig.refineQuerySignatures(qg, 1)
    sb.refineCandidates(queue, qg, dg, sig, cand)
    gm = sb.GMCR(queue)
    gm.generateGMCR(qg, dg, cand)
    off, idx = gm.getGMCR()
    want_total, want_per = oracle.join_wildcard(q, d, cand.getHostCandidates(), off, idx, PROF[prof], ff)
    total = np.zeros(1, np.uint64)
    _, per = sb.joinWildcardCandidates(queue, qg, dg, cand, gm, total, ff, per_pair=True)
    assert len(idx) > 0 and np.array_equal(per, want_per) and int(total[0]) == want_total


@pytest.mark.parametrize("count", [18_912, 18_913, 18_945, 37_887, 37_888, 37_921, 40_033])
@pytest.mark.parametrize("serve", [False, True])
def test_admission_with_two_graphs_per_lane(count, serve):
    """From 592 tiles of 32 graphs on, the admission carries two graphs per
    lane: tile counts on both sides, odd and even, ragged last tiles."""
    d = sb.generate_molecules(count, 3, 9, seed=3301)
    q = sb.generate_queries(10, 2, 6, seed=3302)
    ref = oracle.run_pipeline(q, d, 2, oracle.REF_PTX, False)
    if serve:  # resident planes, gathered
        with sb.Server(d, iterations=2, find_first=False) as srv:
            t = srv.submit(q)
            srv.wait(t)
            matched, total = srv.query_totals(t, q.num_graphs)
        want = np.zeros(q.num_graphs, np.uint64)
        np.add.at(want, ref["indices"].astype(np.int64), ref["per_pair"])
        hits = np.bincount(ref["indices"][ref["per_pair"] > 0], minlength=q.num_graphs)
        assert np.array_equal(total, want) and np.array_equal(matched, hits.astype(np.uint64))
        return
    queue = sb.Queue(0)
    gm = sb.GMCR(queue)
    res = sb.match_batched(queue, sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, d), 2, False, None, gm)
    off, idx = gm.getGMCR()
    assert np.array_equal(off, ref["offsets"]) and np.array_equal(idx, ref["indices"])
    assert np.array_equal(gm.getPairCounts(), ref["per_pair"]) and res["total_matches"] == ref["total"]


@pytest.mark.parametrize("count", [1, 31, 33, 1024, 1025, 8191, 8192, 8193])
def test_segment_offsets_by_graph_count(count):
    """One-launch offsets up to 8,192 data graphs: fewer graphs than threads,
    one per thread, ragged runs, the largest count and the one past it."""
    d = sb.generate_molecules(count, 8, 14, seed=3401)
    q = sb.generate_queries(6, 2, 4, seed=3402).concat(sb.io.parse(_graph(2, [(0, 1)], [1, 1]) + "\n"))
    _check(q, d, 1, "ref-ptx", True)


@pytest.mark.parametrize("prof", ["ref-ptx", "exact"])
@pytest.mark.parametrize("count", [1, 2, 9, 130, 1_111])
def test_bit_sliced_signatures_by_vertex_count(count, prof):
    """Refinement against the oracle's bitset after every pass: vertex counts
    short of one word, of a word group and of a row's padding, and queries with
    more thresholds than a block's table holds."""
    d = sb.generate_molecules(count, 5, 40, seed=3501)
    q = sb.generate_queries(24, 3, 20, seed=3502)
    queue = sb.Queue(0, profile=prof)
    qg, dg = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, d)
    cand = sb.Candidates(queue, qg.total_nodes, dg.total_nodes)
    sig = sb.Signature(queue, dg.total_nodes, qg.total_nodes)
    sig.generateDataSignatures(dg)
    sig.generateQuerySignatures(qg)
    sb.filterCandidates(queue, qg, dg, sig, cand)
    bits = oracle.filter_candidates(q, d)
    assert np.array_equal(cand.getHostCandidates(), bits)
    for r in range(1, 4):
        sig.refineDataSignatures(dg, r)
        sig.refineQuerySignatures(qg, r)
        sb.refineCandidates(queue, qg, dg, sig, cand)
        bits = oracle.refine_candidates(q, d, sig.getQuerySignatures(), sig.getDataSignatures(), bits)
        assert np.array_equal(cand.getHostCandidates(), bits), r
