"""The join's forms in identity order (queries or molecules whose adjacency is
not mirrored), over several mask chunks from the bitset, and out of steps
among the wide pairs."""
import numpy as np
import pytest

import oracle
import sigmo_b200 as sb
from test_gpu_join_forms import MODES, PROF, _check

pytestmark = pytest.mark.gpu


def _with_loops(g, share, seed):
    """A share of the graphs with self-loops at a fifth of their vertices; a
    self-loop's second CSR entry names vertex 0, which does not have it back."""
    rng, out = np.random.default_rng(seed), []
    for line in g.to_text().splitlines():
        head, _, tail = line.partition(" e#")
        n = int(head.split()[0][2:])
        if rng.random() < share:
            count, *rest = tail.split()
            loops = rng.choice(n, max(1, n // 5), replace=False)
            tail = f"{int(count) + len(loops)} " + " ".join(rest + [f"{u} {u} 1" for u in sorted(loops.tolist())])
        out.append(f"{head} e#{tail}")
    return sb.io.parse("\n".join(out) + "\n")


def _chains(sizes):
    return sb.io.parse("".join(f"n#{n} l#1 " + " ".join(f"{i} 8" for i in range(n)) + f" e#{n - 1} " +
                               " ".join(f"{i} {i + 1} 1" for i in range(n - 1)) + "\n" for n in sizes))


def _case(chains, dlo, dhi, count):
    """Carbon chains and small patterns against ring systems and molecules."""
    d = sb.generate_molecules(count, dlo, min(dhi, 64), seed=3801 + dhi, kind=2)
    d = d.concat(sb.generate_molecules(count, dlo, dhi, seed=3802 + dhi, kind=1, median=(dlo + dhi) / 2))
    q = sb.generate_queries(12, 2, 8, seed=3803).concat(_chains(chains)).concat(_chains(chains))
    return _with_loops(q, 0.5, 2), _with_loops(d, 0.6, 1)


CASES = [((3, 6, 9, 10), 8, 64, 120), ((10, 11, 13, 16), 12, 40, 60), ((9, 12, 17, 20), 12, 100, 40), ((8, 16, 18, 33), 20, 256, 30)]


@pytest.mark.parametrize("prof,ff", MODES)
@pytest.mark.parametrize("case", CASES)
def test_unmirrored_graphs(case, prof, ff):
    q, d = _case(*case)
    ref = _check(q, d, 1, prof, ff)
    sizes = q.sizes()[ref["indices"][ref["per_pair"] > 0]]
    assert all((sizes == n).any() for n in case[0])


@pytest.mark.parametrize("prof,ff", MODES)
@pytest.mark.parametrize("case", CASES)
def test_unmirrored_graphs_by_bond_labels(case, prof, ff):
    q, d = _case(*case)
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


@pytest.mark.parametrize("ff", [False, True])
def test_several_mask_chunks_from_the_bitset(ff):
    """Short, long and wide pairs in chunks of 2^20 slots on two streams, from
    the bitset (the stage join and the batched form that materialises it) and
    from the planes, against one chunk."""
    queue = sb.Queue(0)
    d = sb.generate_molecules(32_000, 10, 60, seed=3811)
    q = sb.generate_queries(700, 3, 30, seed=3812, skew_lo=6, skew_hi=15)
    qg, dg = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, d)
    gm, cand = sb.GMCR(queue), sb.Candidates(queue, qg.total_nodes, dg.total_nodes)
    ref = sb.match_batched(queue, qg, dg, 3, ff, None, gm)
    assert ref["admitted_pairs"] > 2 * (1 << 20)  # three chunks
    counts = gm.getPairCounts()
    for serial in (1, 0):
        queue.set_tuning(mask_chunk_slots=1, overflow_serial=serial)
        for bits in (cand, None):
            g2 = sb.GMCR(queue)
            res = sb.match_batched(queue, qg, dg, 3, ff, bits, g2, materialize=bits is not None)
            assert res["total_matches"] == ref["total_matches"] and np.array_equal(g2.getPairCounts(), counts)
            if bits is not None:
                total = np.zeros(1, np.uint64)
                _, per = sb.joinCandidates(queue, qg, dg, cand, g2, total, ff, per_pair=True)
                assert np.array_equal(per, counts) and int(total[0]) == ref["total_matches"]


@pytest.mark.parametrize("prof", ["ref-ptx", "exact"])
def test_budget_spent_among_wide_pairs(prof):
    """Queries of 17 to 20 vertices (the wide join alone): out of steps, then
    without a budget the oracle's counts."""
    ring = sb.generate_molecules(300, 20, 50, seed=3821, kind=2)
    q = _chains((17, 18, 20))
    ref = oracle.run_pipeline(q, ring, 2, PROF[prof], True)
    assert ref["total"] > 0
    queue = sb.Queue(0, profile=prof)
    qg, dg = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, ring)
    for graph in (False, True):
        gm = sb.GMCR(queue)
        queue.set_join_budget(2)
        with pytest.raises(sb.SigmoError) as ei:
            sb.match_batched(queue, qg, dg, 2, True, None, gm, graph=graph)
        assert ei.value.code == 7
        queue.set_join_budget(0)
        res = sb.match_batched(queue, qg, dg, 2, True, None, gm, graph=graph)
        assert res["total_matches"] == ref["total"] and np.array_equal(gm.getPairCounts(), ref["per_pair"])


def _broom(n, leaves, hub):
    """A chain of n vertices whose last one, of label `hub`, carries `leaves` vertices."""
    edges = [(i, i + 1) for i in range(n - 1)] + [(n - 1, n + i) for i in range(leaves)]
    labels = [8] * (n - 1) + [hub] + [8] * leaves
    return (f"n#{n + leaves} l#1 " + " ".join(f"{i} {x}" for i, x in enumerate(labels)) + f" e#{len(edges)} " +
            " ".join(f"{u} {v} 1" for u, v in edges))


@pytest.mark.parametrize("prof,ff", MODES)
@pytest.mark.parametrize("chain,leaves,copies", [(1, 40, 1), (9, 30, 6), (16, 30, 2), (1, 100, 6), (5, 120, 2), (14, 190, 1),
                                                 (3, 9, 300), (3, 9, 1200)])
def test_pairs_with_one_root_candidate(chain, leaves, copies, prof, ff):
    """The hub of a star is one candidate: its pair's parts are shares of the
    next level's.  Patterns of 2 vertices (whose next level is the last), up to
    10, 11 to 16 and more, molecules of one, two and four words, few pairs and
    several batches of wide ones, below vertex 256 and above."""
    patterns = [_broom(1, k, 7) for k in (1, 2, 3)] + [_broom(k, 2, 7) for k in (2, min(chain, 8), chain)]
    q = sb.io.parse("\n".join(patterns) + "\n")
    molecules = [_broom(chain, leaves - i, 7) for i in range(3)] + [_broom(2, 3, 7)]
    d = sb.io.parse("\n".join(molecules * copies + [_broom(30, 3, 0)] * 10 + molecules * copies) + "\n")
    ref = _check(q, d, 1, prof, ff)
    assert ref["total"] > 0
