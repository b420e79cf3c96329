"""Captured batches against what may change between their replays, and calls
that run short of device memory: results equal the oracle's (whole numbers)."""
import numpy as np
import pytest

import oracle
import sigmo_b200 as sb

pytestmark = pytest.mark.gpu


def _equal(gm, res, ref):
    off, idx = gm.getGMCR()
    assert np.array_equal(off, ref["offsets"]) and np.array_equal(idx, ref["indices"])
    assert np.array_equal(gm.getPairCounts(), ref["per_pair"]) and res["total_matches"] == ref["total"]


def test_replay_after_the_query_graph_ran_with_other_iterations():
    """The query graph holds one plane program; a captured batch keeps the one
    that its kernels read."""
    d, q = sb.generate_molecules(1500, 10, 40, seed=3601), sb.generate_queries(60, 3, 20, seed=3602)
    want = {R: oracle.run_pipeline(q, d, R, oracle.REF_PTX, False) for R in (6, 3)}
    assert not np.array_equal(want[6]["offsets"], want[3]["offsets"])
    queue = sb.Queue(0)
    qg, dg = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, d)
    a, b = sb.GMCR(queue), sb.GMCR(queue)
    sb.match_batched(queue, qg, dg, 6, False, None, a, graph=True)  # runs and captures
    for _ in range(2):
        res = sb.match_batched(queue, qg, dg, 3, False, None, b)
        _equal(b, res, want[3])
        others = [sb.createDeviceCSRGraph(queue, q) for _ in range(4)]  # takes memory that was freed
        res = sb.match_batched(queue, qg, dg, 6, False, None, a, graph=True)
        assert res["ms_signatures"] == 0.0  # a replay: its stages are not timed
        _equal(a, res, want[6])
        del others


def test_replay_after_the_query_graph_was_grouped_for_another_set_width():
    """A batch admitted in groups: the groups are planned for one set width, a
    captured batch keeps the ones that its kernels read."""
    R = 6
    two = sb.generate_molecules(300, 6, 120, seed=4903, kind=1, median=22.0)
    four = sb.generate_molecules(60, 130, 250, seed=3612, kind=1, median=150.0)
    assert 64 < two.sizes().max() <= 128 < four.sizes().max()
    q = sb.generate_queries(2000, 3, 64, seed=4901)  # about 200 planes: over one tile of two words
    want = [oracle.run_pipeline(q, d, R, oracle.REF_PTX, True) for d in (two, four)]
    queue = sb.Queue(0)
    qg = sb.createDeviceCSRGraph(queue, q)
    dg = [sb.createDeviceCSRGraph(queue, d) for d in (two, four)]
    gm = [sb.GMCR(queue) for _ in dg]
    for call in range(4):  # run and capture each, then replays
        for i in (0, 1):
            res = sb.match_batched(queue, qg, dg[i], R, True, None, gm[i], graph=True)
            assert (res["ms_signatures"] == 0.0) == (call > 0)
            _equal(gm[i], res, want[i])


def test_replay_after_the_shard_moved():
    """The range masks and the literal join follow a shard's first global
    vertex: a batch captured for one is not replayed for another."""
    d, q = sb.generate_molecules(700, 10, 40, seed=3621), sb.generate_queries(40, 3, 12, seed=3622)
    queue = sb.Queue(0)
    qg, dg = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, d)
    gm, totals = sb.GMCR(queue), []
    for base in (0, 100_003, 100_017):
        dg.set_vertex_base(base)
        plain = sb.GMCR(queue)
        want = sb.match_batched(queue, qg, dg, 4, False, None, plain)
        for call in range(2):
            res = sb.match_batched(queue, qg, dg, 4, False, None, gm, graph=True)
            assert (res["ms_signatures"] == 0.0) == (call > 0)
            assert res["total_matches"] == want["total_matches"] and res["admitted_pairs"] == want["admitted_pairs"]
            assert all(np.array_equal(x, y) for x, y in zip(gm.getGMCR(), plain.getGMCR()))
            assert np.array_equal(gm.getPairCounts(), plain.getPairCounts())
        totals.append(want["total_matches"])
    assert len(set(totals)) == 3


def test_replay_across_a_tuning_field_without_effect():
    d, q = sb.generate_molecules(500, 10, 40, seed=3631), sb.generate_queries(20, 3, 20, seed=3632)
    queue = sb.Queue(0)
    qg, dg, gm = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, d), sb.GMCR(queue)
    first = sb.match_batched(queue, qg, dg, 3, False, None, gm, graph=True)
    for field, replays in (("overflow_split", True), ("overflow_blocks", False)):
        queue.set_tuning(**{field: 5})
        res = sb.match_batched(queue, qg, dg, 3, False, None, gm, graph=True)
        assert (res["ms_signatures"] == 0.0) == replays and res["total_matches"] == first["total_matches"]
