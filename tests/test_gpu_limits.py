"""Calls at the limits of a tile, of device memory and of the forms' sizes:
served, and with the oracle's results (whole numbers: equal)."""
import contextlib
import ctypes
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import oracle
import sigmo_b200 as sb

pytestmark = pytest.mark.gpu


def _graph(n, edges, labels):
    return (f"n#{n} l#1 " + " ".join(f"{i} {labels[i]}" for i in range(n)) + f" e#{len(edges)} " +
            " ".join(f"{u} {v} 1" for u, v in edges))


def _broom(path, leaves, label):
    """A path whose last vertex carries `leaves` vertices of one label: the
    path's vertices have them at every distance up to its length."""
    edges = [(i, i + 1) for i in range(path - 1)] + [(path - 1, path + i) for i in range(leaves)]
    return _graph(path + leaves, edges, [8] * path + [label] * leaves)


def _thresholds(q, R):
    sig, out = oracle.generate_signatures(q), set()
    reach = oracle.new_reach(len(sig), oracle.REF_PTX)
    for r in range(1, R + 1):
        sig = oracle.refine_signatures(q, r, oracle.REF_PTX, sig, reach)
        out.update((r, l, (v >> (4 * l)) & 15) for v in sig.tolist() for l in range(16) if (v >> (4 * l)) & 15)
    return out


class _PoolProps(ctypes.Structure):  # CUmemPoolProps
    _fields_ = [("alloc_type", ctypes.c_int), ("handle_types", ctypes.c_int), ("location_type", ctypes.c_int),
                ("location_id", ctypes.c_int), ("security", ctypes.c_void_p), ("max_size", ctypes.c_size_t),
                ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]


_small_pool = ctypes.c_void_p()  # kept: objects that outlive a test may hold memory of it


@contextlib.contextmanager
def _short_of_memory(free):
    """Stream-ordered allocations come from a pool of 64 MB of which about
    `free` MB are left."""
    cu = ctypes.CDLL("libcuda.so.1")
    ok = lambda rc: rc == 0 or pytest.fail(f"CUDA driver error {rc}")  # noqa: E731
    before, pool = ctypes.c_void_p(), _small_pool
    ok(cu.cuDeviceGetMemPool(ctypes.byref(before), 0))
    if not pool:
        ok(cu.cuMemPoolCreate(ctypes.byref(pool), ctypes.byref(_PoolProps(1, 0, 1, 0, None, 64 << 20, 0))))
    blocks = []
    while len(blocks) < 1024:
        p = ctypes.c_uint64()
        if cu.cuMemAllocFromPoolAsync(ctypes.byref(p), ctypes.c_size_t(1 << 20), pool, None):
            break
        blocks.append(p)
    assert free < len(blocks) < 1024
    for _ in range(free):
        ok(cu.cuMemFreeAsync(blocks.pop(), None))
    ok(cu.cuStreamSynchronize(None))
    ok(cu.cuDeviceSetMemPool(0, pool))
    try:
        yield
    finally:
        ok(cu.cuDeviceSetMemPool(0, before))
        for p in blocks:
            ok(cu.cuMemFreeAsync(p, None))
        ok(cu.cuStreamSynchronize(None))


def _filtered(queue, qg, dg, R):
    cand = sb.Candidates(queue, qg.total_nodes, dg.total_nodes)
    sig = sb.Signature(queue, dg.total_nodes, qg.total_nodes)
    sig.generateDataSignatures(dg)
    sig.generateQuerySignatures(qg)
    sb.filterCandidates(queue, qg, dg, sig, cand)
    for r in range(1, R + 1):
        sig.refineDataSignatures(dg, r)
        sig.refineQuerySignatures(qg, r)
        sb.refineCandidates(queue, qg, dg, sig, cand)
    queue.wait()
    return cand


def test_join_after_the_matching_order_ran_out_of_memory():
    """The matching order's first array fits, its second does not: the call
    fails, and the next one starts over."""
    d, q = sb.generate_molecules(20, 10, 40, seed=3711), sb.generate_queries(60_000, 4, 14, seed=3712)
    assert q.total_nodes * 8 > 3 << 20 > q.total_nodes
    ref = oracle.run_pipeline(q, d, 2, oracle.REF_PTX, True)
    queue = sb.Queue(0)
    qg, dg = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, d)
    cand = _filtered(queue, qg, dg, 2)
    gm = sb.GMCR(queue)
    gm.generateGMCR(qg, dg, cand)
    with _short_of_memory(3):
        with pytest.raises(sb.SigmoError) as ei:
            sb.joinCandidates(queue, qg, dg, cand, gm, np.zeros(1, np.uint64), True)
        assert ei.value.code == 3
    total = np.zeros(1, np.uint64)
    _, per = sb.joinCandidates(queue, qg, dg, cand, gm, total, True, per_pair=True)
    assert np.array_equal(per, ref["per_pair"]) and int(total[0]) == ref["total"]


def test_join_after_the_mapping_ran_out_of_memory():
    """A mapping whose arrays did not all fit is refused by the join."""
    d, q = sb.generate_molecules(20, 10, 40, seed=3711), sb.generate_queries(60_000, 4, 14, seed=3712)
    ref = oracle.run_pipeline(q, d, 2, oracle.REF_PTX, True)
    assert len(ref["indices"]) * 16 > 3 << 20 > len(ref["indices"]) * 4
    queue = sb.Queue(0)
    qg, dg = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, d)
    cand = _filtered(queue, qg, dg, 2)
    gm, total = sb.GMCR(queue), np.zeros(1, np.uint64)
    with _short_of_memory(3):
        with pytest.raises(sb.SigmoError) as ei:
            gm.generateGMCR(qg, dg, cand)
        assert ei.value.code == 3
    with pytest.raises(sb.SigmoError) as ei:
        sb.joinCandidates(queue, qg, dg, cand, gm, total, True)
    assert ei.value.code == 1 and int(total[0]) == 0
    gm.generateGMCR(qg, dg, cand)
    off, idx = gm.getGMCR()
    assert np.array_equal(off, ref["offsets"]) and np.array_equal(idx, ref["indices"])
    _, per = sb.joinCandidates(queue, qg, dg, cand, gm, total, True, per_pair=True)
    assert np.array_equal(per, ref["per_pair"]) and int(total[0]) == ref["total"]


_IN_LITTLE_MEMORY = """
import sys
import numpy as np
import torch
import sigmo_b200 as sb
sys.path.insert(0, "tests")
from test_gpu_limits import _filtered

def stage_join(cand, gm, ff):
    total = np.zeros(1, np.uint64)
    return sb.joinCandidates(queue, qg, dg, cand, gm, total, ff, per_pair=True)[1], int(total[0])

def fill(left):
    torch.cuda.synchronize()
    return torch.empty(torch.cuda.mem_get_info()[0] - (left << 20), dtype=torch.uint8, device="cuda")

profile, long = sys.argv[1], sys.argv[2] == "long"
queue = sb.Queue(0, profile=profile)
hi = 30 if long else 9
for count in (400, 30_000):  # the kernels are loaded before the memory is short
    q = sb.generate_queries(300, 3, hi, seed=3722, skew_lo=6, skew_hi=min(hi, 15))
    qg, dg = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, sb.generate_molecules(count, 10, 60, seed=3721))
    cand, gm = _filtered(queue, qg, dg, 3), sb.GMCR(queue)
    gm.generateGMCR(qg, dg, cand)
    if count == 400:
        stage_join(cand, gm, False)
pairs = gm.total_query_indices
assert pairs * 144 > 128 << 20, pairs  # the pair join's masks
rest = fill(64)
short = [stage_join(cand, gm, ff) for ff in (False, True)]
del rest
torch.cuda.empty_cache()
plenty = sb.GMCR(queue)
for (per, total), ff in zip(short, (False, True)):
    res = sb.match_batched(queue, qg, dg, 3, ff, None, plenty)
    assert np.array_equal(per, plenty.getPairCounts()) and total == res["total_matches"] > 0
# what the temporaries kept is given back to an allocation that needs it
rest = fill(64)
more = sb.Candidates(queue, 1000, 8 * 100_000 * 8 // 5)
print("ok", pairs)
"""


@pytest.mark.parametrize("queries", ["short", "long"])
@pytest.mark.parametrize("profile", ["ref-ptx", "exact"])
def test_stage_join_in_little_memory(profile, queries):
    """The stage join beside its bitset, on a card that is otherwise full: runs
    of fewer pairs, with the counts of the batched form.  In a process of its
    own, whose memory pools hold nothing yet."""
    root = Path(__file__).resolve().parent.parent
    r = subprocess.run([sys.executable, "-c", _IN_LITTLE_MEMORY, profile, queries], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("profile", ["ref-ptx", "exact"])
def test_serving_a_batch_with_more_planes_than_a_tile(wide, profile):
    """16 labels x 15 counts x 6 distances: more planes than a tile of 200 KB
    holds, most of them beyond every count of the database."""
    R = 6
    d = sb.generate_molecules(200, 10, 120 if wide else 40, seed=3701, kind=1 if wide else 0)
    assert (d.sizes().max() > 64) == wide
    d = d.concat(sb.io.parse("\n".join(_broom(6, c, l) for c in (2, 3, 5) for l in (0, 7)) + "\n"))
    q = sb.io.parse("\n".join(_broom(6, c, l) for l in range(16) for c in range(1, 16)) + "\n")
    small = sb.generate_queries(20, 3, 8, seed=3702)
    assert len(_thresholds(q, R)) * 32 * 8 > 225 * 1024
    prof = {"ref-ptx": oracle.REF_PTX, "exact": oracle.EXACT}[profile]
    with sb.Server(d, profile=profile, iterations=R, find_first=False, max_inflight=1) as srv:
        for request in (q, small.concat(q), small):
            t = srv.submit(request, pairs=True)
            assert srv.wait(t)["status"] == 0
            matched, total = srv.query_totals(t, request.num_graphs)
            pairs = srv.pairs(t)
            ref = oracle.run_pipeline(request, d, R, prof, False)
            keep = ref["per_pair"] != 0
            graph = np.repeat(np.arange(d.num_graphs), np.diff(ref["offsets"].astype(np.int64)))
            assert np.array_equal(pairs[0], ref["indices"][keep]) and np.array_equal(pairs[1], graph[keep].astype(np.uint32))
            assert np.array_equal(pairs[2], ref["per_pair"][keep])
            want = np.zeros(request.num_graphs, np.uint64)
            np.add.at(want, ref["indices"].astype(np.int64), ref["per_pair"])
            assert np.array_equal(total, want) and keep.any()
            assert np.array_equal(matched, np.bincount(ref["indices"][keep], minlength=request.num_graphs).astype(np.uint64))


@pytest.mark.parametrize("hi,lists", [(10, 0), (16, 1), (30, 2)])
def test_serving_estimate_holds_the_joins_lists(hi, lists):
    """A batch's projected device bytes: mapping, level masks and, by the
    queries' sizes, the lists of long and of wide pairs, for every pair, the
    result lists and 16 MB."""
    d = sb.generate_molecules(20_000, 10, 40, seed=3731)
    q = sb.generate_queries(12, 3, 8, seed=3732).concat(sb.generate_queries(1, hi, hi, seed=3733))
    assert q.sizes().max() == hi
    pairs = d.num_graphs * q.num_graphs
    with sb.Server(d, iterations=3, max_inflight=1) as srv:
        projected = srv.wait(srv.submit(q))["projected_bytes"]
    need = 4 * d.num_graphs + pairs * (16 + 144 + 4 * lists + 20) + (16 << 20)
    assert need <= projected <= need + (1 << 20)


def _dense(n, degree, seed, loops=()):
    """A random graph; a vertex of `loops` gets a self-loop, whose second CSR
    entry names vertex 0 (an edge that vertex 0 does not have back)."""
    rng = np.random.default_rng(seed)
    u, v = np.nonzero(np.triu(rng.random((n, n)) < degree / n, 1))
    order = rng.permutation(len(u))
    edges = [(int(u[i]), int(v[i])) for i in order] + [(x, x) for x in loops]
    return _graph(n, edges, rng.choice([0, 7, 8], n).tolist())


@pytest.mark.parametrize("profile", [oracle.REF_PTX, oracle.EXACT])
@pytest.mark.parametrize("widest", [64, 128, 256])
def test_graph_creation_by_degree_and_position(widest, profile):
    """Adjacency rows and the mirrored flag (an unmirrored graph is joined in
    identity order): vertices of 8, 9 and more entries beside molecules, graphs
    that lie in one, two and three ranges of 256 vertices, more than 256 empty
    graphs in a row, unmirrored graphs of every kind."""
    from test_gpu_join_forms import _check

    sizes = [n for n in (9, 10, 63, 64, 65, 127, 128, 129, 200, 255, 256) if n <= widest]
    lines = [_graph(n, [(i, j) for i in range(n) for j in range(i + 1, n)], [8] * n) for n in (9, 10)]
    for k, n in enumerate(sizes):
        lines += [_dense(n, 6, k), _dense(n, 14, 100 + k), _dense(n, 14, 200 + k, loops=(3, n - 1)), _dense(n, 3, 300 + k, loops=(5,))]
    lines += ["n#0 l#0 e#0"] * 600 + [_graph(n, [(0, i) for i in range(1, n)], [8] * n) for n in sizes]
    lines += ["n#0 l#0 e#0"] * 300
    molecules = sb.generate_molecules(40, 5, 40, seed=3741)
    dense = sb.io.parse("\n".join(lines) + "\n")
    assert dense.num_graphs > 900 and dense.sizes().max() == widest
    d = dense.concat(molecules).concat(dense).concat(molecules)
    queries = [_graph(2, [(0, 1)], [8, 7]), _graph(3, [(0, 1), (1, 2)], [8, 7, 8]), _graph(3, [(0, 1), (1, 2), (2, 0)], [8, 8, 8]),
               _graph(4, [(0, 1), (0, 2), (0, 3)], [8, 0, 7, 7]), _graph(4, [(0, 1), (1, 2), (2, 3), (3, 0)], [8, 7, 8, 0]),
               _graph(3, [(0, 1), (1, 2), (1, 1)], [8, 7, 8])]
    for ff in (False, True):
        ref = _check(sb.io.parse("\n".join(queries) + "\n"), d, 1, {oracle.REF_PTX: "ref-ptx", oracle.EXACT: "exact"}[profile], ff)
        assert (ref["per_pair"] > 0).sum() > 100


@pytest.mark.parametrize("wg", [32, 128, 1024])
@pytest.mark.parametrize("hi", [9, 32, 33])
def test_literal_search_over_many_graphs(hi, wg):
    """REF_X86 takes the literal search for every molecule: more of them than
    the small blocks are for, work-groups of fewer and more items than a block,
    queries up to the levels that shared memory holds and one past it."""
    d = sb.generate_molecules(300, 5, 64, seed=3751)
    q = sb.generate_queries(60, 2, 9, seed=3752).concat(sb.generate_queries(3, hi, hi, seed=3753))
    assert q.sizes().max() == hi
    queue = sb.Queue(0, profile="ref-x86", join_work_group_size=wg)
    qg, dg = sb.createDeviceCSRGraph(queue, q), sb.createDeviceCSRGraph(queue, d)
    cand, gm = _filtered(queue, qg, dg, 2), sb.GMCR(queue)
    gm.generateGMCR(qg, dg, cand)
    off, idx = gm.getGMCR()
    for ff in (False, True):
        ref = oracle.run_pipeline(q, d, 2, oracle.REF_X86, ff, wg=wg)
        assert np.array_equal(off, ref["offsets"]) and np.array_equal(idx, ref["indices"]) and np.diff(off.astype(int)).max() > 32
        total = np.zeros(1, np.uint64)
        _, per = sb.joinCandidates(queue, qg, dg, cand, gm, total, ff, per_pair=True)
        assert np.array_equal(per, ref["per_pair"]) and int(total[0]) == ref["total"] > 0
