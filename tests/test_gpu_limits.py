"""Calls at the limits of a tile, of device memory and of the forms' sizes:
served, and with the oracle's results (whole numbers: equal)."""
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
