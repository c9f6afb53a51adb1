"""Rows of the device CSR and of the graph store at the lengths where the row
sort changes: one warp (32), one block in shared memory (2048, 16384), chunks
of 16384 merged pairwise (one to eight of them, odd numbers and remainders),
with and without repeated edges.  (Row order and repeats as the reference's
transform leaves them: graph_format_transformer.cc:12-37.)
"""
import numpy as np
import pytest

import fsig_gb300 as F

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 31, 32, 33, 2047, 2048, 2049, 16383, 16384, 16385, 32768, 32769, 49153, 65537, 120000]


def stars(lengths, repeats, rng):
    """One hub per length, its neighbours drawn from the common leaves, edges shuffled."""
    H, leaves = len(lengths), 130000
    parts = []
    for h, n in enumerate(lengths):
        nb = rng.choice(leaves, n, replace=False) + H
        if repeats:
            nb[: n // 3] = nb[n - n // 3:]  # every third neighbour twice
        parts.append(np.stack([np.full(n, h), nb], 1))
    e = np.concatenate(parts)
    e = e[rng.permutation(len(e))]
    flip = rng.random(len(e)) < 0.5
    e[flip] = e[flip][:, ::-1]
    return H + leaves, e.astype(np.uint32)


@pytest.mark.parametrize("lengths", [LENGTHS, [16385], [40000, 5], [120000] * 3, [16384, 2048, 32]])
@pytest.mark.parametrize("repeats", [False, True])
def test_csr_and_store_of_long_rows(engine, lengths, repeats):
    rng = np.random.default_rng(len(lengths) + repeats)
    V, e = stars(lengths, repeats, rng)
    off, adj = engine.build_csr(V, e)
    both = np.concatenate([e, e[:, ::-1]]).astype(np.int64)
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    assert np.array_equal(np.diff(off.astype(np.int64)), np.bincount(both[:, 0], minlength=V))
    assert np.array_equal(adj, both[:, 1])
    # the store: repeats dropped; every edge and every two-edge path found, signatures by the filter's flags
    uniq = np.unique(both, axis=0)
    deg = np.bincount(uniq[:, 0], minlength=V).astype(np.int64)
    lab = (np.arange(V) >= len(lengths)).astype(np.int32)
    engine.load_graph(F.Graph(lab, e))
    info = engine.graph_info()
    assert (info["adj"], info["max_degree"]) == (len(uniq), int(deg.max()))
    r = engine.match(F.Query(np.array([0, 1], np.int32), np.array([[0, 1]], np.uint32)))
    assert r.count == len(uniq) // 2
    hub = deg[: len(lengths)]
    r = engine.match(F.Query(np.array([1, 0, 1], np.int32), np.array([[0, 1], [1, 2]], np.uint32)))
    assert r.count == int((hub * (hub - 1)).sum())
    sig = engine.build_signature(lab, off, adj)
    assert np.count_nonzero(sig.reshape(V, 16)[:, 1:].any(1)) == np.count_nonzero(np.diff(off.astype(np.int64)))
