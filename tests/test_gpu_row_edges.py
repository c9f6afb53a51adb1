"""Rows of the device CSR and of the graph store at the lengths where the
register sort of a warp changes (32 to 512 entries in powers of two) and where
a block's sort in shared memory takes over, with and without repeated edges,
in ascending, descending and random order of the edge list.  (Row order and
repeats as the reference's transform leaves them:
graph_format_transformer.cc:12-37.)
"""
import numpy as np
import pytest

import fsig_gb300 as F

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 15, 16, 17, 31, 32, 33, 63, 64, 65, 95, 127, 128, 129, 191, 255, 256, 257, 383, 511, 512, 513, 640]


@pytest.mark.parametrize("order", ["ascending", "descending", "random"])
@pytest.mark.parametrize("repeats", [False, True])
def test_rows_at_the_sorts_edges(engine, order, repeats):
    rng = np.random.default_rng(5)
    hubs, leaves = len(LENGTHS), 5000
    V = hubs + leaves
    parts = []
    for h, n in enumerate(LENGTHS):
        nb = np.sort(rng.choice(leaves, n, replace=False)) + hubs
        if repeats:
            nb[: n // 2] = nb[n - n // 2:]
            nb.sort()
        parts.append(np.stack([np.full(n, h), nb], 1))
    e = np.concatenate(parts).astype(np.uint32)
    if order == "descending":
        e = e[::-1]
    if order == "random":
        e = e[rng.permutation(len(e))]
    off, adj = engine.build_csr(V, e)
    both = np.concatenate([e, e[:, ::-1]]).astype(np.int64)
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    assert np.array_equal(np.diff(off.astype(np.int64)), np.bincount(both[:, 0], minlength=V))
    assert np.array_equal(adj, both[:, 1])
    uniq = np.unique(both, axis=0)
    deg = np.bincount(uniq[:, 0], minlength=V).astype(np.int64)
    engine.load_graph(F.Graph((np.arange(V) >= hubs).astype(np.int32), np.ascontiguousarray(e)))
    info = engine.graph_info()
    assert (info["adj"], info["max_degree"]) == (len(uniq), int(deg.max()))
    path = F.Query(np.array([1, 0, 1], np.int32), np.array([[0, 1], [1, 2]], np.uint32))
    r, rows = engine.match_embeddings(path)
    hub = deg[:hubs]
    assert r.count == len(rows) == int((hub * (hub - 1)).sum())
    # the middle vertex's neighbours, as the store has them
    for h in range(hubs):
        nb = uniq[uniq[:, 0] == h, 1]
        found = np.unique(rows[rows[:, 1] == h][:, 0])
        assert np.array_equal(found, nb if len(nb) > 1 else nb[:0])
