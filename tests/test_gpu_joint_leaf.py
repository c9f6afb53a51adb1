"""Entries whose leaf hangs on the same earlier vertex have that vertex's
candidates found once: run lengths and group sizes at their edges, ranges up
to and past the length taken this way, no, some and many earlier vertices of
the leaf's label; counts, hashes and per-depth counts against the oracle.
"""
import math

import numpy as np
import pytest

import fsig_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def brooms(centers, arms, others):
    """A root with `centers` neighbours, each with arms of label 2 and others of label 3."""
    labels, edges = [0] + [1] * centers, [(0, 1 + c) for c in range(centers)]
    for c in range(centers):
        for label in [2] * arms + [3] * others:
            labels.append(label)
            edges.append((1 + c, len(labels) - 1))
    return F.Graph(np.array(labels, np.int32), np.array(edges, np.uint32))


@pytest.mark.parametrize("centers,arms,others,k", [
    (1, 1, 1, 1), (6, 3, 2, 2), (5, 31, 7, 1), (5, 32, 33, 1), (3, 33, 32, 2), (40, 2, 5, 1), (700, 1, 3, 1),
    (2, 65, 95, 1), (2, 65, 96, 1), (2, 65, 97, 1), (1, 40, 3000, 1), (1, 20, 20000, 1),
    (6, 2, 0, 2), (6, 33, 0, 2), (4, 96, 0, 2), (4, 97, 0, 2), (2, 128, 0, 2), (2, 40, 0, 3), (1, 1500, 0, 2),
    (3, 6, 0, 5), (3, 7, 0, 6), (2, 9, 0, 7), (1, 9, 0, 9), (1, 10, 0, 10), (2, 7, 3, 6),
])
@pytest.mark.parametrize("index", [F.SEGMENTS_TABLE, F.SEGMENTS_ROWS])
def test_runs_groups_and_ranges(centers, arms, others, k, index):
    g = brooms(centers, arms, others)
    off, adj = g.csr()
    labels = [0, 1] + [2] * k + ([3] if others else [])
    n = len(labels)
    q = F.Query(np.array(labels, np.int32), np.array([(0, 1)] + [(1, i) for i in range(2, n)], np.uint32),
                order=np.arange(n, dtype=np.uint32))
    count, hsh = O.match(g.labels, off, adj, q.labels, q.edges)[:2]
    assert count == centers * math.perm(arms, k) * max(others, 1)
    with F.Engine(0, arena_bytes=2 << 30) as e:
        e.set_segment_index(index)
        e.load_graph(g)
        r = e.match(q, algo=F.ALGO_FUSED)
        assert (r.count, r.hash) == (count, hsh)
        assert r.level_counts == ([1, centers] + [centers * math.perm(arms, i) for i in range(1, k + 1)]
                                  + ([count] if others else []))
        limited = e.match_batch([q], algo=F.ALGO_FUSED, order_source=F.ORDER_GIVEN, max_work=1 << 40)[0]
        assert (limited.count, limited.hash) == (count, hsh)
        assert limited.work == sum(r.level_counts[d] * len_ for d, len_ in
                                   enumerate([centers] + [arms] * k + ([others] if others else [])))
