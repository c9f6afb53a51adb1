"""The buffer of the last depth but one takes more entries than the others when
the leaf's ranges are short: sizes at the edges of both lengths and of the
leaf's groups, ranges short and long, counts, hashes, per-depth counts and
embeddings against the oracle.
"""
import numpy as np
import pytest

import fsig_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def tree(widths):
    """Every vertex of depth i has widths[i] children, labeled by depth."""
    labels, edges, level = [0], [], [0]
    for d, w in enumerate(widths):
        nxt = []
        for v in level:
            for _ in range(w):
                labels.append(d + 1)
                edges.append((v, len(labels) - 1))
                nxt.append(len(labels) - 1)
        level = nxt
    return F.Graph(np.array(labels, np.int32), np.array(edges, np.uint32))


@pytest.mark.parametrize("mid", [1, 31, 32, 33, 127, 128, 129, 160, 500])
@pytest.mark.parametrize("leaves", [1, 3, 23, 24, 70])
@pytest.mark.parametrize("index", [F.SEGMENTS_TABLE, F.SEGMENTS_ROWS])
def test_last_depth_lengths(mid, leaves, index):
    g = tree([4, 8, mid, leaves] if mid * leaves < 4000 else [2, 3, mid, leaves])
    off, adj = g.csr()
    n = 5
    q = F.Query(np.arange(n, dtype=np.int32), np.array([(i, i + 1) for i in range(n - 1)], np.uint32),
                order=np.arange(n, dtype=np.uint32))
    count, hsh = O.match(g.labels, off, adj, q.labels, q.edges)[:2]
    with F.Engine(0, arena_bytes=2 << 30) as e:
        e.set_segment_index(index)
        e.load_graph(g)
        r = e.match(q, algo=F.ALGO_FUSED)
        assert (r.count, r.hash) == (count, hsh)
        assert r.level_counts == [int((g.labels == d).sum()) for d in range(n)]
        _, rows = e.match_embeddings(q, algo=F.ALGO_FUSED)
    assert len(rows) == count
    assert (g.labels[rows] == np.arange(n)).all()
    assert len(np.unique(rows[:, n - 1])) == count
