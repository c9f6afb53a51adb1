"""Any split length gives the same counts, hashes and per-depth counts, from
the shortest pieces to lengths whose sum with a position does not fit 32 bits."""
import numpy as np
import pytest

import fsig_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [32, 33, 256, 1 << 20, 0x7FFFFFFF, 0x80000000, 0xFFFFFF00, 0xFFFFFFFE, 0xFFFFFFFF])
def test_split_lengths(engine, split):
    g = F.gen_rmat(1 << 10, 1 << 13, 0.57, 0.19, 0.19, seed=9, labels=F.gen_labels(1 << 10, 3, "zipf", seed=9))
    off, adj = g.csr()
    engine.load_graph(g)
    qs = [F.gen_query(g, n, F.QUERY_DENSE, seed=n, csr=(off, adj)) for n in (2, 3, 4, 5)]
    want = [O.match(g.labels, off, adj, q.labels, q.edges)[:2] for q in qs]
    for use_graph in (False, True):
        rs = engine.match_batch(qs, algo=F.ALGO_FUSED, split_len=split, use_graph=use_graph)
        assert [(r.count, r.hash) for r in rs] == want
    r, tasks = engine.match_range(qs[-1], F.ALGO_FUSED, split_len=split)
    assert (r.count, r.hash) == want[-1]
    parts = [engine.match_range(qs[-1], F.ALGO_FUSED, t, t + max(tasks // 3, 1), split_len=split)[0]
             for t in range(0, tasks, max(tasks // 3, 1))]
    assert sum(p.count for p in parts) == r.count
    assert sum(p.hash for p in parts) % (1 << 64) == r.hash
