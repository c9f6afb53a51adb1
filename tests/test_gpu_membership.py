"""The membership filter of the graph store's label segments (exact bits for
segments dense in their label class, a Bloom filter for the others) never
changes a result: counts, hashes and per-depth counts with it, without it (an
arena with no room to spare) and after an oversize batch took its room back
are the oracle's, with and without the segment table.  (The reference decides
membership in hashed PCSR units, match/GSI_kernels.cuh:95-213.)
"""
import numpy as np
import pytest

import fsig_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# vertices, edges, labels: an unlabeled graph whose hubs' segments are dense
# and whose other segments are not; classes whose extents are no multiples of
# 32 or 16; many small classes; segments of one or two entries
GRAPHS = [(700, 11200, 1), (333, 2500, 3), (1023, 6000, 5), (4096, 30000, 40), (97, 300, 2)]


def cycle(n, chords=(), labels=None):
    e = [(i, (i + 1) % n) for i in range(n)] + list(chords)
    return F.Query(np.zeros(n, np.int32) if labels is None else np.asarray(labels, np.int32), np.array(e, np.uint32))


@pytest.mark.parametrize("V,E,L", GRAPHS)
@pytest.mark.parametrize("index", [F.SEGMENTS_TABLE, F.SEGMENTS_ROWS])
def test_filter_changes_no_result(V, E, L, index):
    g = F.gen_rmat(V, E, 0.57, 0.19, 0.19, seed=V, labels=F.gen_labels(V, L, "zipf", seed=V))
    off, adj = g.csr()
    qs = [F.gen_query(g, n, F.QUERY_DENSE, seed=50 + n, csr=(off, adj)) for n in ((3, 4) if L < 40 else (3, 4, 5, 6))]
    qs.append(cycle(3))
    if L > 1:
        qs.append(cycle(4, [(0, 2)], [0, 1, 0, 1]))
    want = [O.match(g.labels, off, adj, q.labels, q.edges)[:2] for q in qs]
    levels = []
    # with room for the filter; without; with it until a batch needs its room
    for arena, evict in ((4 << 30, False), (768 << 20, False), ((1 << 30) + (48 << 20), V == 700)):
        with F.Engine(0, arena_bytes=arena) as e:
            e.set_segment_index(index)
            e.load_graph(g)
            if evict:  # root lists, bitmaps and descriptors of more than the arena
                path = F.Query(np.zeros(32, np.int32), np.array([(i, i + 1) for i in range(31)], np.uint32))
                with pytest.raises(F.FsigError) as ei:
                    e.match_batch([path] * 60000, algo=F.ALGO_FUSED)
                assert ei.value.status == F.EADMISSION
            rs = e.match_batch(qs, algo=F.ALGO_FUSED)
            assert [(r.count, r.hash) for r in rs] == want
            levels.append([r.level_counts for r in rs])
    assert levels[0] == levels[1] == levels[2]


def test_cached_graph_has_the_filter_rebuilt(tmp_path):
    g = F.gen_rmat(700, 11200, 0.57, 0.19, 0.19, seed=7, labels=F.gen_labels(700, 2, "uniform", seed=7))
    off, adj = g.csr()
    q = cycle(4, [(0, 2)], [0, 1, 0, 1])
    want = O.match(g.labels, off, adj, q.labels, q.edges)[:2]
    path = tmp_path / "g.fsigcache"
    with F.Engine(0, arena_bytes=2 << 30) as e:
        e.load_graph(g)
        layout = e.graph_layout()
        e.save_graph_cache(path)
    for arena in (2 << 30, 768 << 20):
        with F.Engine(0, arena_bytes=arena) as e:
            e.load_graph_cache(path)
            assert e.graph_layout() == layout
            r = e.match(q, F.ALGO_GSI)
            assert (r.count, r.hash) == want
