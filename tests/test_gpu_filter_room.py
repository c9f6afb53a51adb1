"""A call that needs the membership filter's room gets it, matches without the
filter, and the filter is built again by the next call that leaves the room
free: present, gone and present again, with the oracle's results in every
state, as ordinary launches and as a CUDA graph, with and without the segment
table.  The room is taken by calls that succeed: the largest row buffer that is
accepted ends where the arena does, on top of the filter."""
import numpy as np
import pytest

import fsig_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ARENA = (2 << 30) + 4096


def cycle(n, chords=()):
    return F.Query(np.zeros(n, np.int32), np.array([(i, (i + 1) % n) for i in range(n)] + list(chords), np.uint32))


def largest_buffer(e, q):
    """The most rows a match_embeddings buffer may have."""
    lo, hi = 1, ARENA // (4 * q.num_vertices)
    while lo < hi:
        mid = (lo + hi + 1) // 2
        try:
            e.match_embeddings(q, F.ALGO_FUSED, buffer_rows=mid)
            lo = mid
        except F.FsigError as err:
            assert err.status == F.EADMISSION
            hi = mid - 1
    return lo


@pytest.mark.parametrize("index", [F.SEGMENTS_TABLE, F.SEGMENTS_ROWS])
def test_filter_gives_its_room_and_comes_back(index):
    g = F.gen_rmat(700, 11200, 0.57, 0.19, 0.19, seed=700)
    off, adj = g.csr()
    q = cycle(3)
    batch = [q, cycle(4, [(0, 2)])]
    want = [O.match(g.labels, off, adj, x.labels, x.edges)[:2] for x in batch]
    with F.Engine(0, arena_bytes=ARENA) as e:
        e.set_segment_index(index)
        e.load_graph(g)
        size = e.graph_filter()
        assert size == 2 * 4 * e.graph_info()["adj"]  # four 16-bit words an entry
        rows = largest_buffer(e, q)

        def take_room():
            r, found = e.match_embeddings(q, F.ALGO_FUSED, buffer_rows=rows)
            assert (r.count, r.hash) == want[0] and len(found) == r.count
            assert e.graph_filter() == 0

        def with_filter(**kw):
            rs = e.match_batch(batch, algo=F.ALGO_FUSED, **kw)
            assert [(r.count, r.hash) for r in rs] == want
            assert e.graph_filter() == size
            return [r.level_counts for r in rs], e.last_stats()["kernel_launches"]

        take_room()
        take_room()  # a call that needs the room does not build the filter
        levels, first = with_filter()
        again, second = with_filter()
        assert levels == again and first == second + 1  # built once
        for use_graph in (True, False, True):
            take_room()
            for _ in range(3):
                assert with_filter(use_graph=use_graph)[0] == levels
        # a batch that is refused on the way (2.2 GB of root lists alone; the limit
        # on work is for the case that it is not)
        take_room()
        path = F.Query(np.zeros(32, np.int32), np.array([(i, i + 1) for i in range(31)], np.uint32))
        with pytest.raises(F.FsigError) as ei:
            e.match_batch([path] * 200000, algo=F.ALGO_FUSED, max_work=1)
        assert ei.value.status == F.EADMISSION
        assert with_filter()[0] == levels


def test_no_filter_in_a_small_arena():
    g = F.gen_rmat(700, 11200, 0.57, 0.19, 0.19, seed=700)
    off, adj = g.csr()
    q = cycle(4, [(0, 2)])
    with F.Engine(0, arena_bytes=512 << 20) as e:
        with pytest.raises(F.FsigError) as ei:
            e.graph_filter()
        assert ei.value.status == F.ENOGRAPH
        e.load_graph(g)
        assert e.graph_filter() == 0
        for use_graph in (False, True):
            r, = e.match_batch([q], use_graph=use_graph)
            assert (r.count, r.hash) == O.match(g.labels, off, adj, q.labels, q.edges)[:2]
        assert e.graph_filter() == 0
