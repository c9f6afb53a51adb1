"""What a batch uploads and brings back, by its statistics: no more than its
parts, and every copy counted once."""
import numpy as np
import pytest

import fsig_gb300 as F

pytestmark = pytest.mark.gpu


def triangle():
    return F.Query(np.zeros(3, np.int32), np.array([[0, 1], [1, 2], [2, 0]], np.uint32))


def test_a_batch_uploads_its_descriptors_only():
    g = F.gen_rmat(256, 2048, 0.57, 0.19, 0.19, seed=5)
    with F.Engine(0, arena_bytes=1 << 30) as e:
        e.load_graph(g)
        sizes = []
        for n in (64, 640):
            e.match_batch([triangle()] * n)
            sizes.append(e.last_stats()["h2d_bytes"])
        # parts are padded to 256 bytes, which 64 queries fill.  A vertex: its
        # 112-byte descriptor, label group entry, order, score and first bitmap
        # word (8 bytes); a query: its first vertex
        assert sizes[1] - sizes[0] == 576 * (3 * (112 + 4 + 4 + 4 + 8) + 4)


def test_copies_back_are_counted_once():
    """A graph brings its results back with the first pass and after the last
    one, ordinary launches after every pass; each pass its counters (four lines
    of 128 bytes), each but the last the number of records it left."""
    g = F.gen_rmat(256, 2048, 0.57, 0.19, 0.19, seed=3)
    q = F.Query(np.zeros(5, np.int32), np.array([[0, 1], [1, 2], [2, 3], [3, 4], [4, 0]], np.uint32))
    kw = dict(algo=F.ALGO_FUSED, split_cycles=1000, split_len=32)

    def copied(e, use_graph):
        e.match_batch([q], use_graph=use_graph, **kw)
        st = e.last_stats()
        return st["enum_passes"], st["d2h_bytes"]

    with F.Engine(0, arena_bytes=2 << 30) as e:
        e.load_graph(g)
        for use_graph in (False, True):
            passes, one = copied(e, use_graph)
            assert passes == 1
            results = one - 512
            e.set_queue_waits(idle_wait_ns=1)  # waiting warps leave: their records are later passes'
            for _ in range(5):
                p, b = copied(e, use_graph)
                assert p > 1
                assert b == (2 if use_graph else p) * results + 512 * p + 4 * (p - 1)
            e.set_queue_waits()
