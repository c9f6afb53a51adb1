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
