"""A graph cache whose arrays were changed in the file: the load, which builds
the membership filter from them, reads and writes inside the arrays (such a
store is not matched against here), and the engine then loads the unchanged
file and matches with the oracle's results."""
import numpy as np
import pytest

import fsig_gb300 as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def arrays(v, labels, nadj, table):
    """(name, first byte, words) of the file's arrays behind its 32-byte header."""
    at, out = 32, {}
    for name, words in (("label", v), ("old_of_new", v), ("new_of_old", v), ("base", labels + 1), ("off", v + 1),
                        ("adj", nadj), ("adj_old", nadj if table else 0), ("lseg", v * (labels + 1) if table else 0)):
        out[name] = (at, words)
        at += 4 * words
    return out


@pytest.mark.parametrize("index", [F.SEGMENTS_TABLE, F.SEGMENTS_ROWS])
def test_changed_arrays(tmp_path, index):
    g = F.gen_rmat(700, 11200, 0.57, 0.19, 0.19, seed=7, labels=F.gen_labels(700, 3, "uniform", seed=7))
    off, adj = g.csr()
    q = F.gen_query(g, 4, F.QUERY_DENSE, seed=3, csr=(off, adj))
    want = O.match(g.labels, off, adj, q.labels, q.edges)[:2]
    path, bad = tmp_path / "g.fsigcache", tmp_path / "bad.fsigcache"
    rng = np.random.default_rng(1)
    with F.Engine(0, arena_bytes=2 << 30) as e:
        e.set_segment_index(index)
        e.load_graph(g)
        e.save_graph_cache(path)
        info = e.graph_info()
        data = path.read_bytes()
        table = index == F.SEGMENTS_TABLE
        parts = arrays(info["V"], info["L"], info["adj"], table)
        assert len(data) == 32 + sum(4 * w for _, w in parts.values()) + 64 * info["V"]
        entries = np.frombuffer(data, np.uint8).copy()
        for nadj in (1 << 32, 1 << 62, (1 << 64) - 1):  # more entries than positions have bits for
            entries[16:24] = np.array([nadj], np.uint64).view(np.uint8)
            bad.write_bytes(entries.tobytes())
            with pytest.raises(F.FsigError) as ei:
                e.load_graph_cache(bad)
            assert ei.value.status == F.EIO
        for name in ("label", "off", "adj", "lseg") if table else ("label", "off", "adj"):
            at, words = parts[name]
            for fill in ("ones", "random", "one"):
                changed = np.frombuffer(data, np.uint8).copy()
                part = changed[at: at + 4 * words].view(np.uint32)
                if fill == "one":
                    part[words // 2] = 0xFFFFFFFF
                else:
                    part[:] = 0xFFFFFFFF if fill == "ones" else rng.integers(0, 1 << 32, words, dtype=np.uint32)
                bad.write_bytes(changed.tobytes())
                e.load_graph_cache(bad)
                e.load_graph_cache(path)
                r = e.match(q, F.ALGO_GSI)
                assert (r.count, r.hash) == want
