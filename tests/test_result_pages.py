"""The arrays that transforms' results are copied into by the GPU: their pages
are there before the call (a fake library looks, no GPU), and results that no
call filled are zero."""
import ctypes as C
import mmap

import numpy as np
import pytest

import fsig_gb300 as F

LIBC = C.CDLL(None, use_errno=True)
LIBC.mincore.argtypes = [C.c_void_p, C.c_size_t, C.c_void_p]


def absent_pages(ptr, count):
    """Pages of `count` words at `ptr` that the process never touched."""
    lo = C.cast(ptr, C.c_void_p).value // mmap.PAGESIZE * mmap.PAGESIZE
    hi = C.cast(ptr, C.c_void_p).value + 4 * count
    pages = -(-(hi - lo) // mmap.PAGESIZE)
    seen = (C.c_ubyte * pages)()
    assert LIBC.mincore(lo, hi - lo, seen) == 0
    return pages - sum(b & 1 for b in seen)


class Library:
    def __init__(self, keys=0, lists=0):
        self.keys, self.lists, self.absent = keys, lists, []

    def fsig_build_csr(self, h, v, e, edges, off, adj):
        self.absent += [absent_pages(off, v + 1), absent_pages(adj, max(2 * e, 1))]
        return 0

    def fsig_build_signature(self, h, v, lab, off, adj, column, out):
        self.absent.append(absent_pages(out, 16 * v))
        return 0

    def fsig_build_pcsr(self, h, v, labels, lab, off, adj, unit_keys, unit_edges, table, edges):
        unit_keys[0], unit_edges[0] = self.keys, self.lists
        if table is not None:
            self.absent += [absent_pages(table, 32 * self.keys), absent_pages(edges, self.lists)]
        return 0


def engine(**kw):
    e = F.Engine.__new__(F.Engine)
    e._L, e._h = Library(**kw), None
    return e


@pytest.mark.parametrize("v,edges", [(1, 0), (1000, 5000), (320_000, 1_050_000), (130_000, 3_000_000)])
def test_pages_are_there(v, edges):
    e = engine(keys=v // 2, lists=2 * edges)
    off, adj = e.build_csr(v, np.zeros((edges, 2), np.uint32))
    sig = e.build_signature(np.zeros(v, np.int32), off, adj)
    (k, m, table, lists), = e.build_pcsr(np.zeros(v, np.int32), off, adj, 1)
    assert (len(off), len(adj), len(sig)) == (v + 1, 2 * edges, 16 * v)
    assert (k, m, len(table), len(lists)) == (v // 2, 2 * edges, 32 * (v // 2), 2 * edges)
    big = 32 * (v // 2) * 4 >= 32 << 20  # a mapping of its own, left to the copy
    assert sum(e._L.absent[:3]) == 0 and (big or e._L.absent[3] == 0) and e._L.absent[4] == 0
    assert not (off.any() or adj.any() or sig.any() or lists.any())
