"""Record numbers of the enumeration's queue that wrap from 2^32 - 1 to 0
within a pass (a pass of 2^32 hand-offs): counts, hashes and per-depth counts
are the oracle's, whatever the first number."""
import time

import pytest

import fsig_gb300 as F
from fsig_gb300.workloads import pattern
from oracle import oracle as O

pytestmark = pytest.mark.gpu

WRAP = 1 << 32
# across the ring's end and its next turn, at the wrap itself, a few hand-offs and some thousand records before it
FIRST = [0, 1, (1 << 20) - 1, (1 << 20) - 700, (3 << 20) - 1, WRAP - 1, WRAP - 2, WRAP - 33, WRAP - 700, WRAP - 5000,
         WRAP - (1 << 20), WRAP - (1 << 20) - 1]


@pytest.mark.parametrize("name", ["house", "c5"])
def test_numbers_across_the_wrap(name):
    g = F.gen_rmat(1 << 8, 1 << 11, 0.57, 0.19, 0.19, seed=3)
    off, adj = g.csr()
    q = pattern(name)
    want = O.match(g.labels, off, adj, q.labels, q.edges)[:2]
    levels = set()
    with F.Engine(0, arena_bytes=2 << 30) as e:
        e.load_graph(g)
        for first in FIRST:
            e.set_queue_test(first_record=first)
            for use_graph in (False, True):
                r, = e.match_batch([q], algo=F.ALGO_FUSED, split_cycles=1000, split_len=32, use_graph=use_graph)
                assert (r.status, r.count, r.hash) == (0, *want)
                levels.add(tuple(r.level_counts))
                assert e.last_stats()["enum_records"] > 40
            e.set_queue_waits(idle_wait_ns=1)  # and with records left for later passes
            r, = e.match_batch([q], algo=F.ALGO_FUSED, split_cycles=1000, split_len=32)
            assert (r.status, r.count, r.hash) == (0, *want)
            e.set_queue_waits()
    assert len(levels) == 1


@pytest.mark.parametrize("first", [0, WRAP - 1, WRAP - 300])
def test_a_warp_that_left_does_not_hold_up_the_others(first):
    """One warp leaves at once and its record waits for the next pass; the
    others may wait 30 s for hand-offs, but the pass ends when its work does."""
    g = F.gen_rmat(1 << 8, 1 << 11, 0.57, 0.19, 0.19, seed=3)
    off, adj = g.csr()
    q = pattern("house")
    want = O.match(g.labels, off, adj, q.labels, q.edges)[:2]
    with F.Engine(0, arena_bytes=2 << 30) as e:
        e.load_graph(g)
        kw = dict(algo=F.ALGO_FUSED, split_cycles=1000, split_len=32)
        plain, = e.match_batch([q], **kw)
        e.set_queue_waits(idle_wait_ns=30 * 10**9)
        e.set_queue_test(first_record=first, first_leaves=True)
        passes = []
        for use_graph in (False, True) * 8:
            t = time.perf_counter()
            r, = e.match_batch([q], use_graph=use_graph, **kw)
            assert time.perf_counter() - t < 5.0
            assert (r.status, r.count, r.hash) == (0, *want)
            assert r.level_counts == plain.level_counts
            passes.append(e.last_stats()["enum_passes"])
    # the record of the warp that left (unless it was written before that looked)
    assert max(passes) > 1
