"""Record numbers of the enumeration's queue, on the host: the ready words of
one slot's uses follow each other, across the wrap from 2^32 - 1 to 0 too."""
import hostcu


def test_ready_words_across_the_wrap(tmp_path):
    hostcu.run(tmp_path, r"""
  const uint32_t starts[] = {0u, 1u, kQueueSlots - 1, 5 * kQueueSlots + 77, 0u - kQueueSlots, 0u - 3u, 0xffffffffu};
  for (uint32_t t : starts) {
    uint32_t n = t;
    for (int use = 0; use < 9000; use++, n += kQueueSlots) {  // past a whole turn of the uses
      CHECK(queue_slot(n) == queue_slot(t));
      CHECK(ready_published(n) == ready_free(n) + 1 && (ready_free(n) & 1u) == 0);
      CHECK(ready_next(n) == ready_free(n + kQueueSlots));  // what the next writer of the slot waits for
      CHECK(ready_next(n) != ready_free(n) && ready_next(n) != ready_published(n));
      // a holder that left: the record may still be written, then counts as published, and is never taken
      const uint32_t gone = ready_free(n) | kHolderLeft;
      CHECK(ready_writable(ready_free(n), n) && ready_writable(gone, n) && !ready_writable(ready_published(n), n));
      CHECK(((gone | 1u) & 1u) && (gone | 1u) != ready_published(n) && (ready_free(n) | 1u) == ready_published(n));
      CHECK(!ready_writable(gone | 1u, n) && (ready_published(n) >> 31) == 0);
    }
    for (uint32_t d : {1u, 160u, kQueueSlots, 0x7fffffffu}) CHECK(queue_after(t + d, t) && !queue_after(t, t + d));
    CHECK(!queue_after(t, t));
  }
  CHECK(ready_next(0xffffffffu) == 0 && ready_free(kQueueSlots - 1) == 0);
""")


def test_room_after_a_warp_left(tmp_path):
    # whatever the number of warps: the last number reserved and the last ticket
    # stay within a ring of the first ticket given up
    hostcu.run(tmp_path, r"""
  CHECK(kQueueWarps >= 152 * 4 * 8);  // a GB300's resident warps
  for (uint64_t w = 1; w <= kQueueWarps; w++) {
    const uint64_t limit = queue_room(uint32_t(w));  // beyond the tail when the first warp left
    CHECK(limit > 0 && limit < kQueueSlots);
    const uint64_t tail = limit + w * kHandOff;      // every warp checked the limit, then reserved
    CHECK(tail + w <= kQueueSlots);                  // and took a ticket
    CHECK(w * kHandOff < kQueueSlots);               // numbers between tickets and tail
  }
""")
