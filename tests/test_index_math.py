"""Index arithmetic at the ends of 32 bits, on the host: positions of an
adjacency of up to 2^32 - 1 entries and any piece length a caller gives."""
import hostcu


def test_pieces_of_a_range(tmp_path):
    hostcu.run(tmp_path, r"""
  const uint32_t los[] = {0u, 5u, 1000u, 0x7fffffffu, 0xfffffd00u};
  const uint32_t lens[] = {1u, 31u, 32u, 33u, 64u, 300u, 700u};
  const uint32_t steps[] = {1u, 32u, 256u, 0x7fffffffu, 0xffffff00u, 0xffffffffu};
  for (uint32_t lo : los)
    for (uint32_t len : lens)
      for (uint32_t step : steps) {
        const uint32_t hi = lo + len;
        const uint32_t n = piece_count(len, step);
        uint64_t covered = 0;
        for (uint32_t k = 0; k < n; k++) {
          const uint32_t b = lo + k * step, e = piece_end(b, step, hi);
          CHECK(b >= lo && b < e && e <= hi && e - b <= step);
          covered += e - b;
        }
        CHECK(covered == len);
      }
  CHECK(piece_count(0, 1) == 0 && piece_count(0, 0xffffffffu) == 0);
""")


def test_binary_search_beyond_2_31_entries(tmp_path):
    # a mapping of 2^32 - 1 words of which only the probed pages exist
    hostcu.run(tmp_path, r"""
  const uint64_t n = 0xffffffffull;
  uint32_t* a = static_cast<uint32_t*>(mmap(nullptr, n * 4, PROT_READ | PROT_WRITE,
                                            MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0));
  if (a == MAP_FAILED) return 2;
  const uint32_t los[] = {0u, 0x7ffffff0u, 0x80000000u, 0xc0000000u, 0xfffffc00u};
  for (uint32_t lo : los) {
    const uint32_t hi = lo + 1000;
    for (uint32_t i = lo; i < hi; i++) a[i] = 2 * (i - lo) + 1;  // a row of 1000 odd ids
    for (uint32_t k = 0; k < 1000; k++) {
      CHECK(lower_bound_u32(a, lo, hi, 2 * k) == lo + k);
      CHECK(lower_bound_u32(a, lo, hi, 2 * k + 1) == lo + k);
    }
    CHECK(lower_bound_u32(a, lo, hi, 5000) == hi);
    CHECK(lower_bound_u32(a, hi, hi, 1) == hi);
    for (uint32_t i = lo; i < hi; i++) a[i] = 0;
  }
  a[n - 1] = 7;
  CHECK(lower_bound_u32(a, 0, uint32_t(n), 5) == uint32_t(n - 1));
  CHECK(midpoint(0xfffffff0u, 0xfffffffeu) == 0xfffffff7u && midpoint(5, 6) == 5 && midpoint(0, 0xffffffffu) == 0x7fffffffu);
""")
