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
