// Device-side graph transforms: the resident matching store (renumbered CSR,
// label segments, signatures) and the reference-layout CSR and signature
// tables.  Replaces the host loops of graph_format_transformer.cc:12-37 and
// :217-281 and the per-buffer copies of match/MMatch.cu:14-32.
#include <algorithm>
#include <cstdio>
#include <cstring>

#include "engine.h"
#include "scan.cuh"

namespace fsig {
namespace {

constexpr int kRenumTile = 1024;

// ---- label validation --------------------------------------------------------
__global__ void label_range_kernel(const int32_t* __restrict__ lab, uint32_t V, int32_t* out_max,
                                   uint32_t* out_bad) {
  int32_t mx = -1;
  uint32_t bad = 0;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < V; i += uint64_t(gridDim.x) * blockDim.x) {
    int32_t l = lab[i];
    if (l < 0) bad = 1; else mx = max(mx, l);
  }
  for (int o = 16; o > 0; o >>= 1) {
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    bad |= __shfl_xor_sync(0xffffffffu, bad, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(out_max, mx);
    if (bad) atomicOr(out_bad, 1u);
  }
}

// ---- stable counting sort of vertices by label ---------------------------------
__global__ void __launch_bounds__(kRenumTile) label_tile_hist_kernel(const int32_t* __restrict__ lab, uint32_t V,
                                                                     int32_t L, uint32_t T, uint32_t* counts) {
  extern __shared__ uint32_t h[];
  for (int i = threadIdx.x; i < L; i += blockDim.x) h[i] = 0;
  __syncthreads();
  uint64_t v = uint64_t(blockIdx.x) * kRenumTile + threadIdx.x;
  if (v < V) atomicAdd(&h[lab[v]], 1u);
  __syncthreads();
  for (int i = threadIdx.x; i < L; i += blockDim.x) counts[uint64_t(i) * T + blockIdx.x] = h[i];
}

// counts scanned in (label, tile) order give each tile's first slot per label;
// within a tile, warps take turns so that ranks follow caller ids.
__global__ void __launch_bounds__(kRenumTile) label_tile_rank_kernel(const int32_t* __restrict__ lab, uint32_t V,
                                                                     int32_t L, uint32_t T,
                                                                     const uint32_t* __restrict__ starts,
                                                                     uint32_t* new_of_old, uint32_t* old_of_new,
                                                                     int32_t* label_new) {
  extern __shared__ uint32_t run[];
  for (int i = threadIdx.x; i < L; i += blockDim.x) run[i] = 0;
  __syncthreads();
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t v = uint64_t(blockIdx.x) * kRenumTile + threadIdx.x;
  const bool live = v < V;
  const int32_t l = live ? lab[v] : -1;
  const uint32_t nw = blockDim.x >> 5;
  for (uint32_t w = 0; w < nw; w++) {
    if (warp == w) {
      uint32_t peers = __match_any_sync(0xffffffffu, l);
      uint32_t before = 0;
      if (live) before = run[l];
      __syncwarp();
      if (live) {
        uint32_t rank = __popc(peers & lanemask_lt());
        uint32_t leader = __ffs(peers) - 1;
        uint32_t nid = starts[uint64_t(l) * T + blockIdx.x] + before + rank;
        new_of_old[v] = nid;
        old_of_new[nid] = uint32_t(v);
        label_new[nid] = l;
        if (lane == leader) run[l] = before + __popc(peers);
      }
    }
    __syncthreads();
  }
}

__global__ void base_from_starts_kernel(const uint32_t* __restrict__ starts, int32_t L, uint32_t T, uint32_t V,
                                        uint32_t* base) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < L) base[i] = starts[uint64_t(i) * T];
  if (i == L) base[L] = V;
}

// ---- adjacency -----------------------------------------------------------------
// Degree histogram.  map == nullptr keeps caller ids; drop_loops removes
// self-loops (the matching store) or keeps both copies (the reference CSR).
__global__ void degree_kernel(const uint2* __restrict__ edges, uint64_t E, uint32_t V,
                              const uint32_t* __restrict__ map, bool drop_loops, uint32_t* deg, uint32_t* bad) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < E; i += uint64_t(gridDim.x) * blockDim.x) {
    uint2 e = edges[i];
    if (e.x >= V || e.y >= V) { atomicOr(bad, 2u); continue; }
    if (drop_loops && e.x == e.y) continue;
    uint32_t a = map ? map[e.x] : e.x, b = map ? map[e.y] : e.y;
    atomicAdd(&deg[a], 1u);
    atomicAdd(&deg[b], 1u);
  }
}

__global__ void scatter_kernel(const uint2* __restrict__ edges, uint64_t E, uint32_t V,
                               const uint32_t* __restrict__ map, bool drop_loops, uint32_t* cursor, uint32_t* adj) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < E; i += uint64_t(gridDim.x) * blockDim.x) {
    uint2 e = edges[i];
    if (e.x >= V || e.y >= V) continue;
    if (drop_loops && e.x == e.y) continue;
    uint32_t a = map ? map[e.x] : e.x, b = map ? map[e.y] : e.y;
    adj[atomicAdd(&cursor[a], 1u)] = b;
    adj[atomicAdd(&cursor[b], 1u)] = a;
  }
}

// ---- segmented sort of rows ------------------------------------------------------
// A row of up to kWarpRow entries is sorted by a warp in registers, of up to
// kBlockRow by a small block and of up to kSmemRow by a large one in shared
// memory; longer ones in chunks of kSmemRow.  (A 256-thread block for every row
// above 32 entries spent most of its time in barriers: 135,000 rows of 33 to
// 2048 entries took 1.5 ms, and 0.2 ms with the warps.)
constexpr uint32_t kWarpRow = 512, kBlockRow = 2048, kSmemRow = 16384;

// Rows by class of length, and the longest length.  One atomic per warp and
// class (one per row took 228 us for 2^20 rows, all on five words; this 52 us).
__global__ void classify_rows_kernel(const uint32_t* __restrict__ off, uint32_t V, uint32_t* lists,
                                     uint32_t* counts, uint32_t* max_len) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t longest = 0;
  for (uint64_t base = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) & ~31ull; base < V;
       base += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t v = uint32_t(base) + lane;
    const uint32_t len = v < V ? off[v + 1] - off[v] : 0;
    longest = max(longest, len);
    const int c = len <= 1 ? -1 : (len <= kWarpRow ? 0 : (len <= kBlockRow ? 1 : (len <= kSmemRow ? 2 : 3)));
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t m = __ballot_sync(0xffffffffu, c == k);
      if (!m) continue;
      uint32_t first = 0;
      if (lane == 0) first = atomicAdd(&counts[k], uint32_t(__popc(m)));
      first = __shfl_sync(0xffffffffu, first, 0);
      if (c == k) lists[uint64_t(k) * V + first + __popc(m & lanemask_lt())] = v;
    }
  }
  longest = __reduce_max_sync(0xffffffffu, longest);
  if (lane == 0 && longest) atomicMax(max_len, longest);
}

// Bitonic sort of the up to 32 R entries at p by one warp: entry r * 32 + lane
// in register r of the lane.
template <int R>
__device__ __forceinline__ void warp_sort_row(uint32_t* p, uint32_t len, uint32_t lane) {
  uint32_t x[R];
#pragma unroll
  for (int r = 0; r < R; r++) x[r] = r * 32 + lane < len ? p[r * 32 + lane] : kInvalid;
#pragma unroll
  for (int k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j >= 32; j >>= 1) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int o = r ^ (j >> 5);
        if (o > r) {
          const uint32_t lo = min(x[r], x[o]), hi = max(x[r], x[o]);
          const bool up = ((r * 32) & k) == 0;
          x[r] = up ? lo : hi;
          x[o] = up ? hi : lo;
        }
      }
    }
#pragma unroll
    for (int j = k >> 1 < 16 ? k >> 1 : 16; j > 0; j >>= 1) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x[r], j);
        const bool up = ((r * 32 + lane) & k) == 0, lower = (lane & j) == 0;
        x[r] = lower == up ? min(x[r], y) : max(x[r], y);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++)
    if (r * 32 + lane < len) p[r * 32 + lane] = x[r];
}

__global__ void __launch_bounds__(256) sort_rows_warp_kernel(const uint32_t* __restrict__ rows,
                                                             const uint32_t* __restrict__ count,
                                                             const uint32_t* __restrict__ off, uint32_t* adj) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t n = *count;
  for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t v = rows[r], b = off[v], len = off[v + 1] - b;
    if (len <= 32) warp_sort_row<1>(adj + b, len, lane);
    else if (len <= 64) warp_sort_row<2>(adj + b, len, lane);
    else if (len <= 128) warp_sort_row<4>(adj + b, len, lane);
    else if (len <= 256) warp_sort_row<8>(adj + b, len, lane);
    else warp_sort_row<16>(adj + b, len, lane);
  }
}

// n a power of two; every thread has a pair to compare.
__device__ void block_bitonic(uint32_t* s, uint32_t n) {
  for (uint32_t k = 2; k <= n; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t t = threadIdx.x; t < n >> 1; t += blockDim.x) {
        const uint32_t i = 2 * t - (t & (j - 1)), p = i + j;
        const uint32_t a = s[i], b = s[p];
        const bool up = (i & k) == 0;
        if ((a > b) == up) {
          s[i] = b;
          s[p] = a;
        }
      }
      __syncthreads();
    }
  }
}

// One block per row; the row is sorted in shared memory, padded to a power of two.
__global__ void sort_rows_block_kernel(const uint32_t* __restrict__ rows, const uint32_t* __restrict__ count,
                                       const uint32_t* __restrict__ off, uint32_t* adj) {
  extern __shared__ uint32_t sm[];
  const uint32_t n = *count;
  for (uint32_t r = blockIdx.x; r < n; r += gridDim.x) {
    uint32_t v = rows[r];
    uint32_t b = off[v], len = off[v + 1] - b;
    uint32_t p2 = 1;
    while (p2 < len) p2 <<= 1;
    for (uint32_t i = threadIdx.x; i < p2; i += blockDim.x) sm[i] = i < len ? adj[b + i] : kInvalid;
    __syncthreads();
    block_bitonic(sm, p2);
    for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) adj[b + i] = sm[i];
    __syncthreads();
  }
}

// Rows longer than kSmemRow, in chunks of kSmemRow entries: the chunks are
// sorted in shared memory, then merged pairwise, an entry's place being its own
// index plus its rank in the sibling run by binary search (equal entries: the
// left run's first).  Every entry of every pass is independent, so the longest
// row no longer runs on one block: the 21 rows above 16384 entries of a 2^24-
// edge R-MAT graph took 15 ms by one block's bitonic sort in global memory, and
// 0.27 ms this way.
__global__ void long_chunks_kernel(const uint32_t* __restrict__ rows, uint32_t n, const uint32_t* __restrict__ off,
                                   uint32_t* chunks) {
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    chunks[r] = piece_count(off[rows[r] + 1] - off[rows[r]], kSmemRow);
}

// Row (its first entry, length) and first entry within it of chunk c.
__device__ __forceinline__ void chunk_of(const uint32_t* __restrict__ rows, uint32_t n,
                                         const uint32_t* __restrict__ chunk_off, const uint32_t* __restrict__ off,
                                         uint32_t c, uint32_t& b, uint32_t& len, uint32_t& first) {
  uint32_t lo = 0, hi = n;  // last row with chunk_off <= c
  while (hi - lo > 1) {
    const uint32_t mid = midpoint(lo, hi);
    if (chunk_off[mid] <= c) lo = mid; else hi = mid;
  }
  b = off[rows[lo]];
  len = off[rows[lo] + 1] - b;
  first = (c - chunk_off[lo]) * kSmemRow;
}

__global__ void __launch_bounds__(1024) sort_chunks_kernel(const uint32_t* __restrict__ rows, uint32_t n,
                                                           const uint32_t* __restrict__ chunk_off, uint32_t total,
                                                           const uint32_t* __restrict__ off, uint32_t* adj) {
  extern __shared__ uint32_t sm[];
  for (uint32_t c = blockIdx.x; c < total; c += gridDim.x) {
    uint32_t b, len, first;
    chunk_of(rows, n, chunk_off, off, c, b, len, first);
    const uint32_t m = min(kSmemRow, len - first);
    uint32_t p2 = 1;
    while (p2 < m) p2 <<= 1;
    for (uint32_t i = threadIdx.x; i < p2; i += blockDim.x) sm[i] = i < m ? adj[b + first + i] : kInvalid;
    __syncthreads();
    block_bitonic(sm, p2);
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) adj[b + first + i] = sm[i];
    __syncthreads();
  }
}

// One merge pass over runs of `width` entries (a power of two); width 0 copies.
__global__ void __launch_bounds__(1024) merge_runs_kernel(const uint32_t* __restrict__ rows, uint32_t n,
                                                          const uint32_t* __restrict__ chunk_off, uint32_t total,
                                                          const uint32_t* __restrict__ off, uint64_t width,
                                                          const uint32_t* __restrict__ in, uint32_t* __restrict__ out) {
  for (uint32_t c = blockIdx.x; c < total; c += gridDim.x) {
    uint32_t b, len, first;
    chunk_of(rows, n, chunk_off, off, c, b, len, first);
    const uint32_t count = min(kSmemRow, len - first);
    uint64_t run = 0, lo = len, hi = len;  // the chunk lies in one run; its sibling is [lo, hi)
    if (width) {
      run = first / width;
      lo = min((run ^ 1) * width, uint64_t(len));
      hi = min(lo + width, uint64_t(len));
    }
    for (uint32_t k = threadIdx.x; k < count; k += blockDim.x) {
      const uint32_t i = first + k, x = in[b + i];
      uint32_t to = i;
      if (lo < hi) {
        // entries of the sibling that go first: the smaller ones, and from a left sibling the equal ones
        const bool right = run & 1;
        uint32_t l = uint32_t(lo), h = uint32_t(hi);
        while (l < h) {
          const uint32_t mid = midpoint(l, h);
          const uint32_t y = in[b + mid];
          if (y < x || (right && y == x)) l = mid + 1; else h = mid;
        }
        to = (right ? i - uint32_t(width) : i) + (l - uint32_t(lo));
      }
      out[b + to] = x;
    }
  }
}

// Repeated entries of all sorted rows: equal neighbours in the adjacency, less
// the pairs that straddle two rows.  Most graphs have none, and then nothing of
// the two kernels below runs (a thread walking each row took 1.7 ms on a 2^24-
// edge R-MAT graph, hubs last; this 0.06 ms).
__global__ void repeats_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj, uint32_t V,
                               uint64_t n, unsigned long long* repeats) {
  long long c = 0;
  const uint64_t t0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x, step = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t k = t0 + 1; k < n; k += step) c += adj[k] == adj[k - 1];
  for (uint64_t v = t0; v < V; v += step) {
    const uint32_t b = off[v];
    if (b > 0 && b < off[v + 1]) c -= adj[b] == adj[b - 1];
  }
  c = warp_sum(c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(repeats, (unsigned long long)c);
}

// Unique entries per sorted row, a warp per row.  (Here and below, a lane's
// position is counted from the row's begin or in 64 bits: beyond a row that ends
// at almost 2^32 it may not fit 32.)
__global__ void unique_count_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj, uint32_t V,
                                    uint32_t* ucount) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < V; v += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t* row = adj + off[v];
    const uint32_t len = off[v + 1] - off[v];  // at most 2^31: one entry per edge
    uint32_t c = 0;
    for (uint32_t i = lane; i < len; i += 32) c += i == 0 || row[i] != row[i - 1];
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) ucount[v] = c;
  }
}

__global__ void unique_copy_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj, uint32_t V,
                                   const uint32_t* __restrict__ noff, uint32_t* out) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < V; v += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t* row = adj + off[v];
    const uint32_t len = off[v + 1] - off[v];
    uint32_t w = noff[v];
    for (uint32_t i0 = 0; i0 < len; i0 += 32) {
      const uint32_t i = i0 + lane;
      const uint32_t x = i < len ? row[i] : 0;
      const bool keep = i < len && (i == 0 || x != row[i - 1]);
      const uint32_t m = __ballot_sync(0xffffffffu, keep);
      if (keep) out[w + __popc(m & lanemask_lt())] = x;
      w += __popc(m);
    }
  }
}

// lseg[v*(L+1)+l] = first entry of row v with id >= base[l].
__global__ void label_segments_kernel(const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj,
                                      const uint32_t* __restrict__ base, uint32_t V, int32_t L, uint32_t* lseg) {
  const uint64_t W = uint64_t(L) + 1;
  const uint64_t total = uint64_t(V) * W;
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < total; i += uint64_t(gridDim.x) * blockDim.x) {
    uint32_t v = uint32_t(i / W), l = uint32_t(i % W);
    uint32_t b = off[v], e = off[v + 1];
    lseg[i] = (l == uint32_t(L)) ? e : lower_bound_u32(adj, b, e, base[l]);
  }
}

// Signature of every vertex from its label segments: each segment of c > 0
// neighbours applies min(c, 2) saturating increments to its label's counter.
__global__ void signature_from_segments_kernel(const int32_t* __restrict__ label, const uint32_t* __restrict__ lseg,
                                               uint32_t V, int32_t L, uint4* sig) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    uint32_t w[kSigWords];
#pragma unroll
    for (int i = 0; i < kSigWords; i++) w[i] = 0;
    w[0] = uint32_t(label[v]);
    const uint32_t* s = lseg + uint64_t(v) * (uint32_t(L) + 1);
    for (int32_t l = 0; l < L; l++) {
      uint32_t c = s[l + 1] - s[l];
      if (!c) continue;
      uint32_t word, sh;
      sig_slot(l, word, sh);
      for (uint32_t k = 0; k < min(c, 2u); k++) {
        // registers cannot be indexed dynamically without spilling; select.
#pragma unroll
        for (int i = 1; i < kSigWords; i++) {
          if (uint32_t(i) == word) {
            uint32_t cur = (w[i] >> sh) & 3u;
            w[i] |= (cur == 0 ? 1u : 3u) << sh;
          }
        }
      }
    }
    uint4* o = sig + uint64_t(v) * 4;
    o[0] = make_uint4(w[0], w[1], w[2], w[3]);
    o[1] = make_uint4(w[4], w[5], w[6], w[7]);
    o[2] = make_uint4(w[8], w[9], w[10], w[11]);
    o[3] = make_uint4(w[12], w[13], w[14], w[15]);
  }
}

// Reference-layout signature: one saturating increment per adjacency entry
// (duplicates counted as the reference counts them).
// A warp per row, its counters in shared memory: a neighbour's first increment
// sets the counter's low bit, every later one its high bit, whatever the order.
// (A thread per row walked hubs alone: 514 us for 320k rows of up to 1478
// entries, now 64 us.)
__global__ void __launch_bounds__(256) signature_from_rows_kernel(const int32_t* __restrict__ label,
                                                                  const uint32_t* __restrict__ off,
                                                                  const uint32_t* __restrict__ adj, uint32_t V,
                                                                  int column_oriented, uint32_t* out) {
  __shared__ uint32_t words[8][kSigWords];
  const uint32_t lane = threadIdx.x & 31;
  uint32_t* w = words[threadIdx.x >> 5];
  for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < V; v += (gridDim.x * blockDim.x) >> 5) {
    if (lane < kSigWords) w[lane] = lane == 0 ? uint32_t(label[v]) : 0u;
    __syncwarp();
    const uint32_t end = off[v + 1];
    for (uint64_t e = uint64_t(off[v]) + lane; e < end; e += 32) {
      uint32_t word, sh;
      sig_slot(label[adj[e]], word, sh);
      if ((atomicOr(&w[word], 1u << sh) >> sh) & 1u) atomicOr(&w[word], 2u << sh);
    }
    __syncwarp();
    if (lane < kSigWords) {
      if (column_oriented) out[uint64_t(lane) * V + v] = w[lane];
      else out[uint64_t(v) * kSigWords + lane] = w[lane];
    }
    __syncwarp();
  }
}

// Membership filter (common.cuh), a warp per 256 adjacency entries, one entry
// per lane and step; the lane's row is found from the previous one by
// galloping (rows average a step or two apart).  Bound by the atomics, all to
// words near the entry's own position: L2.  The arrays may be a cache file's, as
// they are in the file, so nothing is read or written outside of them.
constexpr uint32_t kFilterRun = 256;
__global__ void __launch_bounds__(256) membership_filter_kernel(
    const uint32_t* __restrict__ off, const uint32_t* __restrict__ adj, const int32_t* __restrict__ label,
    const uint32_t* __restrict__ base, const uint32_t* __restrict__ lseg, uint32_t V, int32_t L, uint32_t nadj,
    uint32_t shift, uint32_t* __restrict__ filt) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
  for (uint64_t run = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; run * kFilterRun < nadj; run += nwarps) {
    uint32_t lo = 0, hi = V;  // row of the run's first entry: the last v with off[v] <= k
    const uint32_t first = uint32_t(run * kFilterRun);
    while (hi - lo > 1) {
      const uint32_t mid = midpoint(lo, hi);
      if (off[mid] <= first) lo = mid; else hi = mid;
    }
    uint32_t v = lo;
    const uint32_t count = min(kFilterRun, nadj - first);
    for (uint32_t i = lane; i < count; i += 32) {
      const uint32_t k = first + i;
      uint32_t step = 1;
      while (v + step < V && off[v + step] <= k) {
        v += step;
        step <<= 1;
      }
      for (; step; step >>= 1)
        if (v + step < V && off[v + step] <= k) v += step;
      const uint32_t x = adj[k];
      const int32_t l = x < V ? label[x] : -1;
      if (l < 0 || l >= L) continue;
      uint32_t a, b;
      if (lseg) {
        const uint32_t* s = lseg + uint64_t(v) * (uint64_t(L) + 1) + l;
        a = s[0];
        b = s[1];
      } else {
        a = lower_bound_u32(adj, off[v], k, base[l]);
        b = lower_bound_u32(adj, k, min(off[v + 1], nadj), base[l + 1]);
      }
      const uint32_t first_id = base[l] & ~31u, rel = x - first_id;
      const bool dense = b - a >= filter_dense_len(base[l + 1] - first_id, shift);
      const uint32_t w = (a << shift) + filter_word(dense, rel, filter_hash(x), (b - a) << shift);
      if (w < uint64_t(nadj) << shift) atomicOr(&filt[w >> 1], filter_mask(dense, rel, filter_bits(x)) << ((w & 1u) * 16));
    }
  }
}

__global__ void gather_kernel(const uint32_t* __restrict__ idx, uint64_t n, const uint32_t* __restrict__ table,
                              uint32_t* out) {
  for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
    out[i] = table[idx[i]];
}

inline unsigned grid_for(uint64_t n, int threads, int sms) {
  uint64_t b = (n + threads - 1) / threads;
  uint64_t cap = uint64_t(sms) * 32;
  if (b > cap) b = cap;
  return unsigned(b ? b : 1);
}

// Builds offsets/adjacency (rows sorted) from an edge list already on the
// device.  map == nullptr keeps caller ids.  Returns the row data in adj and
// the longest row's length; the edge list's memory serves as scratch.
int build_rows(Engine& e, uint2* d_edges, uint64_t E, uint32_t V, const uint32_t* map, bool drop_loops, uint32_t* off,
               uint32_t* adj, uint32_t* d_flags, uint32_t* longest = nullptr) {
  cudaStream_t s = e.stream;
  uint64_t m = e.arena.mark();
  uint32_t* deg = e.arena.take<uint32_t>(uint64_t(V) + 1);
  uint32_t* lists = e.arena.take<uint32_t>(uint64_t(V) * 4);
  uint32_t* small = e.arena.take<uint32_t>(8);
  if (!deg || !lists || !small) return fail(FSIG_EADMISSION, "graph build scratch does not fit the arena");
  FSIG_CUDA_TRY(cudaMemsetAsync(deg, 0, sizeof(uint32_t) * (uint64_t(V) + 1), s));
  FSIG_CUDA_TRY(cudaMemsetAsync(small, 0, sizeof(uint32_t) * 8, s));
  const int T = 256;
  degree_kernel<<<grid_for(E, T, e.num_sms), T, 0, s>>>(d_edges, E, V, map, drop_loops, deg, d_flags);
  FSIG_CUDA_TRY(cudaGetLastError());
  int rc = device_exclusive_scan<uint32_t>(e.arena, deg, off, uint64_t(V) + 1, nullptr, s);
  if (rc) return rc;
  FSIG_CUDA_TRY(cudaMemcpyAsync(deg, off, sizeof(uint32_t) * V, cudaMemcpyDeviceToDevice, s));
  scatter_kernel<<<grid_for(E, T, e.num_sms), T, 0, s>>>(d_edges, E, V, map, drop_loops, deg, adj);
  FSIG_CUDA_TRY(cudaGetLastError());
  classify_rows_kernel<<<grid_for(V, T, e.num_sms), T, 0, s>>>(off, V, lists, small, small + 4);
  FSIG_CUDA_TRY(cudaGetLastError());
  uint32_t h[8];
  FSIG_CUDA_TRY(cudaMemcpyAsync(h, small, sizeof(h), cudaMemcpyDeviceToHost, s));
  FSIG_CUDA_TRY(cudaStreamSynchronize(s));
  if (h[0]) {
    sort_rows_warp_kernel<<<grid_for(uint64_t(h[0]) * 32, T, e.num_sms), T, 0, s>>>(lists, small + 0, off, adj);
    FSIG_CUDA_TRY(cudaGetLastError());
  }
  if (h[1]) {
    sort_rows_block_kernel<<<std::min<uint32_t>(h[1], e.num_sms * 8), 256, kBlockRow * 4, s>>>(
        lists + uint64_t(V), small + 1, off, adj);
    FSIG_CUDA_TRY(cudaGetLastError());
  }
  if (h[2]) {
    FSIG_CUDA_TRY(cudaFuncSetAttribute(sort_rows_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kSmemRow * 4));
    sort_rows_block_kernel<<<std::min<uint32_t>(h[2], e.num_sms * 2), 1024, kSmemRow * 4, s>>>(
        lists + 2 * uint64_t(V), small + 2, off, adj);
    FSIG_CUDA_TRY(cudaGetLastError());
  }
  if (h[3]) {
    // chunk counts of the long rows and their prefix sums, over the shorter classes' lists
    const uint32_t* rows = lists + 3 * uint64_t(V);
    uint32_t *chunks = deg, *chunk_off = deg;  // deg held the scatter's cursors: done with
    long_chunks_kernel<<<grid_for(h[3], T, e.num_sms), T, 0, s>>>(rows, h[3], off, chunks);
    FSIG_CUDA_TRY(cudaGetLastError());
    rc = device_exclusive_scan<uint32_t>(e.arena, chunks, chunk_off, h[3], small + 5, s);
    if (rc) return rc;
    uint32_t total = 0;
    FSIG_CUDA_TRY(cudaMemcpyAsync(&total, small + 5, sizeof(total), cudaMemcpyDeviceToHost, s));
    FSIG_CUDA_TRY(cudaStreamSynchronize(s));
    FSIG_CUDA_TRY(cudaFuncSetAttribute(sort_chunks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemRow * 4));
    sort_chunks_kernel<<<std::min<uint32_t>(total, e.num_sms * 2), 1024, kSmemRow * 4, s>>>(rows, h[3], chunk_off, total,
                                                                                          off, adj);
    FSIG_CUDA_TRY(cudaGetLastError());
    // the edge list (2E words) is scattered by now: its memory is the other buffer
    uint32_t *in = adj, *out = reinterpret_cast<uint32_t*>(d_edges);
    const unsigned grid = std::min<uint32_t>(total, e.num_sms * 2);
    for (uint64_t width = kSmemRow; width < h[4] || in != adj; width <<= 1) {
      merge_runs_kernel<<<grid, 1024, 0, s>>>(rows, h[3], chunk_off, total, off, width < h[4] ? width : 0, in, out);
      FSIG_CUDA_TRY(cudaGetLastError());
      std::swap(in, out);
    }
  }
  if (longest) *longest = h[4];
  e.arena.release(m);
  return FSIG_OK;
}

__global__ void max_row_kernel(const uint32_t* __restrict__ off, uint32_t V, uint32_t* longest) {
  uint32_t m = 0;
  for (uint64_t v = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; v < V; v += uint64_t(gridDim.x) * blockDim.x)
    m = max(m, off[v + 1] - off[v]);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(longest, m);
}

// Arena bytes left free beside the membership filter when it is built: a
// batch's work queues and room for a batch.
constexpr uint64_t kFilterSpare = 1ull << 30;

// The membership filter in the arena's tail, when there is room for it and
// `spare` bytes; without it the enumeration searches the segments themselves.
int build_membership_filter(Engine& e, DeviceGraph& g, uint64_t spare) {
  const uint32_t shift = filter_shift(g.nadj);
  const uint64_t words32 = ((g.nadj << shift) + 1) / 2;
  uint32_t* filt = words32 ? e.arena.take_tail<uint32_t>(words32, spare) : nullptr;
  if (!filt) return FSIG_OK;
  FSIG_CUDA_TRY(cudaMemsetAsync(filt, 0, sizeof(uint32_t) * words32, e.stream));
  membership_filter_kernel<<<grid_for((g.nadj + kFilterRun - 1) / kFilterRun * 32, 256, e.num_sms), 256, 0, e.stream>>>(
      g.off, g.adj, g.label, g.base, g.lseg, g.V, g.L, uint32_t(g.nadj), shift, filt);
  FSIG_CUDA_TRY(cudaGetLastError());
  g.filt = reinterpret_cast<uint16_t*>(filt);
  return FSIG_OK;
}

}  // namespace

uint64_t filter_bytes(const Engine& e) {
  return e.has_graph && e.arena.tail ? (e.g.nadj << filter_shift(e.g.nadj)) * sizeof(uint16_t) : 0;
}

int restore_membership_filter(Engine& e, uint32_t* launches) {
  if (!e.g.filt || e.arena.tail) return FSIG_OK;
  const int rc = build_membership_filter(e, e.g, 0);
  if (rc) e.arena.tail = 0;
  if (e.arena.tail) *launches += 1;
  return rc;
}

bool use_segment_table(int mode, uint32_t V, int32_t L, uint64_t nadj) {
  if (mode == FSIG_SEGMENTS_TABLE) return true;
  if (mode == FSIG_SEGMENTS_ROWS) return false;
  return uint64_t(V) * (uint64_t(L) + 1) <= 4 * std::max<uint64_t>(nadj, V);
}

uint64_t store_bytes(const DeviceGraph& g) {
  const uint64_t V = g.V, L1 = uint64_t(g.L) + 1;
  uint64_t b = 4 * V * 3 + 4 * L1 + 4 * (V + 1) + 4 * g.nadj + 64 * V;  // label, id maps, base, off, adj, sig
  if (g.lseg) b += 4 * V * L1 + 4 * g.nadj;                           // lseg, adj_old
  return b;
}

int build_device_graph(Engine& e, uint32_t V, const int32_t* h_labels, uint64_t E, const uint32_t* h_edges) {
  cudaStream_t s = e.stream;
  if (V == 0) return fail(FSIG_EINVAL, "graph has no vertices");
  if (2 * E > 0xffffffffull) return fail(FSIG_EINVAL, "graph has 2^31 or more edges");
  // Reset any previous graph.
  e.arena.release(0);
  e.arena.tail = 0;
  e.has_graph = false;
  DeviceGraph g;
  g.V = V;

  // Persistent arrays whose sizes do not depend on L.
  g.label = e.arena.take<int32_t>(V);
  g.old_of_new = e.arena.take<uint32_t>(V);
  g.new_of_old = e.arena.take<uint32_t>(V);
  g.off = e.arena.take<uint32_t>(uint64_t(V) + 1);
  g.adj = e.arena.take<uint32_t>(std::max<uint64_t>(2 * E, 1));
  uint32_t* flags = e.arena.take<uint32_t>(4);
  if (!g.label || !g.old_of_new || !g.new_of_old || !g.off || !g.adj || !flags)
    return fail(FSIG_EADMISSION, "graph does not fit the device arena");
  uint64_t mark_tmp = e.arena.mark();
  int32_t* lab_old = e.arena.take<int32_t>(V);
  uint2* d_edges = e.arena.take<uint2>(std::max<uint64_t>(E, 1));
  if (!lab_old || !d_edges) return fail(FSIG_EADMISSION, "graph staging does not fit the device arena");
  FSIG_CUDA_TRY(cudaMemcpyAsync(lab_old, h_labels, sizeof(int32_t) * V, cudaMemcpyHostToDevice, s));
  if (E) FSIG_CUDA_TRY(cudaMemcpyAsync(d_edges, h_edges, sizeof(uint2) * E, cudaMemcpyHostToDevice, s));
  FSIG_CUDA_TRY(cudaMemsetAsync(flags, 0, 16, s));
  int32_t init_max = -1;
  FSIG_CUDA_TRY(cudaMemcpyAsync(flags + 1, &init_max, 4, cudaMemcpyHostToDevice, s));
  label_range_kernel<<<grid_for(V, 256, e.num_sms), 256, 0, s>>>(lab_old, V, reinterpret_cast<int32_t*>(flags + 1),
                                                                 flags);
  FSIG_CUDA_TRY(cudaGetLastError());
  uint32_t hf[2];
  FSIG_CUDA_TRY(cudaMemcpyAsync(hf, flags, 8, cudaMemcpyDeviceToHost, s));
  FSIG_CUDA_TRY(cudaStreamSynchronize(s));
  if (hf[0] & 1u) return fail(FSIG_EINVAL, "negative vertex label");
  const int32_t L = int32_t(hf[1]) + 1;
  if (L > int32_t(kMaxLabels)) return fail(FSIG_EINVAL, "more than 4096 distinct labels");
  g.L = L;

  // Renumber by (label, caller id).
  const uint32_t T = (V + kRenumTile - 1) / kRenumTile;
  uint32_t* counts = e.arena.take<uint32_t>(uint64_t(L) * T);
  if (!counts) return fail(FSIG_EADMISSION, "renumbering scratch does not fit the arena");
  label_tile_hist_kernel<<<T, kRenumTile, L * 4, s>>>(lab_old, V, L, T, counts);
  FSIG_CUDA_TRY(cudaGetLastError());
  int rc = device_exclusive_scan<uint32_t>(e.arena, counts, counts, uint64_t(L) * T, nullptr, s);
  if (rc) return rc;
  label_tile_rank_kernel<<<T, kRenumTile, L * 4, s>>>(lab_old, V, L, T, counts, g.new_of_old, g.old_of_new, g.label);
  FSIG_CUDA_TRY(cudaGetLastError());
  uint32_t* base_tmp = e.arena.take<uint32_t>(uint64_t(L) + 1);
  if (!base_tmp) return fail(FSIG_EADMISSION, "arena");
  base_from_starts_kernel<<<(L + 1 + 255) / 256, 256, 0, s>>>(counts, L, T, V, base_tmp);
  FSIG_CUDA_TRY(cudaGetLastError());
  g.h_base.resize(size_t(L) + 1);
  FSIG_CUDA_TRY(cudaMemcpyAsync(g.h_base.data(), base_tmp, sizeof(uint32_t) * (L + 1), cudaMemcpyDeviceToHost, s));

  // Rows in new-id space, self-loops dropped, then duplicates removed.
  rc = build_rows(e, d_edges, E, V, g.new_of_old, true, g.off, g.adj, flags, &g.max_deg);
  if (rc) return rc;
  uint32_t* ucount = e.arena.take<uint32_t>(uint64_t(V) + 1);
  uint32_t* noff = e.arena.take<uint32_t>(uint64_t(V) + 1);
  unsigned long long* totals = e.arena.take<unsigned long long>(2);
  if (!ucount || !noff || !totals) return fail(FSIG_EADMISSION, "arena");
  uint32_t h_tot[2] = {0, 0};  // entries without and with repeats
  unsigned long long repeats = 0;
  FSIG_CUDA_TRY(cudaMemcpyAsync(h_tot + 1, g.off + V, 4, cudaMemcpyDeviceToHost, s));
  FSIG_CUDA_TRY(cudaMemcpyAsync(hf, flags, 4, cudaMemcpyDeviceToHost, s));
  FSIG_CUDA_TRY(cudaStreamSynchronize(s));
  if (hf[0] & 2u) return fail(FSIG_EINVAL, "edge endpoint out of range");
  FSIG_CUDA_TRY(cudaMemsetAsync(totals, 0, 16, s));
  repeats_kernel<<<grid_for(std::max<uint64_t>(h_tot[1], V), 256, e.num_sms), 256, 0, s>>>(g.off, g.adj, V, h_tot[1],
                                                                                          totals);
  FSIG_CUDA_TRY(cudaGetLastError());
  FSIG_CUDA_TRY(cudaMemcpyAsync(&repeats, totals, 8, cudaMemcpyDeviceToHost, s));
  FSIG_CUDA_TRY(cudaStreamSynchronize(s));
  h_tot[0] = h_tot[1] - uint32_t(repeats);
  if (repeats) {
    FSIG_CUDA_TRY(cudaMemsetAsync(ucount, 0, sizeof(uint32_t) * (uint64_t(V) + 1), s));
    unique_count_kernel<<<grid_for(uint64_t(V) * 32, 256, e.num_sms), 256, 0, s>>>(g.off, g.adj, V, ucount);
    FSIG_CUDA_TRY(cudaGetLastError());
    rc = device_exclusive_scan<uint32_t>(e.arena, ucount, noff, uint64_t(V) + 1, nullptr, s);
    if (rc) return rc;
    uint32_t* tmp = e.arena.take<uint32_t>(std::max<uint32_t>(h_tot[0], 1));
    if (!tmp) return fail(FSIG_EADMISSION, "arena");
    unique_copy_kernel<<<grid_for(uint64_t(V) * 32, 256, e.num_sms), 256, 0, s>>>(g.off, g.adj, V, noff, tmp);
    FSIG_CUDA_TRY(cudaGetLastError());
    FSIG_CUDA_TRY(cudaMemcpyAsync(g.adj, tmp, sizeof(uint32_t) * h_tot[0], cudaMemcpyDeviceToDevice, s));
    FSIG_CUDA_TRY(cudaMemcpyAsync(g.off, noff, sizeof(uint32_t) * (uint64_t(V) + 1), cudaMemcpyDeviceToDevice, s));
    max_row_kernel<<<grid_for(V, 256, e.num_sms), 256, 0, s>>>(g.off, V, reinterpret_cast<uint32_t*>(totals + 1));
    FSIG_CUDA_TRY(cudaGetLastError());
    FSIG_CUDA_TRY(cudaMemcpyAsync(&g.max_deg, totals + 1, 4, cudaMemcpyDeviceToHost, s));
  }
  g.nadj = h_tot[0];
  FSIG_CUDA_TRY(cudaStreamSynchronize(s));
  e.arena.release(mark_tmp);

  // Persistent label table, segments and signatures.
  const bool table = use_segment_table(e.seg_index, V, L, g.nadj);
  g.base = e.arena.take<uint32_t>(uint64_t(L) + 1);
  g.sig = e.arena.take<uint4>(uint64_t(V) * 4);
  if (table) {
    g.lseg = e.arena.take<uint32_t>(uint64_t(V) * (uint64_t(L) + 1));
    g.adj_old = e.arena.take<uint32_t>(std::max<uint64_t>(g.nadj, 1));
  }
  if (!g.base || !g.sig || (table && (!g.lseg || !g.adj_old)))
    return fail(FSIG_EADMISSION, "graph tables do not fit the device arena");
  FSIG_CUDA_TRY(cudaMemcpyAsync(g.base, g.h_base.data(), sizeof(uint32_t) * (L + 1), cudaMemcpyHostToDevice, s));
  if (table) {
    if (g.nadj) {
      gather_kernel<<<grid_for(g.nadj, 256, e.num_sms), 256, 0, s>>>(g.adj, g.nadj, g.old_of_new, g.adj_old);
      FSIG_CUDA_TRY(cudaGetLastError());
    }
    label_segments_kernel<<<grid_for(uint64_t(V) * (L + 1), 256, e.num_sms), 256, 0, s>>>(g.off, g.adj, g.base, V,
                                                                                         L, g.lseg);
    FSIG_CUDA_TRY(cudaGetLastError());
    signature_from_segments_kernel<<<grid_for(V, 128, e.num_sms), 128, 0, s>>>(g.label, g.lseg, V, L, g.sig);
  } else {
    // one saturating increment per neighbour (rows have no duplicates) gives
    // every label segment's min(count, 2) increments
    signature_from_rows_kernel<<<grid_for(uint64_t(V) * 32, 256, e.num_sms), 256, 0, s>>>(g.label, g.off, g.adj, V, 0,
                                                                           reinterpret_cast<uint32_t*>(g.sig));
  }
  FSIG_CUDA_TRY(cudaGetLastError());
  g.arena_mark = e.arena.mark();
  rc = build_membership_filter(e, g, kFilterSpare);
  if (rc) return rc;
  FSIG_CUDA_TRY(cudaStreamSynchronize(s));
  e.g = g;
  e.has_graph = true;
  return FSIG_OK;
}

// ---------------------------------------------------------------------------
// Binary cache of the resident graph store: a header, then the device arrays
// as they are (renumbered ids, CSR, caller ids, label segments, signatures),
// so that a later load is a file read and host-to-device copies, with no
// parsing, sorting or segment building.
// ---------------------------------------------------------------------------
namespace {
constexpr char kCacheMagic[8] = {'F', 'S', 'I', 'G', 'G', 'S', '0', '1'};

constexpr uint32_t kCacheRows = 1u;  // CacheHeader::flags: a store without lseg and adj_old

struct CacheHeader {
  char magic[8];
  uint32_t V;
  int32_t L;
  uint64_t nadj;
  uint32_t max_deg;
  uint32_t flags;
};

struct CacheArray {
  void* dev;
  uint64_t bytes;
};

std::vector<CacheArray> cache_arrays(const DeviceGraph& g, bool table) {
  const uint64_t V = g.V, L1 = uint64_t(g.L) + 1;
  return {{g.label, 4 * V},
          {g.old_of_new, 4 * V},
          {g.new_of_old, 4 * V},
          {g.base, 4 * L1},
          {g.off, 4 * (V + 1)},
          {g.adj, 4 * g.nadj},
          {g.adj_old, table ? 4 * g.nadj : 0},
          {g.lseg, table ? 4 * V * L1 : 0},
          {g.sig, 64 * V}};
}
}  // namespace

int save_graph_cache(Engine& e, const char* path) {
  if (!e.has_graph) return fail(FSIG_ENOGRAPH, "no data graph loaded");
  const DeviceGraph& g = e.g;
  FILE* f = std::fopen(path, "wb");
  if (!f) return fail(FSIG_EIO, std::string("cannot open ") + path);
  CacheHeader h{};
  std::memcpy(h.magic, kCacheMagic, 8);
  h.V = g.V;
  h.L = g.L;
  h.nadj = g.nadj;
  h.max_deg = g.max_deg;
  h.flags = g.lseg ? 0u : kCacheRows;
  bool ok = std::fwrite(&h, sizeof h, 1, f) == 1;
  std::vector<char> buf;
  for (const CacheArray& a : cache_arrays(g, g.lseg != nullptr)) {
    if (!ok) break;
    buf.resize(a.bytes);
    if (a.bytes) {
      const cudaError_t err = cudaMemcpy(buf.data(), a.dev, a.bytes, cudaMemcpyDeviceToHost);
      if (err != cudaSuccess) {
        std::fclose(f);
        return fail_cuda(err, "cudaMemcpy", __FILE__, __LINE__);
      }
      ok = std::fwrite(buf.data(), 1, a.bytes, f) == a.bytes;
    }
  }
  if (std::fclose(f) != 0) ok = false;
  return ok ? FSIG_OK : fail(FSIG_EIO, std::string("cannot write ") + path);
}

int load_graph_cache(Engine& e, const char* path) {
  FILE* f = std::fopen(path, "rb");
  if (!f) return fail(FSIG_EIO, std::string("cannot open ") + path);
  CacheHeader h{};
  if (std::fread(&h, sizeof h, 1, f) != 1 || std::memcmp(h.magic, kCacheMagic, 8) != 0 || h.V == 0 || h.L < 1 ||
      h.L > int32_t(kMaxLabels) || h.nadj > 0xffffffffull || (h.flags & ~kCacheRows) != 0) {
    std::fclose(f);
    return fail(FSIG_EIO, std::string(path) + " is not a graph cache of this engine");
  }
  e.arena.release(0);
  e.arena.tail = 0;
  e.has_graph = false;
  DeviceGraph g;
  g.V = h.V;
  g.L = h.L;
  g.nadj = h.nadj;
  g.max_deg = h.max_deg;
  const uint64_t V = g.V, L1 = uint64_t(g.L) + 1;
  g.label = e.arena.take<int32_t>(V);
  g.old_of_new = e.arena.take<uint32_t>(V);
  g.new_of_old = e.arena.take<uint32_t>(V);
  g.off = e.arena.take<uint32_t>(V + 1);
  g.adj = e.arena.take<uint32_t>(std::max<uint64_t>(g.nadj, 1));
  const bool table = (h.flags & kCacheRows) == 0;
  g.base = e.arena.take<uint32_t>(L1);
  g.sig = e.arena.take<uint4>(V * 4);
  if (table) {
    g.lseg = e.arena.take<uint32_t>(V * L1);
    g.adj_old = e.arena.take<uint32_t>(std::max<uint64_t>(g.nadj, 1));
  }
  if (!g.label || !g.old_of_new || !g.new_of_old || !g.off || !g.adj || !g.base || !g.sig ||
      (table && (!g.lseg || !g.adj_old))) {
    std::fclose(f);
    e.arena.release(0);
    return fail(FSIG_EADMISSION, "graph does not fit the device arena");
  }
  std::vector<char> buf;
  for (const CacheArray& a : cache_arrays(g, table)) {
    buf.resize(a.bytes);
    if (a.bytes && std::fread(buf.data(), 1, a.bytes, f) != a.bytes) {
      std::fclose(f);
      e.arena.release(0);
      return fail(FSIG_EIO, std::string(path) + " is truncated");
    }
    if (a.bytes) FSIG_CUDA_TRY(cudaMemcpy(a.dev, buf.data(), a.bytes, cudaMemcpyHostToDevice));
  }
  std::fclose(f);
  g.h_base.resize(L1);
  FSIG_CUDA_TRY(cudaMemcpy(g.h_base.data(), g.base, 4 * L1, cudaMemcpyDeviceToHost));
  g.arena_mark = e.arena.mark();
  const int rc = build_membership_filter(e, g, kFilterSpare);
  if (rc) return rc;
  FSIG_CUDA_TRY(cudaStreamSynchronize(e.stream));
  e.g = g;
  e.has_graph = true;
  return FSIG_OK;
}

int build_reference_csr(Engine& e, uint32_t V, uint64_t E, const uint32_t* h_edges, uint32_t* h_off,
                        uint32_t* h_adj) {
  cudaStream_t s = e.stream;
  if (2 * E > 0xffffffffull) return fail(FSIG_EINVAL, "graph has 2^31 or more edges");
  uint64_t m = e.arena.mark();
  uint32_t* off = e.arena.take<uint32_t>(uint64_t(V) + 1);
  uint32_t* adj = e.arena.take<uint32_t>(std::max<uint64_t>(2 * E, 1));
  uint2* d_edges = e.arena.take<uint2>(std::max<uint64_t>(E, 1));
  uint32_t* flags = e.arena.take<uint32_t>(4);
  if (!off || !adj || !d_edges || !flags) { e.arena.release(m); return fail(FSIG_EADMISSION, "CSR does not fit the arena"); }
  if (E) FSIG_CUDA_TRY(cudaMemcpyAsync(d_edges, h_edges, sizeof(uint2) * E, cudaMemcpyHostToDevice, s));
  FSIG_CUDA_TRY(cudaMemsetAsync(flags, 0, 16, s));
  int rc = build_rows(e, d_edges, E, V, nullptr, false, off, adj, flags);
  if (rc) { e.arena.release(m); return rc; }
  uint32_t hf = 0;
  FSIG_CUDA_TRY(cudaMemcpyAsync(&hf, flags, 4, cudaMemcpyDeviceToHost, s));
  FSIG_CUDA_TRY(cudaMemcpyAsync(h_off, off, sizeof(uint32_t) * (uint64_t(V) + 1), cudaMemcpyDeviceToHost, s));
  if (E) FSIG_CUDA_TRY(cudaMemcpyAsync(h_adj, adj, sizeof(uint32_t) * 2 * E, cudaMemcpyDeviceToHost, s));
  FSIG_CUDA_TRY(cudaStreamSynchronize(s));
  e.arena.release(m);
  if (hf & 2u) return fail(FSIG_EINVAL, "edge endpoint out of range");
  return FSIG_OK;
}

int build_reference_signature(Engine& e, uint32_t V, const int32_t* h_labels, const uint32_t* h_off,
                              const uint32_t* h_adj, int column_oriented, uint32_t* h_sig) {
  cudaStream_t s = e.stream;
  uint64_t nadj = h_off[V];
  uint64_t m = e.arena.mark();
  int32_t* lab = e.arena.take<int32_t>(V);
  uint32_t* off = e.arena.take<uint32_t>(uint64_t(V) + 1);
  uint32_t* adj = e.arena.take<uint32_t>(std::max<uint64_t>(nadj, 1));
  uint32_t* sig = e.arena.take<uint32_t>(uint64_t(V) * kSigWords);
  if (!lab || !off || !adj || !sig) { e.arena.release(m); return fail(FSIG_EADMISSION, "signature does not fit the arena"); }
  FSIG_CUDA_TRY(cudaMemcpyAsync(lab, h_labels, sizeof(int32_t) * V, cudaMemcpyHostToDevice, s));
  FSIG_CUDA_TRY(cudaMemcpyAsync(off, h_off, sizeof(uint32_t) * (uint64_t(V) + 1), cudaMemcpyHostToDevice, s));
  if (nadj) FSIG_CUDA_TRY(cudaMemcpyAsync(adj, h_adj, sizeof(uint32_t) * nadj, cudaMemcpyHostToDevice, s));
  signature_from_rows_kernel<<<grid_for(uint64_t(V) * 32, 256, e.num_sms), 256, 0, s>>>(lab, off, adj, V, column_oriented, sig);
  FSIG_CUDA_TRY(cudaGetLastError());
  FSIG_CUDA_TRY(cudaMemcpyAsync(h_sig, sig, sizeof(uint32_t) * kSigWords * V, cudaMemcpyDeviceToHost, s));
  FSIG_CUDA_TRY(cudaStreamSynchronize(s));
  e.arena.release(m);
  return FSIG_OK;
}

}  // namespace fsig
