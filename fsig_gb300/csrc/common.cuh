// Shared device helpers, the device arena and error plumbing for libfsig.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/fsig.h"

namespace fsig {

constexpr uint32_t kInvalid = 0xffffffffu;
constexpr int kSigWords = 16;          // 512-bit signature, word 0 = label
constexpr uint32_t kMurmurSeed = 17;   // HASHSEED of the reference

// ---------------------------------------------------------------------------
// hashing
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ uint64_t fmix64(uint64_t k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ull;
  k ^= k >> 33;
  return k;
}

// MurmurHash2 (Appleby) of one little-endian 32-bit word with seed 17, the
// key hash of the reference's PCSR buckets and signature slots.
__host__ __device__ __forceinline__ uint32_t murmur2_u32(uint32_t k) {
  const uint32_t m = 0x5bd1e995u;
  uint32_t h = kMurmurSeed ^ 4u;
  k *= m;
  k ^= k >> 24;
  k *= m;
  h = (h * m) ^ k;
  h ^= h >> 13;
  h *= m;
  h ^= h >> 15;
  return h;
}

// Signature counter position for a neighbour label: word 1 + a, shift s.
// The shift is (2*b) & 31 with b = (2*slot) % 32 (see the signature builder).
__host__ __device__ __forceinline__ void sig_slot(int32_t label, uint32_t& word, uint32_t& shift) {
  uint32_t hp = murmur2_u32(uint32_t(label)) % 240u;
  word = 1u + (2u * hp) / 32u;
  shift = (2u * ((2u * hp) % 32u)) & 31u;
}

// ---------------------------------------------------------------------------
// membership filter of the adjacency's label segments: 1 << s words of 16 bits
// per entry, the block of segment [lo, hi) being words [lo << s, hi << s).  A
// segment that is dense in its label class (class extent at most as many ids as
// its block has bits) holds one bit per id of the class, which is exact; another
// is a Bloom filter whose element x sets two bits of one word, so that with one
// word an entry 2-3 % of the ids that are not in it pass.  One
// probe of a word settles most candidates that a binary search took 7-8
// dependent loads to refuse: the 512-query batch on 2^26 edges 377 -> 197 ms (247
// without it and 128 with it by now), house counting on 700 vertices (dense
// segments) 93 -> 63 ms.  The filter lies
// in arena room that a request which needs it takes back, so what fitted an arena
// still fits, and is built again once that room is free.  One word an entry is
// half the adjacency; graphs of at most kFilterSmall entries get four (32 MB
// then, well inside the L2), which makes segments from a quarter of that length on
// exact.  (Four measured better at 2.1 M entries and below; one is for graphs whose
// filter would outgrow the L2, measured at 2^27.  Where between them the line
// lies best was not measured.)
// ---------------------------------------------------------------------------
constexpr uint64_t kFilterSmall = 1ull << 22;
__host__ __device__ __forceinline__ uint32_t filter_shift(uint64_t nadj) { return nadj <= kFilterSmall ? 2 : 0; }
// the shortest dense segment of a class of this extent
__device__ __forceinline__ uint32_t filter_dense_len(uint32_t extent, uint32_t shift) {
  return ((extent - 1) >> (4 + shift)) + 1;
}
__device__ __forceinline__ uint32_t filter_hash(uint32_t x) { return x * 0x9e3779b1u; }
__device__ __forceinline__ uint32_t filter_bits(uint32_t x) {
  const uint32_t h = x * 0x85ebca6bu;
  return (1u << (h >> 28)) | (1u << ((h >> 24) & 15u));
}
// word of x within its segment's block of `words`; rel = x - first id of the class's extent
__device__ __forceinline__ uint32_t filter_word(bool dense, uint32_t rel, uint32_t hash, uint32_t words) {
  return dense ? rel >> 4 : __umulhi(hash, words);
}
__device__ __forceinline__ uint32_t filter_mask(bool dense, uint32_t rel, uint32_t bits) {
  return dense ? 1u << (rel & 15u) : bits;
}

// ---------------------------------------------------------------------------
// device arena: one cudaMalloc, bump allocation with marks
// ---------------------------------------------------------------------------
struct Arena {
  char* base = nullptr;
  uint64_t cap = 0;
  uint64_t top = 0;
  uint64_t peak = 0;
  uint64_t tail = 0;  // bytes at the end lent to what can do without them (take_tail)

  static constexpr uint64_t kAlign = 256;
  // Returns nullptr when the request does not fit (admission failure).
  template <class T>
  T* take(uint64_t count) {
    uint64_t bytes = (count * sizeof(T) + kAlign - 1) & ~(kAlign - 1);
    if (bytes == 0) bytes = kAlign;
    if (top + bytes > cap) return nullptr;
    if (top + bytes > cap - tail) tail = 0;  // the tail's room is needed: its holder sees tail == 0
    T* p = reinterpret_cast<T*>(base + top);
    top += bytes;
    if (top > peak) peak = top;
    return p;
  }
  // Room at the end, beyond `spare` free bytes, that the next take() that needs
  // it gets back; nullptr when there is not that much.
  template <class T>
  T* take_tail(uint64_t count, uint64_t spare) {
    const uint64_t bytes = (count * sizeof(T) + kAlign - 1) & ~(kAlign - 1);
    const uint64_t end = cap & ~(kAlign - 1);
    if (bytes == 0 || top + bytes + spare > end) return nullptr;
    tail = cap - (end - bytes);
    return reinterpret_cast<T*>(base + (end - bytes));
  }
  uint64_t mark() const { return top; }
  void release(uint64_t m) { top = m; }
  uint64_t free_bytes() const { return cap - top; }
};

// ---------------------------------------------------------------------------
// warp helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }
__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}
__device__ __forceinline__ uint32_t lanemask_le() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_le;" : "=r"(m));
  return m;
}
template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// End of the piece of at most `step` entries that begins at lo in [lo, hi): the
// sum lo + step may not fit 32 bits (any step a caller gives, positions of large
// adjacencies).
__host__ __device__ __forceinline__ uint32_t piece_end(uint32_t lo, uint32_t step, uint32_t hi) {
  return hi - lo > step ? lo + step : hi;
}
// Pieces of at most `step` entries in `len` entries.
__host__ __device__ __forceinline__ uint32_t piece_count(uint32_t len, uint32_t step) {
  return len ? (len - 1) / step + 1 : 0;
}

// between lo and hi; their sum may not fit 32 bits
__host__ __device__ __forceinline__ uint32_t midpoint(uint32_t lo, uint32_t hi) { return lo + ((hi - lo) >> 1); }

// first index in [lo, hi) of sorted a[] with a[i] >= key
__host__ __device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t* __restrict__ a, uint32_t lo, uint32_t hi,
                                                             uint32_t key) {
  while (lo < hi) {
    const uint32_t mid = midpoint(lo, hi);
#ifdef __CUDA_ARCH__
    const uint32_t x = __ldg(a + mid);
#else
    const uint32_t x = a[mid];
#endif
    if (x < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

}  // namespace fsig

#define FSIG_CUDA_TRY(expr)                                                        \
  do {                                                                              \
    cudaError_t _e = (expr);                                                        \
    if (_e != cudaSuccess) {                                                        \
      return ::fsig::fail_cuda(_e, #expr, __FILE__, __LINE__);                      \
    }                                                                               \
  } while (0)

namespace fsig {
// Records the CUDA error text in a thread-local slot; the C ABI copies it to
// the engine's last-error string.
int fail_cuda(cudaError_t e, const char* what, const char* file, int line);
int fail(int status, const std::string& msg);
const std::string& thread_error();
void clear_thread_error();
}  // namespace fsig
