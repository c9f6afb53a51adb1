// Enumeration kernel: depth-first extension of partial embeddings, one warp
// per task, with work stealing.  Included by match.cu.
//
// A task is (query q, depth d, mapped vertices f[0..d), driver range
// [lo, hi) at depth d).  Pass 0 takes implicit tasks: every root candidate of
// every query, with its depth-1 driver range cut into chunks of `split`
// entries.  Later passes (normally none) take explicit task records.
//
// A warp extends up to 32 partial embeddings at a time, one per lane.  For
// every depth it keeps a buffer of up to 32 mapped vertices in shared memory,
// each with the slot of its parent in the previous depth's buffer; an entry's
// earlier vertices are found by walking its parents.  Lane j holds depth j's
// cursor (cnt_j entries, it_j the first one not wholly extended, off_j how
// much of that one's driver range is examined).
//
// Filling the buffer of depth i from depth i-1's entries: each lane takes one
// entry, finds the label-l(i) segments of its backward neighbours' rows
// (bounds into shared memory) and picks the shortest as its driver.  The
// drivers of all entries, end to end, are then examined 32 candidates at a
// time, one per lane, whichever entry they belong to: the lanes' owners come
// from the bits where a driver begins in this window.  A candidate passes
// when its bit in depth i's candidate bitmap is set, it differs from the
// entry's earlier vertices of the same label (adjacent ones differ anyway),
// and it lies in each of the entry's other backward segments, two per-lane
// binary searches in lockstep (two independent loads in flight).  Candidates
// that pass the first two tests are appended to depth i's buffer and searched
// for once it is full, so that the searches run on all lanes; those found stay.
// A buffer with enough entries is extended in turn, and later the fill goes on
// where it stopped.  At the leaf the passing candidates are counted and hashed.
//
// What bounds it: instructions and L2 latency (the working set is L2
// resident), so the aim is full lanes.  A warp per entry, as before, ran 11 of
// 32 lanes at the leaf of the 320k-vertex workloads (one range of 11-12
// neighbours after another) and paid the set-up of a range, some 300
// instructions, for each.  200 eight-vertex queries there 115 -> 34 ms of
// kernel, 512 queries of 4-32 vertices 69 -> 34 ms, 253 instructions a window
// at 79 % of the issue rate.  On 2^26 edges, where the searches dominate, it is
// bound by their latency at 24 warps an SM (49 % of the issue rate).
//
// Work stealing: a warp that runs out of input takes a ticket, one atomicAdd
// on the queue's head, and waits for the record of that number, polling the
// record's own ready word.  A busy warp checks every 64 steps whether more
// tickets than records are out; if so it hands its shallowest pending depth
// (buffered candidates and the remaining driver range) to the queue as task
// records and carries on with the rest.  One counter holds the warps at work
// plus the records not taken yet; the pass is over when it reaches zero.
// (Tickets replaced a compare-and-swap on the head by every idle warp for
// every record: up to 2048 warps retrying on one word served a record in
// 0.4-1.0 us whatever the work in it, which bounded every batch but the
// largest.  One 4-vertex query on a 10k-vertex graph 3.8 -> 0.37 ms, 100 of
// them 37 -> 2.5 ms, 37 refined queries on 2^26 edges 78 -> 29 ms, a
// 512-query batch there 390 -> 305 ms.)  Waiting is bounded: a warp that waits too long leaves, which
// never loses work -- the records nobody took are the next pass's input.
// Every value that steers a warp's control flow is read by lane 0 and
// broadcast.
#pragma once

namespace fsig {
namespace {

struct TaskRec {
  uint32_t f[kMaxQ];
  uint32_t q, d, lo, hi;  // lo == hi == kInvalid: the whole driver range
};

struct EnumArgs {
  GraphView g;
  const Plan* __restrict__ plans;
  const uint32_t* __restrict__ pool;
  uint32_t Q;
  // pass-0 implicit tasks
  const uint32_t* __restrict__ roots;
  const uint32_t* __restrict__ root_q;
  const uint32_t* __restrict__ chunk_off;  // [nroots + 1]
  const uint32_t* __restrict__ nroots_ptr;  // number of roots (device)
  uint32_t split;
  uint32_t t_end;  // pass-0 tasks [initial ctr[0], t_end) (a range of the task space)
  // explicit input tasks (passes >= 1)
  const TaskRec* __restrict__ in_tasks;
  const uint32_t* __restrict__ in_index;  // [in_count] records of in_tasks
  uint32_t in_count;
  // work queue
  TaskRec* out_tasks;
  uint32_t* out_ready;
  uint32_t out_cap;  // a power of two
  uint32_t* ctr;  // counters, kCtrStride apart: [0] input grab, [1] queue tail (records reserved) and,
                  // in the next word, tickets taken, [2] warps at work + records not taken yet,
                  // [3] error bits, [4] fault injection's one-shot, [5] once a waiting warp has left,
                  // the record number from which on no more are reserved
  uint32_t chunk;
  long long budget;  // cycles on a task before it may be split while warps are idle
  QueryResult* res;
  unsigned long long work_cap;  // per-query limit on examined driver entries (0: none)
  unsigned long long* algo_bytes;
  unsigned long long* ev;       // event counters: tasks, records popped, hand-offs, records written, examines
  unsigned long long seed;
  // optional embedding output (single-query batches): rows of n caller ids,
  // column u = the data vertex of query vertex u; emit_ctr counts every
  // embedding found, rows past emit_cap are not written
  uint32_t* emit;
  unsigned long long emit_cap;
  unsigned long long* emit_ctr;
  // bounded waits (nanoseconds of the GPU's global timer): how long a warp
  // waits for a record it took to be published, and how long an idle warp
  // waits for hand-offs before it leaves (its queued work runs in a later pass)
  unsigned long long ready_wait_ns;
  unsigned long long idle_wait_ns;
  // fault injection for tests: the first record handed off in the pass is
  // written but never published, so the warp that takes it waits out
  // ready_wait_ns and the pass reports a timeout
  uint32_t unpublished;
  uint32_t levels;  // depths with a buffer: the batch's largest query minus one, at least 1
};

constexpr uint32_t kErrTimeout = 1u;
constexpr uint32_t kCtrStride = 32;        // one 128-byte line per counter
// The queue is a ring: record number t lies in slot t mod out_cap, use
// g = t / out_cap of that slot.  The slot's ready word is 2g while it is free
// for that use, 2g + 1 from the record's publication until its ticket holder
// has read it, then 2g + 2 (= free for use g + 1).  Records are reserved only
// while warps wait, so at most (warps) x (records of one hand-off) numbers lie
// between the tickets and the tail, far below the ring's 2^20 slots: a
// reserved slot's previous record always has a ticket holder.

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr uint32_t kBuf = 32;        // entries of a depth's buffer
constexpr uint32_t kScratch = 384;   // words for the segments and earlier vertices of the entries being extended
// Candidate windows one fill examines before it returns, so that the periodic
// checks and hand-offs come in time on long driver ranges.
constexpr uint32_t kFillWindows = 64;
// Windows between two checks of the work limit and of the waiting warps.
constexpr uint32_t kCheckWindows = 32;

// Per warp; followed by cand[levels][kBuf] and par[levels][kBuf], levels = the
// batch's largest query minus one.
struct WarpSmem {
  Plan plan;
  uint2 owner[kBuf];                // entries with a driver: its place relative to the window index, the entry
  unsigned long long sown[kBuf];    // leaf: partial hash of each entry being extended
  unsigned long long sbase[kBuf];   // partial hashes of depth n-3's buffer
  uint32_t scratch[kScratch];
  uint8_t drv[kBuf];                // driver of each entry being extended (its place in scratch)
};

constexpr size_t warp_smem_bytes(uint32_t levels) {
  return (sizeof(WarpSmem) + size_t(levels) * kBuf * 5 + 15) & ~size_t(15);
}

// Segment [lo, hi) of row v's neighbours with label l (0 <= l < L): two loads
// from the dense table, or, in a graph store without one (kRows), two binary
// searches in the row for the first ids of label classes l and l + 1.
template <bool kRows>
__device__ __forceinline__ void row_segment(const GraphView& g, uint32_t v, int32_t l, uint64_t W1, uint32_t& lo,
                                            uint32_t& hi) {
  if constexpr (kRows) {
    const uint32_t b = __ldg(g.off + v), e = __ldg(g.off + v + 1);
    lo = lower_bound_u32(g.adj, b, e, __ldg(g.base + l));
    hi = lower_bound_u32(g.adj, lo, e, __ldg(g.base + l + 1));
  } else {
    const uint32_t* s = g.lseg + uint64_t(v) * W1 + l;
    lo = s[0];
    hi = s[1];
  }
}

// Whether x lies in both sorted segments a[lo0, hi0) and a[lo1, hi1) (in the
// first alone without `two`): two binary searches in lockstep, so that a step
// has two independent loads in flight.
__device__ __forceinline__ bool in_segments(const uint32_t* __restrict__ a, uint32_t lo0, uint32_t hi0, uint32_t lo1,
                                            uint32_t hi1, bool two, uint32_t x, uint32_t& bytes) {
  uint32_t n0 = hi0 - lo0, n1 = two ? hi1 - lo1 : 1;
  if (n0 == 0 || n1 == 0) return false;
#pragma unroll 1
  while (n0 > 1 || n1 > 1) {
    const uint32_t h0 = n0 >> 1, h1 = n1 >> 1;
    const uint32_t y0 = __ldg(a + lo0 + h0), y1 = __ldg(a + lo1 + h1);
    if (y0 <= x) lo0 += h0;
    if (y1 <= x) lo1 += h1;
    n0 -= h0;
    n1 -= h1;
    bytes += 8;
  }
  bytes += 8;
  return __ldg(a + lo0) == x && (!two || __ldg(a + lo1) == x);
}

// kRows: the graph store has no segment table (GraphView::lseg is null) and
// no caller-id copy of the adjacency (adj_old); segments are found in the
// rows and a leaf's caller id is looked up once it survives.
template <bool kRows>
__global__ void __launch_bounds__(kEnumWarps * 32, kEnumMinBlocks) enumerate_kernel(EnumArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WarpSmem& ws = *reinterpret_cast<WarpSmem*>(smem_raw + warp_smem_bytes(A.levels) * (threadIdx.x >> 5));
  uint32_t* const cand = reinterpret_cast<uint32_t*>(&ws + 1);              // [levels][kBuf]
  uint8_t* const par = reinterpret_cast<uint8_t*>(cand + A.levels * kBuf);  // [levels][kBuf]
  const uint32_t lane = threadIdx.x & 31;
  const GraphView& g = A.g;
  const uint64_t W1 = uint64_t(g.L) + 1;
  const uint32_t nroots = A.in_tasks ? 0u : *A.nroots_ptr;
  const uint32_t T_in = A.in_tasks ? A.in_count : min(A.chunk_off[nroots], A.t_end);

  // lane-distributed level state; f is the task's prefix (lane j: f_j)
  uint32_t f = 0, cnt = 0, it = 0, off = 0;
  unsigned long long my_hash = 0;
  bool s_valid = false;  // sbase holds depth n-3's current buffer
  unsigned long long lc = 0;  // lane j: partial embeddings of length j + 1 found (lane n-1: embeddings)
  uint32_t bytes = 0;         // drained into the 64-bit total before it can overflow
  uint32_t pend = 0;          // driver entries examined, not yet published to res.work (lane 0)
  // event counters (lane 0); a warp's share of one launch fits 32 bits
  uint32_t n_tasks = 0, n_pops = 0, n_handoffs = 0, n_recs = 0, n_examine = 0;
  uint32_t cur_q = kInvalid;

  // Publishes the driver entries this warp examined for the current query.
  // The total a query examines does not depend on how its work was split
  // (every driver entry counts once), so whether it exceeds the limit does not
  // either.
  auto publish = [&]() {
    if (lane == 0 && pend) {
      const unsigned long long tot = atomicAdd(&A.res[cur_q].work, (unsigned long long)pend) + pend;
      pend = 0;
      if (tot > A.work_cap) atomicExch(&A.res[cur_q].aborted, 1u);
    }
  };

  // Prefix of the entry in slot `slot` of depth p's buffer: lane j <= p gets f_j.
  auto prefix = [&](uint32_t p, uint32_t slot) {
    uint32_t v = 0;
#pragma unroll 1
    for (uint32_t k = p;; k--) {
      const uint32_t x = cand[k * kBuf + slot];
      if (lane == k) v = x;
      if (k == 0) break;
      slot = par[k * kBuf + slot];
    }
    return v;
  };

  // Hands the shallowest depth from d0 - 1 to last that still has entries to
  // extend to the queue -- each entry a record, the rest of a partly extended
  // entry's driver range in pieces for the waiting warps -- and marks that depth
  // done here.  [lo_set, hi_set): the task's own driver range at depth d0, if
  // it has one.  Returns false when no records may be reserved.
  auto donate = [&](uint32_t d0, uint32_t last, uint32_t hungry, uint32_t lo_set, uint32_t hi_set) -> bool {
    const uint32_t has = __ballot_sync(kFull, lane + 1 >= d0 && lane <= last && it < cnt);
    if (!has) return true;
    const uint32_t l = __ffs(has) - 1;
    const uint32_t c_l = __shfl_sync(kFull, cnt, l), i_l = __shfl_sync(kFull, it, l), o_l = __shfl_sync(kFull, off, l);
    // the current entry's driver range, when it is partly examined or given
    const bool given = l + 1 == d0 && lo_set != kInvalid;
    const bool part = given || o_l > 0;
    uint32_t lo = lo_set, hi = hi_set, fp = 0;
    if (part) {
      fp = prefix(l, i_l);
      if (!given) {  // the choice a fill makes: the shortest segment, the latest depth on ties
        uint32_t a = 0, b = 0, len = kInvalid;
        if ((ws.plan.bwd[l + 1] >> lane) & 1u) {
          row_segment<kRows>(g, fp, ws.plan.lab[l + 1], W1, a, b);
          len = b - a;
        }
        const uint32_t shortest = __reduce_min_sync(kFull, len);
        const uint32_t j = 31 - __clz(__ballot_sync(kFull, len == shortest));
        lo = __shfl_sync(kFull, a, j);
        hi = __shfl_sync(kFull, b, j);
      }
      lo += o_l;
    }
    const uint32_t rest = part ? hi - lo : 0u, takers = min(hungry, 32u);
    const uint32_t hand = max(32u, (rest + takers - 1) / takers);
    const uint32_t pieces = (rest + hand - 1) / hand;
    const uint32_t first = part ? i_l + 1 : i_l;
    const uint32_t total = pieces + (c_l - first);
    uint32_t base = 0;
    if (lane == 0) {
      const uint32_t limit = *(volatile uint32_t*)&A.ctr[5 * kCtrStride];
      if (limit && *(volatile uint32_t*)&A.ctr[1 * kCtrStride] + total > limit) {
        base = kInvalid;
      } else {
        base = atomicAdd(&A.ctr[1 * kCtrStride], total);
        atomicAdd(&A.ctr[2 * kCtrStride], total);
      }
    }
    base = __shfl_sync(kFull, base, 0);
    if (base == kInvalid) return false;
    // the slots' previous records are read by now, or about to be (see above)
    {
      const uint32_t mask = A.out_cap - 1, shift = 31 - __clz(A.out_cap);
      const unsigned long long t0 = global_ns();
#pragma unroll 1
      for (uint32_t k = base + lane; k < base + total; k += 32) {
        while (*(volatile uint32_t*)&A.out_ready[k & mask] != 2 * (k >> shift)) {
          if (global_ns() - t0 > A.ready_wait_ns) {
            atomicOr(&A.ctr[3 * kCtrStride], kErrTimeout);
            break;
          }
        }
      }
      __syncwarp();
    }
    uint32_t slot = base;
#pragma unroll 1
    for (uint32_t k = 0; k < pieces; k++) {
      TaskRec* r = A.out_tasks + (slot++ & (A.out_cap - 1));
      if (lane <= l) r->f[lane] = fp;
      if (lane == 0) { r->q = cur_q; r->d = l + 1; r->lo = lo + k * hand; r->hi = min(lo + (k + 1) * hand, hi); }
    }
#pragma unroll 1
    for (uint32_t k = first; k < c_l; k++) {
      TaskRec* r = A.out_tasks + (slot++ & (A.out_cap - 1));
      const uint32_t fk = prefix(l, k);
      if (lane <= l) r->f[lane] = fk;
      if (lane == 0) { r->q = cur_q; r->d = l + 1; r->lo = kInvalid; r->hi = kInvalid; }
    }
    if (lane == l) {
      it = cnt;
      off = 0;
    }
    __threadfence();
    __syncwarp();
    int hold = 0;  // test hook: keep the pass's first handed-off record unpublished
    if (A.unpublished && lane == 0) hold = atomicCAS(&A.ctr[4 * kCtrStride], 0u, 1u) == 0u;
    hold = __shfl_sync(kFull, hold, 0);
#pragma unroll 1
    for (uint32_t k = base + lane; k < base + total; k += 32)
      if (!(hold && k == base))
        atomicExch(&A.out_ready[k & (A.out_cap - 1)], 2 * (k >> (31 - __clz(A.out_cap))) + 1);
    if (lane == 0) { n_handoffs++; n_recs += total; }
    return true;
  };

  // How many warps wait for records that nobody has reserved (tickets minus
  // records), 0 while this task is younger than its budget.  Decided by lane 0
  // alone and broadcast.
  auto waiting_warps = [&](uint32_t t_start) -> uint32_t {
    uint32_t w = 0;
    if (lane == 0 && A.out_cap) {
      uint32_t tail, tickets;
      asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(tail), "=r"(tickets) : "l"(A.ctr + kCtrStride));
      if (int32_t(tickets - tail) > 0 && (long long)(uint32_t(clock()) - t_start) > A.budget) w = tickets - tail;
    }
    return __shfl_sync(kFull, w, 0);
  };

  // Writes the embeddings completed by one leaf window: lanes in m hold a
  // leaf's caller id in xo and its entry's slot in depth n-2's buffer.
  auto emit_rows = [&](uint32_t m, uint32_t n, uint32_t xo, uint32_t slot) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(A.emit_ctr, (unsigned long long)__popc(m));
    base = __shfl_sync(kFull, base, 0);
    const unsigned long long row = base + __popc(m & lanemask_lt());
    if (((m >> lane) & 1u) && row < A.emit_cap) {
      uint32_t* dst = A.emit + row * n;
      dst[ws.plan.qv[n - 1]] = xo;
#pragma unroll 1
      for (uint32_t k = n - 1; k-- > 0;) {
        dst[ws.plan.qv[k]] = __ldg(g.old_of_new + cand[k * kBuf + slot]);
        slot = par[k * kBuf + slot];
      }
    }
  };

  // Extends depth lv - 1's entries to depth lv (see the top of this file): into
  // depth lv's buffer until it is about full, or, at the leaf, into counts and
  // hashes.  [lo_set, hi_set), unless kInvalid, is the driver range of the one
  // entry there is.  Returns the windows examined; the cursors of depths lv - 1
  // and lv say where it stopped.
  auto fill = [&](uint32_t lv, uint32_t lo_set, uint32_t hi_set) -> uint32_t {
    const bool leaf = lv + 1 == ws.plan.n;
    const uint32_t p = lv - 1;
    const uint32_t bwd = ws.plan.bwd[lv], inj = ws.plan.same[lv] & ~bwd;
    const int32_t lab = ws.plan.lab[lv];
    const uint32_t nb = __popc(bwd), ni = __popc(inj);
    const uint32_t stride = min(kBuf, kScratch / (2 * nb + ni));  // entries per group
    const uint32_t bmbase = ws.plan.bmbase[lv];
    const uint32_t* __restrict__ bm = A.pool + ws.plan.bmoff[lv];
    const uint32_t cntp = __shfl_sync(kFull, cnt, p);
    uint32_t itp = __shfl_sync(kFull, it, p), offp = __shfl_sync(kFull, off, p);
    uint32_t have = 0, sure = 0, used = 0;  // entries appended; of them, searched for in every segment
    bool stop = false;
    if (leaf && !s_valid && lv >= 2) {  // partial hashes of depth n-3's entries
      const uint32_t c = __shfl_sync(kFull, cnt, lv - 2);
      if (lane < c) {
        unsigned long long sum = 0;
        uint32_t slot = lane;
#pragma unroll 1
        for (uint32_t k = lv - 1; k-- > 0;) {
          sum += fmix64((uint64_t(ws.plan.qv[k]) << 32) | __ldg(g.old_of_new + cand[k * kBuf + slot]));
          slot = par[k * kBuf + slot];
        }
        ws.sbase[lane] = sum;
      }
      s_valid = true;
      __syncwarp();
    }
    while (itp < cntp && !stop) {
      // the group: lane c takes entry itp + c
      uint32_t group = min(cntp - itp, stride);
      uint32_t dlo = 0, dhi = 0, drv = 0;
      if (lane < group) {
        uint32_t slot = itp + lane, need = bwd | inj, wb = 0, wi = 2 * nb, best = kInvalid;
#pragma unroll 1
        for (uint32_t k = p;; k--) {
          if ((bwd >> k) & 1u) {
            uint32_t a, b;
            row_segment<kRows>(g, cand[k * kBuf + slot], lab, W1, a, b);
            ws.scratch[wb * stride + lane] = a;
            ws.scratch[(wb + 1) * stride + lane] = b;
            if (b - a < best) {
              best = b - a;
              dlo = a;
              dhi = b;
              drv = wb;
            }
            wb += 2;
            bytes += 8;
          } else if ((inj >> k) & 1u) {
            ws.scratch[wi++ * stride + lane] = cand[k * kBuf + slot];
          }
          need &= ~(1u << k);
          if (!need) break;
          slot = par[k * kBuf + slot];
        }
        if (lo_set != kInvalid) {
          dlo = lo_set;
          dhi = hi_set;
        }
        if (lane == 0) dlo = min(dlo + offp, dhi);
        if (leaf) {
          unsigned long long sum =
              fmix64((uint64_t(ws.plan.qv[p]) << 32) | __ldg(g.old_of_new + cand[p * kBuf + itp + lane]));
          if (p > 0) sum += ws.sbase[par[p * kBuf + itp + lane]];
          ws.sown[lane] = sum;
          bytes += 4;
        }
      }
      uint32_t len = dhi - dlo;
      if (__any_sync(kFull, len >= (1u << 27))) {  // the group's total has to fit 32 bits
        group = 1;
        if (lane) len = 0;
      }
      uint32_t incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane >= uint32_t(o)) incl += y;
      }
      const uint32_t start = incl - len, T = __shfl_sync(kFull, incl, 31);
      const uint32_t full = __ballot_sync(kFull, len > 0);
      if (len > 0) ws.owner[__popc(full & lanemask_lt())] = make_uint2(dlo - start, lane);
      ws.drv[lane] = uint8_t(drv);
      __syncwarp();
      uint32_t pos = 0, begun = 0;  // begun: drivers that start before pos
      while (pos < T && !stop) {
        const uint32_t at = start - pos;
        const uint32_t heads = __reduce_or_sync(kFull, (len > 0 && start >= pos && at < 32) ? 1u << at : 0u);
        const uint32_t r = begun + __popc(heads & (lanemask_lt() | (1u << lane))) - 1;
        const uint32_t e = pos + lane;
        bool pred = e < T;
        uint32_t x = 0xffffffffu, xo = 0, c = 0;
        if (pred) {
          const uint2 o = ws.owner[r];
          c = o.y;
          x = __ldg(g.adj + (o.x + e));
          if (leaf && !kRows) xo = __ldg(g.adj_old + (o.x + e));
          const uint32_t bit = x - bmbase;
          bytes += leaf ? 12 : 8;
          pred = (__ldg(bm + (bit >> 5)) >> (bit & 31)) & 1u;
        }
#pragma unroll 1
        for (uint32_t i = 0; i < ni; i++) pred = pred && x != ws.scratch[(2 * nb + i) * stride + c];
        uint32_t step = min(32u, T - pos);
        bool searching = leaf && nb > 1;
        used++;
        if (!leaf) {
          uint32_t m = __ballot_sync(kFull, pred);
          const uint32_t got = __popc(m), rank = __popc(m & lanemask_lt());
          if (have + got > kBuf) {  // take what fits; go on from the first one that does not
            step = __ffs(__ballot_sync(kFull, pred && have + rank == kBuf)) - 1;
            m &= (1u << step) - 1;
          }
          if ((m >> lane) & 1u) {
            cand[lv * kBuf + have + rank] = x;
            par[lv * kBuf + have + rank] = uint8_t(itp + c);
          }
          have += __popc(m);
          searching = nb > 1 && have > sure && (have == kBuf || pos + step >= T || used >= kFillWindows);
          __syncwarp();
          if (searching) {  // the entries not yet searched for, one per lane
            pred = lane >= sure && lane < have;
            if (pred) {
              x = cand[lv * kBuf + lane];
              c = par[lv * kBuf + lane] - itp;
            }
          }
        }
        if (searching && pred) {
          // the entry's other segments, two at a time
          const uint32_t dseg = ws.drv[c];
          uint32_t s = dseg == 0 ? 2 : 0;
#pragma unroll 1
          while (pred && s < 2 * nb) {
            const uint32_t s1 = s + 2 == dseg ? s + 4 : s + 2;
            const bool two = s1 < 2 * nb;
            const uint32_t s2 = two ? s1 : s;
            pred = in_segments(g.adj, ws.scratch[s * stride + c], ws.scratch[(s + 1) * stride + c],
                               ws.scratch[s2 * stride + c], ws.scratch[(s2 + 1) * stride + c], two, x, bytes);
            s = s1 + 2 == dseg ? s1 + 4 : s1 + 2;
          }
        }
        __syncwarp();
        if (leaf) {
          const uint32_t m = __ballot_sync(kFull, pred);
          if (pred) {
            if (kRows) xo = __ldg(g.old_of_new + x);
            my_hash += fmix64(A.seed + ws.sown[c] + fmix64((uint64_t(ws.plan.qv[lv]) << 32) | xo));
          }
          if (A.emit && m) emit_rows(m, lv + 1, xo, itp + c);
          if (lane == lv) lc += __popc(m);
        } else {
          if (searching) {
            const uint32_t m = __ballot_sync(kFull, pred);
            have = sure + __popc(m);
            if (pred) {
              cand[lv * kBuf + sure + __popc(m & lanemask_lt())] = x;
              par[lv * kBuf + sure + __popc(m & lanemask_lt())] = uint8_t(itp + c);
            }
            sure = have;
            __syncwarp();
          }
          // enough entries: with further segments to search the room that is
          // left decides how many lanes search
          if (nb == 1) sure = have;
          stop = sure >= (nb > 1 ? kBuf / 2 : kBuf - 8);
        }
        if (lane == 0) {
          n_examine++;
          if (A.work_cap) pend += step;
        }
        begun += __popc(step < 32 ? heads & ((1u << step) - 1) : heads);
        pos += step;
        stop = stop || used >= kFillWindows;
      }
      if (pos >= T) {
        itp += group;
        offp = 0;
      } else {  // inside the last driver begun at or before pos
        const uint32_t o = 31 - __clz(__ballot_sync(kFull, len > 0 && start <= pos));
        offp = pos - __shfl_sync(kFull, start, o) + (o == 0 ? offp : 0u);
        itp += o;
      }
      __syncwarp();
    }
    if (lane == p) {
      it = itp;
      off = offp;
    }
    if (!leaf) {
      if (lane == lv) {
        cnt = have;
        it = 0;
        off = 0;
        lc += have;
      }
      if (lv + 3 == ws.plan.n) s_valid = false;
    }
    return used;
  };

  uint32_t t = 0, t_last = 0;  // input tasks in hand: [t, t_last)
#pragma unroll 1
  for (;;) {
    // ---- the next task: query q, depth d, mapped f (lane-distributed, lanes
    // < d), driver range [lo, hi) at depth d (kInvalid: the whole one).  One
    // place for every kind of task, and one copy of the code that runs it: an
    // earlier form with a copy per kind (250 KB of code) spent two thirds of
    // its issue slots waiting for instructions.
    uint32_t q = kInvalid, d = 1, lo = kInvalid, hi = kInvalid, root = kInvalid, chunk = 0;
    const TaskRec* rec = nullptr;
    uint32_t* ready = nullptr;
    uint32_t free_word = 0;
    if (t == t_last) {  // input tasks (after an error every task ends at its first check)
      uint32_t t0 = T_in;
      if (lane == 0 && *(volatile uint32_t*)&A.ctr[0 * kCtrStride] < T_in)
        t0 = atomicAdd(&A.ctr[0 * kCtrStride], A.chunk);
      t = __shfl_sync(kFull, t0, 0);
      t_last = t < T_in ? min(t + A.chunk, T_in) : t;
    }
    if (t < t_last) {
      if (A.in_tasks) {
        rec = A.in_tasks + A.in_index[t];
      } else {
        // implicit: root i, chunk of its depth-1 driver range
        uint32_t a = 0, b = nroots;  // last i with chunk_off[i] <= t
#pragma unroll 1
        while (b - a > 1) {
          const uint32_t mid = (a + b) >> 1;
          if (A.chunk_off[mid] <= t) a = mid; else b = mid;
        }
        chunk = t - A.chunk_off[a];
        q = A.root_q[a];
        root = A.roots[a];
      }
      t++;
    } else {
      // input exhausted: take a ticket and wait for its record while others work
      uint32_t slot = kInvalid;
      if (lane == 0) {
        const uint32_t mine = atomicAdd(&A.ctr[1 * kCtrStride + 1], 1u);
        atomicSub(&A.ctr[2 * kCtrStride], 1u);
        const unsigned long long t_idle = global_ns();
        unsigned long long t_reserved = 0;  // when the record of this ticket was first seen reserved
        uint32_t sleep_ns = 32;
        volatile uint32_t* word = A.out_ready + (mine & (A.out_cap - 1));
        const uint32_t published = 2 * (mine >> (31 - __clz(A.out_cap))) + 1;
#pragma unroll 1
        for (;;) {
          if (*word == published) {
            slot = mine;
            break;
          }
          // finished when nobody works and every record is taken
          if (*(volatile uint32_t*)&A.ctr[2 * kCtrStride] == 0 || *(volatile uint32_t*)&A.ctr[3 * kCtrStride]) break;
          const unsigned long long now = global_ns();
          const uint32_t tail = *(volatile uint32_t*)&A.ctr[1 * kCtrStride];
          if (int32_t(tail - mine) > 0) {
            if (!t_reserved) {
              t_reserved = now;
            } else if (now - t_reserved > A.ready_wait_ns) {
              atomicOr(&A.ctr[3 * kCtrStride], kErrTimeout);
              break;
            }
          } else if (now - t_idle >= A.idle_wait_ns) {
            // leave: this ticket's record, if it comes, waits for the next pass,
            // so no slot from here on may be used again
            atomicCAS(&A.ctr[5 * kCtrStride], 0u, max(tail + A.out_cap / 2, 1u));
            break;
          }
          __nanosleep(sleep_ns);
          if (sleep_ns < 1024) sleep_ns <<= 1;
        }
      }
      slot = __shfl_sync(kFull, slot, 0);
      if (slot != kInvalid) {
        __threadfence();
        if (lane == 0) n_pops++;
        rec = A.out_tasks + (slot & (A.out_cap - 1));
        ready = A.out_ready + (slot & (A.out_cap - 1));
        free_word = 2 * (slot >> (31 - __clz(A.out_cap))) + 2;
      }
    }
    if (rec) {
      // the header is read by lane 0 and broadcast, like every other value that
      // steers the warp's control flow; records popped in this launch were
      // written by another SM, so they are read through L2 (ld.cg)
      if (lane == 0) {
        q = __ldcg(&rec->q);
        d = __ldcg(&rec->d);
        lo = __ldcg(&rec->lo);
        hi = __ldcg(&rec->hi);
      }
      q = __shfl_sync(kFull, q, 0);
      d = __shfl_sync(kFull, d, 0);
      lo = __shfl_sync(kFull, lo, 0);
      hi = __shfl_sync(kFull, hi, 0);
      if (lane < d) f = __ldcg(&rec->f[lane]);
      if (ready) {  // the record is read: its slot is free again
        __threadfence();
        __syncwarp();
        if (lane == 0) *(volatile uint32_t*)ready = free_word;
      }
    }
    // ---- its query
    if (q != cur_q || q == kInvalid) {
      if (cur_q != kInvalid) {
        publish();
        const unsigned long long h = warp_sum(my_hash);
        if (lane == 0 && h) atomicAdd(&A.res[cur_q].hash, h);
        if (lane < ws.plan.n && lc) {
          atomicAdd(&A.res[cur_q].levels[lane], lc);
          if (lane + 1 == ws.plan.n) atomicAdd(&A.res[cur_q].count, lc);
        }
        my_hash = lc = 0;
      }
      if (q == kInvalid) break;
      __syncwarp();
      const uint32_t* src = reinterpret_cast<const uint32_t*>(A.plans + q);
      uint32_t* dst = reinterpret_cast<uint32_t*>(&ws.plan);
#pragma unroll 1
      for (uint32_t i = lane; i < sizeof(Plan) / 4; i += 32) dst[i] = src[i];
      __syncwarp();
      cur_q = q;
    }
    const uint32_t n = ws.plan.n;
    if (root != kInvalid) {
      if (lane == 0) {
        f = root;
        lc += chunk == 0;  // the root itself, once
      }
      if (n > 1) {
        row_segment<kRows>(g, root, ws.plan.lab[1], W1, lo, hi);
        lo += chunk * A.split;
        hi = min(lo + A.split, hi);
      }
    }
    if (lane == 0) n_tasks++;
    if (d == n) {  // a complete embedding (single-vertex queries)
      if (lane == 0) {
        const uint32_t xo = __ldg(g.old_of_new + f);
        my_hash += fmix64(A.seed + fmix64((uint64_t(ws.plan.qv[0]) << 32) | xo));
        bytes += 4;
        if (A.emit) {
          const unsigned long long row = atomicAdd(A.emit_ctr, 1ull);
          if (row < A.emit_cap) A.emit[row] = xo;
        }
      }
      continue;
    }
    // ---- run it
    const uint32_t t_start = uint32_t(clock());
    __syncwarp();
    if (lane < d) {
      cand[lane * kBuf] = f;
      par[lane * kBuf] = 0;
    }
    cnt = lane < d ? 1u : 0u;
    it = lane + 1 < d ? 1u : 0u;
    off = 0;
    s_valid = false;
    __syncwarp();
    uint32_t lv = d, windows = kCheckWindows, used = 0;
#pragma unroll 1
    for (;;) {
      if (windows >= kCheckWindows) {
        // at the start and every kCheckWindows windows: the query's work limit,
        // the pass's error word (the call will fail anyway), and waiting warps
        windows = 0;
        if (__any_sync(kFull, bytes >= (1u << 30))) {
          const unsigned long long b = warp_sum((unsigned long long)bytes);
          if (lane == 0) atomicAdd(A.algo_bytes, b);
          bytes = 0;
        }
        int stop = 0;
        if (A.work_cap) {
          publish();
          if (lane == 0) stop = *(volatile unsigned int*)&A.res[cur_q].aborted != 0;
        }
        if (lane == 0) stop |= *(volatile uint32_t*)&A.ctr[3 * kCtrStride] != 0;
        if (__shfl_sync(kFull, stop, 0)) break;
        // (never before the first window: a task handed on untouched would go round)
        const uint32_t hungry = used ? waiting_warps(t_start) : 0u;
        if (hungry) {
          // the entries of the leaf's ranges are handed off only when those are long
          const uint32_t last = (lv + 1 == n && used >= kFillWindows) ? n - 1 : n - 2;  // plus one
          if (last >= d) donate(d, min(lv, last - 1), hungry, lo, hi);
        }
      }
      if (__shfl_sync(kFull, it, lv - 1) >= __shfl_sync(kFull, cnt, lv - 1)) {
        if (lv == d) break;
        lv--;
        continue;
      }
      used = fill(lv, lv == d ? lo : kInvalid, hi);
      windows += used + 1;
      if (lv + 1 < n && __shfl_sync(kFull, cnt, lv) > 0) lv++;
    }
  }
  const unsigned long long all_bytes = warp_sum((unsigned long long)bytes);
  if (lane == 0) {
    atomicAdd(A.algo_bytes, all_bytes);
    atomicAdd(&A.ev[0], (unsigned long long)n_tasks);
    atomicAdd(&A.ev[1], (unsigned long long)n_pops);
    atomicAdd(&A.ev[2], (unsigned long long)n_handoffs);
    atomicAdd(&A.ev[3], (unsigned long long)n_recs);
    atomicAdd(&A.ev[4], (unsigned long long)n_examine);
  }
}

}  // namespace
}  // namespace fsig
