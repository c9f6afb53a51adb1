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
// earlier vertices are found by walking its parents.  LevelState is a depth's
// cursor.
//
// Filling the buffer of depth i from depth i-1's entries: each lane takes one
// entry, finds the label-l(i) segments of its backward neighbours' rows
// (bounds into shared memory) and picks the shortest as its driver.  The
// drivers of all entries, end to end, are then examined 32 candidates at a
// time, one per lane, whichever entry they belong to: the lanes' owners come
// from the bits where a driver begins in this window.  A candidate passes
// when its bit in depth i's candidate bitmap is set, it differs from the
// entry's earlier vertices of the same label (adjacent ones differ anyway),
// and it lies in each of the entry's other backward segments.  The store's
// membership filter settles most of these by one load (common.cuh); candidates
// that pass every filter are appended to depth i's buffer and, where a filter
// is not exact, searched for once the buffer is full, so that the searches (two
// per-lane binary searches in lockstep) run on all lanes; those found stay.
// A buffer with enough entries is extended in turn, and later the fill goes on
// where it stopped.  At the leaf the passing candidates are counted and hashed.
// A leaf that hangs on an earlier vertex than its parent in the order has the
// same range for each entry below that vertex, one after another in the buffer:
// its candidates and their hashes are then found once, and the pairs of a
// candidate and an entry take the lanes (joint, in fill).
//
// What bounds it: instructions and L2 latency (the working set is L2
// resident), so the aim is full lanes and few instructions a window.  A warp per
// entry ran 11 of 32 lanes at the leaf of the 320k-vertex workloads (one range of
// 11-12 neighbours after another) and paid the set-up of a range, some 300
// instructions, for each: 200 eight-vertex queries there took 115 ms of kernel,
// 512 queries of 4-32 vertices 69, 512 queries of 12-32 vertices on 2^26 edges 305,
// house counting on 700 vertices 104.  Now 19.8, 15.2, 126 and 32 ms, 243
// instructions a window at 69 % of the issue rate on 2^26 edges.  (Buffers of one
// pool per warp leave room for 4 blocks an SM also for 32-vertex queries; 32
// entries for each depth, for 3.  Loading a window ahead gains nothing.)
//
// Work stealing: a warp that runs out of input takes a ticket, one atomicAdd
// on the queue's head, and waits for the record of that number, polling the
// record's own ready word.  A busy warp checks every 32 windows whether
// more tickets than records are out; if so it hands its shallowest pending depth
// (buffered candidates and the remaining driver range) to the queue as task
// records and carries on with the rest.  One counter holds the warps at work
// plus the records not taken yet; the pass is over when it reaches zero.
// (With a compare-and-swap on the head by every idle warp for every record, up
// to 2048 warps retrying on one word served a record in 0.4-1.0 us whatever the
// work in it, which bounded every batch but the largest: one 4-vertex query on a
// 10k-vertex graph 3.8 ms, 0.37 with tickets.)  Waiting is bounded: a warp that
// waits too long leaves, which never loses work -- its record, if it is written,
// is the next pass's input.
// Every value that steers a warp's control flow is read by lane 0 and
// broadcast.
#pragma once

#include "queue.cuh"

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
  uint32_t* ctr;  // counters, kCtrStride apart: [0] input grab, [1] queue tail (records reserved) and,
                  // in the next word, tickets taken, [2] warps at work + records not taken yet and,
                  // in the next word, records whose holders left (not counted in the former),
                  // [3] error bits, [4] fault injection's one-shot, [5] once a waiting warp has left,
                  // the record number from which on no more are reserved
  uint32_t room;  // queue_room of the launch's warps
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
  // for tests: number of the pass's first record and ticket; whether the warp
  // that takes that ticket leaves at once
  uint32_t first_record, first_leaves;
};

constexpr uint32_t kErrTimeout = 1u;
constexpr uint32_t kCtrStride = 32;        // one 128-byte line per counter
// Records (queue.cuh) are reserved only while warps wait, so at most (warps) x
// (records of one hand-off) numbers lie between the tickets and the tail, fewer
// than the ring's 2^20 slots: a reserved slot's previous record always has a
// ticket holder, or one that left, whose slot does not come round (queue_room).

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr uint32_t kBuf = 32;        // entries of a depth's buffer
// Depth n-2, whose entries the leaf loop takes 32 at a time, may keep up to
// kLastBuf when it has no second segment itself: a fill that ends
// at 32 entries has set up 32 parents and used three or four of them where each
// has ten children (200 eight-vertex queries on 320k vertices 25.4 -> 22.9 ms
// with 128, 23.4 with 64, 22.3 with 192).  It does not where the leaf's ranges are
// long (from kLongLeaf / 8 windows an entry on, in its last fill), since fewer,
// longer buffers then only keep work from the warps that wait: 37 queries on
// 2^26 edges 11.6 ms, 12.5 with 128 always; nor while warps wait.
constexpr uint32_t kLastBuf = 128;
constexpr uint32_t kLongLeaf = 6;
static_assert(kHandOff == 32 + kLastBuf, "a hand-off is a range's pieces and a buffer");
constexpr uint32_t kScratch = 384;   // words for the segments and earlier vertices of the entries being extended
// Candidate windows one fill examines before it returns, so that the periodic
// checks and hand-offs come in time on long driver ranges.
// (64: 139 ms for 512 queries on 2^26 edges, 96: 136; 128 and 256 are slower for
// batches of a few queries.)
constexpr uint32_t kFillWindows = 96;
// Driver entries of a group up to which its entries' shared ranges are taken
// together: four fills' worth, since such a group is not interrupted (512 queries
// on 2^26 edges 131 ms with 3072, 129 with 6144, 126 with this and with eight times
// it; 200 eight-vertex queries on 320k vertices 19.9 ms with each, 21.0 with 1536).
constexpr uint32_t kJointEntries = 4 * 32 * kFillWindows;
// Windows between two checks of the work limit and of the waiting warps.
constexpr uint32_t kCheckWindows = 32;

constexpr uint32_t kPool = 384;      // entries of all buffers of a warp (see below)

// What a fill needs to know of its depth, in two 16-byte loads; made from the
// query's Plan when a warp turns to it.  (Read field by field, with the levels'
// cursors in registers of lanes, 200 eight-vertex queries on 320k vertices took
// 26.6 ms instead of 25.4, 512 queries on 2^26 edges 136 instead of 132.)
struct alignas(16) LevelPlan {
  const uint32_t* bm;  // candidate bitmap
  uint32_t bwd;        // earlier depths adjacent to this one
  uint32_t inj;        // earlier depths of the same label that are not
  uint32_t bmbase;     // first id of the bitmap
  uint32_t dense;      // segments from this length on have an exact filter (in filter words)
  int32_t lab;
  uint8_t nb, n4;      // segments; earlier vertices to compare, in fours
  uint8_t stride;      // entries extended at a time
  uint8_t qv;          // query vertex
};
struct alignas(16) LevelState {
  uint32_t cnt, it, off;  // entries, the first one not wholly extended, how much of its driver range is examined
  uint32_t sp;            // where the buffer starts in the pool
};

// Per warp.  The depths' buffers lie one after another in the pool, each as
// long as it is filled; a fill takes at most kBuf entries (kLastBuf at depth n-2)
// and leaves one for each depth below it.  (A fixed 32 entries for each of 31
// depths would allow 3 blocks an SM instead of 4.)
struct WarpSmem {
  LevelPlan plan[kMaxQ];
  LevelState lev[kMaxQ];
  uint2 owner[kBuf];                // entries with a driver: its place relative to the window index, the entry
  unsigned long long sown[kBuf];    // leaf: partial hash of each entry being extended
  unsigned long long sbase[kBuf];   // partial hashes of depth n-3's buffer
  // per entry being extended: its earlier vertices of the same label, four in a
  // word; then its segments (start, length, as filter words)
  alignas(16) uint2 scratch[kScratch / 2];
  uint32_t cand[kPool];             // mapped vertex
  uint8_t par[kPool];               // its parent's place in the previous depth's buffer
  // What only fills, tasks and hand-offs touch is kept here for the registers.
  unsigned long long found[kMaxQ];  // partial embeddings of each length, of the current query, not yet published
  unsigned long long loads;         // 4-byte loads of the windows, filters and searches
  uint32_t ev[5];                   // events: tasks, records popped, hand-offs, records written, windows
  uint32_t pend;                    // driver entries examined, not yet published to res.work
  uint32_t task_lo, task_hi;        // driver range of the task at its first depth
  uint32_t t, t_last;               // input tasks in hand: [t, t_last)
  uint32_t query, n;
  uint32_t room, pad;               // longest buffer of depth n-2
};
static_assert(sizeof(WarpSmem) % 16 == 0, "the next warp's part is aligned");

// 1 << s, 0 for s >= 32
__device__ __forceinline__ uint32_t bit_or_zero(uint32_t s) {
  uint32_t r;
  asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(1u), "r"(s));
  return r;
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

// Whether x lies in both sorted segments a[lo0, lo0 + n0) and a[lo1, lo1 + n1)
// (in the first alone without `two`): two binary searches in lockstep, so that a step
// has two independent loads in flight.
__device__ __forceinline__ bool in_segments(const uint32_t* __restrict__ a, uint32_t lo0, uint32_t n0, uint32_t lo1,
                                            uint32_t n1, bool two, uint32_t x, uint32_t& loads) {
  if (!two) n1 = 1;
  if (n0 == 0 || n1 == 0) return false;
#pragma unroll 1
  while (n0 > 1 || n1 > 1) {
    const uint32_t h0 = n0 >> 1, h1 = n1 >> 1;
    const uint32_t y0 = __ldg(a + lo0 + h0), y1 = __ldg(a + lo1 + h1);
    if (y0 <= x) lo0 += h0;
    if (y1 <= x) lo1 += h1;
    n0 -= h0;
    n1 -= h1;
    loads += 2;
  }
  loads += 2;
  return __ldg(a + lo0) == x && (!two || __ldg(a + lo1) == x);
}

// kRows: the graph store has no segment table (GraphView::lseg is null) and
// no caller-id copy of the adjacency (adj_old); segments are found in the
// rows and a leaf's caller id is looked up once it survives.
template <bool kRows>
__global__ void __launch_bounds__(kEnumWarps * 32, kEnumMinBlocks) enumerate_kernel(EnumArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WarpSmem& ws = reinterpret_cast<WarpSmem*>(smem_raw)[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31;
  const GraphView& g = A.g;
  const uint64_t W1 = uint64_t(g.L) + 1;
  const uint32_t nroots = A.in_tasks ? 0u : *A.nroots_ptr;
  const uint32_t T_in = A.in_tasks ? A.in_count : min(A.chunk_off[nroots], A.t_end);

  unsigned long long my_hash = 0;
  bool s_valid = false;  // sbase holds depth n-3's current buffer
  ws.found[lane] = 0;
  if (lane < 5) ws.ev[lane] = 0;
  if (lane == 0) {
    ws.loads = 0;
    ws.pend = 0;
    ws.t = ws.t_last = 0;
    ws.query = kInvalid;
  }
  __syncwarp();

  // Publishes the driver entries this warp examined for the current query.
  // The total a query examines does not depend on how its work was split
  // (every driver entry counts once), so whether it exceeds the limit does not
  // either.
  auto publish = [&]() {
    if (lane == 0 && A.work_cap && ws.pend) {
      const unsigned long long tot = atomicAdd(&A.res[ws.query].work, (unsigned long long)ws.pend) + ws.pend;
      ws.pend = 0;
      if (tot > A.work_cap) atomicExch(&A.res[ws.query].aborted, 1u);
    }
  };

  // Prefix of the entry in slot `slot` of depth p's buffer: lane j <= p gets f_j.
  auto prefix = [&](uint32_t p, uint32_t slot) {
    uint32_t v = 0;
#pragma unroll 1
    for (uint32_t k = p;; k--) {
      const uint32_t at = ws.lev[k].sp + slot;
      const uint32_t x = ws.cand[at];
      if (lane == k) v = x;
      if (k == 0) break;
      slot = ws.par[at];
    }
    return v;
  };

  // Hands the shallowest depth from d0 - 1 to last that still has entries to
  // extend to the queue -- each entry a record, the rest of a partly extended
  // entry's driver range in pieces for the waiting warps -- and marks that depth
  // done here.  [lo_set, hi_set): the task's own driver range at depth d0, if
  // it has one.  Returns false when no records may be reserved.
  auto donate = [&](uint32_t d0, uint32_t last, uint32_t hungry, uint32_t lo_set, uint32_t hi_set) -> bool {
    const LevelState mine = ws.lev[lane];
    const uint32_t has = __ballot_sync(kFull, lane + 1 >= d0 && lane <= last && mine.it < mine.cnt);
    if (!has) return true;
    const uint32_t l = __ffs(has) - 1;
    const uint32_t c_l = ws.lev[l].cnt, i_l = ws.lev[l].it, o_l = ws.lev[l].off;
    // the current entry's driver range, when it is partly examined or given
    const bool given = l + 1 == d0 && lo_set != kInvalid;
    const bool part = given || o_l > 0;
    uint32_t lo = lo_set, hi = hi_set, fp = 0;
    if (part) {
      fp = prefix(l, i_l);
      if (!given) {  // the choice a fill makes: the shortest segment, the latest depth on ties
        uint32_t a = 0, b = 0, len = kInvalid;
        if ((ws.plan[l + 1].bwd >> lane) & 1u) {
          row_segment<kRows>(g, fp, ws.plan[l + 1].lab, W1, a, b);
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
    const uint32_t hand = max(32u, piece_count(rest, takers));
    const uint32_t pieces = piece_count(rest, hand);
    const uint32_t first = part ? i_l + 1 : i_l;
    const uint32_t total = pieces + (c_l - first);
    uint32_t base = 0;  // any number, 2^32 - 1 too
    bool full = false;
    if (lane == 0) {
      const uint32_t limit = *(volatile uint32_t*)&A.ctr[5 * kCtrStride];
      full = limit && queue_after(*(volatile uint32_t*)&A.ctr[1 * kCtrStride] + total, limit);
      if (!full) {
        base = atomicAdd(&A.ctr[1 * kCtrStride], total);
        atomicAdd(&A.ctr[2 * kCtrStride], total);
      }
    }
    if (__any_sync(kFull, full)) return false;
    base = __shfl_sync(kFull, base, 0);
    // the slots' previous records are read by now, or about to be (see above); a
    // record that is not must not be written over while its holder may read it
    {
      const unsigned long long t0 = global_ns();
      bool late = false;
#pragma unroll 1
      for (uint32_t k = lane; k < total && !late; k += 32) {
        while (!late && !ready_writable(*(volatile uint32_t*)&A.out_ready[queue_slot(base + k)], base + k))
          late = global_ns() - t0 > A.ready_wait_ns;
      }
      if (late) atomicOr(&A.ctr[3 * kCtrStride], kErrTimeout);
      if (__any_sync(kFull, late)) return false;
    }
    uint32_t slot = base;
#pragma unroll 1
    for (uint32_t k = 0; k < pieces; k++) {
      TaskRec* r = A.out_tasks + queue_slot(slot++);
      if (lane <= l) r->f[lane] = fp;
      if (lane == 0) { r->q = ws.query; r->d = l + 1; r->lo = lo + k * hand; r->hi = piece_end(lo + k * hand, hand, hi); }
    }
#pragma unroll 1
    for (uint32_t k = first; k < c_l; k++) {
      TaskRec* r = A.out_tasks + queue_slot(slot++);
      const uint32_t fk = prefix(l, k);
      if (lane <= l) r->f[lane] = fk;
      if (lane == 0) { r->q = ws.query; r->d = l + 1; r->lo = kInvalid; r->hi = kInvalid; }
    }
    __syncwarp();
    if (lane == 0) {
      ws.lev[l].it = c_l;
      ws.lev[l].off = 0;
    }
    __threadfence();
    __syncwarp();
    int hold = 0;  // test hook: keep the pass's first handed-off record unpublished
    if (A.unpublished && lane == 0) hold = atomicCAS(&A.ctr[4 * kCtrStride], 0u, 1u) == 0u;
    hold = __shfl_sync(kFull, hold, 0);
    uint32_t left = 0;  // records whose holders left
#pragma unroll 1
    for (uint32_t k = lane; k < total; k += 32)
      if (!(hold && k == 0)) left += atomicOr(&A.out_ready[queue_slot(base + k)], 1u) >> 31;
    left = __reduce_add_sync(kFull, left);
    if (lane == 0) {
      if (left) {  // the next pass's: nobody here has to wait for them
        atomicAdd(&A.ctr[2 * kCtrStride + 1], left);
        atomicSub(&A.ctr[2 * kCtrStride], left);
      }
      ws.ev[2]++;
      ws.ev[3] += total;
    }
    return true;
  };

  // How many warps wait for records that nobody has reserved (tickets minus
  // records), 0 while this task is younger than its budget.  Decided by lane 0
  // alone and broadcast.
  auto waiting_warps = [&](uint32_t t_start) -> uint32_t {
    uint32_t w = 0;
    if (lane == 0) {
      uint32_t tail, tickets;
      asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(tail), "=r"(tickets) : "l"(A.ctr + kCtrStride));
      if (queue_after(tickets, tail) && (long long)(uint32_t(clock()) - t_start) > A.budget) w = tickets - tail;
    }
    return __shfl_sync(kFull, w, 0);
  };

  // Writes the embeddings completed by one leaf window: lanes in m hold a
  // leaf's caller id in xo and its entry's place in depth n-2's buffer.
  auto emit_rows = [&](uint32_t m, uint32_t n, uint32_t xo, uint32_t slot) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(A.emit_ctr, (unsigned long long)__popc(m));
    base = __shfl_sync(kFull, base, 0);
    const unsigned long long row = base + __popc(m & lanemask_lt());
    const bool mine = ((m >> lane) & 1u) && row < A.emit_cap;
    uint32_t* dst = A.emit + row * n;
    if (mine) dst[ws.plan[n - 1].qv] = xo;
#pragma unroll 1
    for (uint32_t k = n - 1; k-- > 0;) {
      const uint32_t at = ws.lev[k].sp + slot;
      if (mine) {
        dst[ws.plan[k].qv] = __ldg(g.old_of_new + ws.cand[at]);
        slot = ws.par[at];
      }
    }
  };

  // Extends depth lv - 1's entries to depth lv (see the top of this file): into
  // depth lv's buffer until it is about full, or, at the leaf, into counts and
  // hashes.  [lo_set, hi_set), unless kInvalid, is the driver range of the one
  // entry there is.  Returns the windows examined; the cursors of depths lv - 1
  // and lv say where it stopped.
  uint32_t made = 0;  // entries the last fill appended
  auto fill = [&](uint32_t lv, uint32_t lo_set, uint32_t hi_set) -> uint32_t {
    const uint32_t n = ws.n, p = lv - 1;
    const bool leaf = lv + 1 == n;
    const LevelPlan lp = ws.plan[lv];
    const LevelState from = ws.lev[p];
    const uint32_t bwd = lp.bwd, inj = lp.inj, nb = lp.nb, n4 = lp.n4, stride = lp.stride;
    const uint32_t bmbase = lp.bmbase, dense = lp.dense;
    const int32_t lab = lp.lab;
    const uint32_t* __restrict__ bm = lp.bm;
    uint4* const other = reinterpret_cast<uint4*>(ws.scratch);  // [n4][stride], padded with kInvalid
    uint2* const segs = ws.scratch + 2 * n4 * stride;           // [nb][stride]
    // whether x is none of entry c's earlier vertices
    auto fresh = [&](uint32_t x, uint32_t c) {
      bool yes = true;
#pragma unroll 1
      for (uint32_t k = 0; k < n4; k++) {
        const uint4 o = other[k * stride + c];
        yes = yes && x != o.x && x != o.y && x != o.z && x != o.w;
      }
      return yes;
    };
    const uint32_t fs = g.filt ? g.fshift : 0;  // segments are kept in units of their filter's words
    const uint32_t cntp = from.cnt, spp = from.sp, spl = spp + cntp;  // spl: depth lv's buffer
    const uint32_t longest = lv + 2 == n && nb == 1 ? ws.room : kBuf;
    const uint32_t room = min(longest, kPool - spl - (n - 2 - min(lv, n - 2)));
    // Entries that end a fill.  With further segments to search the room left
    // decides how many lanes search, so half the buffer is enough.
    const uint32_t enough = nb > 1 || room < 16 ? (room + 1) / 2 : room - 8;
    uint32_t itp = from.it, offp = from.off;
    uint32_t have = 0, sure = 0;  // entries appended; of them, searched for in every segment
    uint32_t used = 0, seen = 0, hits = 0, loads = 0;  // loads: 4-byte loads of the filters and searches
    bool stop = false;
    if (leaf && !s_valid && lv >= 2) {  // partial hashes of depth n-3's entries
      unsigned long long sum = 0;
      uint32_t slot = min(lane, ws.lev[lv - 2].cnt - 1);
#pragma unroll 1
      for (uint32_t k = lv - 1; k-- > 0;) {
        const uint32_t at = ws.lev[k].sp + slot;
        sum += fmix64((uint64_t(ws.plan[k].qv) << 32) | __ldg(g.old_of_new + ws.cand[at]));
        slot = ws.par[at];
      }
      ws.sbase[lane] = sum;
      s_valid = true;
      __syncwarp();
    }
    while (itp < cntp && !stop) {
      // the group: lane c takes entry itp + c (lanes past the group repeat its last one)
      uint32_t group = min(cntp - itp, stride);
      const bool mine = lane < group;
      const uint32_t own = spp + itp + min(lane, group - 1);
      uint32_t dlo = 0, len = kInvalid, drv = 0, anc = 0;  // anc: where the driver's vertex lies in the pool
      {
        uint32_t at = own, need = bwd | inj, wb = 0, wi = 0;
        if (mine) {
#pragma unroll 1
          for (uint32_t k = 0; k < n4; k++) other[k * stride + lane] = make_uint4(kInvalid, kInvalid, kInvalid, kInvalid);
        }
#pragma unroll 1
        for (uint32_t k = p;; k--) {
          const uint32_t v = ws.cand[at];
          if ((bwd >> k) & 1u) {
            uint32_t a, b;
            row_segment<kRows>(g, v, lab, W1, a, b);
            if (mine) segs[wb * stride + lane] = make_uint2(a << fs, (b - a) << fs);
            if (b - a < len) {
              len = b - a;
              dlo = a;
              drv = wb;
              anc = at;
            }
            wb++;
          } else if ((inj >> k) & 1u) {
            if (mine) reinterpret_cast<uint32_t*>(&other[(wi >> 2) * stride + lane])[wi & 3] = v;
            wi++;
          }
          need &= ~(1u << k);
          if (!need) break;
          at = ws.lev[k - 1].sp + ws.par[at];
        }
        if (mine && drv) segs[drv * stride + lane] = segs[lane];  // the others: places 1 .. nb - 1
        if (lo_set != kInvalid) {
          dlo = lo_set;
          len = hi_set - lo_set;
        }
        if (lane == 0) {
          dlo += offp;
          len -= offp;
        }
        if (!mine) len = 0;
      }
      if (leaf) {
        unsigned long long sum = fmix64((uint64_t(ws.plan[p].qv) << 32) | __ldg(g.old_of_new + ws.cand[own]));
        if (p > 0) sum += ws.sbase[ws.par[own]];
        ws.sown[lane] = sum;
      }
      if (__any_sync(kFull, len >= (1u << 27))) {  // the group's total has to fit 32 bits
        group = 1;
        if (lane) len = 0;
      }
      // Entries next to one another whose driver belongs to the same vertex: its
      // candidates are found once for all of them (joint, below).  This pays from
      // two entries a range on: then the pair loop has no loads from memory and
      // one hash instead of two.  88 % of the entries of 512 queries of 4-32
      // vertices on 320k vertices have such a leaf, 27 to a range: 19.5 -> 15.3
      // ms; of 200 eight-vertex queries 80 %, 14 to a range: 23.0 -> 19.9 ms.  (With
      // leaves of two segments as well it cost spills and 3 % everywhere, for no
      // gain on any of these.)
      uint32_t joint = 0, run = 0;  // joint: driver entries of the group, before they are shared
      if (leaf && nb == 1 && !(bwd >> p) && n4 <= 2 && !A.emit && !offp && lo_set == kInvalid) {
        const uint32_t before = __shfl_up_sync(kFull, anc, 1);
        const uint32_t firsts = __ballot_sync(kFull, mine && (lane == 0 || anc != before)) | bit_or_zero(group);
        const uint32_t all = __reduce_add_sync(kFull, len);
        if (2 * __popc(firsts) <= group + 2 && all <= kJointEntries) {
          joint = all;
          const uint32_t later = firsts & ~lanemask_le();
          run = (later ? __ffs(later) - 1 : 32u) - lane;
          if (!((firsts >> lane) & 1u)) len = 0;
        }
      }
      uint32_t incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane >= uint32_t(o)) incl += y;
      }
      const uint32_t T = __shfl_sync(kFull, incl, 31);
      const uint32_t start = len ? incl - len : kInvalid;
      {
        const uint32_t rank = __popc(__ballot_sync(kFull, len != 0) & lanemask_lt());
        if (len) ws.owner[rank] = make_uint2(dlo - start, lane | run << 8);
      }
      __syncwarp();
      const bool filtered = nb > 1 && g.filt;
      uint32_t pos = 0, begun = kInvalid;  // begun: drivers that start before pos, minus one
      if (joint) {
        uint4* const cands = reinterpret_cast<uint4*>(ws.scratch) + 2 * kBuf;  // candidate, its hash, first entry less first pair
        const uint64_t tq = uint64_t(lp.qv) << 32;
#pragma unroll 1
        while (pos < T) {
          const uint32_t heads = __reduce_or_sync(kFull, bit_or_zero(start - pos));
          const uint2 o = ws.owner[begun + __popc(heads & lanemask_le())];
          const uint32_t e = pos + lane, at = o.x + min(e, T - 1);
          const uint32_t x = __ldg(g.adj + at);
          const uint32_t xo = kRows ? __ldg(g.old_of_new + x) : __ldg(g.adj_old + at);
          const uint32_t bit = x - bmbase;
          const bool pred = e < T && ((__ldg(bm + (bit >> 5)) >> (bit & 31)) & 1u);
          const uint32_t pairs = pred ? o.y >> 8 : 0u;
          uint32_t upto = pairs;
#pragma unroll
          for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, upto, d);
            if (lane >= uint32_t(d)) upto += y;
          }
          const uint32_t P = __shfl_sync(kFull, upto, 31);
          const uint32_t first = pred ? upto - pairs : kInvalid;
          const uint32_t rank = __popc(__ballot_sync(kFull, pred) & lanemask_lt());
          if (pred) {
            const uint64_t h = fmix64(tq | xo);
            cands[rank] = make_uint4(x, uint32_t(h), uint32_t(h >> 32), (o.y & 255u) - first);
          }
          __syncwarp();
          uint32_t k = kInvalid;
#pragma unroll 1
          for (uint32_t i = 0; i < P; i += 32) {
            const uint32_t hd = __reduce_or_sync(kFull, bit_or_zero(first - i));
            const uint4 y = cands[k + __popc(hd & lanemask_le())];
            const uint32_t c = y.w + min(i + lane, P - 1);
            bool yes = i + lane < P;
            if (n4) yes = yes && fresh(y.x, c);
            const uint64_t h = fmix64(A.seed + ws.sown[c] + (uint64_t(y.z) << 32 | y.y));
            my_hash += yes ? h : 0;
            hits += yes;
            k += __popc(hd);
            used++;
          }
          __syncwarp();
          begun += __popc(heads);
          pos += 32;
          used++;
        }
        stop = used >= kFillWindows;
        if (lane == 0) loads -= 3 * (joint - T);  // counted with the entries seen
        pos = T;
        seen += joint;
      } else if (leaf && !A.emit && (nb == 1 || (nb == 2 && filtered))) {
        // the common leaves: at most one segment to look up, all lanes alike
        const uint64_t tq = uint64_t(lp.qv) << 32;
#pragma unroll 1
        while (pos < T && !stop) {
          const uint32_t heads = __reduce_or_sync(kFull, bit_or_zero(start - pos));
          const uint2 o = ws.owner[begun + __popc(heads & lanemask_le())];
          const uint32_t e = pos + lane, at = o.x + min(e, T - 1);
          const uint32_t x = __ldg(g.adj + at);
          const uint32_t xo = kRows ? __ldg(g.old_of_new + x) : __ldg(g.adj_old + at);
          const uint32_t bit = x - bmbase;
          const uint32_t word = __ldg(bm + (bit >> 5));
          bool pred = e < T && ((word >> (bit & 31)) & 1u);
          if (nb == 2) {
            const uint2 a = segs[stride + o.y];
            const bool da = a.y >= dense;
            const uint32_t w = __ldg(g.filt + (a.x + filter_word(da, bit, filter_hash(x), a.y)));
            pred = pred && (~w & filter_mask(da, bit, filter_bits(x))) == 0;
            if (__any_sync(kFull, pred && !da)) {
              if (pred && !da) pred = in_segments(g.adj, a.x >> fs, a.y >> fs, a.x >> fs, 1, false, x, loads);
              __syncwarp();
            }
          }
          if (n4) pred = pred && fresh(x, o.y);
          const uint64_t h = fmix64(A.seed + ws.sown[o.y] + fmix64(tq | xo));
          my_hash += pred ? h : 0;
          hits += pred;
          begun += __popc(heads);
          pos += 32;
          stop = ++used >= kFillWindows;
        }
        pos = min(pos, T);
        seen += pos;
      }
#pragma unroll 1
      while (pos < T && !stop) {
        const uint32_t heads = __reduce_or_sync(kFull, bit_or_zero(start - pos));
        const uint2 o = ws.owner[begun + __popc(heads & lanemask_le())];
        const uint32_t e = pos + lane, at = o.x + min(e, T - 1);
        uint32_t x = __ldg(g.adj + at), c = o.y;
        const uint32_t bit = x - bmbase;
        const uint32_t word = __ldg(bm + (bit >> 5));
        bool pred = e < T;
        const uint32_t hash = filter_hash(x), bits = filter_bits(x);
        if (filtered) {  // the first of the other segments' filters, beside the candidate bit
          const uint2 a = segs[stride + c];
          const bool da = a.y >= dense;
          const uint32_t w = __ldg(g.filt + (a.x + filter_word(da, bit, hash, a.y)));
          pred = pred && (~w & filter_mask(da, bit, bits)) == 0;
        }
        pred = pred && ((word >> (bit & 31)) & 1u);
        uint32_t step = min(32u, T - pos);
        used++;
        const bool final = used >= kFillWindows;
        if (__any_sync(kFull, pred)) {
          if (n4) pred = pred && fresh(x, c);
          if (filtered) {  // the other filters, two at a time
#pragma unroll 1
            for (uint32_t k = 2; k < nb && __any_sync(kFull, pred); k += 2) {
              const uint2 a = segs[k * stride + c], b = segs[min(k + 1, nb - 1) * stride + c];
              const bool da = a.y >= dense, db = b.y >= dense;
              uint32_t wa = 0, wb = 0;
              if (pred) {
                wa = __ldg(g.filt + (a.x + filter_word(da, bit, hash, a.y)));
                wb = __ldg(g.filt + (b.x + filter_word(db, bit, hash, b.y)));
              }
              loads++;
              pred = ((~wa & filter_mask(da, bit, bits)) | (~wb & filter_mask(db, bit, bits))) == 0;
            }
          }
          if (!leaf) {
            uint32_t m = __ballot_sync(kFull, pred);
            const uint32_t rank = have + __popc(m & lanemask_lt());
            if (have + __popc(m) > room) {  // take what fits; go on from the first one that does not
              step = __ffs(__ballot_sync(kFull, pred && rank == room)) - 1;
              m &= (1u << step) - 1;
            }
            if ((m >> lane) & 1u) {
              ws.cand[spl + rank] = x;
              ws.par[spl + rank] = uint8_t(itp + c);
            }
            have += __popc(m);
          }
        }
        bool searching = leaf && nb > 1;
        if (!leaf) {
          searching = nb > 1 && have > sure && (have == room || pos + step >= T || final);
          if (searching) {  // the entries not yet searched for, one per lane
            __syncwarp();
            pred = lane >= sure && lane < have;
            if (pred) {
              x = ws.cand[spl + lane];
              c = ws.par[spl + lane] - itp;
            }
          }
        }
        if (searching && pred) {
          // the other segments whose filter is not exact, two at a time
          uint32_t k = 1;
#pragma unroll 1
          while (pred && k < nb) {
            uint2 a = segs[k++ * stride + c];
            if (a.y >= dense) continue;
            uint2 b = a;
            bool two = false;
#pragma unroll 1
            while (k < nb && !two) {
              b = segs[k++ * stride + c];
              two = b.y < dense;
            }
            pred = in_segments(g.adj, a.x >> fs, a.y >> fs, b.x >> fs, b.y >> fs, two, x, loads);
          }
        }
        __syncwarp();
        if (leaf) {
          const uint32_t xo = kRows ? __ldg(g.old_of_new + x) : __ldg(g.adj_old + at);
          const uint64_t h = fmix64(A.seed + ws.sown[c] + fmix64((uint64_t(lp.qv) << 32) | xo));
          my_hash += pred ? h : 0;
          hits += pred;
          if (A.emit) {
            const uint32_t m = __ballot_sync(kFull, pred);
            if (m) emit_rows(m, n, xo, itp + c);
          }
        } else {
          if (searching) {
            const uint32_t m = __ballot_sync(kFull, pred);
            if (pred) {
              const uint32_t to = spl + sure + __popc(m & lanemask_lt());
              ws.cand[to] = x;
              ws.par[to] = uint8_t(itp + c);
            }
            have = sure + __popc(m);
            __syncwarp();
          }
          if (searching || nb == 1) sure = have;
          stop = sure >= enough;
        }
        begun += __popc(step < 32 ? heads & ((1u << step) - 1) : heads);
        pos += step;
        seen += step;
        stop = stop || final;
      }
      if (pos >= T) {
        itp += group;
        offp = 0;
      } else {  // inside the last driver begun at or before pos
        const uint32_t o = 31 - __clz(__ballot_sync(kFull, start <= pos));
        offp = pos - __shfl_sync(kFull, start, o) + (o == 0 ? offp : 0u);
        itp += o;
      }
      __syncwarp();
    }
    if (leaf) have = __reduce_add_sync(kFull, hits);
    if (lv + 3 == n) s_valid = false;
    if (nb > 1) loads = __reduce_add_sync(kFull, loads);
    if (lane == 0) {
      ws.lev[p].it = itp;
      ws.lev[p].off = offp;
      if (!leaf) ws.lev[lv] = LevelState{have, 0, 0, spl};
      ws.found[lv] += have;
      ws.ev[4] += used;
      ws.pend += seen;
      ws.loads += loads + seen * ((leaf ? 3 : 2) + (nb > 1 && g.filt ? 1 : 0));
    }
    __syncwarp();
    made = have;
    return used;
  };

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
    uint32_t free_word = 0, f = 0;
    uint32_t t = ws.t, t_last = ws.t_last;
    __syncwarp();
    if (t == t_last) {  // input tasks (after an error every task ends at its first check)
      uint32_t t0 = T_in;
      if (lane == 0 && *(volatile uint32_t*)&A.ctr[0 * kCtrStride] < T_in)
        t0 = atomicAdd(&A.ctr[0 * kCtrStride], A.chunk);
      t = __shfl_sync(kFull, t0, 0);
      t_last = t < T_in ? min(t + A.chunk, T_in) : t;
    }
    if (lane == 0) {
      ws.t = min(t + 1, t_last);
      ws.t_last = t_last;
    }
    if (t < t_last) {
      if (A.in_tasks) {
        rec = A.in_tasks + A.in_index[t];
      } else {
        // implicit: root i, chunk of its depth-1 driver range
        uint32_t a = 0, b = nroots;  // last i with chunk_off[i] <= t
#pragma unroll 1
        while (b - a > 1) {
          const uint32_t mid = midpoint(a, b);
          if (A.chunk_off[mid] <= t) a = mid; else b = mid;
        }
        chunk = t - A.chunk_off[a];
        q = A.root_q[a];
        root = A.roots[a];
      }
    } else {
      // input exhausted: take a ticket and wait for its record while others work
      uint32_t mine = 0;
      bool got = false;
      if (lane == 0) {
        mine = atomicAdd(&A.ctr[1 * kCtrStride + 1], 1u);
        atomicSub(&A.ctr[2 * kCtrStride], 1u);
        const unsigned long long t_idle = global_ns();
        unsigned long long t_reserved = 0;  // when the record of this ticket was first seen reserved
        uint32_t sleep_ns = 32;
        volatile uint32_t* word = A.out_ready + queue_slot(mine);
#pragma unroll 1
        for (;;) {
          if (*word == ready_published(mine)) {
            got = true;
            break;
          }
          // finished when nobody works and every record is taken
          if (*(volatile uint32_t*)&A.ctr[2 * kCtrStride] == 0 || *(volatile uint32_t*)&A.ctr[3 * kCtrStride]) break;
          const unsigned long long now = global_ns();
          const uint32_t tail = *(volatile uint32_t*)&A.ctr[1 * kCtrStride];
          if (queue_after(tail, mine)) {
            if (!t_reserved) {
              t_reserved = now;
            } else if (now - t_reserved > A.ready_wait_ns) {
              atomicOr(&A.ctr[3 * kCtrStride], kErrTimeout);
              break;
            }
          } else if (now - t_idle >= (A.first_leaves && mine == A.first_record ? 0ull : A.idle_wait_ns)) {
            // leave: this ticket's record, if it comes, waits for the next pass.
            // (Unmarked, such a record kept the counter from zero: every other
            // waiting warp then waited out its own idle_wait at the pass's end.)
            atomicCAS(&A.ctr[5 * kCtrStride], 0u, max(tail + A.room, 1u));
            const uint32_t was =
                atomicCAS(const_cast<uint32_t*>(word), ready_free(mine), ready_free(mine) | kHolderLeft);
            if (was == ready_free(mine)) break;
            // published meanwhile, or the slot's previous record is still being read
            if (now - t_idle >= A.idle_wait_ns + A.ready_wait_ns && was != ready_published(mine)) break;
          }
          __nanosleep(sleep_ns);
          if (sleep_ns < 1024) sleep_ns <<= 1;
        }
      }
      if (__any_sync(kFull, got)) {
        mine = __shfl_sync(kFull, mine, 0);
        __threadfence();
        if (lane == 0) ws.ev[1]++;
        rec = A.out_tasks + queue_slot(mine);
        ready = A.out_ready + queue_slot(mine);
        free_word = ready_next(mine);
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
    __syncwarp();
    const uint32_t cur_q = ws.query;
    if (q != cur_q || q == kInvalid) {
      if (cur_q != kInvalid) {
        publish();
        const unsigned long long h = warp_sum(my_hash), c = ws.found[lane];
        if (lane == 0 && h) atomicAdd(&A.res[cur_q].hash, h);
        if (lane < ws.n && c) {
          atomicAdd(&A.res[cur_q].levels[lane], c);
          if (lane + 1 == ws.n) atomicAdd(&A.res[cur_q].count, c);
        }
        my_hash = 0;
        ws.found[lane] = 0;
      }
      if (q == kInvalid) break;
      __syncwarp();
      const Plan& pl = A.plans[q];
      const uint32_t n = pl.n;
      if (lane < n) {
        LevelPlan x;
        x.bm = A.pool + pl.bmoff[lane];
        x.bwd = pl.bwd[lane];
        x.inj = pl.same[lane] & ~x.bwd;
        x.bmbase = pl.bmbase[lane];
        x.lab = pl.lab[lane];
        x.nb = uint8_t(__popc(x.bwd));
        x.n4 = uint8_t((__popc(x.inj) + 3) / 4);
        const uint32_t words = 2 * x.nb + 4 * x.n4;
        x.stride = uint8_t(words <= kScratch / kBuf ? kBuf : kScratch / words);
        x.qv = uint8_t(pl.qv[lane]);
        x.dense = kInvalid;
        if (g.filt && x.lab >= 0 && x.lab < g.L)
          x.dense = filter_dense_len(__ldg(g.base + x.lab + 1) - x.bmbase, g.fshift) << g.fshift;
        ws.plan[lane] = x;
      }
      if (lane == 0) {
        ws.n = n;
        ws.pend = 0;
      }
      if (lane == 0) ws.query = q;
      __syncwarp();
    }
    const uint32_t n = ws.n;
    if (root != kInvalid) {
      if (lane == 0) {
        f = root;
        ws.found[0] += chunk == 0;  // the root itself, once
      }
      if (n > 1) {
        row_segment<kRows>(g, root, ws.plan[1].lab, W1, lo, hi);
        lo += chunk * A.split;
        hi = piece_end(lo, A.split, hi);
      }
    }
    if (lane == 0) ws.ev[0]++;
    if (d == n) {  // a complete embedding (single-vertex queries)
      if (lane == 0) {
        const uint32_t xo = __ldg(g.old_of_new + f);
        my_hash += fmix64(A.seed + fmix64((uint64_t(ws.plan[0].qv) << 32) | xo));
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
      ws.cand[lane] = f;
      ws.par[lane] = 0;
    }
    if (lane == 0) {
      ws.task_lo = lo;
      ws.task_hi = hi;
      ws.room = kBuf;
    }
    ws.lev[lane] = LevelState{lane < d ? 1u : 0u, lane + 1 < d ? 1u : 0u, 0u, lane};
    s_valid = false;
    __syncwarp();
    uint32_t lv = d, windows = kCheckWindows, used = 0, hungry = 1;
#pragma unroll 1
    for (;;) {
      if (windows >= kCheckWindows) {
        // at the start and every kCheckWindows windows: the query's work limit,
        // the pass's error word (the call will fail anyway), and waiting warps
        windows = 0;
        int stop = 0;
        if (A.work_cap) {
          publish();
          if (lane == 0) stop = *(volatile unsigned int*)&A.res[ws.query].aborted != 0;
        }
        if (lane == 0) stop |= *(volatile uint32_t*)&A.ctr[3 * kCtrStride] != 0;
        if (__shfl_sync(kFull, stop, 0)) break;
        // (never before the first window: a task handed on untouched would go round)
        if (used) hungry = waiting_warps(t_start);
        if (used && hungry) {
          // the entries of the leaf's ranges are handed off only when those are long
          const uint32_t last = (lv + 1 == n && used >= kFillWindows) ? n - 1 : n - 2;  // plus one
          if (last >= d) donate(d, min(lv, last - 1), hungry, ws.task_lo, ws.task_hi);
        }
      }
      const uint32_t before = ws.lev[lv - 1].it;
      if (before >= ws.lev[lv - 1].cnt) {
        if (lv == d) break;
        lv--;
        continue;
      }
      used = fill(lv, lv == d ? ws.task_lo : kInvalid, ws.task_hi);
      windows += used + 1;
      if (lv + 1 == n) {
        if (lane == 0) ws.room = hungry || 8 * used >= kLongLeaf * (ws.lev[lv - 1].it - before) ? kBuf : kLastBuf;
        __syncwarp();
      }
      if (lv + 1 < n && made > 0) lv++;
    }
  }
  if (lane == 0) {
    atomicAdd(A.algo_bytes, 4 * ws.loads);
#pragma unroll 1
    for (int i = 0; i < 5; i++) atomicAdd(&A.ev[i], (unsigned long long)ws.ev[i]);
  }
}

}  // namespace
}  // namespace fsig
