// Batched window query (replaces bfs_frontier, src/rtree_bfs_frontier.cuh:292-529,
// and bfs_thrust, src/rtree_bfs_thrust.cuh:59-256).
//
// Semantics kept from the reference: the root is never tested; a node whose
// children are nodes passes on the children whose MBR intersects the window
// (src/rtree_bfs_frontier.cuh:110-124); a leaf-parent (pos >= R_sz) tests its
// boxes at slots [pos - R_sz, pos - R_sz + len) (count_hit/write_hit,
// :191-289); a hit emits (fid = sorted box's id, tid = window index).
//
// Traversal: one warp per window.  The warp keeps its frontier in shared
// memory as a stack of node indices.  Each step pops up to K = 32 / fanout
// nodes (one child per lane, children read in SoA layout, coalesced), tests
// the children, compacts the intersecting inner children back onto the stack
// with a ballot/popc prefix, and emits leaf hits warp-collectively.  Popping
// the top K entries and pushing shallower parents' children first keeps the
// stack ordered by depth, so it never holds more than K*fanout entries per
// level: (levels - 1) * K * fanout + 1 in total, which the host sizes exactly.
//
// Three forms:
//   plain       one warp per window in input order, a count pass, an int64
//               exclusive scan and a write pass: output grouped by window.
//   dense       the drop-in query's small batches: one warp (or several) per
//               window, one traversal, pairs in no order.
//   persistent  #SM x occupancy CTAs; warps take windows from an atomic ticket
//               in Morton order of the window centres (neighbouring windows
//               share tree paths, so the tree stays in L2); the top tree levels
//               are staged in shared memory with bulk async copies; hits go to
//               chunks a warp reserves with one atomic, and a
//               compaction pass moves the tail of the array into the unused
//               ends of each warp's last chunk so the output is dense.
//               On sorted windows over packed trees the windows are classed by
//               the boxes they can be expected to meet: huge ones are shared
//               by several warps, small ones go to a kernel that takes 32
//               neighbours per warp (small_windows_kernel).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "internal.h"
#include "profile.h"
#include "traverse.cuh"

namespace crt {

// Device-side counters of one query (int64 words; zeroed before a launch).
struct QueryCounters {
  unsigned long long ticket;  // next large window (persistent)
  unsigned long long small_ticket;  // next small window (persistent)
  unsigned long long nhuge;         // windows of the huge class (first in the sorted order)
  unsigned long long nlarge;        // windows of the huge and large classes
  unsigned long long next;    // next unreserved output slot
  unsigned long long hits;    // exact pair count
  unsigned long long nholes;  // unused chunk ends recorded
  int error;
  int pad;
  unsigned long long nq;      // window count (read by graph replays)
};

// query_stats and the allocation-free entry point keep the counters in the
// first 256 bytes of their scratch.
static_assert(sizeof(QueryCounters) <= 256, "counters fit their scratch slot");

struct Hole {
  long long start;
  long long len;
};

// ---------------------------------------------------------------------------
// Emitters: warp-collective; `hit` and `id` are per lane.
// ---------------------------------------------------------------------------
struct CountEmit {
  static constexpr bool kCountsTests = false;
  static constexpr int kSmall = kSmallRange;
  long long hits = 0;
  __device__ __forceinline__ void begin(int) {}
  __device__ __forceinline__ void operator()(bool hit, int) { hits += __popc(__ballot_sync(0xffffffffu, hit)); }
  __device__ __forceinline__ void range(const int*, long long, long long count) { hits += count; }
  __device__ __forceinline__ void small_ranges(const int*, bool mine, long long, int count)
  {
    hits += __reduce_add_sync(0xffffffffu, mine ? (unsigned)count : 0u);
  }
  __device__ __forceinline__ void big_ranges(const int* bid, bool mine, long long first, long long count)
  {
    emit_ranges_each(*this, bid, mine, first, count);
  }
};

// Counts hits and the leaf boxes tested (workload statistics).
struct StatEmit {
  static constexpr bool kCountsTests = true;
  static constexpr int kSmall = kSmallRange;
  long long hits = 0;
  long long tested = 0;
  __device__ __forceinline__ void begin(int) {}
  __device__ __forceinline__ void operator()(bool hit, int) { hits += __popc(__ballot_sync(0xffffffffu, hit)); }
  long long range_hits = 0;
  __device__ __forceinline__ void leaf_tests(int n) { tested += n; }
  __device__ __forceinline__ void range(const int*, long long, long long count)
  {
    hits += count;
    range_hits += count;
  }
  __device__ __forceinline__ void small_ranges(const int*, bool mine, long long, int count)
  {
    const unsigned n = __reduce_add_sync(0xffffffffu, mine ? (unsigned)count : 0u);
    hits += n;
    range_hits += n;
  }
  __device__ __forceinline__ void big_ranges(const int* bid, bool mine, long long first, long long count)
  {
    emit_ranges_each(*this, bid, mine, first, count);
  }
};

// Writes at precomputed per-window offsets (plain write pass).
struct OffsetEmit {
  static constexpr bool kCountsTests = false;
  static constexpr int kSmall = kSmallRange;
  int32_t* fid;
  int32_t* tid;
  long long base;
  long long cap;
  int q;
  __device__ __forceinline__ void begin(int qq) { q = qq; }
  __device__ __forceinline__ void operator()(bool hit, int id)
  {
    uint32_t m = __ballot_sync(0xffffffffu, hit);
    if (!m) return;
    long long slot = base + __popc(m & lanemask_lt());
    if (hit && slot < cap) {
      __stcs(fid + slot, id);
      if (tid) __stcs(tid + slot, q);  // no window column: CSR output
    }
    base += __popc(m);
  }
  __device__ __forceinline__ void range(const int* bid, long long first, long long count)
  {
    copy_range(bid, first, count, fid, tid, base, cap, q);
    base += count;
  }
  __device__ __forceinline__ void small_ranges(const int* bid, bool mine, long long first, int count)
  {
    emit_small_ranges(*this, bid, mine, first, count);
  }
  __device__ __forceinline__ void big_ranges(const int* bid, bool mine, long long first, long long count)
  {
    emit_ranges_each(*this, bid, mine, first, count);
  }
};

// ---------------------------------------------------------------------------
// Range sharing (persistent form).  One window can own a contained subtree of
// millions of boxes; copied by one warp it leaves the rest of the GPU idle at
// the end of a batch.  The warp that finds such a range reserves its output,
// cuts it into kPiece-id pieces, publishes them in a job queue and goes on
// with its window.  Warps that find no window left claim queue indices with
// one fetch-and-add each and copy the pieces as they are published, so the
// tail of a batch runs on every warp of the GPU.  A claimed index that no
// window will ever fill ends the claimer's wait once every window is done.
// ---------------------------------------------------------------------------
struct RangeJob {
  long long first;  // first sorted slot
  long long slot;   // first output slot
  int count;
  int q;
  unsigned ready;   // 1 once published; the taker clears it
  int pad;
};
// The queue's counters, each on its own 128-byte line: waiting warps poll
// them, and they must not share a line with the ticket and output counters
// every busy warp updates.
struct JobQueue {
  unsigned long long tail;  // pieces reserved
  unsigned long long pad0[15];
  unsigned long long head;  // queue indices claimed
  unsigned long long pad1[15];
  unsigned long long active;  // warps not yet past their ticket loop
  unsigned long long pad2[15];
  RangeJob entries[1];  // kJobs
};
constexpr int kJobs = 1 << 18;         // queue entries per launch (8 MiB)
constexpr int kPiece = 16384;          // ids per piece
constexpr int kShareMin = 2 * kPiece;  // ranges shorter than this stay with their finder
constexpr size_t kJobQueueBytes = offsetof(JobQueue, entries) + sizeof(RangeJob) * kJobs;
constexpr int kQueue = 64;  // contained runs a warp can queue (ChunkEmit)

__device__ __forceinline__ void fence_sc_gpu() { asm volatile("fence.sc.gpu;" ::: "memory"); }

// Waits (lane 0) until queue index h is published, and takes the piece; 0 when
// h will never be published (every ticket is taken, no warp still works on
// one, and h was not reserved) or the bounded wait ran out (an error is
// recorded).  ntickets: the ticket count of the launch.
__device__ __forceinline__ int wait_piece(JobQueue* Q, const QueryCounters* ctr,
                                          unsigned long long ntickets, long long h, RangeJob& out,
                                          int* err)
{
  RangeJob* J = Q->entries + h;
  uint32_t nap = 64;
  for (uint32_t spin = 0; spin < kSpinLimit / 16; spin++) {
    if (ld_acquire_u32(&J->ready)) {
      out.first = J->first;
      out.slot = J->slot;
      out.count = J->count;
      out.q = J->q;
      J->ready = 0;
      return 1;
    }
    if (ld_relaxed_ull(&Q->tail) <= (unsigned long long)h) {
      // not reserved yet: can any window still reserve it?
      fence_sc_gpu();
      const unsigned long long t = ld_relaxed_ull(&ctr->ticket);
      fence_sc_gpu();
      const unsigned long long a = ld_relaxed_ull(&Q->active);
      if (t >= ntickets && a == 0) {
        fence_sc_gpu();
        if (ld_relaxed_ull(&Q->tail) <= (unsigned long long)h) return 0;
      }
    }
    __nanosleep(nap);
    nap = min(2u * nap, 8192u);
  }
  raise_error(err, CRT_ERR_DEVICE_TIMEOUT);
  return 0;
}

// Warp-reserved output chunks (persistent form).  kQueued: the warp queues
// contained runs.
template <bool kQueued>
struct ChunkEmit {
  static constexpr bool kCountsTests = false;
  // runs of 64 boxes and more are queued (32: the same, 128: 2% slower, 256: 6%)
  static constexpr int kSmall = kQueued ? 64 : kSmallRange;
  int32_t* fid;
  int32_t* tid;
  long long cap;
  unsigned long long* next;
  long long cur = 0, end = 0;
  long long hits = 0;
  int chunk;
  int q;
  JobQueue* jobs = nullptr;  // null: no range sharing
  __device__ __forceinline__ void begin(int qq) { q = qq; }
  __device__ __forceinline__ void operator()(bool hit, int id)
  {
    uint32_t m = __ballot_sync(0xffffffffu, hit);
    if (!m) return;
    const int nh = __popc(m);
    const int r = __popc(m & lanemask_lt());
    hits += nh;
    long long slot;
    if (cur + nh <= end) {
      slot = cur + r;
      cur += nh;
    } else {
      const long long left = end - cur;
      unsigned long long nb = 0;
      if (lane_id() == 0) nb = atomicAdd(next, (unsigned long long)chunk);
      nb = __shfl_sync(0xffffffffu, nb, 0);
      slot = r < left ? cur + r : (long long)nb + (r - left);
      cur = (long long)nb + (nh - left);
      end = (long long)nb + chunk;
    }
    if (hit && slot < cap) {
      __stcs(fid + slot, id);
      __stcs(tid + slot, q);
    }
  }
  __device__ __forceinline__ void small_ranges(const int* bid, bool mine, long long first, int count)
  {
    if (cur >= cap && cur < end) {  // past the output: only the count matters
      hits += __reduce_add_sync(0xffffffffu, mine ? (unsigned)count : 0u);
      return;
    }
    emit_small_ranges(*this, bid, mine, first, count);
  }
  // Large contained runs go to exact reservations (no unused chunk end), 32 of
  // them in one: the warp queues them and reserves for all when 32 wait, or when
  // its window ends.  Every warp reserves from one counter, and that counter
  // takes about one atomic per 1.6 ns: with one per range 10M boxes x 250k
  // windows of side 1e-2..1e-1 took 21 ms, with one per step 12.4 (and 1M
  // mixed windows 17.0 ms where runs down to 64 boxes came here, 11.2 queued).
  // Without a queue (persist_shape) a step's runs share one reservation: a kernel
  // of its own, since a branch here cost the 16-warp shape (40 registers) 3%.
  int2* queue = nullptr;  // kQueue entries of this warp: first slot, count
  int queued = 0;
  __device__ __forceinline__ void big_ranges(const int* bid, bool mine, long long first, long long count)
  {
    const uint32_t m = __ballot_sync(0xffffffffu, mine);
    const int lane = (int)lane_id();
    int2 r = make_int2((int)first, (int)count);
    if constexpr (!kQueued) {  // this step's runs to the first lanes
      const int at = (int)__fns(m, 0, lane + 1) & 31;
      r = make_int2(__shfl_sync(0xffffffffu, r.x, at), __shfl_sync(0xffffffffu, r.y, at));
      if (lane >= __popc(m)) r = make_int2(0, 0);
      place_ranges(bid, r, __popc(m));
      return;
    }
    if (mine) queue[queued + __popc(m & lanemask_lt())] = r;
    queued += __popc(m);
    __syncwarp();
    if (queued >= 32) {
      flush_ranges(bid);
      // the entries past the first 32 move down
      int2 rest = make_int2(0, 0);
      if (lane < queued) rest = queue[32 + lane];
      __syncwarp();
      if (lane < queued) queue[lane] = rest;
      __syncwarp();
    }
  }
  // Places the first 32 queued ranges (all, when there are fewer).
  __device__ __forceinline__ void flush_ranges(const int* bid)
  {
    const int n = min(queued, 32);
    if (n == 0) return;
    place_ranges(bid, (int)lane_id() < n ? queue[lane_id()] : make_int2(0, 0), n);
    queued -= n;
  }
  // Places the ranges of the first n lanes in one reservation (the other lanes'
  // are empty).
  __device__ __forceinline__ void place_ranges(const int* bid, int2 r, int n)
  {
    const int lane = (int)lane_id();
    long long x = r.y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    unsigned long long nb = 0;
    if (lane == 31) nb = atomicAdd(next, (unsigned long long)x);
    nb = __shfl_sync(0xffffffffu, nb, 31);
    const long long excl = x - r.y;
    for (int i = 0; i < n; i++)
      place(bid, __shfl_sync(0xffffffffu, r.x, i), __shfl_sync(0xffffffffu, r.y, i),
            (long long)nb + __shfl_sync(0xffffffffu, excl, i));
  }
  // Copies a contained subtree's ids to its reservation at output slot nb
  // (large ones cut into pieces that idle warps copy).
  __device__ __forceinline__ void place(const int* bid, long long first, long long count,
                                        long long nb)
  {
    hits += count;
    if (nb >= cap) return;  // past the output: only the count matters
    if (!jobs || count < kShareMin) {
      copy_range_realign(bid, first, count, fid, tid, nb, cap, q);
      return;
    }
    // publish the pieces; the ones the queue has no room for are copied here
    const long long np = (count + kPiece - 1) / kPiece;
    unsigned long long j0 = 0;
    if (lane_id() == 0) j0 = atomicAdd(&jobs->tail, (unsigned long long)np);
    j0 = __shfl_sync(0xffffffffu, j0, 0);
    const long long own = max(0ll, min(np, (long long)kJobs - (long long)j0));
    for (long long p = lane_id(); p < own; p += 32) {
      RangeJob& J = jobs->entries[(long long)j0 + p];
      const long long off = p * kPiece;
      J.first = first + off;
      J.slot = (long long)nb + off;
      J.count = (int)min((long long)kPiece, count - off);
      J.q = q;
      st_release_u32(&J.ready, 1u);
    }
    if (own < np)
      copy_range(bid, first + own * kPiece, count - own * kPiece, fid, tid,
                 (long long)nb + own * kPiece, cap, q);
  }
};

// ---------------------------------------------------------------------------
// Plain form: count pass / write pass, one warp per window in input order
// ---------------------------------------------------------------------------
constexpr int kPlainWarps = 8;

__global__ void __launch_bounds__(kPlainWarps * 32)
    plain_count_kernel(TreeView T, WindowView W, int K, int stack_cap,
                       long long* __restrict__ counts, QueryCounters* ctr)
{
  extern __shared__ FrontierEntry s_stack[];
  const int warp = threadIdx.x >> 5;
  const long long q = (long long)blockIdx.x * kPlainWarps + warp;
  if (q >= W.n) return;
  int lg, lc;
  lane_map(T.fanout, lg, lc);
  NodeCache C{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0};
  CountEmit emit;
  traverse(T, C, K, lg, lc, W.xmin[q], W.ymin[q], W.xmax[q], W.ymax[q],
           s_stack + warp * stack_cap, stack_cap, emit, &ctr->error);
  if (lane_id() == 0) counts[q] = emit.hits;
}

__global__ void __launch_bounds__(kPlainWarps * 32)
    plain_write_kernel(TreeView T, WindowView W, int K, int stack_cap,
                       const long long* __restrict__ offsets, int32_t* fid, int32_t* tid,
                       long long cap, const QueryCounters* ctr, int* err)
{
  extern __shared__ FrontierEntry s_stack[];
  const int warp = threadIdx.x >> 5;
  const long long q = (long long)blockIdx.x * kPlainWarps + warp;
  if (q >= W.n) return;
  if (ctr->error) {  // the offsets are not to be used
    raise_error(err, ctr->error);
    return;
  }
  if (offsets[W.n] > cap) return;  // overflow: the host reports the required size
  int lg, lc;
  lane_map(T.fanout, lg, lc);
  NodeCache C{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0};
  OffsetEmit emit{fid, tid, offsets[q], cap, (int)q};
  traverse(T, C, K, lg, lc, W.xmin[q], W.ymin[q], W.xmax[q], W.ymax[q],
           s_stack + warp * stack_cap, stack_cap, emit, err);
}

template <bool kContain>
__global__ void __launch_bounds__(kPlainWarps * 32)
    stats_kernel(TreeView T, WindowView W, int K, int stack_cap, long long* __restrict__ hits,
                 long long* __restrict__ tested, unsigned long long* __restrict__ totals,
                 QueryCounters* ctr)
{
  extern __shared__ FrontierEntry s_stack[];
  const int warp = threadIdx.x >> 5;
  const long long q = (long long)blockIdx.x * kPlainWarps + warp;
  if (q >= W.n) return;
  int lg, lc;
  lane_map(T.fanout, lg, lc);
  NodeCache C{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0};
  StatEmit emit;
  traverse<StatEmit, kContain>(T, C, K, lg, lc, W.xmin[q], W.ymin[q], W.xmax[q], W.ymax[q],
                               s_stack + warp * stack_cap, stack_cap, emit, &ctr->error);
  if (lane_id() == 0) {
    if (hits) hits[q] = emit.hits;
    if (tested) tested[q] = emit.tested;
    atomicAdd(&totals[0], (unsigned long long)emit.hits);
    atomicAdd(&totals[1], (unsigned long long)emit.tested);
    atomicAdd(&totals[2], (unsigned long long)emit.range_hits);
  }
}

// int64 exclusive scan (counts -> offsets[0..n]) and the result block, one
// launch: a CTA takes 1024 counts in ticket order and looks back over the
// tiles before it, 32 at a time (decoupled look-back, one 64-bit status word
// per tile, zeroed before).  Block sums, their scan, an apply pass and a
// result kernel, mostly launch latency for the batches of a plain query, took
// 16 us for 20k windows with the gaps between them; this takes 3.5.
constexpr int kScanThreads = 1024;
constexpr unsigned long long kTileAgg = 1ull << 62;
constexpr unsigned long long kTileIncl = 2ull << 62;
constexpr unsigned long long kTileFlags = 3ull << 62;

__global__ void __launch_bounds__(kScanThreads)
    scan_kernel(const long long* __restrict__ counts, long long n, long long* __restrict__ offsets,
                unsigned long long* __restrict__ status, QueryCounters* __restrict__ ctr,
                long long cap, crt_query_result* __restrict__ res)
{
  __shared__ long long s_warp[32];
  __shared__ long long s_before;
  __shared__ int s_tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_tile = (int)atomicAdd(&ctr->ticket, 1ull);
  __syncthreads();
  const int tile = s_tile;
  const long long i = (long long)tile * kScanThreads + threadIdx.x;
  const long long v = i < n ? counts[i] : 0;
  long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const long long t = s_warp[lane];
    long long w = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    s_warp[lane] = w - t;
    const long long total = __shfl_sync(0xffffffffu, w, 31);
    if (lane == 0) st_relaxed_u64((uint64_t*)&status[tile], (tile ? kTileAgg : kTileIncl) | (uint64_t)total);
    long long before = 0;
    uint32_t spins = 0;
    for (int t0 = tile - 1; t0 >= 0;) {
      // lane l: tile t0 - l (before tile 0: an inclusive zero)
      const unsigned long long st = t0 >= lane ? ld_relaxed_u64((const uint64_t*)&status[t0 - lane]) : kTileIncl;
      const uint32_t open = __ballot_sync(0xffffffffu, (st & kTileFlags) == 0);
      const uint32_t incl = __ballot_sync(0xffffffffu, (st & kTileFlags) == kTileIncl);
      // the tiles up to the first inclusive one, if none before it is missing
      const int stop = incl ? __ffs(incl) : 32;
      if (open & (stop == 32 ? 0xffffffffu : (1u << stop) - 1)) {
        if (++spins > kSpinLimit || ld_relaxed_i32(&ctr->error) != 0) {
          if (lane == 0) raise_error(&ctr->error, CRT_ERR_DEVICE_TIMEOUT);
          break;
        }
        if (spins > 64) __nanosleep(64);
        continue;
      }
      long long part = lane < stop ? (long long)(st & ~kTileFlags) : 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      before += part;
      if (incl) break;
      t0 -= 32;
    }
    if (lane == 0) {
      if (tile) st_relaxed_u64((uint64_t*)&status[tile], kTileIncl | (uint64_t)(before + total));
      s_before = before;
      if (tile == (int)gridDim.x - 1) {
        const long long all = before + total;
        offsets[n] = all;
        res->required = all;
        res->overflow = all > cap ? 1 : 0;
        res->count = all > cap ? 0 : all;
        res->error = ld_relaxed_i32(&ctr->error);
      }
    }
  }
  __syncthreads();
  if (i < n) offsets[i] = s_before + s_warp[warp] + x - v;
}

// ---------------------------------------------------------------------------
// Persistent form
// ---------------------------------------------------------------------------
struct PersistParams {
  TreeView T;
  WindowView W;
  const uint32_t* order0;  // sorted window order candidates (vals[0], vals[1])
  const uint32_t* order1;
  const SortCtrl* sort_ctrl;  // n_active picks the buffer; null: input order
  int K;
  int stack_cap;
  int stage_n;  // nodes staged in shared memory (multiple of 4), 0 = none
  int parts;    // warps sharing one window (shares of the root's children)
  bool classes;  // the windows are sorted by class: huge, large, small
  int split_height;  // nodes of this height are dealt out among a huge window's warps
  int chunk;
  int32_t* fid;
  int32_t* tid;
  long long cap;
  QueryCounters* ctr;
  Hole* holes;
  long long max_holes;
  JobQueue* jobs;  // counters and kJobs entries, zeroed before the launch
};

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
  return (uint32_t)__cvta_generic_to_shared(p);
}

// One bulk async copy global -> shared (16-byte aligned, size a multiple of
// 16), completing on the mbarrier at `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint32_t bar)
{
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// Warps sharing a huge window, each walking the levels above the split height
// and then its own share of the nodes of that height.  A window of side 0.1 on
// 10M boxes keeps one warp busy for 1.2 ms, so a batch with few such windows
// waits for the slowest; many of them fill the GPU by themselves, and then the
// levels walked twice only cost.  Traversal of mixed batches (sides 1e-5 ..
// 0.1, 10M boxes, 16 warps per CTA) with 1, 2, 4 and 8 warps per huge window:
//     5k windows (0.1 per warp)  1243    -   411   315 us
//    60k         (1.5)           1649    -  1189  1216
//   250k         (6)             4050  3745  3805  4168
//     1M         (24)           13240 13350 14100     -
// Road geometry (20k windows, a tenth covering over 1%): 3490 -> 1215 us.
__device__ __forceinline__ int split_parts_for(long long nhuge, long long warps)
{
  return 2 * nhuge < warps ? 8 : nhuge < 2 * warps ? 4 : nhuge < 12 * warps ? 2 : 1;
}

// kShare: range sharing (the job queue).  Its code needs registers the
// tighter CTA shapes do not have, so only the 8-warp shape (64 registers)
// shares ranges; the autotuner weighs the shapes against each other.  kQueued:
// the warps have queues of contained runs.
template <int kThreads, int kMinBlocks, bool kShare, bool kQueued>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
    persistent_kernel(PersistParams P)
{
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long s_mbar;
  __shared__ int s_stage_ok;
  chain_next();  // the small windows' kernel
  const int warps = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5;
  // layout: [staged nodes: 6 arrays x stage_n x 4 B][stacks: warps x stack_cap
  // entries][queued ranges: warps x kQueue, or none]
  float* c_xmin = (float*)smem_raw;
  float* c_ymin = c_xmin + P.stage_n;
  float* c_xmax = c_ymin + P.stage_n;
  float* c_ymax = c_xmax + P.stage_n;
  int* c_pos = (int*)(c_ymax + P.stage_n);
  int* c_len = c_pos + P.stage_n;
  FrontierEntry* stacks = (FrontierEntry*)(c_len + P.stage_n);
  NodeCache C{c_xmin, c_ymin, c_xmax, c_ymax, c_pos, c_len, 0};

  if (P.stage_n > 0) {
    // bulk async copies of the top levels into shared memory, one mbarrier
    const uint32_t bar = smem_addr(&s_mbar);
    const uint32_t bytes = (uint32_t)P.stage_n * 4u;
    if (threadIdx.x == 0) {
      s_stage_ok = 1;
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                   "r"(6u * bytes)
                   : "memory");
      bulk_load(c_xmin, P.T.nxmin, bytes, bar);
      bulk_load(c_ymin, P.T.nymin, bytes, bar);
      bulk_load(c_xmax, P.T.nxmax, bytes, bar);
      bulk_load(c_ymax, P.T.nymax, bytes, bar);
      bulk_load(c_pos, P.T.npos, bytes, bar);
      bulk_load(c_len, P.T.nlen, bytes, bar);
    }
    // bounded wait for phase 0 (twice the usual limit: after a timeout the
    // copies must not still be landing when the CTA leaves)
    uint32_t done = 0;
    for (uint32_t spin = 0; spin < 2 * kSpinLimit; spin++) {
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n selp.u32 %0, 1, 0, p;\n}"
          : "=r"(done)
          : "r"(bar)
          : "memory");
      if (done) break;
    }
    if (!done) {
      if (threadIdx.x == 0) s_stage_ok = 0;
      raise_error(&P.ctr->error, CRT_ERR_DEVICE_TIMEOUT);
    }
    __syncthreads();
    if (!s_stage_ok) return;
    C.n = P.stage_n;
  }

  FrontierEntry* stack = stacks + warp * P.stack_cap;
  int lg, lc;
  lane_map(P.T.fanout, lg, lc);
  const uint32_t* order = nullptr;
  if (P.sort_ctrl) {
    const int na = P.sort_ctrl->n_active;
    order = na == 0 ? nullptr : ((na & 1) ? P.order1 : P.order0);
  }
  const long long nq = (long long)P.ctr->nq;
  const int parts = P.parts;
  // one ticket per (window, share); the small windows are small_windows_kernel's
  const long long nhuge = P.classes ? (long long)P.ctr->nhuge : 0;
  const int split_parts = split_parts_for(nhuge, (long long)gridDim.x * warps);
  const long long nsplit = nhuge * split_parts;
  const long long ntickets = nsplit + ((P.classes ? (long long)P.ctr->nlarge : nq) - nhuge) * parts;
  ChunkEmit<kQueued> emit;
  emit.fid = P.fid;
  emit.tid = P.tid;
  emit.cap = P.cap;
  emit.next = &P.ctr->next;
  emit.chunk = P.chunk;
  if constexpr (kQueued) emit.queue = (int2*)(stacks + warps * P.stack_cap) + warp * kQueue;
  emit.jobs = kShare ? P.jobs : nullptr;
  JobQueue* Q = kShare ? P.jobs : nullptr;
  // a warp counts as active from before its first ticket until it has left
  // the ticket loop, so a waiting warp that sees the tickets gone and no
  // warp active knows no window can publish any more
  if (Q && lane_id() == 0) {
    atomicAdd(&Q->active, 1ull);
    fence_sc_gpu();
  }
  while (true) {
    unsigned long long t = 0;
    if (lane_id() == 0) t = atomicAdd(&P.ctr->ticket, 1ull);
    t = __shfl_sync(0xffffffffu, t, 0);
    if ((long long)t >= ntickets) break;
    long long qi = (long long)t;
    int part = 0, nparts = 1;
    Split split;
    if ((long long)t < nsplit) {
      qi = (long long)t / split_parts;
      split.height = P.split_height;
      split.mask = split_parts - 1;
      split.part = (int)t & (split_parts - 1);
    } else {
      qi -= nsplit;
      if (parts > 1) {
        nparts = parts;
        part = (int)(qi % parts);
        qi /= parts;
      }
      qi += nhuge;
    }
    int q = order ? (int)order[qi] : (int)qi;
    if (q < 0 || (long long)q >= nq) q = (int)qi;  // only after a sort error (reported)
    emit.begin(q);
    traverse(P.T, C, P.K, lg, lc, P.W.xmin[q], P.W.ymin[q], P.W.xmax[q], P.W.ymax[q], stack,
             P.stack_cap, emit, &P.ctr->error, part, nparts, split);
    if constexpr (kQueued) emit.flush_ranges(P.T.bid);
  }
  if (Q) {
    __syncwarp();
    if (lane_id() == 0) {
      fence_sc_gpu();  // this warp's reservations before it stops counting
      atomicAdd(&Q->active, ~0ull);  // -1
    }
  }
  // No window left: copy published pieces until no window can publish more.
  if (Q) {
    while (true) {
      long long h = 0;
      if (lane_id() == 0) h = (long long)atomicAdd(&Q->head, 1ull);
      h = __shfl_sync(0xffffffffu, h, 0);
      if (h >= kJobs) break;  // past the queue: never published
      RangeJob J{};
      int got = 0;
      if (lane_id() == 0) got = wait_piece(Q, P.ctr, (unsigned long long)ntickets, h, J, &P.ctr->error);
      if (!__shfl_sync(0xffffffffu, got, 0)) break;
      const long long first = __shfl_sync(0xffffffffu, J.first, 0);
      const long long slot = __shfl_sync(0xffffffffu, J.slot, 0);
      const int count = __shfl_sync(0xffffffffu, J.count, 0);
      const int jq = __shfl_sync(0xffffffffu, J.q, 0);
      copy_range(P.T.bid, first, count, P.fid, P.tid, slot, P.cap, jq);
    }
  }
  if (lane_id() == 0) {
    if (emit.hits) atomicAdd(&P.ctr->hits, (unsigned long long)emit.hits);
    if (emit.end > emit.cur) {
      unsigned long long h = atomicAdd(&P.ctr->nholes, 1ull);
      if ((long long)h < P.max_holes) {
        P.holes[h].start = emit.cur;
        P.holes[h].len = emit.end - emit.cur;
      } else {
        raise_error(&P.ctr->error, CRT_ERR_NOT_SUPPORTED);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Small windows (persistent form, windows sorted)
// ---------------------------------------------------------------------------
// A window that meets a handful of boxes walks some 20 frontier entries to
// find them, most of them on the upper levels and the same for its
// neighbours; one window per warp spent 1600 warp instructions on each (10M
// boxes, fanout 10, sides up to 1e-3: 1.80 ms per 1M windows, 77% of the
// issue slots).  Here a warp takes up to 32 windows that are neighbours in
// Morton order (the same batch: 0.67 ms) and
//   1. descends once with their bounding box, level by level, while the nodes
//      it meets fit the frontier (kFrontier): that frontier holds every node
//      of its level that any of the windows meets;
//   2. tests every window (one per lane) against the frontier's MBRs;
//   3. takes the (window, node) pairs K at a time: leaf-parents' boxes are
//      tested at once, other nodes go on through traverse_group's stack.
// Only for packed trees over ordinary boxes: a node excluded by the bounding
// box is excluded by each window, and (NaN aside) a child that a window meets
// lies under nodes that it meets, so skipping those tests changes nothing: a
// node's MBR bounds its children's and its boxes, as in every tree a build made,
// which the tables' test (level_tables) does not look at.  A
// NaN in a window opens that side of the bounding box.  Hits are staged in
// shared memory and flushed densely, one reservation per flush, so nothing is
// left for the compaction pass.
constexpr int kSmallWarps = 8;
constexpr int kFrontier = 96;     // nodes (64: 770, 96: 674, 128: 705 us for the batch above)
constexpr int kSmallStage = 128;  // staged pairs per warp
constexpr int kSmallSets = 2;     // pairs tested per step, in multiples of K
constexpr int kPairChunk = 32;  // frontier nodes whose pairs are listed at a time

struct StageEmit {
  static constexpr bool kCountsTests = false;
  static constexpr int kSmall = kSmallRange;
  int2* s_out;  // this warp's staging, kSmallStage pairs
  int n = 0;
  int q = 0;  // the window, where the warp walks one at a time
  int32_t* fid;
  int32_t* tid;
  long long cap;
  unsigned long long* next;
  long long total = 0;
  __device__ __forceinline__ long long reserve(long long count)
  {
    unsigned long long b = 0;
    if (lane_id() == 0) b = atomicAdd(next, (unsigned long long)count);
    total += count;
    return (long long)__shfl_sync(0xffffffffu, b, 0);
  }
  __device__ __forceinline__ void flush()
  {
    __syncwarp();
    if (n > 0) {
      const long long b = reserve(n);
      for (int i = (int)lane_id(); i < n; i += 32) {
        const int2 v = s_out[i];
        put_pair(fid, tid, b + i, cap, v.x, v.y);
      }
      n = 0;
    }
    __syncwarp();
  }
  // The lanes of mask m (hit) emit (id, window q).
  __device__ __forceinline__ void hits(uint32_t m, bool hit, int id, int q)
  {
    const int c = __popc(m);
    if (n + c > kSmallStage) flush();
    if (hit) s_out[n + __popc(m & lanemask_lt())] = make_int2(id, q);
    n += c;
  }
  // Every lane's slot range, 32 ids per warp pass (as emit_small_ranges), each
  // with its range's window.
  __device__ __forceinline__ void small_ranges(const int* __restrict__ bid, bool mine, long long first,
                                               int count, int q)
  {
    const int lane = (int)lane_id();
    const int c = mine ? count : 0;
    int x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const int all = __shfl_sync(0xffffffffu, x, 31);
    const int base = (int)first - (x - c);  // sorted slots are below 2^31
    for (int t0 = 0; t0 < all; t0 += 32) {
      const int t = t0 + lane;
      int j = 0;  // lanes whose inclusive prefix is <= t: the owner of t
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const int v = __shfl_sync(0xffffffffu, x, j + s - 1);
        if (v <= t) j += s;
      }
      const int b = __shfl_sync(0xffffffffu, base, j);
      const int w = __shfl_sync(0xffffffffu, q, j);
      const bool ok = t < all;
      hits(__ballot_sync(0xffffffffu, ok), ok, ok ? __ldg(bid + b + t) : 0, w);
    }
  }
  __device__ __forceinline__ void big_ranges(const int* bid, bool mine, long long first, long long count,
                                             int q)
  {
    uint32_t im = __ballot_sync(0xffffffffu, mine);
    while (im) {
      const int src = __ffs(im) - 1;
      im &= im - 1;
      const long long c = __shfl_sync(0xffffffffu, count, src);
      copy_range(bid, __shfl_sync(0xffffffffu, first, src), c, fid, tid, reserve(c), cap,
                 __shfl_sync(0xffffffffu, q, src));
    }
  }
  // the emitter of traverse(): every lane's window is q
  __device__ __forceinline__ void operator()(bool hit, int id)
  {
    const uint32_t m = __ballot_sync(0xffffffffu, hit);
    if (m) hits(m, hit, id, q);
  }
  __device__ __forceinline__ void small_ranges(const int* bid, bool mine, long long first, int count)
  {
    small_ranges(bid, mine, first, count, q);
  }
  __device__ __forceinline__ void big_ranges(const int* bid, bool mine, long long first, long long count)
  {
    big_ranges(bid, mine, first, count, q);
  }
};

// Shared memory of one warp.  The pair list and the stack follow each other;
// both are free while the frontier is expanded, which uses their room for the
// next level's nodes.
struct SmallSmem {
  static constexpr size_t kWin = 0;                                     // float4 x 32
  static constexpr size_t kQ = kWin + 16 * kGroupWindows;               // int x 32
  static constexpr size_t kMbr = kQ + 4 * kGroupWindows;                // float4 x kFrontier
  static constexpr size_t kLink = kMbr + 16 * kFrontier;                // int2 x kFrontier
  static constexpr size_t kOut = kLink + 8 * kFrontier;                 // int2 x kSmallStage
  static constexpr size_t kPairs = kOut + 8 * kSmallStage;              // uint16 x pairs
  static constexpr size_t kStack = kPairs + 2 * kGroupWindows * kPairChunk;
  static_assert(kMbr % 16 == 0 && kPairs % 16 == 0 && kStack % 16 == 0, "16-byte parts");
  static size_t bytes(int stack_cap)
  {
    const size_t a = kStack + sizeof(FrontierEntry) * (size_t)stack_cap;
    const size_t b = kPairs + 24 * (size_t)kFrontier;
    return ((a > b ? a : b) + 15) / 16 * 16;
  }
};

__global__ void __launch_bounds__(kSmallWarps * 32, 3)
    small_windows_kernel(PersistParams P, int warp_bytes)
{
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int lane = (int)lane_id(), warp = threadIdx.x >> 5;
  unsigned char* my = smem_raw + (size_t)warp * warp_bytes;
  float4* s_win = (float4*)(my + SmallSmem::kWin);
  int* s_q = (int*)(my + SmallSmem::kQ);
  float4* f_mbr = (float4*)(my + SmallSmem::kMbr);
  int2* f_link = (int2*)(my + SmallSmem::kLink);  // {first child, children}
  uint16_t* s_pair = (uint16_t*)(my + SmallSmem::kPairs);
  FrontierEntry* stack = (FrontierEntry*)(my + SmallSmem::kStack);
  float4* g_mbr = (float4*)(my + SmallSmem::kPairs);  // the next level, while expanding
  int2* g_link = (int2*)(my + SmallSmem::kPairs + 16 * kFrontier);
  const TreeView& T = P.T;
  const int K = P.K;
  const uint32_t lt = lanemask_lt();
  int lg, lc;
  lane_map(T.fanout, lg, lc);
  const int na = P.sort_ctrl->n_active;
  const uint32_t* order = na == 0 ? nullptr : ((na & 1) ? P.order1 : P.order0);
  const long long nlarge = (long long)P.ctr->nlarge, nq = (long long)P.ctr->nq;
  const long long nsmall = nq - nlarge;
  // batches shrink towards the end (guided self-scheduling, Polychronopoulos
  // and Kuck, 1987)
  const long long share = (long long)gridDim.x * kSmallWarps * 2;
  // and there are some sixteen batches a warp: 32 neighbours on dense data can hold
  // 300k pairs (uniform boxes, 1M windows of 10: batches of 32 720 us, of 17 626,
  // of 4 790; 1M windows of 1200 on clustered boxes 14.9 ms with eight, 12.7
  // with sixteen)
  const long long most = max(2ll, min((long long)kGroupWindows, nsmall / (8 * share)));
  StageEmit emit;
  emit.s_out = (int2*)(my + SmallSmem::kOut);
  emit.fid = P.fid;
  emit.tid = P.tid;
  emit.cap = P.cap;
  emit.next = &P.ctr->next;
  unsigned long long t = 0;
  while (true) {
    const int want = (int)max(1ll, min(most, (nsmall - (long long)t) / share));
    if (lane == 0) t = atomicAdd(&P.ctr->small_ticket, (unsigned long long)want);
    t = __shfl_sync(0xffffffffu, t, 0);
    if ((long long)t >= nsmall) break;
    const int nw = (int)min((long long)want, nsmall - (long long)t);
    // the windows, and their bounding box (a NaN opens its side)
    const float inf = __int_as_float(0x7f800000);
    float4 w = make_float4(inf, inf, -inf, -inf);
    if (lane < nw) {
      const long long qi = nlarge + (long long)t + lane;
      int q = order ? (int)order[qi] : (int)qi;
      if (q < 0 || (long long)q >= nq) q = (int)qi;  // only after a sort error (reported)
      w = make_float4(P.W.xmin[q], P.W.ymin[q], P.W.xmax[q], P.W.ymax[q]);
      s_q[lane] = q;
    }
    s_win[lane] = w;
    float4 box = make_float4(isnan(w.x) ? -inf : w.x, isnan(w.y) ? -inf : w.y,
                             isnan(w.z) ? inf : w.z, isnan(w.w) ? inf : w.w);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      box.x = fminf(box.x, __shfl_xor_sync(0xffffffffu, box.x, o));
      box.y = fminf(box.y, __shfl_xor_sync(0xffffffffu, box.y, o));
      box.z = fmaxf(box.z, __shfl_xor_sync(0xffffffffu, box.z, o));
      box.w = fmaxf(box.w, __shfl_xor_sync(0xffffffffu, box.w, o));
    }
    // 1. the frontier: from the root (never tested), level by level
    if (lane == 0) f_link[0] = make_int2(__ldg(T.npos), __ldg(T.nlen));
    __syncwarp();
    int nf = 1;
    int height = T.nlev - 1;  // of the frontier's nodes (0: leaf-parents)
    while (height > 0) {
      int ng = 0;
      for (int e0 = 0; e0 < nf && ng <= kFrontier; e0 += K) {
        const int e = e0 + lg;
        bool ok = lg < K && e < nf;
        const int2 link = f_link[ok ? e : 0];
        const int i = link.x + lc;
        ok = ok && lc < link.y && i < T.rsz;
        float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
        int2 l = make_int2(0, 0);
        if (ok) {
          m = make_float4(__ldg(T.nxmin + i), __ldg(T.nymin + i), __ldg(T.nxmax + i), __ldg(T.nymax + i));
          l = make_int2(__ldg(T.npos + i), __ldg(T.nlen + i));
        }
        const bool hit = ok && intersects(box.x, box.y, box.z, box.w, m.x, m.y, m.z, m.w);
        const uint32_t hm = __ballot_sync(0xffffffffu, hit);
        const int at = ng + __popc(hm & lt);
        if (hit && at < kFrontier) {
          g_mbr[at] = m;
          g_link[at] = l;
        }
        ng += __popc(hm);
      }
      __syncwarp();
      if (ng > kFrontier) break;  // the level does not fit: stay above it
      for (int i = lane; i < ng; i += 32) {
        f_mbr[i] = g_mbr[i];
        f_link[i] = g_link[i];
      }
      __syncwarp();
      nf = ng;
      height--;
      if (nf == 0) break;
    }
    // 2./3. pairs of windows and frontier nodes, kPairChunk nodes at a time
    const bool top = height == T.nlev - 1;  // the root itself: never tested
    for (int c0 = 0; c0 < nf; c0 += kPairChunk) {
      const int nc = min(kPairChunk, nf - c0);
      uint32_t mine = 0;
      if (lane < nw) {
        if (top) {
          mine = 1u;
        } else {
          for (int i = 0; i < nc; i++) {
            const float4 m = f_mbr[c0 + i];
            if (intersects(w.x, w.y, w.z, w.w, m.x, m.y, m.z, m.w)) mine |= 1u << i;
          }
        }
      }
      const int cnt = __popc(mine);
      int x = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      const int np = __shfl_sync(0xffffffffu, x, 31);
      for (int at = x - cnt; mine; mine &= mine - 1)
        s_pair[at++] = (uint16_t)(lane << 8 | (c0 + __ffs(mine) - 1));
      __syncwarp();
      if (height == 0) {
        // leaf-parents: test their boxes
        for (int p0 = 0; p0 < np; p0 += kSmallSets * K) {
          float m1[kSmallSets], n1[kSmallSets], m2[kSmallSets], n2[kSmallSets];
          int id[kSmallSets], wl[kSmallSets];
          bool ok[kSmallSets];
#pragma unroll
          for (int s = 0; s < kSmallSets; s++) {
            const int p = p0 + s * K + lg;
            ok[s] = lg < K && p < np;
            const uint32_t pr = s_pair[ok[s] ? p : 0];
            wl[s] = pr >> 8;
            const int2 link = f_link[pr & 0xFFu];
            const int j = link.x - T.rsz + lc;
            ok[s] = ok[s] && lc < link.y && j < T.nbox;
            m1[s] = n1[s] = m2[s] = n2[s] = 0.f;
            id[s] = 0;
            if (ok[s]) {
              m1[s] = __ldg(T.bxmin + j);
              n1[s] = __ldg(T.bymin + j);
              m2[s] = __ldg(T.bxmax + j);
              n2[s] = __ldg(T.bymax + j);
              id[s] = __ldg(T.bid + j);
            }
          }
#pragma unroll
          for (int s = 0; s < kSmallSets; s++) {
            const float4 v = s_win[wl[s]];
            const bool hit = ok[s] && intersects(v.x, v.y, v.z, v.w, m1[s], n1[s], m2[s], n2[s]);
            const uint32_t hm = __ballot_sync(0xffffffffu, hit);
            if (hm) emit.hits(hm, hit, id[s], s_q[wl[s]]);
          }
        }
      } else {
        int p = 0;
        traverse_group<kSmallSets>(
            T, K, lg, lc, s_win, s_q, stack, P.stack_cap, emit,
            [&](int sp) {
              const int m = min(kGroupWindows, np - p);
              if (m <= 0) return sp;
              if (lane < m) {
                const uint32_t pr = s_pair[p + lane];
                const int2 link = f_link[pr & 0xFFu];
                stack[sp + lane] = group_entry(link.x, link.y, (int)(pr >> 8), height - 1);
              }
              p += m;
              __syncwarp();
              return sp + m;
            },
            &P.ctr->error);
      }
      __syncwarp();
    }
  }
  emit.flush();
  if (lane == 0 && emit.total) atomicAdd(&P.ctr->hits, (unsigned long long)emit.total);
  chain_wait();  // what follows this kernel needs the persistent kernel's output too
}

// ---------------------------------------------------------------------------
// Dense form (the drop-in query's small batches)
// ---------------------------------------------------------------------------
// One traversal per window in input order, hits staged per warp and flushed
// densely: no second traversal, no scan, no window order and no compaction, so
// a batch costs three launches.  The pairs come in no order, which is all the
// drop-in query promises.  Batches that leave the GPU short of warps give each
// window kDenseParts of them (Split).  10k windows on 1M boxes (384k pairs):
// one traversal of 30 us instead of 23 + 29 and a scan.
constexpr int kDenseParts = 8;

__global__ void __launch_bounds__(kPlainWarps * 32)
    dense_kernel(TreeView T, WindowView W, int K, int stack_cap, int parts, int split_height,
                 int32_t* fid, int32_t* tid, long long cap, QueryCounters* ctr)
{
  extern __shared__ FrontierEntry s_stack[];  // stacks, then kSmallStage pairs per warp
  const int warp = threadIdx.x >> 5;
  const long long t = (long long)blockIdx.x * kPlainWarps + warp;
  const long long q = t / parts;
  if (q >= W.n) return;
  Split split;
  if (parts > 1) {
    split.part = (int)(t - q * parts);
    if (*T.lvl_odd == 0) {  // entries carry their height only with the shortcut on
      split.height = split_height;
      split.mask = parts - 1;
    } else if (split.part != 0) {
      return;
    }
  }
  int lg, lc;
  lane_map(T.fanout, lg, lc);
  NodeCache C{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0};
  StageEmit emit;
  emit.s_out = s_stack + kPlainWarps * stack_cap + warp * kSmallStage;
  emit.q = (int)q;
  emit.fid = fid;
  emit.tid = tid;
  emit.cap = cap;
  emit.next = &ctr->next;
  traverse(T, C, K, lg, lc, W.xmin[q], W.ymin[q], W.xmax[q], W.ymax[q], s_stack + warp * stack_cap,
           stack_cap, emit, &ctr->error, 0, 1, split);
  emit.flush();
}

// Sorts the recorded holes by start and makes the exclusive prefix of their
// lengths: a hole's rank is the number of holes before it (starts are
// distinct: holes do not overlap) and its prefix their total length.  A CTA
// takes kRankHoles holes, one per lane, and deals all holes out among its
// warps, which read each from shared memory once for 32 comparisons.  Bound by
// the issue of n^2 / 32 comparisons: 28 us for 7104 holes; one thread per hole
// with a serial loop, and a prefix pass of its own, took 94 us.
constexpr int kRankHoles = 32;
constexpr int kRankWarps = 8;
constexpr int kRankTile = 1024;

__global__ void __launch_bounds__(kRankWarps * 32)
    hole_rank_kernel(const Hole* __restrict__ holes, Hole* __restrict__ sorted,
                     long long* __restrict__ cum, const QueryCounters* __restrict__ ctr,
                     long long max_holes)
{
  __shared__ __align__(16) Hole s_hole[kRankTile];
  __shared__ int s_rank[kRankHoles];
  __shared__ unsigned long long s_before[kRankHoles];
  const int nh = (int)min((long long)ctr->nholes, max_holes);
  const int lane = (int)lane_id(), warp = threadIdx.x >> 5;
  const int i0 = blockIdx.x * kRankHoles;
  if (i0 >= nh) {  // whole CTA idle
    if (nh == 0 && blockIdx.x == 0 && threadIdx.x == 0) cum[0] = 0;
    return;
  }
  if (threadIdx.x < kRankHoles) {
    s_rank[threadIdx.x] = 0;
    s_before[threadIdx.x] = 0;
  }
  const Hole my = holes[min(i0 + lane, nh - 1)];
  int r = 0;
  unsigned long long before = 0;
  for (int t0 = 0; t0 < nh; t0 += kRankTile) {
    const int m = min(kRankTile, nh - t0);
    __syncthreads();
    for (int k = threadIdx.x; k < m; k += blockDim.x) s_hole[k] = holes[t0 + k];
    __syncthreads();
    const int k1 = min(m, (warp + 1) * (kRankTile / kRankWarps));
    for (int k = warp * (kRankTile / kRankWarps); k < k1; k++) {
      const Hole h = s_hole[k];
      if (h.start < my.start) {
        r++;
        before += (unsigned long long)h.len;
      }
    }
  }
  __syncthreads();
  atomicAdd(&s_rank[lane], r);
  atomicAdd(&s_before[lane], before);
  __syncthreads();
  if (threadIdx.x < kRankHoles && i0 + lane < nh) {
    const int rank = s_rank[lane];
    sorted[rank] = my;
    cum[rank] = (long long)s_before[lane];
    if (rank == nh - 1) cum[nh] = (long long)s_before[lane] + my.len;
  }
}

// First index of [0, n) at which `pred` (true, then false) is false, n if
// none: the CTA tests one pivot per thread and round, two rounds for 2^16
// indices, instead of a chain of log2 n dependent loads.  Every thread calls.
template <class Pred>
__device__ __forceinline__ int block_partition(int n, Pred pred)
{
  int lo = 0, end = n;
  while (lo < end) {
    const int step = (end - lo + (int)blockDim.x - 1) / (int)blockDim.x;
    const int i = lo + ((int)threadIdx.x + 1) * step - 1;
    const int c = __syncthreads_count(i < end && pred(i));
    end = min(end, lo + (c + 1) * step - 1);
    lo += c * step;
  }
  return lo;
}

// Moves every pair stored at or above `hits` (T) into the holes below it, so
// the output is dense [0, T); then writes the result block.  The B pairs to
// move are the data slots of [T, next) in order, and their destinations the
// hole slots below T in order: both are runs, so each CTA takes a piece of
// kMovePiece consecutive moves, finds the hole it starts to fill and the data
// it starts from, and then copies run by run with coalesced accesses.  Bound
// by the latency of a piece's searches and runs, so pieces are short: 3.6M
// moves over 7104 holes take 37 us; with binary searches nested in one another
// and pieces of 8192 they took 96 us.
constexpr int kMovePiece = 2048;

__global__ void __launch_bounds__(256)
    compact_kernel(const Hole* __restrict__ h, const long long* __restrict__ cum,
                   QueryCounters* __restrict__ ctr, long long max_holes, int32_t* fid,
                   int32_t* tid, long long cap, const SortCtrl* __restrict__ sort,
                   crt_query_result* __restrict__ res)
{
  // a window order that was not finished names some windows twice
  const int error = ctr->error ? ctr->error : sort ? sort->error : 0;
  const int nh = (int)min((long long)ctr->nholes, max_holes);
  const long long T = (long long)ctr->hits;
  const long long R = (long long)ctr->next;
  const bool overflow = R > cap;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    res->required = T;
    res->overflow = overflow ? 1 : 0;
    res->count = overflow ? 0 : T;
    res->error = error;
  }
  if (overflow || error || nh == 0) return;
  // holes [0, above) start below T; B hole slots lie below T
  const int above = block_partition(nh, [&](int i) { return h[i].start < T; });
  long long B = 0;
  if (above > 0) B = cum[above - 1] + min(T - h[above - 1].start, h[above - 1].len);
  for (long long r0 = (long long)blockIdx.x * kMovePiece; r0 < B;
       r0 += (long long)gridDim.x * kMovePiece) {
    long long rem = min((long long)kMovePiece, B - r0);
    // destination of move r0: the r0-th hole slot, in the last hole with at
    // most r0 hole slots before it
    int a = block_partition(above, [&](int i) { return cum[i] <= r0; }) - 1;
    if (a < 0) a = 0;
    long long d = h[a].start + (r0 - cum[a]);
    // source of move r0: hole `above + i` has (start - T) - (cum - B) data
    // slots of [T, ...) before it; the r0-th lies past those with at most r0
    int jn = above + block_partition(nh - above, [&](int i) {
      return h[above + i].start - T - (cum[above + i] - B) <= r0;
    });  // next hole above the source
    long long s = T + r0 + (cum[jn] - B);
    while (rem > 0) {
      const long long src_end = jn < nh ? h[jn].start : R;
      const long long dst_end = min(h[a].start + h[a].len, T);
      const long long n = min(rem, min(src_end - s, dst_end - d));
      if (n <= 0 || d < 0 || s + n > R || d + n > T) {  // inconsistent holes: report, stop
        if (threadIdx.x == 0) raise_error(&res->error, CRT_ERR_CUDA);
        break;
      }
      for (long long i = threadIdx.x; i < n; i += blockDim.x) {
        fid[d + i] = fid[s + i];
        tid[d + i] = tid[s + i];
      }
      s += n;
      d += n;
      rem -= n;
      while (jn < nh && s == h[jn].start) {  // skip the hole(s) above the source
        s = h[jn].start + h[jn].len;
        jn++;
      }
      if (rem > 0 && d == dst_end) {
        if (++a >= nh) {
          if (threadIdx.x == 0) raise_error(&res->error, CRT_ERR_CUDA);
          break;
        }
        d = h[a].start;
      }
    }
  }
}

// Window keys and digit histograms: the boxes' Morton key, below two class
// bits when the windows are classed (huge, large, small; the key's two lowest
// bits make room).  The class is by the boxes the window may meet, taken twice:
// at the density of the root's MBR, and at the density where the window lies
// (local_hits), as boxes may lie in clusters, along lines, or far from one
// another.  It only decides which kernel answers the window, but the wrong one is
// slow: small_windows_kernel gives a warp up to 32 neighbours, and with the
// root's density alone, windows on dense data (10M clustered boxes, 300k windows
// of 2600 boxes each) took 10.9 ms there, where one window per warp takes 4.8 and
// the queries before the classes took 6.1.
//   small  at most 256 boxes at the root's density (64, 256 and 1024 measured
//          within 4% on mixed batches) and 128 where it lies: places denser than
//          the rest are where the estimate is worst (256: 50k windows of
//          7300 clustered boxes in a far larger domain 1.59 ms, 128: 1.43).
//   huge   more than 4096 (4k, 8k, 16k boxes and more split took 60k mixed windows
//          1.31, 1.43 and 1.48 ms); where it lies 12k (50k windows of 7300 boxes,
//          all huge by 4k, 1.05 ms, large 1.00).
// A window that is not ordered, or has a NaN, is never small.
constexpr float kSmallHits = 256.f, kSmallLocal = 128.f;
constexpr float kHugeHits = 4096.f, kHugeLocal = 3 * kHugeHits;

// Boxes that the density where the window lies gives it: the boxes in the Morton
// cell that holds its centre and is one to two of its sides wide (in key units),
// times the window's share of the cell.  The count comes from the keys of
// kSamples boxes, every n / kSamples-th one in slot order, read as a piecewise
// linear count over the keys: the boxes are sorted, so in a dense place the
// samples lie close together.  A set in another order gives a useless number,
// and its windows a kernel that may not suit them.  Two searches in shared memory:
// 1M windows 10 to 15 us of 620.
constexpr int kSamples = 8192;
__device__ __forceinline__ int sample_at(int i) { return i + (i >> 5); }  // apart in the banks

__device__ __forceinline__ float local_hits(const uint32_t* s_key, uint32_t key, float w, float h,
                                            float per_sample)
{
  const float side = fmaxf(fmaxf(w, h), 1.f);
  const int k = min(((__float_as_int(side) + 0x7FFFFF) >> 23) - 127, 16);  // 2^k >= side
  const float cell = (float)(1 << k);
  const float part = fminf(1.f, w / cell) * fminf(1.f, h / cell);
  if (k == 16) return (float)kSamples * per_sample * part;
  const uint32_t lo = key & ~((1u << 2 * k) - 1u), hi = lo + (1u << 2 * k) - 1u;
  int a = 0;  // samples below lo (the last one is not looked at)
#pragma unroll
  for (int step = kSamples / 2; step; step >>= 1)
    if (s_key[sample_at(a + step - 1)] < lo) a += step;
  int b = a, step = 1;  // samples up to hi
  while (b + step < kSamples && s_key[sample_at(b + step - 1)] <= hi) {
    b += step;
    step <<= 1;
  }
  for (step >>= 1; step; step >>= 1)
    if (b + step < kSamples && s_key[sample_at(b + step - 1)] <= hi) b += step;
  // between the samples around each end of the cell
  const auto within = [&](int i, uint32_t v) {  // v lies above sample i - 1, not above sample i
    if (i == 0) return 1.f;
    const uint32_t below = s_key[sample_at(i - 1)], span = s_key[sample_at(i)] - below;
    return span ? fminf((float)(v - below) / (float)span, 1.f) : 1.f;
  };
  return fmaxf(0.f, (float)(b - a) + within(b, hi) - within(a, lo)) * per_sample * part;
}

__global__ void window_key_kernel(WindowView W, TreeView T, bool classes, const uint32_t* __restrict__ samples,
                                  QueryCounters* __restrict__ qc, uint32_t* __restrict__ keys,
                                  SortCtrl* __restrict__ ctrl)
{
  __shared__ uint32_t s_key[kSamples + kSamples / 32];
  __shared__ uint32_t sh[kDigits][kBins];
  for (int i = threadIdx.x; i < kDigits * kBins; i += blockDim.x) (&sh[0][0])[i] = 0;
  classes = classes && T.lvl_odd != nullptr && *T.lvl_odd == 0;
  float root_w = 0.f, root_h = 0.f;
  if (classes) {
    root_w = __ldg(T.nxmax) - __ldg(T.nxmin);
    root_h = __ldg(T.nymax) - __ldg(T.nymin);
  }
  const bool local = classes && T.nbox >= kSamples;
  if (local)
    for (int i = 4 * threadIdx.x; i < kSamples; i += 4 * blockDim.x) {
      const uint4 v = *reinterpret_cast<const uint4*>(samples + i);
      uint32_t* at = s_key + sample_at(i);
      at[0] = v.x;
      at[1] = v.y;
      at[2] = v.z;
      at[3] = v.w;
    }
  unsigned huge = 0, large = 0;  // large counts both
  __syncthreads();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < W.n;
       i += (long long)gridDim.x * blockDim.x) {
    const float x1 = W.xmin[i], y1 = W.ymin[i], x2 = W.xmax[i], y2 = W.ymax[i];
    uint32_t k = sort_key(x1, y1, x2, y2);
    bool small = false;
    if (classes) {
      const float part = fminf(1.f, (x2 - x1) / root_w) * fminf(1.f, (y2 - y1) / root_h);
      const bool box = x2 >= x1 && y2 >= y1;
      const float hits = part * (float)T.nbox;
      float near = 0.f;
      if (local && box && hits <= kHugeHits)
        near = local_hits(s_key, k, x2 - x1, y2 - y1, (float)T.nbox / kSamples);
      small = hits <= kSmallHits && near <= kSmallLocal && box;
      const bool big = T.nlev > 1 && !(hits <= kHugeHits && near <= kHugeLocal);
      k = k >> 2 | (small ? 0xC0000000u : big ? 0u : 0x40000000u);
      huge += big;
    }
    large += !small;
    keys[i] = k;
#pragma unroll
    for (int d = 0; d < kDigits; d++) atomicAdd(&sh[d][key_digit(k, d)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kDigits * kBins; i += blockDim.x) {
    uint32_t v = (&sh[0][0])[i];
    if (v) atomicAdd(&ctrl->hist[i], v);
  }
  large = __reduce_add_sync(0xffffffffu, large);
  huge = __reduce_add_sync(0xffffffffu, huge);
  if (large && (threadIdx.x & 31) == 0) atomicAdd(&qc->nlarge, (unsigned long long)large);
  if (huge && (threadIdx.x & 31) == 0) atomicAdd(&qc->nhuge, (unsigned long long)huge);
  sort_plan(ctrl, W.n, kDigits);
}

__global__ void set_nq_kernel(QueryCounters* ctr, long long nq) { ctr->nq = (unsigned long long)nq; }

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static TreeView make_view(const crt_rtree_f32& rt, const crt_bbox_f32& rb)
{
  TreeView T;
  T.nxmin = rt.xmin; T.nymin = rt.ymin; T.nxmax = rt.xmax; T.nymax = rt.ymax;
  T.npos = rt.pos; T.nlen = rt.len; T.rsz = rt.sz; T.fanout = rt.fanout;
  T.bxmin = rb.xmin; T.bymin = rb.ymin; T.bxmax = rb.xmax; T.bymax = rb.ymax; T.bid = rb.id;
  T.nbox = rb.sz;
  T.nlev = 0;
  T.lvl_first = nullptr;
  T.lvl_span = nullptr;
  T.lvl_odd = nullptr;
  return T;
}

// The tables hold only for the reference's packed layout, which a tree has
// exactly when its node count is the packed count for its box count.
LevelTables level_tables(const crt_rtree_f32& rt, int64_t nbox)
{
  LevelTables t;
  if (rt.sz <= 0 || rt.fanout < 2 || rt.fanout > kLenMask) return t;
  std::vector<int64_t> lv;
  const int L = tree_levels(nbox, rt.fanout, lv);
  if (L <= 0 || L > kMaxLevels) return t;
  int64_t rsz = 0;
  for (auto x : lv) rsz += x;
  if (rsz != rt.sz) return t;
  int64_t start = rsz;
  long long sp = rt.fanout;
  for (int h = 0; h < L; h++) {
    start -= lv[h];
    t.first[h] = (int)start;
    t.span[h] = sp;
    sp = sp > (1ll << 40) ? sp : sp * rt.fanout;
  }
  t.nlev = L;
  return t;
}

// One launch prepares a query: CTA 0 writes the tables (passed by value, so
// the host never waits on a pageable transfer and the write can be recorded in
// a CUDA graph) and the window count, and all CTAs scan the boxes for one that
// is not ordinary (*odd was zeroed before; every thread that sees one stores
// the same value).  kVec: the four arrays are 16-byte aligned; eight 16-byte
// loads per thread are then in flight (10M boxes: 53 us with 4-byte loads, 30
// so; the read alone takes 25).  Given `samples`, also the keys of kSamples boxes.
template <bool kVec>
__global__ void __launch_bounds__(256)
    prepare_kernel(LevelTables t, int* __restrict__ first, long long* __restrict__ span,
                   int* __restrict__ odd, const float* __restrict__ xmin,
                   const float* __restrict__ ymin, const float* __restrict__ xmax,
                   const float* __restrict__ ymax, int64_t n, QueryCounters* __restrict__ ctr,
                   long long nq, uint32_t* __restrict__ samples)
{
  if (blockIdx.x == 0) {
    if (first && threadIdx.x < kMaxLevels) {
      first[threadIdx.x] = t.first[threadIdx.x];
      span[threadIdx.x] = t.span[threadIdx.x];
    }
    if (ctr && threadIdx.x == 0) ctr->nq = (unsigned long long)nq;
  }
  if (n <= 0) return;
  bool bad = false;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t at = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (samples && n >= kSamples)
    for (int64_t i = at; i < kSamples; i += stride) {
      const int64_t j = i * n / kSamples;
      samples[i] = sort_key(xmin[j], ymin[j], xmax[j], ymax[j]);
    }
  int64_t done = 0;
  if (kVec) {
    const auto odd4 = [](float4 a, float4 b) {
      return !(a.x <= b.x && a.y <= b.y && a.z <= b.z && a.w <= b.w);
    };
    const int64_t n4 = n >> 2;
    for (int64_t i = at; i < n4; i += 2 * stride) {
      const int64_t j = min(i + stride, n4 - 1);
      const float4 a0 = reinterpret_cast<const float4*>(xmin)[i], b0 = reinterpret_cast<const float4*>(xmax)[i];
      const float4 c0 = reinterpret_cast<const float4*>(ymin)[i], d0 = reinterpret_cast<const float4*>(ymax)[i];
      const float4 a1 = reinterpret_cast<const float4*>(xmin)[j], b1 = reinterpret_cast<const float4*>(xmax)[j];
      const float4 c1 = reinterpret_cast<const float4*>(ymin)[j], d1 = reinterpret_cast<const float4*>(ymax)[j];
      bad |= odd4(a0, b0) | odd4(c0, d0) | odd4(a1, b1) | odd4(c1, d1);
    }
    done = n4 << 2;
  }
  for (int64_t i = done + at; i < n; i += stride)
    bad |= !(xmin[i] <= xmax[i] && ymin[i] <= ymax[i]);
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) *odd = 1;
}

static void launch_prepare(const LevelTables& t, int* first, long long* span, int* odd,
                           const float* xmin, const float* ymin, const float* xmax,
                           const float* ymax, int64_t n, QueryCounters* ctr, int64_t nq,
                           uint32_t* samples, cudaStream_t stream)
{
  const bool vec = ((((uintptr_t)xmin) | ((uintptr_t)ymin) | ((uintptr_t)xmax) | ((uintptr_t)ymax)) & 15) == 0;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(cdiv(n, vec ? 2048 : 256), (int64_t)sm_count() * 8));
  if (vec)
    prepare_kernel<true><<<grid, 256, 0, stream>>>(t, first, span, odd, xmin, ymin, xmax, ymax, n, ctr, nq, samples);
  else
    prepare_kernel<false><<<grid, 256, 0, stream>>>(t, first, span, odd, xmin, ymin, xmax, ymax, n, ctr, nq, samples);
  CRT_LAUNCHED(1);
}

void launch_odd_boxes(const float* xmin, const float* ymin, const float* xmax, const float* ymax,
                      int64_t n, int* odd, cudaStream_t stream)
{
  cudaMemsetAsync(odd, 0, sizeof(int), stream);
  if (n > 0)
    launch_prepare(LevelTables(), nullptr, nullptr, odd, xmin, ymin, xmax, ymax, n, nullptr, 0, nullptr, stream);
}

// Puts the tables at `dev` (kLevelTableBytes, 8-byte aligned, its flag word
// zeroed by the caller), checks the view's boxes for the shortcut, points the
// view at both, and sets ctr->nq when ctr is given.
static void attach_levels(TreeView& T, const LevelTables& t, void* dev, QueryCounters* ctr, int64_t nq,
                          uint32_t* samples, cudaStream_t stream)
{
  if (t.nlev == 0) {
    if (ctr) launch_prepare(t, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, ctr, nq, nullptr, stream);
    return;
  }
  int* first = (int*)dev;
  long long* span = (long long*)((char*)dev + sizeof(int) * kMaxLevels);
  int* odd = (int*)((char*)dev + kLevelOddOffset);
  launch_prepare(t, first, span, odd, T.bxmin, T.bymin, T.bxmax, T.bymax, T.nbox, ctr, nq, samples, stream);
  T.nlev = t.nlev;
  T.lvl_first = first;
  T.lvl_span = span;
  T.lvl_odd = odd;
}

// Counters and tables, the head of every query's scratch: zeroed in one piece.
constexpr size_t kHeadTables = 256;
constexpr size_t kHeadBytes = (kHeadTables + kLevelTableBytes + 255) / 256 * 256;

// Number of levels of a tree with R_sz nodes over nbox boxes at this fanout
// (1 when the root is the only level).
static int levels_of(int64_t nbox, int fanout)
{
  std::vector<int64_t> lv;
  int L = tree_levels(std::max<int64_t>(nbox, 1), std::max(fanout, 2), lv);
  return std::max(L, 1);
}

struct TraversalShape {
  int K;
  int stack_cap;
};

static TraversalShape traversal_shape(int64_t nbox, int fanout)
{
  const int L = levels_of(nbox, fanout);
  TraversalShape s;
  s.K = fanout <= 32 ? std::max(1, 32 / fanout) : 1;
  // at most K*fanout entries per pushed level (levels 1 .. L-1), plus the root
  s.stack_cap = (L - 1) * s.K * fanout + 1;
  s.stack_cap = (s.stack_cap + 31) / 32 * 32;
  return s;
}

// Chunk of a query that names none; the capacity it asks for (query_capacity)
// leaves room for 4096-slot chunks.  A chunk's unused end is moved by the
// compaction: 213M pairs of a road batch leave 72 us of moves at 1024 slots,
// 145 at 4096, with the same traversal time.
constexpr int kDefaultChunk = 1024;
constexpr int kDefaultChunkRoom = 4096;

// Persistent traversal variants: CTA width and CTAs per SM, which fix the
// register budget (65536 / (threads x CTAs)).  Wider CTAs share one staged
// copy of the top levels among more warps; narrower ones get more registers.
struct PersistVariant {
  int threads;
  int min_blocks;
  bool share;         // range sharing
  const void* fn[2];  // without and with queues of contained runs
};

#define CRT_VARIANT(T, B, S) \
  {T, B, S, {(const void*)persistent_kernel<T, B, S, false>, (const void*)persistent_kernel<T, B, S, true>}}
static const PersistVariant kVariants[] = {
    CRT_VARIANT(1024, 2, false),  // 64 warps/SM, 32 registers
    CRT_VARIANT(512, 3, false),   // 48 warps/SM, 40 registers
    CRT_VARIANT(256, 4, true),    // 32 warps/SM, 64 registers
};

static const PersistVariant& variant_for(int warps_per_cta)
{
  for (const auto& v : kVariants)
    if (v.threads / 32 == warps_per_cta) return v;
  return kVariants[2];  // default: 8 warps per CTA
}

// Shared memory of the persistent traversal: the staged top levels (6 arrays),
// one frontier stack per warp and the warps' queues of contained runs.  When
// that does not let the variant's CTAs share an SM, staging is dropped, then the
// CTAs per SM, and last the queues (fanout 2 in 32-warp CTAs above 2^25 boxes);
// a stack too deep for that too is an error.  The queues go last: where they
// cost one of an SM's CTAs (deep trees of fanout 2 to 4) batches of 50k mixed
// windows took, with the queues and without: fanout 3, 10M boxes, 32 warps 688
// and 711 us; fanout 2, 200k boxes, 16 warps 155 and 162; fanout 4, 30M boxes,
// 32 warps 1090 and 1128 (100k windows of one size, side 1e-2: 1960 and 1815,
// 274 and 285, 3620 and 3600).
struct PersistShape {
  const PersistVariant* v;
  int stage_n;
  bool queue;
  size_t smem;
  const void* fn() const { return v->fn[queue]; }
};

static PersistShape persist_shape(int stack_cap, int stage_n, int warps_per_cta)
{
  const PersistVariant& v = variant_for(warps_per_cta);
  const size_t per_sm = 227 * 1024;
  const int warps = v.threads / 32;
  for (int pass = 0; pass < 4; pass++) {
    const int sn = pass == 0 ? stage_n : 0;
    const bool queue = pass < 3;
    const size_t smem = (size_t)sn * 24 + (size_t)warps * (stack_cap * sizeof(FrontierEntry) +
                                                           (queue ? kQueue * sizeof(int2) : 0));
    const size_t limit = pass < 2 ? per_sm / v.min_blocks - 1024 : 220 * 1024;
    if (smem <= limit) return PersistShape{&v, sn, queue, smem};
  }
  return PersistShape{nullptr, 0, false, 0};
}

static int persistent_grid(const PersistShape& p)
{
  int per_sm = 0;
  allow_smem(p.fn(), 1024);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p.fn(), p.v->threads, p.smem);
  if (per_sm < 1) per_sm = 1;
  return per_sm * sm_count();
}

// The shape above for tests: {shared memory (0: refused), nodes staged, whether
// the warps have queues}.
void persist_shape_of(int64_t nbox, int fanout, int stage_n, int warps_per_cta, int out[3])
{
  const PersistShape p = persist_shape(traversal_shape(nbox, fanout).stack_cap, stage_n, warps_per_cta);
  out[0] = (int)p.smem;
  out[1] = p.stage_n;
  out[2] = p.queue;
}

int64_t query_capacity(int64_t pairs, const crt_query_opts& o)
{
  if (o.mode == CRT_QUERY_PLAIN) return pairs;
  const int chunk = o.chunk > 0 ? o.chunk : kDefaultChunkRoom;
  // every resident warp may leave one partly used chunk
  const int64_t warps = (int64_t)sm_count() * 64;  // resident warps per SM at most
  return pairs + warps * chunk;
}

struct PersistScratch {
  QueryCounters* ctr;
  Hole* holes;
  Hole* sorted;
  long long* cum;
  void* sort_zero;
  SortCols cols;
  uint32_t* samples;  // kSamples keys of the boxes
  long long max_holes;
  JobQueue* jobs;
  size_t bytes;
};

static size_t persist_scratch_bytes(int64_t max_nq, long long max_holes, bool sort)
{
  auto al = [](size_t x) { return (x + 255) / 256 * 256; };
  size_t b = kHeadBytes + 2 * al(sizeof(Hole) * max_holes) +
             al(sizeof(long long) * (max_holes + 1)) + al(kJobQueueBytes);
  if (sort) b += al(4 * kSamples) + al(sort_zero_bytes(max_nq)) + 4 * al(4 * (size_t)std::max<int64_t>(max_nq, 1));
  return b;
}

static void persist_scratch_carve(char* base, int64_t max_nq, long long max_holes, bool sort,
                                  PersistScratch& S)
{
  auto al = [](size_t x) { return (x + 255) / 256 * 256; };
  size_t off = 0;
  S.ctr = (QueryCounters*)(base + off); off += kHeadBytes;
  S.holes = (Hole*)(base + off); off += al(sizeof(Hole) * max_holes);
  S.sorted = (Hole*)(base + off); off += al(sizeof(Hole) * max_holes);
  S.cum = (long long*)(base + off); off += al(sizeof(long long) * (max_holes + 1));
  S.jobs = (JobQueue*)(base + off); off += al(kJobQueueBytes);
  S.sort_zero = nullptr;
  S.cols = SortCols{};
  S.samples = nullptr;
  if (sort) {
    S.sort_zero = base + off; off += al(sort_zero_bytes(max_nq));
    size_t kv = al(4 * (size_t)std::max<int64_t>(max_nq, 1));
    S.cols.key[0] = (uint32_t*)(base + off); off += kv;
    S.cols.key[1] = (uint32_t*)(base + off); off += kv;
    S.cols.val[0] = (uint32_t*)(base + off); off += kv;
    S.cols.val[1] = (uint32_t*)(base + off); off += kv;
    S.samples = (uint32_t*)(base + off); off += al(4 * kSamples);
    S.cols.make_values = S.cols.drop_keys = true;
  }
  S.max_holes = max_holes;
  S.bytes = off;
}

// A persistent query is three stages on one stream, none synchronising the
// host: `pre` (order the windows; the counters were reset), the traversal kernel,
// and `post` (sort the unused chunk ends, compact, write the result block).
// A plan records all three as one CUDA graph.
static void enqueue_pre(const TreeView& T, const WindowView& W, int64_t max_nq,
                        const PersistScratch& S, bool sort, bool classes, bool share,
                        cudaStream_t stream)
{
  // the job queue's ready flags (where ranges are shared) and the sort's zeroed
  // block, which follows them
  const bool order = sort && max_nq > 0;
  char* z0 = share ? (char*)S.jobs : (char*)S.sort_zero;
  char* z1 = order ? (char*)S.sort_zero + sort_zero_bytes(max_nq) : (char*)S.jobs + kJobQueueBytes;
  if (share || order) cudaMemsetAsync(z0, 0, (size_t)(z1 - z0), stream);
  if (order) {
    const int sms = sm_count();
    int g = (int)std::min<int64_t>(cdiv(max_nq, 256), (int64_t)sms * 4);
    window_key_kernel<<<std::max(g, 1), 256, 0, stream>>>(W, T, classes, S.samples, S.ctr, S.cols.key[0],
                                                          sort_ctrl(S.sort_zero));
    sort_passes(S.cols, W.n, kDigits, S.sort_zero, stream);
    CRT_LAUNCHED(1);
  }
}

// Nodes of this height are dealt out among the warps sharing a window: the
// first height whose nodes hold 256 boxes, at most the root's children's.
static int split_height(const TreeView& T)
{
  int h = 0;
  for (int64_t span = T.fanout; span < 256 && h < T.nlev - 2; span *= T.fanout) h++;
  return h;
}

struct TraverseLaunch {
  PersistParams P;
  size_t smem;
  int grid;
  int threads;
  const void* fn;
  // the small windows' launch (P.classes)
  PersistParams small;
  int small_grid;
  int small_warp_bytes;
};

// Whether the windows are classed: sorted, and a packed tree of fanout <= 32
// whose boxes were scanned (a box that is not ordinary makes every window
// large, on the device).
static bool window_classes(const TreeView& T, bool sort)
{
  return sort && T.nlev > 0 && T.lvl_odd != nullptr && T.fanout <= 32 && T.rsz > 0;
}

static TraverseLaunch make_traverse(const TreeView& T, const WindowView& W,
                                    const PersistScratch& S, bool sort, int stage_n,
                                    int32_t* fid, int32_t* tid, long long cap, int chunk,
                                    int warps_per_cta, int parts)
{
  const TraversalShape sh = traversal_shape(T.nbox, T.fanout);
  const PersistShape ps = persist_shape(sh.stack_cap, stage_n, warps_per_cta);
  TraverseLaunch L;
  PersistParams& P = L.P;
  P.T = T;
  P.W = W;
  P.order0 = S.cols.val[0];
  P.order1 = S.cols.val[1];
  P.sort_ctrl = sort ? sort_ctrl(S.sort_zero) : nullptr;
  P.K = sh.K;
  P.stack_cap = sh.stack_cap;
  P.stage_n = ps.stage_n;
  P.parts = parts;
  P.classes = window_classes(T, sort);
  P.split_height = split_height(T);
  P.chunk = chunk;
  P.fid = fid;
  P.tid = tid;
  P.cap = cap;
  P.ctr = S.ctr;
  P.holes = S.holes;
  P.max_holes = S.max_holes;
  P.jobs = S.jobs;
  L.smem = ps.smem;
  L.threads = ps.v->threads;
  L.fn = ps.fn();
  L.grid = persistent_grid(ps);
  if (P.classes) {
    L.small = P;
    // as one window's stack, with kSmallSets sets per step, a refill and the
    // entries left when it ran
    const int cap = (levels_of(T.nbox, T.fanout) - 1) * kSmallSets * sh.K * T.fanout + kGroupWindows +
                    kSmallSets * sh.K;
    L.small.stack_cap = (cap + 31) / 32 * 32;
    L.small_warp_bytes = (int)SmallSmem::bytes(L.small.stack_cap);
    const size_t smem = (size_t)L.small_warp_bytes * kSmallWarps;
    int per_sm = 0;
    allow_smem(small_windows_kernel);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, small_windows_kernel, kSmallWarps * 32, smem);
    L.small_grid = std::max(per_sm, 1) * sm_count();
  }
  return L;
}

static cudaError_t launch_traverse(const TraverseLaunch& L, cudaStream_t stream)
{
  ProfScope ps("traverse_persistent", stream);
  void* args[] = {(void*)&L.P};
  cudaError_t e = cudaLaunchKernel(L.fn, dim3(L.grid), dim3(L.threads), args, L.smem, stream);
  CRT_LAUNCHED(1);
  if (e == cudaSuccess && L.P.classes) {
    // its CTAs start as the persistent kernel's leave (they share nothing but
    // the output counters), and end after it: 60k mixed windows 1.05 -> 1.01
    // ms, 5k 0.26 -> 0.24
    e = launch_beside(small_windows_kernel, (unsigned)L.small_grid, kSmallWarps * 32,
                      (size_t)L.small_warp_bytes * kSmallWarps, stream, L.small, L.small_warp_bytes);
    CRT_LAUNCHED(1);
  }
  return e;
}

static void enqueue_post(const PersistScratch& S, int32_t* fid, int32_t* tid, long long cap,
                         crt_query_result* res, cudaStream_t stream)
{
  const int sms = sm_count();
  hole_rank_kernel<<<std::max(1, (int)cdiv(S.max_holes, kRankHoles)), kRankWarps * 32, 0, stream>>>(
      S.holes, S.sorted, S.cum, S.ctr, S.max_holes);
  compact_kernel<<<sms * 8, 256, 0, stream>>>(S.sorted, S.cum, S.ctr, S.max_holes, fid, tid, cap,
                                              S.sort_zero ? sort_ctrl(S.sort_zero) : nullptr, res);
  CRT_LAUNCHED(2);
}

// Nodes of the root and the `levels` whole tree levels below it, rounded up
// to a multiple of 4 (16-byte bulk copies; the extra nodes are staged too)
// and at most R_sz rounded down to one; 0 when staging is off or the node
// arrays are not 16-byte aligned.
static int stage_nodes_for(const crt_rtree_f32& rt, int64_t nbox, int levels)
{
  if (levels <= 0 || rt.sz <= 0) return 0;
  const void* arrs[6] = {rt.xmin, rt.ymin, rt.xmax, rt.ymax, rt.pos, rt.len};
  for (auto p : arrs)
    if (((uintptr_t)p & 15u) != 0) return 0;
  std::vector<int64_t> lv;  // leaf-parent level first, root last
  const int L = tree_levels(std::max<int64_t>(nbox, 1), std::max(rt.fanout, 2), lv);
  int64_t n = 0;
  for (int i = 0; i <= levels && i < L; i++) n += lv[L - 1 - i];
  n = std::min<int64_t>((int64_t)rt.sz & ~(int64_t)3, (n + 3) & ~(int64_t)3);
  return (int)n;
}

// The deepest staging (at most `levels` levels) whose nodes fit beside the
// warps' stacks at the variant's full occupancy.
static int fit_stage_nodes(const crt_rtree_f32& rt, int64_t nbox, int levels, int stack_cap,
                           int warps_per_cta)
{
  for (int k = levels; k > 0; k--) {
    const int sn = stage_nodes_for(rt, nbox, k);
    if (sn > 0 && persist_shape(stack_cap, sn, warps_per_cta).stage_n == sn) return sn;
  }
  return 0;
}

static long long max_holes_for(int stack_cap, int stage_n, int warps_per_cta)
{
  const PersistShape ps = persist_shape(stack_cap, stage_n, warps_per_cta);
  return (long long)persistent_grid(ps) * (ps.v->threads / 32);
}

// Warps per window of the persistent form (0 = 1); -1 for an unsupported value.
static int window_parts(const crt_query_opts& o)
{
  const int w = o.warps_per_window <= 0 ? 1 : o.warps_per_window;
  return (w == 1 || w == 2 || w == 4) ? w : -1;
}

// Whether the dense form's shared memory fits a CTA (it stages pairs beside
// the stacks; a fanout in the thousands leaves no room).
static size_t dense_smem(int stack_cap)
{
  return (size_t)kPlainWarps * (stack_cap + kSmallStage) * sizeof(FrontierEntry);
}
bool query_dense_fits(int64_t nbox, int fanout)
{
  return dense_smem(traversal_shape(nbox, fanout).stack_cap) <= 227 * 1024;
}

// The dense form into caller-owned columns of `cap` slots each: *pairs is the
// pair count, more than cap when the output was too small (nothing past it is
// written).  Synchronises the stream.
int query_dense(const crt_rtree_f32& rt, const crt_bbox_f32& rbox, const crt_bbox_f32& qbox,
                int32_t* fid, int32_t* tid, int64_t cap, int64_t* pairs, cudaStream_t stream)
{
  NvtxRange range("crt_query_dense");
  *pairs = 0;
  if (qbox.sz <= 0) return CRT_OK;
  TreeView T = make_view(rt, rbox);
  WindowView W{qbox.xmin, qbox.ymin, qbox.xmax, qbox.ymax, qbox.sz};
  const TraversalShape sh = traversal_shape(rbox.sz, rt.fanout);
  char* scr = nullptr;
  if (cudaMallocAsync((void**)&scr, kHeadBytes, stream) != cudaSuccess) {
    cudaGetLastError();
    return fail(CRT_ERR_OOM, "query: scratch allocation failed");
  }
  QueryCounters* ctr = (QueryCounters*)scr;
  cudaMemsetAsync(scr, 0, kHeadBytes, stream);
  attach_levels(T, level_tables(rt, rbox.sz), scr + kHeadTables, nullptr, 0, nullptr, stream);
  // kPlainWarps x 4 warps per SM is what the traversal's shared memory allows
  const bool few = T.nlev > 1 && W.n * kDenseParts <= (int64_t)sm_count() * kPlainWarps * 4;
  const int parts = few ? kDenseParts : 1;
  const size_t smem = dense_smem(sh.stack_cap);
  allow_smem(dense_kernel);
  {
    ProfScope ps("traverse_dense", stream);
    dense_kernel<<<(unsigned)cdiv(W.n * parts, kPlainWarps), kPlainWarps * 32, smem, stream>>>(
        T, W, sh.K, sh.stack_cap, parts, split_height(T), fid, tid, cap, ctr);
    CRT_LAUNCHED(1);
  }
  QueryCounters h{};
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, ctr, sizeof(h), cudaMemcpyDeviceToHost, stream);
  cudaFreeAsync(scr, stream);
  const cudaError_t es = cudaStreamSynchronize(stream);
  if (e == cudaSuccess) e = es;
  if (e != cudaSuccess) return cuda_fail(e, "query");
  if (h.error) return fail(h.error, "query: device-side error");
  *pairs = (int64_t)h.next;
  return CRT_OK;
}

// Scratch of a plain query: the head (counters and tables) and behind it the
// scan's status words, one count per window, the offsets.
struct PlainScratch {
  char* head;
  unsigned long long* status;
  long long* counts;
  long long* offsets;
};
constexpr int64_t plain_tiles(int64_t nq) { return nq < 1 ? 1 : (nq + kScanThreads - 1) / kScanThreads; }
// Bytes of the head and the status words, zeroed together.
constexpr size_t plain_zero_bytes(int64_t nq)
{
  return (kHeadBytes + 8 * (size_t)plain_tiles(nq) + 255) / 256 * 256;
}

// The plain query's launches: reset, prepare, count, scan (with the result
// block), write.
static void enqueue_plain(TreeView T, const LevelTables& lt, const WindowView& W, const PlainScratch& S,
                          int32_t* fid, int32_t* tid, int64_t capacity, crt_query_result* res,
                          cudaStream_t stream)
{
  const TraversalShape sh = traversal_shape(T.nbox, T.fanout);
  QueryCounters* ctr = (QueryCounters*)S.head;
  const int64_t nq = W.n;
  cudaMemsetAsync(S.head, 0, plain_zero_bytes(nq), stream);
  attach_levels(T, lt, S.head + kHeadTables, nullptr, 0, nullptr, stream);
  const size_t smem = (size_t)kPlainWarps * sh.stack_cap * sizeof(FrontierEntry);
  allow_smem(plain_count_kernel);
  allow_smem(plain_write_kernel);
  const unsigned g = (unsigned)cdiv(nq, kPlainWarps);
  if (nq > 0) {
    ProfScope ps("traverse_plain", stream);
    plain_count_kernel<<<g, kPlainWarps * 32, smem, stream>>>(T, W, sh.K, sh.stack_cap, S.counts, ctr);
    CRT_LAUNCHED(1);
  }
  scan_kernel<<<(unsigned)plain_tiles(nq), kScanThreads, 0, stream>>>(
      S.counts, nq, S.offsets, S.status, ctr, capacity, res);
  CRT_LAUNCHED(1);
  if (nq > 0) {
    ProfScope ps("traverse_plain", stream);
    plain_write_kernel<<<g, kPlainWarps * 32, smem, stream>>>(T, W, sh.K, sh.stack_cap, S.offsets, fid,
                                                              tid, capacity, ctr, &res->error);
    CRT_LAUNCHED(1);
  }
}

int query_into(const crt_rtree_f32& rt, const crt_bbox_f32& rbox, const crt_bbox_f32& qbox,
               int32_t* fid, int32_t* tid, int64_t capacity, crt_query_result* d_result,
               int64_t* d_offsets, const crt_query_opts& opts, cudaStream_t stream)
{
  NvtxRange range(opts.mode == CRT_QUERY_PLAIN ? "crt_query_plain" : "crt_query_persistent");
  if (!d_result) return fail(CRT_ERR_INVALID_ARG, "query: result block is required");
  if (qbox.sz < 0 || rbox.sz < 0 || rt.sz < 0)
    return fail(CRT_ERR_INVALID_ARG, "query: negative size");
  if (rt.sz > 0 && rt.fanout < 2) return fail(CRT_ERR_INVALID_ARG, "query: fanout < 2");
  if (capacity > 0 && !fid) return fail(CRT_ERR_INVALID_ARG, "query: null output");
  // without a window column the output is CSR: only the plain form with offsets
  if (capacity > 0 && !tid && (opts.mode != CRT_QUERY_PLAIN || !d_offsets))
    return fail(CRT_ERR_INVALID_ARG, "query: null window column outside PLAIN with offsets");
  TreeView T = make_view(rt, rbox);
  const LevelTables lt = opts.no_contain ? LevelTables() : level_tables(rt, rbox.sz);
  WindowView W{qbox.xmin, qbox.ymin, qbox.xmax, qbox.ymax, qbox.sz};
  const int64_t nq = qbox.sz;

  if (opts.mode == CRT_QUERY_PLAIN) {
    const size_t zero = plain_zero_bytes(nq);
    const size_t per = 8 * (size_t)(nq + 1);
    char* scr = nullptr;
    if (cudaMallocAsync((void**)&scr, zero + (d_offsets ? 1 : 2) * per, stream) != cudaSuccess) {
      cudaGetLastError();
      return fail(CRT_ERR_OOM, "query: scratch allocation failed");
    }
    PlainScratch S;
    S.head = scr;
    S.status = (unsigned long long*)(scr + kHeadBytes);
    S.counts = (long long*)(scr + zero);
    S.offsets = d_offsets ? (long long*)d_offsets : (long long*)(scr + zero + per);
    enqueue_plain(T, lt, W, S, fid, tid, capacity, d_result, stream);
    cudaFreeAsync(scr, stream);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "query (plain)");
    return CRT_OK;
  }

  // persistent
  const TraversalShape sh = traversal_shape(rbox.sz, rt.fanout);
  const bool sort = opts.sort_windows != 0 && nq > 1;
  const int stage_n = fit_stage_nodes(rt, rbox.sz, opts.stage_levels, sh.stack_cap,
                                      opts.warps_per_cta);
  const int chunk = opts.chunk >= 64 ? opts.chunk : kDefaultChunk;
  const int parts = window_parts(opts);
  if (parts < 0) return fail(CRT_ERR_INVALID_ARG, "query: warps_per_window must be 1, 2 or 4");
  if (!persist_shape(sh.stack_cap, stage_n, opts.warps_per_cta).v)
    return fail(CRT_ERR_NOT_SUPPORTED, "query: traversal stack too large");
  const long long max_holes = max_holes_for(sh.stack_cap, stage_n, opts.warps_per_cta);
  const size_t bytes = persist_scratch_bytes(nq, max_holes, sort);
  char* scr = nullptr;
  if (cudaMallocAsync((void**)&scr, bytes, stream) != cudaSuccess) {
    cudaGetLastError();
    return fail(CRT_ERR_OOM, "query: scratch allocation failed");
  }
  PersistScratch S;
  persist_scratch_carve(scr, nq, max_holes, sort, S);
  cudaMemsetAsync(scr, 0, kHeadBytes, stream);
  attach_levels(T, lt, scr + kHeadTables, S.ctr, nq, S.samples, stream);
  enqueue_pre(T, W, nq, S, sort, window_classes(T, sort), variant_for(opts.warps_per_cta).share, stream);
  cudaError_t e = launch_traverse(make_traverse(T, W, S, sort, stage_n, fid, tid, capacity, chunk,
                                                opts.warps_per_cta, parts),
                                  stream);
  enqueue_post(S, fid, tid, capacity, d_result, stream);
  cudaFreeAsync(scr, stream);
  if (e == cudaSuccess) e = cudaGetLastError();
  else cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "query (persistent)");
  return CRT_OK;
}

// ---------------------------------------------------------------------------
// Plain query without allocation
// ---------------------------------------------------------------------------
// Some callers cannot allocate device memory while they run: a process whose
// device memory is owned by another allocator (an engine that reserves the
// GPU's memory up front and must account for every byte), or a
// latency-critical loop that cannot afford cudaMalloc's implicit device
// synchronisation.  For them the plain query has a variant whose scratch --
// counters, per-window counts, scan partials, offsets and containment tables
// -- lives in this fixed device array instead of the stream-ordered pool.
//
// The array is a module global: every GPU that loads the library holds its
// 1 MiB until the process exits.  In host code `g_noalloc_scratch` is only a
// host-side stand-in; the device address comes from cudaGetSymbolAddress,
// looked up once per device (the first call on a device does it, with that
// device current).  All calls share the array and it keeps the last call's
// contents, so the counters are cleared on every call; calls whose work
// overlaps on the GPU (different streams, or another thread) race on it and
// must be serialised by the caller.
constexpr int64_t kNoAllocMaxWindows = 1 << 16;
constexpr size_t kNoAllocCountsOff = plain_zero_bytes(kNoAllocMaxWindows);
constexpr size_t kNoAllocOffsetsOff = kNoAllocCountsOff + 8 * (size_t)kNoAllocMaxWindows;
constexpr size_t kNoAllocBytes =
    (kNoAllocOffsetsOff + 8 * (size_t)(kNoAllocMaxWindows + 1) + 255) / 256 * 256;
static_assert(kNoAllocBytes <= (1u << 20) + 4096, "no-alloc scratch stays near 1 MiB");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

static int noalloc_scratch_address(char** out)
{
  static std::mutex mu;
  static std::vector<std::pair<int, char*>> addr;  // device -> device address of the array
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "query_plain_noalloc: cudaGetDevice");
  std::lock_guard<std::mutex> lk(mu);
  for (auto& a : addr)
    if (a.first == dev) {
      *out = a.second;
      return CRT_OK;
    }
  void* p = nullptr;
  e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess) return cuda_fail(e, "query_plain_noalloc: cudaGetSymbolAddress");
  addr.emplace_back(dev, (char*)p);
  *out = (char*)p;
  return CRT_OK;
}

int query_plain_noalloc(const crt_rtree_f32& rt, const crt_bbox_f32& rbox,
                        const crt_bbox_f32& qbox, int32_t* fid, int32_t* tid, int64_t capacity,
                        crt_query_result* d_result, cudaStream_t stream)
{
  if (!d_result) return fail(CRT_ERR_INVALID_ARG, "query_plain_noalloc: result block is required");
  if (qbox.sz < 0 || rbox.sz < 0 || rt.sz < 0 || capacity < 0)
    return fail(CRT_ERR_INVALID_ARG, "query_plain_noalloc: negative size");
  if (qbox.sz > kNoAllocMaxWindows)
    return fail(CRT_ERR_INVALID_ARG,
                "query_plain_noalloc: at most 65536 windows per call (fixed scratch); "
                "split the batch or use crt_query_into_f32");
  if (rt.sz > 0 && rt.fanout < 2) return fail(CRT_ERR_INVALID_ARG, "query_plain_noalloc: fanout < 2");
  if (capacity > 0 && (!fid || !tid))
    return fail(CRT_ERR_INVALID_ARG, "query_plain_noalloc: null output");
  char* scr = nullptr;
  int rc = noalloc_scratch_address(&scr);
  if (rc != CRT_OK) return rc;
  TreeView T = make_view(rt, rbox);
  WindowView W{qbox.xmin, qbox.ymin, qbox.xmax, qbox.ymax, qbox.sz};
  PlainScratch S;
  S.head = scr;
  S.status = (unsigned long long*)(scr + kHeadBytes);
  S.counts = (long long*)(scr + kNoAllocCountsOff);
  S.offsets = (long long*)(scr + kNoAllocOffsetsOff);
  enqueue_plain(T, level_tables(rt, rbox.sz), W, S, fid, tid, capacity, d_result, stream);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "query_plain_noalloc");
  return CRT_OK;
}

// The windows' classes for tests: {huge, large, small} windows of a sorted query
// with the library's defaults.
int window_class_counts(const crt_rtree_f32& rt, const crt_bbox_f32& rbox, const crt_bbox_f32& qbox,
                        int64_t out[3], cudaStream_t stream)
{
  TreeView T = make_view(rt, rbox);
  const WindowView W{qbox.xmin, qbox.ymin, qbox.xmax, qbox.ymax, qbox.sz};
  char* scr = nullptr;
  if (cudaMallocAsync((void**)&scr, persist_scratch_bytes(W.n, 1, true), stream) != cudaSuccess) {
    cudaGetLastError();
    return fail(CRT_ERR_OOM, "window_class_counts: scratch allocation failed");
  }
  PersistScratch S;
  persist_scratch_carve(scr, W.n, 1, true, S);
  cudaMemsetAsync(scr, 0, kHeadBytes, stream);
  attach_levels(T, level_tables(rt, rbox.sz), scr + kHeadTables, S.ctr, W.n, S.samples, stream);
  enqueue_pre(T, W, W.n, S, true, window_classes(T, true), false, stream);
  QueryCounters c{};
  cudaMemcpyAsync(&c, S.ctr, sizeof(c), cudaMemcpyDeviceToHost, stream);
  cudaFreeAsync(scr, stream);
  const cudaError_t e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_fail(e, "window_class_counts");
  out[0] = (int64_t)c.nhuge;
  out[1] = (int64_t)(c.nlarge - c.nhuge);
  out[2] = W.n - (int64_t)c.nlarge;
  return CRT_OK;
}

// The result block of a persistent query without pairs whose traversal and window
// order left these errors, for tests: its error, or a negative status.
int persist_result_error(int traversal, int order, cudaStream_t stream)
{
  char* scr = nullptr;
  const size_t bytes = persist_scratch_bytes(2, 1, true);
  if (cudaMallocAsync((void**)&scr, bytes + sizeof(crt_query_result), stream) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  PersistScratch S;
  persist_scratch_carve(scr, 2, 1, true, S);
  crt_query_result* res = (crt_query_result*)(scr + bytes);
  crt_query_result h{};
  cudaMemsetAsync(scr, 0, bytes, stream);
  cudaMemcpyAsync(&S.ctr->error, &traversal, sizeof(int), cudaMemcpyHostToDevice, stream);
  cudaMemcpyAsync(&sort_ctrl(S.sort_zero)->error, &order, sizeof(int), cudaMemcpyHostToDevice, stream);
  enqueue_post(S, nullptr, nullptr, 0, res, stream);
  cudaMemcpyAsync(&h, res, sizeof(h), cudaMemcpyDeviceToHost, stream);
  cudaFreeAsync(scr, stream);
  return cudaStreamSynchronize(stream) == cudaSuccess ? h.error : -1;
}

int query_stats(const crt_rtree_f32& rt, const crt_bbox_f32& rbox, const crt_bbox_f32& qbox,
                int64_t* d_hits, int64_t* d_tested, int64_t* h_totals, cudaStream_t stream)
{
  TreeView T = make_view(rt, rbox);
  WindowView W{qbox.xmin, qbox.ymin, qbox.xmax, qbox.ymax, qbox.sz};
  const TraversalShape sh = traversal_shape(rbox.sz, rt.fanout);
  char* scr = nullptr;
  if (cudaMallocAsync((void**)&scr, 1024 + kLevelTableBytes, stream) != cudaSuccess) {
    cudaGetLastError();
    return fail(CRT_ERR_OOM, "query_stats: scratch allocation failed");
  }
  QueryCounters* ctr = (QueryCounters*)scr;
  unsigned long long* tot = (unsigned long long*)(scr + 256);  // [3] box-by-box, [3] containment
  cudaMemsetAsync(scr, 0, 1024 + kLevelTableBytes, stream);
  const size_t smem = (size_t)kPlainWarps * sh.stack_cap * sizeof(FrontierEntry);
  allow_smem(stats_kernel<false>);
  allow_smem(stats_kernel<true>);
  if (qbox.sz > 0) {
    const unsigned g = (unsigned)cdiv(qbox.sz, kPlainWarps);
    // the reference algorithm: every leaf box under an intersecting node is tested
    stats_kernel<false><<<g, kPlainWarps * 32, smem, stream>>>(
        T, W, sh.K, sh.stack_cap, (long long*)d_hits, (long long*)d_tested, tot, ctr);
    // this library's: contained subtrees are emitted by slot range
    TreeView Tc = T;
    attach_levels(Tc, level_tables(rt, rbox.sz), scr + 1024, nullptr, 0, nullptr, stream);
    stats_kernel<true><<<g, kPlainWarps * 32, smem, stream>>>(Tc, W, sh.K, sh.stack_cap, nullptr,
                                                              nullptr, tot + 3, ctr);
    CRT_LAUNCHED(2);
  }
  unsigned long long h[6] = {0, 0, 0, 0, 0, 0};
  int err = 0;
  cudaMemcpyAsync(h, tot, sizeof(h), cudaMemcpyDeviceToHost, stream);
  cudaMemcpyAsync(&err, &ctr->error, sizeof(int), cudaMemcpyDeviceToHost, stream);
  cudaFreeAsync(scr, stream);
  cudaError_t e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_fail(e, "query_stats");
  if (err) return fail(err, "query_stats: device-side error");
  if (h[0] != h[3]) return fail(CRT_ERR_CUDA, "query_stats: the two traversals disagree on the pair count");
  if (h_totals) {
    h_totals[0] = (int64_t)h[0];  // hits
    h_totals[1] = (int64_t)h[1];  // leaf boxes tested box by box
    h_totals[2] = (int64_t)h[4];  // leaf boxes tested with containment
    h_totals[3] = (int64_t)h[5];  // hits emitted by contained slot ranges
  }
  return CRT_OK;
}

// ---------------------------------------------------------------------------
// Persistent plan captured in a CUDA graph
// ---------------------------------------------------------------------------
// The whole query -- counter reset, window ordering, the persistent traversal
// and the output compaction -- is one graph, replayed with one
// cudaGraphLaunch.  Two event-record nodes bracket the traversal: they record
// the plan's own events, or, while kernel timing is on, a fresh event pair
// per launch (set into the instantiated graph before the launch), so the
// traversal's duration is measured inside the replay.
struct Plan {
  TreeView T;
  WindowView W;
  int64_t max_nq;
  PersistScratch S;
  char* scratch = nullptr;
  bool sort;
  int stage_n;
  int chunk;
  int32_t* fid;
  int32_t* tid;
  long long cap;
  crt_query_result* res;
  TraverseLaunch traverse;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaEvent_t own[2] = {nullptr, nullptr};         // recorded when timing is off
  cudaGraphNode_t ev_node[2] = {nullptr, nullptr};  // the event-record nodes
};

int plan_destroy(void* hp);

// The event-record node of `graph` that records `ev`.
static cudaGraphNode_t find_event_node(cudaGraph_t graph, cudaEvent_t ev)
{
  size_t n = 0;
  if (cudaGraphGetNodes(graph, nullptr, &n) != cudaSuccess || n == 0) return nullptr;
  std::vector<cudaGraphNode_t> nodes(n);
  if (cudaGraphGetNodes(graph, nodes.data(), &n) != cudaSuccess) return nullptr;
  for (auto nd : nodes) {
    cudaGraphNodeType t;
    cudaEvent_t e = nullptr;
    if (cudaGraphNodeGetType(nd, &t) == cudaSuccess && t == cudaGraphNodeTypeEventRecord &&
        cudaGraphEventRecordNodeGetEvent(nd, &e) == cudaSuccess && e == ev)
      return nd;
  }
  return nullptr;
}

int plan_create(const crt_rtree_f32& rt, const crt_bbox_f32& rbox, const crt_bbox_f32& qbox,
                int64_t max_nq, int32_t* fid, int32_t* tid, int64_t capacity,
                crt_query_result* res, const crt_query_opts& opts, cudaStream_t stream,
                void** out)
{
  if (!res || max_nq < 0) return fail(CRT_ERR_INVALID_ARG, "plan: bad arguments");
  Plan* p = new Plan();
  p->T = make_view(rt, rbox);
  p->W = WindowView{qbox.xmin, qbox.ymin, qbox.xmax, qbox.ymax, max_nq};
  p->max_nq = max_nq;
  p->sort = opts.sort_windows != 0 && max_nq > 1;
  p->chunk = opts.chunk >= 64 ? opts.chunk : kDefaultChunk;
  const int parts = window_parts(opts);
  if (parts < 0) {
    delete p;
    return fail(CRT_ERR_INVALID_ARG, "plan: warps_per_window must be 1, 2 or 4");
  }
  p->fid = fid;
  p->tid = tid;
  p->cap = capacity;
  p->res = res;
  const TraversalShape sh = traversal_shape(rbox.sz, rt.fanout);
  p->stage_n = fit_stage_nodes(rt, rbox.sz, opts.stage_levels, sh.stack_cap, opts.warps_per_cta);
  if (!persist_shape(sh.stack_cap, p->stage_n, opts.warps_per_cta).v) {
    delete p;
    return fail(CRT_ERR_NOT_SUPPORTED, "plan: traversal stack too large");
  }
  const long long max_holes = max_holes_for(sh.stack_cap, p->stage_n, opts.warps_per_cta);
  const size_t bytes = persist_scratch_bytes(max_nq, max_holes, p->sort);
  if (cudaMalloc((void**)&p->scratch, bytes) != cudaSuccess) {
    cudaGetLastError();
    delete p;
    return fail(CRT_ERR_OOM, "plan: scratch allocation failed");
  }
  persist_scratch_carve(p->scratch, max_nq, max_holes, p->sort, p->S);
  cudaMemsetAsync(p->scratch, 0, kHeadBytes, stream);
  attach_levels(p->T, opts.no_contain ? LevelTables() : level_tables(rt, rbox.sz),
                p->scratch + kHeadTables, p->S.ctr, max_nq, p->S.samples, stream);
  p->traverse = make_traverse(p->T, p->W, p->S, p->sort, p->stage_n, fid, tid, capacity, p->chunk,
                              opts.warps_per_cta, parts);
  // capture the whole query on a private stream; a window-sorting plan
  // orders exactly max_nq windows, so it only runs with nq == max_nq
  // (plan_set_nq enforces it); without sorting the kernel reads the live
  // count from ctr->nq
  cudaStream_t cs = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&p->own[0]);
  if (e == cudaSuccess) e = cudaEventCreate(&p->own[1]);
  if (e == cudaSuccess) e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    // each replay resets the counters (nq stays)
    cudaMemsetAsync(p->S.ctr, 0, offsetof(QueryCounters, nq), cs);
    enqueue_pre(p->T, p->W, max_nq, p->S, p->sort, window_classes(p->T, p->sort),
                variant_for(opts.warps_per_cta).share, cs);
    cudaError_t le = cudaEventRecordWithFlags(p->own[0], cs, cudaEventRecordExternal);
    if (le == cudaSuccess) le = launch_traverse(p->traverse, cs);
    if (le == cudaSuccess) le = cudaEventRecordWithFlags(p->own[1], cs, cudaEventRecordExternal);
    enqueue_post(p->S, fid, tid, capacity, res, cs);
    e = cudaStreamEndCapture(cs, &p->graph);
    if (e == cudaSuccess && le != cudaSuccess) e = le;
  }
  if (e == cudaSuccess) {
    p->ev_node[0] = find_event_node(p->graph, p->own[0]);
    p->ev_node[1] = find_event_node(p->graph, p->own[1]);
    if (!p->ev_node[0] || !p->ev_node[1]) e = cudaErrorInvalidValue;
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&p->exec, p->graph, 0);
  cudaStreamSynchronize(stream);
  if (cs) cudaStreamDestroy(cs);
  if (e != cudaSuccess) {
    cudaGetLastError();
    plan_destroy(p);
    return cuda_fail(e, "plan: graph capture");
  }
  *out = p;
  return CRT_OK;
}

int plan_set_nq(void* hp, int64_t nq, cudaStream_t stream)
{
  Plan* p = (Plan*)hp;
  if (nq < 0 || nq > p->max_nq) return fail(CRT_ERR_INVALID_ARG, "plan: nq out of range");
  if (p->sort && nq != p->max_nq)
    return fail(CRT_ERR_NOT_SUPPORTED, "plan: a window-sorting plan runs exactly max_nq windows");
  set_nq_kernel<<<1, 1, 0, stream>>>(p->S.ctr, nq);
  CRT_LAUNCHED(1);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CRT_OK : cuda_fail(e, "plan_set_nq");
}

int plan_launch(void* hp, cudaStream_t stream)
{
  NvtxRange range("crt_plan_launch");
  Plan* p = (Plan*)hp;
  cudaEvent_t a = p->own[0], b = p->own[1];
  cudaError_t e = cudaSuccess;
  if (prof_register("traverse_persistent", &a, &b)) {
    // this launch records a fresh pair (read and destroyed when the timings
    // are collected); the nodes go back to the plan's own events right after,
    // so the instantiated graph never refers to a destroyed event
    e = cudaGraphExecEventRecordNodeSetEvent(p->exec, p->ev_node[0], a);
    if (e == cudaSuccess) e = cudaGraphExecEventRecordNodeSetEvent(p->exec, p->ev_node[1], b);
    if (e == cudaSuccess) e = cudaGraphLaunch(p->exec, stream);
    cudaError_t r = cudaGraphExecEventRecordNodeSetEvent(p->exec, p->ev_node[0], p->own[0]);
    if (r == cudaSuccess) r = cudaGraphExecEventRecordNodeSetEvent(p->exec, p->ev_node[1], p->own[1]);
    if (e == cudaSuccess) e = r;
  } else {
    e = cudaGraphLaunch(p->exec, stream);
  }
  if (e != cudaSuccess) return cuda_fail(e, "plan_launch");
  // window keys and four sort passes; the traversal; hole ranks and
  // compaction
  CRT_LAUNCHED((p->sort ? 5 : 0) + 1 + (p->traverse.P.classes ? 1 : 0) + 2);
  return CRT_OK;
}

int plan_destroy(void* hp)
{
  Plan* p = (Plan*)hp;
  if (!p) return CRT_OK;
  if (p->exec) cudaGraphExecDestroy(p->exec);
  if (p->graph) cudaGraphDestroy(p->graph);
  for (auto ev : p->own)
    if (ev) cudaEventDestroy(ev);
  if (p->scratch) cudaFree(p->scratch);
  delete p;
  return CRT_OK;
}

}  // namespace crt
