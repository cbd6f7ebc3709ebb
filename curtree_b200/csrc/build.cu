// Z-order bulk load (replaces build_rtree, src/rtree_bulkload_thrust.cuh:62-213).
//
// Pipeline, all on one stream, no host synchronisation until the end:
//   1. encode      read the box SoA (float4 loads where aligned), write the
//                  flipped 32-bit Morton key and the slot of a 32-byte AoS
//                  record of each box (records of a 4096-box tile grouped by
//                  the key's top byte, in large sets in blocks per top byte),
//                  and count all four 8-bit key digits.
//   2. plan        the encoder's last CTA: which digit passes are non-uniform (a
//                  uniform digit leaves a stable order unchanged, so its pass is
//                  skipped) and the global bucket start of every digit value.
//   3. 4 x sweep    (sort.cu) stable LSD radix passes over (key, slot) with decoupled
//                  look-back across tiles: one read and one write of the pairs
//                  per pass.  The first active pass reads the encoder's slots,
//                  the last one writes only slots.
//   4. leaf level  gather each sorted box's record (runs of one top digit per
//                  tile, so lines are shared by neighbouring records), write the permuted
//                  SoA, and reduce every run of `fanout` boxes into its
//                  leaf-parent node.
//   5. upper levels  reduce runs of `fanout` nodes, up to the root: a launch that
//                  fits one wave makes every level above its own.
// Node order, pos and len follow the reference exactly (root at 0, levels
// downward, children contiguous, leaf-parent pos = R_sz + first slot).
#include <cuda_runtime.h>

#include <cstdio>
#include <vector>

#include "internal.h"
#include "profile.h"

namespace crt {

struct alignas(32) Box32 {
  float4 mbr;  // xmin, ymin, xmax, ymax
  int4 idp;    // id, 0, 0, 0
};

// ---------------------------------------------------------------------------
// 1. encode
// ---------------------------------------------------------------------------
// Each CTA takes tiles of kEncTile boxes.  Per box it writes the key and, in
// input order, the slot of the box's 32-byte record; the records of a tile
// are placed in its own slot range (in large sets in blocks, below) grouped by
// the key's top digit.  The sort
// then carries those slots (its first pass reads them instead of making
// input indices), and the leaf level's gather in sorted order, which walks
// one top digit at a time, reads each tile's run for that digit (about
// kEncTile / 256 records, often several whole 128-byte lines) instead of
// single records scattered over the whole copy.  Order inside a run does not
// matter: ties in the sort keep input order because the (key, slot) pairs
// start in input order.
constexpr int kEncThreads = 256;
constexpr int kEncGroups = 4;                            // float4 groups per thread
constexpr int kEncTile = 4 * kEncGroups * kEncThreads;   // 4096 boxes
constexpr int kGroups = 256;                             // record runs: by the key's top byte
static_assert(kGroups <= kEncThreads, "one thread per run");

// Where the records of a large set lie (kBlocks): each top byte fills blocks of
// records (2^16 of them at 33 M boxes and more, a 2 MB page), handed out as its
// runs come in, so the leaf level's gather for a top byte walks that byte's
// pages.  With the records of a tile in the tile's own slots every page holds
// records of every top byte, and the gather of a large set waits for address
// translation (finer grouping inside the tile changes nothing).  100 M clustered
// boxes: levels 2158 -> 1612 us for 80 us more in the encoder (the wait for the
// run's place and shorter runs), build 5.65 -> 5.16 ms; 10 M: levels 177 -> 154,
// encoder +7, build 626 -> 613 us.
struct BlockTable {
  uint32_t* cursor;  // per top byte: records placed so far (zeroed)
  uint32_t* block;   // per top byte and its k-th block: number + 1, 0 = none yet (zeroed)
  uint32_t* used;    // blocks handed out (zeroed)
  uint32_t stride;   // blocks per top byte in `block`
  uint32_t most;     // blocks there are
  uint32_t bits;     // log2 of the records in a block (at least a tile's)
};

// Block k of top byte d: handed out by the thread whose run holds its first
// record, awaited by the threads of the later runs in it.
__device__ __forceinline__ uint32_t take_block(const BlockTable& B, int d, uint32_t k, int* err)
{
  uint32_t b = atomicAdd(B.used, 1u);
  if (b >= B.most) {  // cannot happen: `most` counts every full block and a part-filled one per top byte
    raise_error(err, CRT_ERR_NOT_SUPPORTED);
    b = 0;
  }
  st_release_u32(&B.block[(size_t)d * B.stride + k], b + 1);
  return b;
}
__device__ __forceinline__ uint32_t wait_block(const BlockTable& B, int d, uint32_t k, int* err)
{
  for (uint32_t spin = 0; spin < kSpinLimit; spin++) {
    const uint32_t b = ld_acquire_u32(&B.block[(size_t)d * B.stride + k]);
    if (b) return b - 1;
    if (spin > 64) __nanosleep(64);
  }
  raise_error(err, CRT_ERR_DEVICE_TIMEOUT);
  return 0;
}

struct BoxIn {
  const float* __restrict__ xmin;
  const float* __restrict__ ymin;
  const float* __restrict__ xmax;
  const float* __restrict__ ymax;
  const int* __restrict__ id;
};

// Loads boxes j..j+3 (those below n); kVec: the arrays are 16-byte aligned.
template <bool kVec>
__device__ __forceinline__ void load4(const BoxIn& in, int64_t j, int64_t n, float4& a, float4& b,
                                      float4& c, float4& d, int4& e)
{
  if (kVec && j + 3 < n) {
    a = reinterpret_cast<const float4*>(in.xmin)[j >> 2];
    b = reinterpret_cast<const float4*>(in.ymin)[j >> 2];
    c = reinterpret_cast<const float4*>(in.xmax)[j >> 2];
    d = reinterpret_cast<const float4*>(in.ymax)[j >> 2];
    e = reinterpret_cast<const int4*>(in.id)[j >> 2];
    return;
  }
  float* pa = &a.x;
  float* pb = &b.x;
  float* pc = &c.x;
  float* pd = &d.x;
  int* pe = &e.x;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const bool v = j + k < n;
    pa[k] = v ? in.xmin[j + k] : 0.f;
    pb[k] = v ? in.ymin[j + k] : 0.f;
    pc[k] = v ? in.xmax[j + k] : 0.f;
    pd[k] = v ? in.ymax[j + k] : 0.f;
    pe[k] = v ? in.id[j + k] : 0;
  }
}

template <bool kVec, bool kBlocks>
__global__ void __launch_bounds__(kEncThreads) encode_kernel(BoxIn in, int64_t n,
                                                             uint32_t* __restrict__ keys,
                                                             uint32_t* __restrict__ slots,
                                                             Box32* __restrict__ aos,
                                                             SortCtrl* __restrict__ ctrl, BlockTable B)
{
  // digit histograms over all of this CTA's tiles (the last digit is the top
  // byte: it is added from the tile's top-byte counts)
  __shared__ uint32_t sh[kDigits][kBins];
  __shared__ uint32_t s_run[kGroups];  // this tile: count, then run start, per top byte
  __shared__ uint32_t s_wsum[kGroups / 32];
  __shared__ uint32_t s_part[kBlocks ? kGroups : 1];  // records of the run in its first block
  __shared__ uint32_t s_more[kBlocks ? kGroups : 1];  // start of the others, less that count
  __shared__ uint32_t s_dr[kEncTile];  // per box of the tile: top byte << 16 | rank in its run
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kDigits * kBins; i += kEncThreads) (&sh[0][0])[i] = 0;
  const int64_t ntiles = (n + kEncTile - 1) / kEncTile;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    if (tid < kGroups) s_run[tid] = 0;
    __syncthreads();
    const int64_t base = t * kEncTile;
#pragma unroll
    for (int g = 0; g < kEncGroups; g++) {
      const int i0 = 4 * (tid + g * kEncThreads);  // first box of the group in the tile
      const int64_t j = base + i0;
      float4 a, b, c, d;
      int4 e;
      load4<kVec>(in, j, n, a, b, c, d, e);
      const float* pa = &a.x;
      const float* pb = &b.x;
      const float* pc = &c.x;
      const float* pd = &d.x;
      uint32_t kk[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        kk[k] = sort_key(pa[k], pb[k], pc[k], pd[k]);
        if (j + k < n) {
          const uint32_t top = kk[k] >> 24;
          s_dr[i0 + k] = top << 16 | atomicAdd(&s_run[top], 1u);
#pragma unroll
          for (int dg = 0; dg < kDigits - 1; dg++) atomicAdd(&sh[dg][key_digit(kk[k], dg)], 1u);
        }
      }
      if (j + 3 < n) {
        *reinterpret_cast<uint4*>(keys + j) = make_uint4(kk[0], kk[1], kk[2], kk[3]);
      } else {
        for (int k = 0; k < 4; k++)
          if (j + k < n) keys[j + k] = kk[k];
      }
    }
    __syncthreads();
    // run starts: exclusive prefix of the tile's top-byte counts
    uint32_t cnt = 0, x = 0;
    if (tid < kGroups) {
      cnt = s_run[tid];
      if (cnt) atomicAdd(&sh[kDigits - 1][tid], cnt);
      if (kBlocks) {
        // the run's place in its top byte's blocks.  All lanes hand out the
        // blocks whose first record is theirs before any lane waits, so every
        // wait is for a running thread that waits for nothing.
        const uint32_t v = cnt ? atomicAdd(&B.cursor[tid], cnt) : 0u;
        const uint32_t k = v >> B.bits, off = v & ((1u << B.bits) - 1);
        const uint32_t part = min(cnt, (1u << B.bits) - off);
        uint32_t more = 0, b = 0;
        if (part < cnt) more = take_block(B, tid, k + 1, &ctrl->error) << B.bits;
        if (cnt && off == 0) b = take_block(B, tid, k, &ctrl->error);
        __syncwarp();
        if (off != 0) b = wait_block(B, tid, k, &ctrl->error);
        s_run[tid] = (b << B.bits) + off;
        s_part[tid] = part;
        s_more[tid] = more - part;
      } else {
        x = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        if (lane == 31) s_wsum[warp] = x;
      }
    }
    __syncthreads();
    if (!kBlocks) {
      if (tid < kGroups) {
        uint32_t start = x - cnt;
        for (int w = 0; w < warp; w++) start += s_wsum[w];
        s_run[tid] = (uint32_t)base + start;
      }
      __syncthreads();
    }
    // records into their runs; slots in input order
#pragma unroll
    for (int g = 0; g < kEncGroups; g++) {
      const int i0 = 4 * (tid + g * kEncThreads);
      const int64_t j = base + i0;
      float4 a, b, c, d;
      int4 e;
      load4<kVec>(in, j, n, a, b, c, d, e);  // second read of the tile: from L2
      const float* pa = &a.x;
      const float* pb = &b.x;
      const float* pc = &c.x;
      const float* pd = &d.x;
      const int* pe = &e.x;
      uint32_t sl[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t dr = j + k < n ? s_dr[i0 + k] : 0u;
        const uint32_t g = dr >> 16, r = dr & 0xFFFFu;
        sl[k] = (kBlocks && r >= s_part[g] ? s_more[g] : s_run[g]) + r;
        if (j + k < n) {
          Box32 bx;
          bx.mbr = make_float4(pa[k], pb[k], pc[k], pd[k]);
          bx.idp = make_int4(pe[k], 0, 0, 0);
          aos[sl[k]] = bx;
        }
      }
      if (j + 3 < n) {
        *reinterpret_cast<uint4*>(slots + j) = make_uint4(sl[0], sl[1], sl[2], sl[3]);
      } else {
        for (int k = 0; k < 4; k++)
          if (j + k < n) slots[j + k] = sl[k];
      }
    }
    __syncthreads();
  }
  chain_next();
  for (int i = tid; i < kDigits * kBins; i += kEncThreads) {
    const uint32_t v = (&sh[0][0])[i];
    if (v) atomicAdd(&ctrl->hist[i], v);
  }
  sort_plan(ctrl, n, kDigits);
}

// ---------------------------------------------------------------------------
// 4./5. level reductions
// ---------------------------------------------------------------------------
constexpr int kLevelThreads = 256;
constexpr int kLevelChunk = 2048;  // children staged per round
constexpr int kUpMax = 12;         // levels a CTA makes above its own parents
constexpr int kTailMax = 32;       // levels the last CTA makes
constexpr int64_t kTailNodes = 16384;  // most children it starts from

struct NodeOut {
  float* __restrict__ xmin;
  float* __restrict__ ymin;
  float* __restrict__ xmax;
  float* __restrict__ ymax;
  int* __restrict__ pos;
  int* __restrict__ len;
};

// One launch of the level kernel: a level of nparent parents over nchild
// children, the up_n levels above it that each CTA makes from its own parents,
// and the tail_n levels above those that the last CTA to finish makes alone.
struct LevelArgs {
  int nodes_per_cta;  // a multiple of fanout^up_n
  int fanout;
  int64_t nchild, nparent;
  uint32_t nslots;   // record slots (leaf level)
  int parent_start;  // first node of the parents' level
  int pos_base;      // pos of the first parent
  int child_start;   // first node of the children's level (inner levels)
  int up_n;
  int up_start[kUpMax];
  int tail_n;
  int tail_child;        // first node and node count of the level below the tail
  int tail_nchild;
  int tail_start[kTailMax];
  int* done;  // CTAs finished (zeroed)
};

__device__ __forceinline__ void put_node(const NodeOut& N, int o, float4 m, int pos, int len)
{
  N.xmin[o] = m.x;
  N.ymin[o] = m.y;
  N.xmax[o] = m.z;
  N.ymax[o] = m.w;
  N.pos[o] = pos;
  N.len[o] = len;
}

// reduce_op (src/rtree_bulkload_thrust.cuh:38-50) of one more child.
__device__ __forceinline__ float4 merge_box(float4 a, float4 m)
{
  return make_float4(fminf(a.x, m.x), fminf(a.y, m.y), fmaxf(a.z, m.z), fmaxf(a.w, m.w));
}

// Reduces runs of `fanout` consecutive children into parent nodes
// (reduce_op, src/rtree_bulkload_thrust.cuh:38-50: min, min, max, max of the
// MBR, first child index, child count).  kLeaf: children are the sorted boxes,
// gathered from the AoS copy through the sorted slot order, and the permuted
// SoA is written on the way; otherwise children are nodes at child_start.
// The leaf level is bound by its gathers: 100M clustered boxes take 1.53 ms with
// the records in blocks (2.1 in the tiles' own slots), 0.64 of the copy
// bandwidth for its 64 bytes a box, and 0.86 with the records read in order.
// Tile shapes, records per thread in flight and 32-byte loads measured no
// difference.  A level above
// it is a few microseconds of launch and latency, so a CTA goes on upwards over
// the parents it holds in shared memory, and the last CTA makes the top of the
// tree: one or two launches instead of one per level (all levels of 20k boxes,
// fanout 10: 19 us with the gaps between the launches, 10 now; 1M: 37, now 25).
//
// kFuse: the launch makes the levels above its own too.
template <bool kLeaf, bool kFuse>
__global__ void __launch_bounds__(kLevelThreads, 3)  // 80 registers (12 bytes spilled): three CTAs per SM
    level_kernel(LevelArgs A, NodeOut N,
                 // leaf inputs/outputs
                 const uint32_t* __restrict__ vals0, const uint32_t* __restrict__ vals1,
                 const SortCtrl* __restrict__ ctrl, const Box32* __restrict__ aos,
                 float* __restrict__ oxmin, float* __restrict__ oymin,
                 float* __restrict__ oxmax, float* __restrict__ oymax, int* __restrict__ oid)
{
  __shared__ float4 s_mbr[kLevelChunk];
  __shared__ int s_last;
  chain_wait();
  // 32-bit indices: children and parents are below 2^31, their sums with a
  // fanout below 2^32
  const uint32_t fanout = (uint32_t)A.fanout;
  const uint32_t nchild = (uint32_t)A.nchild;
  const uint32_t p0 = blockIdx.x * (uint32_t)A.nodes_per_cta;
  const uint32_t p1 = min((uint32_t)A.nparent, p0 + (uint32_t)A.nodes_per_cta);
  const uint32_t c0 = p0 * fanout;
  const uint32_t c1 = min(nchild, p1 * fanout);
  const uint32_t* sorted = nullptr;
  if (kLeaf) {
    // record slots in sorted order (the encoder's slots when no pass ran)
    int na = ctrl->n_active;
    sorted = (na & 1) ? vals1 : vals0;
  }
  // this thread's parent (if any) and its child range
  const uint32_t my = p0 + threadIdx.x;
  const bool have = my < p1;
  const uint32_t my_c0 = my * fanout;
  const uint32_t my_c1 = min(nchild, my_c0 + fanout);
  float4 box = make_float4(0.f, 0.f, 0.f, 0.f);
  bool init = false;
  for (uint32_t cb = c0; cb < c1; cb += kLevelChunk) {
    const uint32_t ce = min(c1, cb + (uint32_t)kLevelChunk);
    if (kLeaf) {
      // all slot loads, then all 32-byte record loads, then the stores: each
      // thread keeps kGather record reads in flight
      constexpr int kGather = kLevelChunk / kLevelThreads;
      uint32_t src[kGather];
#pragma unroll
      for (int u = 0; u < kGather; u++) {
        const uint32_t s = cb + threadIdx.x + u * kLevelThreads;
        src[u] = s < ce ? sorted[s] : 0u;
        if (src[u] >= A.nslots) src[u] = s < ce ? s : 0u;  // only after a sort error (reported)
      }
      Box32 bx[kGather];
#pragma unroll
      for (int u = 0; u < kGather; u++)
        if (cb + threadIdx.x + u * kLevelThreads < ce) bx[u] = aos[src[u]];
#pragma unroll
      for (int u = 0; u < kGather; u++) {
        const uint32_t s = cb + threadIdx.x + u * kLevelThreads;
        if (s < ce) {
          const float4 m = bx[u].mbr;
          __stcs(oxmin + s, m.x);
          __stcs(oymin + s, m.y);
          __stcs(oxmax + s, m.z);
          __stcs(oymax + s, m.w);
          __stcs(oid + s, bx[u].idp.x);
          s_mbr[s - cb] = m;
        }
      }
    } else {
      for (uint32_t s = cb + threadIdx.x; s < ce; s += kLevelThreads) {
        const uint32_t i = (uint32_t)A.child_start + s;
        s_mbr[s - cb] = make_float4(N.xmin[i], N.ymin[i], N.xmax[i], N.ymax[i]);
      }
    }
    __syncthreads();
    if (have) {
      const uint32_t lo = max(my_c0, cb), hi = min(my_c1, ce);
      for (uint32_t s = lo; s < hi; s++) {
        const float4 m = s_mbr[s - cb];
        box = init ? merge_box(box, m) : m;
        init = true;
      }
    }
    __syncthreads();
  }
  if (have)
    put_node(N, (int)(A.parent_start + my), box, (int)(A.pos_base + my_c0), (int)(my_c1 - my_c0));
  chain_next();
  if constexpr (!kFuse) return;
  // the levels above, over this CTA's parents
  if (A.up_n > 0) {
    if (have) s_mbr[threadIdx.x] = box;
    int cnt = (int)(p1 - p0);
    int first = (int)p0;  // index in its level of the CTA's first node
    int below = A.parent_start;
    for (int k = 0; k < A.up_n; k++) {
      __syncthreads();
      const int np = (cnt + (int)fanout - 1) / (int)fanout;
      const int lo = (int)threadIdx.x * (int)fanout, hi = min(cnt, lo + (int)fanout);
      float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
      if ((int)threadIdx.x < np) {
        m = s_mbr[lo];
        for (int i = lo + 1; i < hi; i++) m = merge_box(m, s_mbr[i]);
      }
      __syncthreads();
      if ((int)threadIdx.x < np) {
        s_mbr[threadIdx.x] = m;
        put_node(N, (int)(A.up_start[k] + first / (int)fanout + (int)threadIdx.x), m, (int)(below + first + lo),
                 hi - lo);
      }
      first /= (int)fanout;
      below = A.up_start[k];
      cnt = np;
    }
  }
  // the top of the tree, by the CTA that finishes last
  if (A.tail_n > 0) {
    __threadfence();  // this thread's nodes before the count
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(A.done, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    int below = A.tail_child, cnt = A.tail_nchild;
    for (int k = 0; k < A.tail_n; k++) {
      const int np = (cnt + (int)fanout - 1) / (int)fanout;
      // threads that share a parent's children: a level of few parents is a chain
      // of loads through L2 for the one thread of each (1M boxes, fanout 1000, 1000
      // children: build 189 us with one thread, 136 now; fanout 300
      // 158 and 129; fanouts 10 and 16 the same)
      int g = 1;
      while (2 * g * np <= kLevelThreads && 2 * g <= (int)fanout) g *= 2;
      const int l = (int)threadIdx.x & (g - 1);
      for (int p0 = 0; p0 < np; p0 += kLevelThreads / g) {
        const int p = p0 + (int)threadIdx.x / g;
        const bool ok = p < np;
        const int lo = ok ? p * (int)fanout : 0, hi = ok ? min(cnt, lo + (int)fanout) : 1;
        const auto child = [&](int i) {  // another CTA's, or written a level ago: through L2
          const int j = below + i;
          return make_float4(__ldcg(N.xmin + j), __ldcg(N.ymin + j), __ldcg(N.xmax + j), __ldcg(N.ymax + j));
        };
        float4 m = child(min(lo + l, hi - 1));
#pragma unroll 4
        for (int i = lo + l + g; i < hi; i += g) m = merge_box(m, child(i));
        for (int o = min(g, 32) >> 1; o > 0; o >>= 1)
          m = merge_box(m, make_float4(__shfl_xor_sync(0xffffffffu, m.x, o), __shfl_xor_sync(0xffffffffu, m.y, o),
                                       __shfl_xor_sync(0xffffffffu, m.z, o), __shfl_xor_sync(0xffffffffu, m.w, o)));
        if (g > 32) {
          const int warp = (int)threadIdx.x >> 5;
          if ((threadIdx.x & 31) == 0) s_mbr[warp] = m;
          __syncthreads();
          if (l == 0)
            for (int w = 1; w < g >> 5; w++) m = merge_box(m, s_mbr[warp + w]);
          __syncthreads();
        }
        if (ok && l == 0) put_node(N, A.tail_start[k] + p, m, below + lo, hi - lo);
      }
      __syncthreads();
      below = A.tail_start[k];
      cnt = np;
    }
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
int tree_levels(int64_t n, int fanout, std::vector<int64_t>& lv)
{
  lv.clear();
  if (n < 1 || fanout < 2) return -1;
  int64_t len = n;
  while (len != 1) {
    len = (len + fanout - 1) / fanout;
    lv.push_back(len);
  }
  return (int)lv.size();
}

static bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// Sets of at least this many boxes keep their records in blocks.  Build in
// blocks against the tiles' own slots: 4.2 M boxes 328 to 320 us, 5 M 374 to
// 368, 10 M 602 to 611 (uniform) and 613 to 626 (clustered).
constexpr int64_t kBlocksMin = 1 << 23;
// Records per block: the largest power of two up to 2^16 with at least
// kBlockShare of them in the set, so the part-filled blocks (one per top byte)
// add at most half to the copy.  10 M boxes: 2^14 154 us of levels, 2^13 162,
// 2^12 170; 30 M: 2^16 405, 2^15 423, 2^14 536.  A set of kBlocksMin has 2^14.
constexpr int64_t kBlockShare = 512;
constexpr int kBlockBitsMost = 16;
constexpr int kBlockBitsLeast = 14;
static_assert(kBlocksMin >> kBlockBitsLeast >= kBlockShare, "the least suits the smallest set");
static_assert(kEncTile <= 1 << kBlockBitsLeast, "a run crosses into at most one block");

// Builds the tree of `n` boxes.  in_* may alias out_* (in-place build).
// Node arrays must hold R_sz entries.  Synchronises `stream` at the end and
// reports device-side errors.
int build_tree(const float* in_xmin, const float* in_ymin, const float* in_xmax,
               const float* in_ymax, const int* in_id, int64_t n, int fanout, float* out_xmin,
               float* out_ymin, float* out_xmax, float* out_ymax, int* out_id, float* nxmin,
               float* nymin, float* nxmax, float* nymax, int* npos, int* nlen,
               cudaStream_t stream)
{
  NvtxRange range("crt_build");
  std::vector<int64_t> lv;
  if (tree_levels(n, fanout, lv) < 0)
    return fail(CRT_ERR_INVALID_ARG, "build: need n >= 1 and fanout >= 2");
  int64_t rsz = 0;
  for (auto x : lv) rsz += x;
  if (n + rsz > INT32_MAX)
    return fail(CRT_ERR_INVALID_ARG, "build: n + R_sz exceeds the int32 pos range of RTREE");

  // scratch: the sort's control block and status words and the record blocks'
  // table (zeroed), then keys/vals/aos.  Large sets keep their records in blocks
  // where there is room for that, other sets in the tiles' own slots.
  const size_t sort_bytes = (sort_zero_bytes(n) + 255) / 256 * 256;
  const size_t kv_bytes = ((size_t)n * 4 + 255) / 256 * 256;
  bool blocks = n >= kBlocksMin;
  BlockTable B{};
  size_t zero_bytes = 0;
  uint32_t nslots = 0;
  char* scratch = nullptr;
  cudaError_t e = cudaSuccess;
  for (;; blocks = false) {
    size_t table = 0;
    nslots = (uint32_t)n;
    if (blocks) {
      B.bits = kBlockBitsLeast;
      while (B.bits < kBlockBitsMost && (n >> (B.bits + 1)) >= kBlockShare) B.bits++;
      B.stride = (uint32_t)(n >> B.bits) + 2;
      B.most = (uint32_t)(n >> B.bits) + kGroups;
      nslots = B.most << B.bits;
      table = sizeof(uint32_t) * (kGroups * ((size_t)B.stride + 1) + 1);
    }
    zero_bytes = (sort_bytes + table + 255) / 256 * 256;
    e = cudaMallocAsync((void**)&scratch, zero_bytes + 4 * kv_bytes + (size_t)nslots * sizeof(Box32) + 256,
                        stream);
    if (e == cudaSuccess) break;
    cudaGetLastError();
    if (!blocks) return fail(CRT_ERR_OOM, "build: scratch allocation failed");
  }
  B.cursor = (uint32_t*)(scratch + sort_bytes);
  B.block = B.cursor + kGroups;
  B.used = B.block + kGroups * (size_t)B.stride;
  size_t off = zero_bytes;
  SortCtrl* ctrl = sort_ctrl(scratch);
  SortCols cols{};
  cols.key[0] = (uint32_t*)(scratch + off); off += kv_bytes;
  cols.key[1] = (uint32_t*)(scratch + off); off += kv_bytes;
  cols.val[0] = (uint32_t*)(scratch + off); off += kv_bytes;
  cols.val[1] = (uint32_t*)(scratch + off); off += kv_bytes;
  cols.drop_keys = true;
  Box32* aos = (Box32*)(scratch + off);

  int rc = CRT_OK;
  do {
    if ((e = cudaMemsetAsync(scratch, 0, zero_bytes, stream)) != cudaSuccess) break;
    const int sms = sm_count();
    const bool vec = aligned16(in_xmin) && aligned16(in_ymin) && aligned16(in_xmax) &&
                     aligned16(in_ymax) && aligned16(in_id);
    int grid = (int)std::min<int64_t>(cdiv(n, kEncTile), (int64_t)sms * 3);
    if (grid < 1) grid = 1;
    const BoxIn bin{in_xmin, in_ymin, in_xmax, in_ymax, in_id};
    {
    ProfScope ps("encode", stream);
    const auto encode = vec ? (blocks ? encode_kernel<true, true> : encode_kernel<true, false>)
                            : (blocks ? encode_kernel<false, true> : encode_kernel<false, false>);
    encode<<<grid, kEncThreads, 0, stream>>>(bin, n, cols.key[0], cols.val[0], aos, ctrl, B);
    }
    CRT_LAUNCHED(1);
    sort_passes(cols, n, kDigits, scratch, stream);

    // the levels, leaf-parents first: start[l] is level l's first node
    std::vector<int64_t> start(lv.size());
    int64_t at = rsz;
    for (size_t l = 0; l < lv.size(); l++) start[l] = at -= lv[l];
    const NodeOut nodes{nxmin, nymin, nxmax, nymax, npos, nlen};
    int launch = 0;
    for (size_t l = 0; l < lv.size(); launch++) {
      LevelArgs A{};
      A.fanout = fanout;
      A.nchild = l ? lv[l - 1] : n;
      A.nparent = lv[l];
      A.nslots = nslots;
      A.parent_start = (int)start[l];
      A.child_start = l ? (int)start[l - 1] : 0;
      A.pos_base = l ? A.child_start : (int)rsz;
      // a launch of one wave goes on upwards: whole subtrees per CTA as far as
      // its parents go.  In longer launches the extra steps (and the last CTA's
      // fence) cost every wave more than the launches they save (10M boxes,
      // fanout 16: leaf level 176 us with them, 165 without).
      const int64_t most = std::max<int64_t>(1, std::min<int64_t>(kLevelThreads, kLevelChunk / fanout));
      const bool fuse = cdiv(A.nparent, most) <= (int64_t)sms * 4;
      int64_t sub = 1;
      while (fuse && A.up_n < kUpMax && l + 1 + A.up_n < lv.size() && sub * fanout <= most) {
        sub *= fanout;
        A.up_start[A.up_n] = (int)start[l + 1 + A.up_n];
        A.up_n++;
      }
      A.nodes_per_cta = (int)(most / sub * sub);
      size_t top = l + A.up_n;  // the last level made so far
      if (fuse && lv[top] <= kTailNodes && launch < (int)(sizeof(ctrl->level_done) / sizeof(int))) {
        A.tail_child = (int)start[top];
        A.tail_nchild = (int)lv[top];
        while (A.tail_n < kTailMax && top + 1 < lv.size()) A.tail_start[A.tail_n++] = (int)start[++top];
        A.done = &ctrl->level_done[launch];
      }
      const unsigned g = (unsigned)cdiv(A.nparent, A.nodes_per_cta);
      ProfScope ps("level", stream);
      if (l == 0)
        launch_after(fuse ? level_kernel<true, true> : level_kernel<true, false>, g, kLevelThreads, 0,
                     stream, A, nodes, cols.val[0], cols.val[1], ctrl, aos, out_xmin, out_ymin, out_xmax,
                     out_ymax, out_id);
      else
        launch_after(fuse ? level_kernel<false, true> : level_kernel<false, false>, g, kLevelThreads, 0,
                     stream, A, nodes, nullptr, nullptr, ctrl, nullptr, nullptr, nullptr, nullptr,
                     nullptr, nullptr);
      CRT_LAUNCHED(1);
      l = top + 1;
    }
    if (lv.empty()) {
      // one box, no nodes: the sorted box set is the input itself
      if (out_xmin != in_xmin) {
        cudaMemcpyAsync(out_xmin, in_xmin, 4, cudaMemcpyDeviceToDevice, stream);
        cudaMemcpyAsync(out_ymin, in_ymin, 4, cudaMemcpyDeviceToDevice, stream);
        cudaMemcpyAsync(out_xmax, in_xmax, 4, cudaMemcpyDeviceToDevice, stream);
        cudaMemcpyAsync(out_ymax, in_ymax, 4, cudaMemcpyDeviceToDevice, stream);
        cudaMemcpyAsync(out_id, in_id, 4, cudaMemcpyDeviceToDevice, stream);
      }
    }
    if ((e = cudaGetLastError()) != cudaSuccess) break;
    int dev_err = 0;
    if ((e = cudaMemcpyAsync(&dev_err, &ctrl->error, sizeof(int), cudaMemcpyDeviceToHost,
                             stream)) != cudaSuccess)
      break;
    if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) break;
    if (dev_err) rc = fail(dev_err, "build: device-side wait timed out in the radix sort");
  } while (0);
  cudaFreeAsync(scratch, stream);
  if (e != cudaSuccess) return cuda_fail(e, "build");
  return rc;
}

}  // namespace crt
