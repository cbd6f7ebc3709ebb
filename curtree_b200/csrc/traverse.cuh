// Warp-cooperative traversal of one window, shared by the batch query
// (query.cu) and the serving loop (server.cu).
//
// Semantics kept from the reference: the root is never tested; a node whose
// children are nodes passes on the children whose MBR intersects the window
// (src/rtree_bfs_frontier.cuh:110-124); a leaf-parent (pos >= R_sz) tests its
// boxes at slots [pos - R_sz, pos - R_sz + len) (count_hit/write_hit,
// src/rtree_bfs_frontier.cuh:191-289); a hit emits (fid = sorted box's id,
// tid = window index).
//
// The warp keeps its frontier in shared memory as a stack of node indices.
// Each step pops up to K = 32 / fanout nodes (one child per lane, children
// read in SoA layout, coalesced), tests the children, compacts the
// intersecting inner children back onto the stack with a ballot/popc prefix,
// and emits leaf hits warp-collectively.  Popping the top K entries and
// pushing shallower parents' children first keeps the stack ordered by depth,
// so it never holds more than K*fanout entries per level: (levels - 1) * K *
// fanout + 1 in total, which the host sizes exactly.
#pragma once

#include "common.cuh"

namespace crt {

// Deepest tree the containment shortcut handles (a tree of 2^31 boxes at
// fanout 2 has 31 levels).
constexpr int kMaxLevels = 40;

struct TreeView {
  const float* __restrict__ nxmin;
  const float* __restrict__ nymin;
  const float* __restrict__ nxmax;
  const float* __restrict__ nymax;
  const int* __restrict__ npos;
  const int* __restrict__ nlen;
  int rsz;
  int fanout;
  const float* __restrict__ bxmin;
  const float* __restrict__ bymin;
  const float* __restrict__ bxmax;
  const float* __restrict__ bymax;
  const int* __restrict__ bid;
  int nbox;
  // Packed-layout tables for the containment shortcut (nlev == 0: off).  In
  // the reference's bulk-load layout the subtree of the g-th node of height h
  // (h = 0: leaf-parents) holds the sorted slots
  // [g * span[h], min(nbox, (g + 1) * span[h])), span[h] = fanout^(h + 1).
  int nlev;
  const int* __restrict__ lvl_first;        // first node index of height h
  const long long* __restrict__ lvl_span;   // boxes under a full node of height h
  // Non-zero word: some box is not ordinary, and the shortcut is off (null:
  // every box was found ordinary when the tables were made).
  const int* __restrict__ lvl_odd;
};

// Host image of the containment tables: kMaxLevels ints (first node of each
// height) then kMaxLevels int64 (boxes under a full node of that height).  On
// the device a flag word follows them: set when some box is not ordinary.
struct LevelTables {
  int nlev = 0;
  int first[kMaxLevels];
  long long span[kMaxLevels];
};
constexpr size_t kLevelOddOffset = sizeof(int) * kMaxLevels + sizeof(long long) * kMaxLevels;
constexpr size_t kLevelTableBytes = kLevelOddOffset + 16;
// Tables of a tree in the reference's packed layout; nlev == 0 otherwise.
LevelTables level_tables(const crt_rtree_f32& rt, int64_t nbox);
// Zeroes *odd, then sets it when some of the n boxes is not ordinary
// (xmin <= xmax and ymin <= ymax, which a NaN coordinate also fails).
void launch_odd_boxes(const float* xmin, const float* ymin, const float* xmax, const float* ymax,
                      int64_t n, int* odd, cudaStream_t stream);

struct WindowView {
  const float* __restrict__ xmin;
  const float* __restrict__ ymin;
  const float* __restrict__ xmax;
  const float* __restrict__ ymax;
  int64_t n;
};

// Top tree levels staged in shared memory (node index < n), or none.
struct NodeCache {
  const float* xmin;
  const float* ymin;
  const float* xmax;
  const float* ymax;
  const int* pos;
  const int* len;
  int n;
};

__device__ __forceinline__ void load_node_box(const TreeView& T, const NodeCache& C, int i,
                                              float& a, float& b, float& c, float& d)
{
  if (i < C.n) {
    a = C.xmin[i]; b = C.ymin[i]; c = C.xmax[i]; d = C.ymax[i];
  } else {
    a = __ldg(T.nxmin + i); b = __ldg(T.nymin + i); c = __ldg(T.nxmax + i); d = __ldg(T.nymax + i);
  }
}
__device__ __forceinline__ void load_node_link(const TreeView& T, const NodeCache& C, int i,
                                               int& p, int& l)
{
  if (i < C.n) {
    p = C.pos[i]; l = C.len[i];
  } else {
    p = __ldg(T.npos + i); l = __ldg(T.nlen + i);
  }
}

// ---------------------------------------------------------------------------
// Warp traversal of one window
// ---------------------------------------------------------------------------
// One frontier entry: the children range [pos, pos + len) of a node that
// intersected the window.  Carrying the range on the stack (it is loaded with
// the node's MBR when the node is tested) saves a dependent load per level.
// With the containment shortcut on, the high 8 bits of `len` hold the height
// of the nodes in the range.
typedef int2 FrontierEntry;
constexpr int kLenBits = 24;
constexpr int kLenMask = (1 << kLenBits) - 1;

// Emits every box of the sorted slot range [first, first + count) as a hit,
// 32 at a time (warp-collective); emitters with a faster bulk path override it.
template <class Emit>
__device__ __forceinline__ void emit_range_default(Emit& emit, const int* __restrict__ bid,
                                                   long long first, long long count)
{
  const int lane = (int)lane_id();
  for (long long base = 0; base < count; base += 32) {
    const long long i = base + lane;
    const bool hit = i < count;
    emit(hit, hit ? __ldg(bid + first + i) : 0);
  }
}

// Emits every lane's slot range one after the other through emit.range
// (warp-collective).
template <class Emit>
__device__ __forceinline__ void emit_ranges_each(Emit& emit, const int* __restrict__ bid, bool mine,
                                                 long long first, long long count)
{
  uint32_t im = __ballot_sync(0xffffffffu, mine);
  while (im) {
    const int src = __ffs(im) - 1;
    im &= im - 1;
    emit.range(bid, __shfl_sync(0xffffffffu, first, src), __shfl_sync(0xffffffffu, count, src));
  }
}

// Contained runs of slots below Emit::kSmall boxes (a leaf-parent holds
// `fanout`) are emitted together, all of one step's at once; longer ones go
// through the emitter's big_ranges.  kSmallRange is the line of the emitters
// that place a long run into an output reservation of its own.
constexpr int kSmallRange = 256;

// Emits the ids of every lane's slot range [first, first + count) (count <
// Emit::kSmall; a lane with mine == false adds none), 32 ids per warp pass
// whatever the ranges' sizes: each lane finds the range holding its id by a
// binary search over the lanes' inclusive count prefix (warp-collective).
template <class Emit>
__device__ __forceinline__ void emit_small_ranges(Emit& emit, const int* __restrict__ bid, bool mine,
                                                  long long first, int count)
{
  const int lane = (int)lane_id();
  const int c = mine ? count : 0;
  int x = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  const int total = __shfl_sync(0xffffffffu, x, 31);
  // element t of the concatenation, inside lane j's range, is id bid[base_j + t]
  const long long base = first - (x - c);
  for (int t0 = 0; t0 < total; t0 += 32) {
    const int t = t0 + lane;
    int j = 0;  // lanes whose inclusive prefix is <= t: the owner of t
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      const int v = __shfl_sync(0xffffffffu, x, j + s - 1);
      if (v <= t) j += s;
    }
    const long long b = __shfl_sync(0xffffffffu, base, j);
    const bool ok = t < total;
    emit(ok, ok ? __ldg(bid + b + t) : 0);
  }
}

// Pair stores use the evict-first hint (st.global.cs): the output streams
// through L2 once, and keeping it out of the way leaves L2 to the tree's
// boxes and ids (measured: 1-3% on the uniform batch, 7-10% on road
// geometry).
__device__ __forceinline__ void put_pair(int32_t* __restrict__ fid, int32_t* __restrict__ tid,
                                         long long slot, long long cap, int id, int q)
{
  if (slot < cap) {
    __stcs(fid + slot, id);
    if (tid) __stcs(tid + slot, q);  // no window column: CSR output
  }
}

// Four pairs at output slot sl (16-byte aligned in fid and tid), or one by
// one where they reach cap.
__device__ __forceinline__ void put_pairs4(int32_t* __restrict__ fid, int32_t* __restrict__ tid,
                                           long long sl, long long cap, int4 v, int q)
{
  if (sl + 3 < cap) {
    __stcs(reinterpret_cast<int4*>(fid + sl), v);
    if (tid) __stcs(reinterpret_cast<int4*>(tid + sl), make_int4(q, q, q, q));
  } else {
    put_pair(fid, tid, sl + 0, cap, v.x, q);
    put_pair(fid, tid, sl + 1, cap, v.y, q);
    put_pair(fid, tid, sl + 2, cap, v.z, q);
    put_pair(fid, tid, sl + 3, cap, v.w, q);
  }
}

// Writes the pairs (bid[first + i], q) to output slots slot0 + i for
// i < count, skipping slots at or past `cap` (warp-collective).  A contained
// subtree can hold millions of boxes, so the ids are read as 16-byte vectors
// (128 ids per warp step, kRangeUnroll steps in flight) instead of one 4-byte
// load per lane; one step keeps the kernels within their register budgets.
// Where the output is not 16-byte aligned with the source the stores are
// single; this form needs fewer registers than copy_range_realign (below),
// and the plain and serving kernels run faster with it.
constexpr int kRangeUnroll = 1;

__device__ __forceinline__ void copy_range(const int* __restrict__ bid, long long first,
                                           long long count, int32_t* __restrict__ fid,
                                           int32_t* __restrict__ tid, long long slot0,
                                           long long cap, int q)
{
  const int lane = (int)lane_id();
  const int* src = bid + first;
  // head: ids before the first 16-byte boundary of the source
  long long head = (long long)((4 - (((uintptr_t)src >> 2) & 3)) & 3);
  if (head > count) head = count;
  if (lane < head) put_pair(fid, tid, slot0 + lane, cap, __ldg(src + lane), q);
  const int4* v = reinterpret_cast<const int4*>(src + head);
  const long long nv = (count - head) >> 2;
  const long long s = slot0 + head;
  for (long long g0 = 0; g0 < nv; g0 += 32 * kRangeUnroll) {
    int4 r[kRangeUnroll];
#pragma unroll
    for (int u = 0; u < kRangeUnroll; u++) {
      const long long g = g0 + u * 32 + lane;
      if (g < nv) r[u] = __ldg(v + g);
    }
#pragma unroll
    for (int u = 0; u < kRangeUnroll; u++) {
      const long long g = g0 + u * 32 + lane;
      if (g < nv) {
        const long long sl = s + 4 * g;
        const uintptr_t al = (uintptr_t)(fid + sl) | (tid ? (uintptr_t)(tid + sl) : (uintptr_t)0);
        if (sl + 3 < cap && (al & 15) == 0) {
          __stcs(reinterpret_cast<int4*>(fid + sl), r[u]);
          if (tid) __stcs(reinterpret_cast<int4*>(tid + sl), make_int4(q, q, q, q));
        } else {
          put_pair(fid, tid, sl + 0, cap, r[u].x, q);
          put_pair(fid, tid, sl + 1, cap, r[u].y, q);
          put_pair(fid, tid, sl + 2, cap, r[u].z, q);
          put_pair(fid, tid, sl + 3, cap, r[u].w, q);
        }
      }
    }
  }
  // tail: the last (count - head) % 4 ids
  const long long done = head + 4 * nv;
  if (lane < count - done) put_pair(fid, tid, slot0 + done + lane, cap, __ldg(src + done + lane), q);
}

// copy_range with 16-byte stores wherever the reservation starts (the
// persistent kernel's large-subtree reservations start anywhere in a
// 16-byte line): the output is aligned first (up to 3 ids one by one); when
// the source then sits at another offset within its 16 bytes, each lane's
// four ids come from its own aligned source vector and its neighbour's (one
// shuffle per component), so loads and stores both stay 16-byte accesses.
// Only aligned vectors inside [bid, bid + first + count) are read.
__device__ __forceinline__ void copy_range_realign(const int* __restrict__ bid, long long first,
                                                   long long count, int32_t* __restrict__ fid,
                                                   int32_t* __restrict__ tid, long long slot0,
                                                   long long cap, int q)
{
  const int lane = (int)lane_id();
  if (count <= 0) return;
  const uintptr_t fa = (uintptr_t)(fid + slot0);
  // vectors need bid 16-byte aligned and fid, tid at one offset within 16 bytes
  const bool vec = ((uintptr_t)bid & 15) == 0 &&
                   (!tid || (((uintptr_t)(tid + slot0) ^ fa) & 15) == 0);
  if (!vec) {
    for (long long i = lane; i < count; i += 32)
      put_pair(fid, tid, slot0 + i, cap, __ldg(bid + first + i), q);
    return;
  }
  // head: ids before the output's first 16-byte boundary
  long long head = (long long)((4 - ((fa >> 2) & 3)) & 3);
  if (head > count) head = count;
  if (lane < head) put_pair(fid, tid, slot0 + lane, cap, __ldg(bid + first + lane), q);
  const long long f1 = first + head;  // first source id of the body
  const long long s1 = slot0 + head;  // its output slot, 16-byte aligned
  const long long end = first + count;
  const int r = (int)(f1 & 3);  // source offset within its 16 bytes
  const long long B = f1 - r;   // the aligned source vector holding f1
  const int4* __restrict__ v = reinterpret_cast<const int4*>(bid + B);
  long long ng;  // output vectors of the body
  if (r == 0) {
    ng = (end - f1) >> 2;
    for (long long g = lane; g < ng; g += 32) put_pairs4(fid, tid, s1 + 4 * g, cap, __ldg(v + g), q);
  } else {
    // output vector g takes source vectors g and g + 1, both inside [B, end)
    // for g < ng
    ng = end - B >= 8 ? ((end - B - 8) >> 2) + 1 : 0;
    for (long long g0 = 0; g0 < ng; g0 += 32) {
      const long long g = g0 + lane;
      int4 x = make_int4(0, 0, 0, 0);
      if (g <= ng) x = __ldg(v + g);
      int4 n;
      n.x = __shfl_down_sync(0xffffffffu, x.x, 1);
      n.y = __shfl_down_sync(0xffffffffu, x.y, 1);
      n.z = __shfl_down_sync(0xffffffffu, x.z, 1);
      n.w = __shfl_down_sync(0xffffffffu, x.w, 1);
      if (lane == 31 && g + 1 <= ng) n = __ldg(v + g + 1);
      if (g < ng) {
        int4 o;
        if (r == 1) o = make_int4(x.y, x.z, x.w, n.x);
        else if (r == 2) o = make_int4(x.z, x.w, n.x, n.y);
        else o = make_int4(x.w, n.x, n.y, n.z);
        put_pairs4(fid, tid, s1 + 4 * g, cap, o, q);
      }
    }
  }
  // tail: the ids past the body (fewer than 8)
  for (long long i = f1 + 4 * ng + lane; i < end; i += 32)
    put_pair(fid, tid, s1 + (i - f1), cap, __ldg(bid + i), q);
}

// Outcome of testing one child slot of a step.
struct ChildTest {
  bool valid, hit, push, inside;
  int hid, cpos, clen;
  int rfirst, rcount;  // slots of a contained node
  bool leaf;  // a box slot (counted as a leaf test)
};

// A window shared by several warps below the root: every warp walks the nodes
// above `height`, and a node of that height (or a contained one above it)
// belongs to the warp `part` that its index names.  mask == 0: not shared.
struct Split {
  int height = 0;
  int mask = 0;  // parts - 1, parts a power of two
  int part = 0;
};

// Tests child c of popped entry g (of k popped; lane e of the warp holds
// entry e): a leaf box against the window, or an inner node (intersects:
// push its children range; contained: emit its boxes' slot range).
__device__ __forceinline__ void test_child(const TreeView& T, const NodeCache& C, FrontierEntry e,
                                           int k, int g, int c, bool contain, float x1, float y1,
                                           float x2, float y2, const Split& split, ChildTest& t)
{
  const int gs = min(g, k - 1);
  const int pos = __shfl_sync(0xffffffffu, e.x, gs);
  const int ey = __shfl_sync(0xffffffffu, e.y, gs);
  const int len = contain ? (ey & kLenMask) : ey;
  const int hc = contain ? (ey >> kLenBits) : 0;  // height of the nodes [pos, pos+len)
  t.valid = g < k && c < len;
  const int child = pos + c;
  t.hit = t.push = t.inside = t.leaf = false;
  t.hid = t.cpos = t.clen = 0;
  t.rfirst = t.rcount = 0;
  if (!t.valid) return;
  if (pos >= T.rsz) {
    const int s = child - T.rsz;
    if (s < T.nbox) {
      t.leaf = true;
      // the id is loaded with the box (one round trip; most tested boxes of
      // a leaf-parent that straddles the window hit)
      const float m1 = __ldg(T.bxmin + s), n1 = __ldg(T.bymin + s);
      const float m2 = __ldg(T.bxmax + s), n2 = __ldg(T.bymax + s);
      const int id = __ldg(T.bid + s);
      t.hit = intersects(x1, y1, x2, y2, m1, n1, m2, n2);
      t.hid = id;
    }
  } else if (child < T.rsz) {
    float a, b, cc, d;
    load_node_box(T, C, child, a, b, cc, d);
    load_node_link(T, C, child, t.cpos, t.clen);
    t.push = intersects(x1, y1, x2, y2, a, b, cc, d);
    const bool inside = contain && t.push && x1 <= a && cc <= x2 && y1 <= b && d <= y2;
    // another warp's share of the window
    if (split.mask && (hc == split.height || (inside && hc > split.height)) &&
        (child & split.mask) != split.part) {
      t.push = false;
    } else if (inside) {
      t.inside = true;
      t.push = false;
      const long long span = __ldg(T.lvl_span + hc);
      const long long first = (long long)(child - __ldg(T.lvl_first + hc)) * span;
      t.rfirst = (int)first;
      t.rcount = (int)min((long long)T.nbox - first, span);
    } else if (contain) {
      t.clen |= max(hc - 1, 0) << kLenBits;
    }
  }
}

// Tests the boxes of k popped leaf-parents (lane e of the warp holds entry e;
// at most kSets * K of them, fanout <= 32) and emits the hits.  Three steps of
// four pop leaf-parents only: without the inner nodes' loads, containment test,
// push and ranges such a step issues less than half the instructions, and two
// sets of boxes are in flight (1M mixed windows on 10M boxes: 13.1 -> 12.5 ms;
// one set 12.8).
template <int kSets, class Emit>
__device__ __forceinline__ void leaf_step(const TreeView& T, FrontierEntry e, int k, int K, int lane_g,
                                          int lane_c, bool contain, float x1, float y1, float x2,
                                          float y2, Emit& emit)
{
  float m1[kSets], n1[kSets], m2[kSets], n2[kSets];
  int id[kSets];
  bool ok[kSets];
#pragma unroll
  for (int s = 0; s < kSets; s++) {
    const int g = s * K + lane_g;
    ok[s] = lane_g < K && g < k;
    const int slot = __shfl_sync(0xffffffffu, e.x, ok[s] ? g : 0) - T.rsz + lane_c;
    const int ey = __shfl_sync(0xffffffffu, e.y, ok[s] ? g : 0);
    ok[s] = ok[s] && lane_c < (contain ? (ey & kLenMask) : ey) && slot < T.nbox;
    m1[s] = n1[s] = m2[s] = n2[s] = 0.f;
    id[s] = 0;
    if (ok[s]) {
      m1[s] = __ldg(T.bxmin + slot);
      n1[s] = __ldg(T.bymin + slot);
      m2[s] = __ldg(T.bxmax + slot);
      n2[s] = __ldg(T.bymax + slot);
      id[s] = __ldg(T.bid + slot);
    }
  }
#pragma unroll
  for (int s = 0; s < kSets; s++) {
    if constexpr (Emit::kCountsTests) emit.leaf_tests(__popc(__ballot_sync(0xffffffffu, ok[s])));
    emit(ok[s] && intersects(x1, y1, x2, y2, m1[s], n1[s], m2[s], n2[s]), id[s]);
  }
}

// part / nparts: this warp takes the part-th of nparts equal shares of the
// root's children (several warps sharing one window); the shares' subtrees
// are disjoint, so their hits together are the window's.
template <class Emit, bool kContain = true, int kLeafSets = 2>
__device__ __forceinline__ void traverse(const TreeView& T, const NodeCache& C, int K,
                                         int lane_g, int lane_c, float x1, float y1, float x2,
                                         float y2, FrontierEntry* stack, int stack_cap,
                                         Emit& emit, int* err, int part = 0, int nparts = 1,
                                         Split split = Split())
{
  const int lane = (int)lane_id();
  const uint32_t lt = lanemask_lt();
  const int f = T.fanout;
  if (T.rsz == 0) {
    if (part != 0) return;
    // one-box (or empty) tree: no nodes, test the boxes directly
    for (int base = 0; base < T.nbox; base += 32) {
      int s = base + lane;
      bool hit = s < T.nbox &&
                 intersects(x1, y1, x2, y2, T.bxmin[s], T.bymin[s], T.bxmax[s], T.bymax[s]);
      if constexpr (Emit::kCountsTests) emit.leaf_tests(min(32, T.nbox - base));
      emit(hit, hit ? T.bid[s] : 0);
    }
    return;
  }
  // A window that contains a node's MBR hits every ordinary box under it:
  // x1 <= MBR.xmin <= xmin <= xmax <= MBR.xmax <= x2, and the same in y, so
  // none of the predicate's four exclusions holds.  The subtree's slot range
  // is then emitted without descending.  A box that is not ordinary (xmin >
  // xmax, ymin > ymax, or a NaN coordinate, which the MBR's min/max skip) can
  // fail the predicate under a contained MBR, so any such box in the set
  // turns the shortcut off.  A NaN in the window or the MBR fails the
  // containment test and takes the normal path.
  const bool contain = kContain && T.nlev > 0 && (T.lvl_odd == nullptr || *T.lvl_odd == 0);
  // the root is never tested: its children range starts the frontier
  {
    int rp, rl;
    load_node_link(T, C, 0, rp, rl);
    if (nparts > 1) {
      const int a = (int)((long long)rl * part / nparts);
      const int b = (int)((long long)rl * (part + 1) / nparts);
      rp += a;
      rl = b - a;
    }
    if (contain) rl |= max(T.nlev - 2, 0) << kLenBits;
    if (lane == 0) stack[0] = make_int2(rp, rl);
  }
  int sp = 1;
  __syncwarp();
  while (sp > 0) {
    if (f <= 32) {
      // leaf-parents are the deepest entries, so they lie on top
      const int k = min(sp, kLeafSets * K);
      FrontierEntry e = make_int2(T.rsz, 0);
      if (lane < k) e = stack[sp - k + lane];
      if (__all_sync(0xffffffffu, e.x >= T.rsz)) {
        sp -= k;
        leaf_step<kLeafSets>(T, e, k, K, lane_g, lane_c, contain, x1, y1, x2, y2, emit);
        __syncwarp();
        continue;
      }
    }
    const int k = min(sp, K);
    sp -= k;
    // popped entries stack[sp .. sp+k): lower index = shallower; lane g holds entry g
    FrontierEntry e = make_int2(0, 0);
    if (lane < k) e = stack[sp + lane];
    __syncwarp();
    const int span = f <= 32 ? 32 : f;  // children covered per node group
    for (int base = 0; base < span; base += 32) {
      ChildTest t;
      if (f <= 32) test_child(T, C, e, k, lane_g, lane_c, contain, x1, y1, x2, y2, split, t);
      else test_child(T, C, e, k, 0, base + lane, contain, x1, y1, x2, y2, split, t);
      if constexpr (Emit::kCountsTests) emit.leaf_tests(__popc(__ballot_sync(0xffffffffu, t.leaf)));
      const uint32_t pm = __ballot_sync(0xffffffffu, t.push);
      if (pm) {
        const int np = __popc(pm);
        if (sp + np > stack_cap) {
          // cannot happen with the host-sized stack; never write past it
          raise_error(err, CRT_ERR_NOT_SUPPORTED);
          return;
        }
        if (t.push) stack[sp + __popc(pm & lt)] = make_int2(t.cpos, t.clen);
        sp += np;
      }
      emit(t.hit, t.hid);
      if (contain) {
        const uint32_t im = __ballot_sync(0xffffffffu, t.inside);
        if (im) {
          // contained siblings next to each other hold one run of slots: its
          // first lane emits them all (the same batch: 12.5 -> 12.2 ms)
          const int end = t.rfirst + t.rcount;
          const int before = __shfl_up_sync(0xffffffffu, end, 1);
          const bool join = t.inside && lane > 0 && ((im >> (lane - 1)) & 1u) && before == t.rfirst;
          const uint32_t jm = __ballot_sync(0xffffffffu, join);
          const uint32_t next = ~jm & (0xfffffffeu << lane);  // lanes above that start anew
          const int run = __shfl_sync(0xffffffffu, end, next ? __ffs(next) - 2 : 31) - t.rfirst;
          const bool head = t.inside && !join;
          const bool small = head && run < Emit::kSmall;
          if (__any_sync(0xffffffffu, small)) emit.small_ranges(T.bid, small, t.rfirst, run);
          const bool big = head && !small;
          if (__any_sync(0xffffffffu, big)) emit.big_ranges(T.bid, big, t.rfirst, run);
        }
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Warp traversal of several windows at once (fanout <= 32)
// ---------------------------------------------------------------------------
// The warp's stack holds entries of up to 32 windows (each entry names its
// window); a step pops kSets * K entries of any of them, and the loads of all
// their children are in flight together.  An entry's `y` is: children count
// (bits 0-7), window (bits 8-12), height of the nodes in the range (bits
// 24-31).  refill(sp) may push entries when a step would not be full (sp <
// kSets * K) and returns the new stack size; below its entries the stack keeps
// the depth order of one window's, so it never holds more than kSets * K *
// fanout entries per level, plus the refill's kGroupWindows and the kSets * K
// left when it ran.  Only for packed trees over ordinary boxes.
constexpr int kGroupWindows = 32;
constexpr int kGroupLenMask = 0xFF;

__device__ __forceinline__ FrontierEntry group_entry(int pos, int len, int window, int height)
{
  // at most 32 children are looked at (lane_c < fanout)
  return make_int2(pos, min(max(len, 0), 32) | window << 8 | height << 24);
}

template <int kSets, class Emit, class Refill>
__device__ __forceinline__ void traverse_group(const TreeView& T, int K, int lane_g, int lane_c,
                                               const float4* s_win, const int* s_q,
                                               FrontierEntry* stack, int stack_cap, Emit& emit,
                                               Refill refill, int* err)
{
  const uint32_t lt = lanemask_lt();
  int sp = 0;
  while (true) {
    if (sp < kSets * K) sp = refill(sp);
    if (sp == 0) return;
    const int k = min(sp, kSets * K);
    sp -= k;
    // popped entries stack[sp .. sp+k): lower index = shallower.  Every set's
    // loads are issued before the first test; boxes and nodes share them, so
    // a step that meets both waits one round trip.
    float m1[kSets], n1[kSets], m2[kSets], n2[kSets];
    int ref[kSets], len[kSets], child[kSets], ey[kSets];
    bool ok[kSets], leaf[kSets];
#pragma unroll
    for (int s = 0; s < kSets; s++) {
      const int at = s * K + lane_g;
      ok[s] = lane_g < K && at < k;
      const FrontierEntry e = stack[sp + (ok[s] ? at : 0)];
      ey[s] = e.y;
      child[s] = e.x + lane_c;
      leaf[s] = e.x >= T.rsz;
      const int j = leaf[s] ? child[s] - T.rsz : child[s];
      ok[s] = ok[s] && lane_c < (e.y & kGroupLenMask) && j < (leaf[s] ? T.nbox : T.rsz);
      m1[s] = n1[s] = m2[s] = n2[s] = 0.f;
      ref[s] = len[s] = 0;
      if (ok[s]) {
        m1[s] = __ldg((leaf[s] ? T.bxmin : T.nxmin) + j);
        n1[s] = __ldg((leaf[s] ? T.bymin : T.nymin) + j);
        m2[s] = __ldg((leaf[s] ? T.bxmax : T.nxmax) + j);
        n2[s] = __ldg((leaf[s] ? T.bymax : T.nymax) + j);
        ref[s] = __ldg((leaf[s] ? T.bid : T.npos) + j);  // a box's id, a node's first child
        if (!leaf[s]) len[s] = __ldg(T.nlen + j);
      }
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < kSets; s++) {
      const int wl = (ey[s] >> 8) & (kGroupWindows - 1);
      const float4 w = s_win[wl];
      const bool meets = ok[s] && intersects(w.x, w.y, w.z, w.w, m1[s], n1[s], m2[s], n2[s]);
      const bool inside = meets && !leaf[s] && w.x <= m1[s] && m2[s] <= w.z && w.y <= n1[s] && n2[s] <= w.w;
      const bool push = meets && !leaf[s] && !inside;
      const int h = (int)((uint32_t)ey[s] >> 24);
      const uint32_t pm = __ballot_sync(0xffffffffu, push);
      if (pm) {
        const int np = __popc(pm);
        if (sp + np > stack_cap) {
          // cannot happen with the host-sized stack; never write past it
          raise_error(err, CRT_ERR_NOT_SUPPORTED);
          return;
        }
        if (push) stack[sp + __popc(pm & lt)] = group_entry(ref[s], len[s], wl, max(h - 1, 0));
        sp += np;
      }
      const uint32_t hm = __ballot_sync(0xffffffffu, meets && leaf[s]);
      if (hm) emit.hits(hm, meets && leaf[s], ref[s], s_q[wl]);
      if (__any_sync(0xffffffffu, inside)) {
        long long first = 0, count = 0;
        if (inside) {
          const long long span = __ldg(T.lvl_span + h);
          first = (long long)(child[s] - __ldg(T.lvl_first + h)) * span;
          count = min((long long)T.nbox - first, span);
        }
        const bool small = inside && count < Emit::kSmall;
        if (__any_sync(0xffffffffu, small)) emit.small_ranges(T.bid, small, first, (int)count, s_q[wl]);
        const bool big = inside && !small;
        if (__any_sync(0xffffffffu, big)) emit.big_ranges(T.bid, big, first, count, s_q[wl]);
      }
    }
    __syncwarp();
  }
}

// Lane -> (node group, child) of its first child slot, for fanout <= 32;
// lanes past the last whole group get group 32 (never valid).
__device__ __forceinline__ void lane_map(int f, int& g, int& c)
{
  const int lane = (int)lane_id();
  if (f <= 32) {
    g = lane / f;
    c = lane - g * f;
    if (g >= 32 / f) { g = 32; c = 0; }
  } else {
    g = 0;
    c = lane;
  }
}

}  // namespace crt
