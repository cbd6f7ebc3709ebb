// Z-order bulk load (replaces build_rtree, src/rtree_bulkload_thrust.cuh:62-213).
//
// Pipeline, all on one stream, no host synchronisation until the end:
//   1. encode      read the box SoA (float4 loads where aligned), write the
//                  flipped 32-bit Morton key and the slot of a 32-byte AoS
//                  record of each box (records of a 4096-box tile grouped by
//                  the key's top digit), and count all four 8-bit key digits.
//   2. plan        one CTA: which digit passes are non-uniform (a uniform digit
//                  leaves a stable order unchanged, so its pass is skipped) and
//                  the global bucket start of every digit value.
//   3. 4 x onesweep  stable LSD radix passes over (key, slot) with decoupled
//                  look-back across tiles: one read and one write of the pairs
//                  per pass.  The first active pass reads the encoder's slots,
//                  the last one writes only slots.
//   4. leaf level  gather each sorted box's record (runs of one top digit per
//                  tile, so lines are shared by neighbouring records), write the permuted
//                  SoA, and reduce every run of `fanout` boxes into its
//                  leaf-parent node.
//   5. upper levels  reduce runs of `fanout` nodes, level by level up to the root.
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
// are placed in its own slot range grouped by the key's top digit.  The sort
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

template <bool kVec>
__global__ void __launch_bounds__(kEncThreads) encode_kernel(BoxIn in, int64_t n,
                                                             uint32_t* __restrict__ keys,
                                                             uint32_t* __restrict__ slots,
                                                             Box32* __restrict__ aos,
                                                             SortCtrl* __restrict__ ctrl)
{
  // digit histograms over all of this CTA's tiles (the last digit is the top
  // byte: it is added from the tile's top-byte counts)
  __shared__ uint32_t sh[kDigits][kBins];
  __shared__ uint32_t s_run[kGroups];  // this tile: count, then run start, per top byte
  __shared__ uint32_t s_wsum[kGroups / 32];
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
      x = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) s_wsum[warp] = x;
    }
    __syncthreads();
    if (tid < kGroups) {
      uint32_t start = x - cnt;
      for (int w = 0; w < warp; w++) start += s_wsum[w];
      s_run[tid] = start;
    }
    __syncthreads();
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
        sl[k] = (uint32_t)base + s_run[dr >> 16] + (dr & 0xFFFFu);
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

// Reduces runs of `fanout` consecutive children into parent nodes
// (reduce_op, src/rtree_bulkload_thrust.cuh:38-50: min, min, max, max of the
// MBR, first child index, child count).  kLeaf: children are the sorted boxes,
// gathered from the AoS copy through the sorted slot order, and the permuted
// SoA is written on the way; otherwise children are nodes at child_start.
template <bool kLeaf>
__global__ void __launch_bounds__(kLevelThreads, 3)  // 80 registers: three CTAs per SM
    level_kernel(int nodes_per_cta, int fanout, int64_t nchild, int64_t nparent,
                 int64_t parent_start, int64_t pos_base,
                 // leaf inputs/outputs
                 const uint32_t* __restrict__ vals0, const uint32_t* __restrict__ vals1,
                 const SortCtrl* __restrict__ ctrl, const Box32* __restrict__ aos,
                 float* __restrict__ oxmin, float* __restrict__ oymin,
                 float* __restrict__ oxmax, float* __restrict__ oymax, int* __restrict__ oid,
                 // node arrays
                 float* __restrict__ nxmin, float* __restrict__ nymin,
                 float* __restrict__ nxmax, float* __restrict__ nymax, int* __restrict__ npos,
                 int* __restrict__ nlen, int64_t child_start)
{
  __shared__ float4 s_mbr[kLevelChunk];
  const int64_t p0 = (int64_t)blockIdx.x * nodes_per_cta;
  const int64_t p1 = min(nparent, p0 + nodes_per_cta);
  if (p0 >= p1) return;
  const int64_t c0 = p0 * fanout;
  const int64_t c1 = min(nchild, p1 * fanout);
  const uint32_t* sorted = nullptr;
  if (kLeaf) {
    // record slots in sorted order (the encoder's slots when no pass ran)
    int na = ctrl->n_active;
    sorted = (na & 1) ? vals1 : vals0;
  }
  // this thread's parent (if any) and its child range
  const int64_t my = p0 + threadIdx.x;
  const bool have = my < p1;
  const int64_t my_c0 = my * fanout;
  const int64_t my_c1 = min(nchild, my_c0 + fanout);
  float a = 0.f, b = 0.f, c = 0.f, d = 0.f;
  bool init = false;
  for (int64_t cb = c0; cb < c1; cb += kLevelChunk) {
    const int64_t ce = min(c1, cb + (int64_t)kLevelChunk);
    if (kLeaf) {
      // all slot loads, then all 32-byte record loads, then the stores: each
      // thread keeps kGather record reads in flight
      constexpr int kGather = kLevelChunk / kLevelThreads;
      uint32_t src[kGather];
#pragma unroll
      for (int u = 0; u < kGather; u++) {
        const int64_t s = cb + threadIdx.x + u * kLevelThreads;
        src[u] = s < ce ? sorted[s] : 0u;
        if ((int64_t)src[u] >= nchild) src[u] = s < ce ? (uint32_t)s : 0u;  // only after a sort error (reported)
      }
      Box32 bx[kGather];
#pragma unroll
      for (int u = 0; u < kGather; u++)
        if (cb + threadIdx.x + u * kLevelThreads < ce) bx[u] = aos[src[u]];
#pragma unroll
      for (int u = 0; u < kGather; u++) {
        const int64_t s = cb + threadIdx.x + u * kLevelThreads;
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
      for (int64_t s = cb + threadIdx.x; s < ce; s += kLevelThreads) {
        const int64_t i = child_start + s;
        s_mbr[s - cb] = make_float4(nxmin[i], nymin[i], nxmax[i], nymax[i]);
      }
    }
    __syncthreads();
    if (have) {
      const int64_t lo = max(my_c0, cb), hi = min(my_c1, ce);
      for (int64_t s = lo; s < hi; s++) {
        float4 m = s_mbr[s - cb];
        if (!init) {
          a = m.x; b = m.y; c = m.z; d = m.w;
          init = true;
        } else {
          a = fminf(a, m.x);
          b = fminf(b, m.y);
          c = fmaxf(c, m.z);
          d = fmaxf(d, m.w);
        }
      }
    }
    __syncthreads();
  }
  if (have) {
    const int64_t o = parent_start + my;
    nxmin[o] = a;
    nymin[o] = b;
    nxmax[o] = c;
    nymax[o] = d;
    npos[o] = (int)(pos_base + my_c0);
    nlen[o] = (int)(my_c1 - my_c0);
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

  // scratch: [ctrl | hist | status] (zeroed) then keys/vals/aos
  const size_t zero_bytes = sort_zero_bytes(n);
  const size_t kv_bytes = ((size_t)n * 4 + 255) / 256 * 256;
  const size_t aos_bytes = (size_t)n * sizeof(Box32);
  const size_t total = (zero_bytes + 255) / 256 * 256 + 4 * kv_bytes + aos_bytes + 256;
  char* scratch = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&scratch, total, stream);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(CRT_ERR_OOM, "build: scratch allocation failed");
  }
  size_t off = (zero_bytes + 255) / 256 * 256;
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
    if (vec)
      encode_kernel<true><<<grid, kEncThreads, 0, stream>>>(bin, n, cols.key[0], cols.val[0], aos,
                                                            ctrl);
    else
      encode_kernel<false><<<grid, kEncThreads, 0, stream>>>(bin, n, cols.key[0], cols.val[0], aos,
                                                             ctrl);
    }
    CRT_LAUNCHED(1);
    sort_passes(cols, n, kDigits, scratch, stream);

    // leaf-parent level
    int64_t parent_start = rsz;
    int64_t child_start = 0, nchild = n;
    for (size_t l = 0; l < lv.size(); l++) {
      const int64_t np = lv[l];
      parent_start -= np;
      int npc = (int)std::max<int64_t>(1, std::min<int64_t>(kLevelThreads, kLevelChunk / fanout));
      unsigned g = (unsigned)cdiv(np, npc);
      ProfScope ps("level", stream);
      if (l == 0)
        level_kernel<true><<<g, kLevelThreads, 0, stream>>>(
            npc, fanout, nchild, np, parent_start, rsz, cols.val[0], cols.val[1], ctrl, aos,
            out_xmin, out_ymin, out_xmax, out_ymax, out_id, nxmin, nymin, nxmax, nymax, npos,
            nlen, 0);
      else
        level_kernel<false><<<g, kLevelThreads, 0, stream>>>(
            npc, fanout, nchild, np, parent_start, child_start, nullptr, nullptr, ctrl, nullptr,
            nullptr, nullptr, nullptr, nullptr, nullptr, nxmin, nymin, nxmax, nymax, npos, nlen,
            child_start);
      CRT_LAUNCHED(1);
      child_start = parent_start;
      nchild = np;
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
