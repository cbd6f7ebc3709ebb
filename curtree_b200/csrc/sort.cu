// Stable LSD radix sort of (key, value) pairs of 32-bit words, shared by the
// bulk load (Morton keys), the window ordering and the canonical pair order.
// The caller's key kernel fills the digit histograms and its last CTA plans
// the passes (sort_plan, sort.cuh); every pass then is one launch that reads
// and writes the pairs once, with decoupled look-back across tiles (Merrill and
// Garland, "Single-pass parallel prefix scan with decoupled look-back", 2016;
// Adinets and Merrill, "Onesweep: a faster least significant digit radix sort
// for GPUs", 2022, put it under a radix sort's passes).
//
// A pass is bound by instruction issue, the shared-memory pipe and the chain
// ticket -> keys -> ranks -> bin scan -> look-back -> stores inside a tile, not
// by DRAM: 100M pairs take 0.57 ms per pass, 2.8 TB/s.  What shortened the
// chain (0.67 ms before): the values go through registers, on their way while
// the bins are scanned, instead of through a third shared-memory buffer; the
// look-back comes after the staging, when the predecessors have mostly
// published; no second launch to plan the passes.  CTAs that stay resident
// and fetch their next tile's ticket and keys early measured slower (2.94
// against 2.30 ms then): a claimed tile waits for its CTA, and every successor's
// look-back waits for that tile.
#include <cuda_runtime.h>

#include <algorithm>

#include "profile.h"
#include "sort.cuh"

namespace crt {

constexpr uint64_t kFlagAgg = 1ull << 62;
constexpr uint64_t kFlagIncl = 2ull << 62;
constexpr uint64_t kFlagMask = 3ull << 62;
// Predecessors a look-back reads per round trip (100M keys, four passes: 1 2.33,
// 2 2.32, 4 2.30, 8 2.42 ms).
constexpr int kLook = 4;

// Shared memory of one pass: keys and values staged in destination order, the
// per-warp digit counters (16-bit: at most a tile's keys), the per-warp lane
// masks of every digit, the bins' global offsets and the warp sums of the bin
// scan.
template <int kThreads, int kIpt>
struct SweepSmem {
  static constexpr int kTile = kThreads * kIpt;
  static constexpr int kWarps = kThreads / 32;
  static constexpr size_t kKeys = 0;
  static constexpr size_t kVals = kKeys + 4 * (size_t)kTile;
  static constexpr size_t kHist = kVals + 4 * (size_t)kTile;
  static constexpr size_t kMask = kHist + 2 * (size_t)kWarps * kBins;
  static constexpr size_t kGbase = kMask + 4 * (size_t)kWarps * kBins;
  static constexpr size_t kWsum = kGbase + 4 * (size_t)kBins;
  static constexpr size_t kBytes = kWsum + 4 * 32;
};

// Ranks this thread's keys inside its warp, stably (rounds in order, lanes in
// order), two 16-bit ranks per word.  kFull: every item of the tile is valid
// (no bounds checks).  The lanes that hold the same digit find each other
// through a mask word per digit in shared memory (each sets its bit; the lowest
// lane clears the word again): some 15 instructions where one ballot per digit
// bit takes 45 (four passes of 10M uniform keys 296 -> 272 us, 100M clustered
// 2.30 -> 2.28 ms; __match_any_sync was slower than the ballots).
template <bool kFull, int kIpt>
__device__ __forceinline__ void rank_keys(const uint32_t (&key)[kIpt], uint32_t (&rank)[kIpt / 2],
                                          uint16_t* wh, uint32_t* wm, int wbase, int tile_n, int shift,
                                          uint32_t flip)
{
  const uint32_t lt = lanemask_lt();
  const uint32_t me = 1u << lane_id();
#pragma unroll
  for (int i = 0; i < kIpt; i++) {
    const bool v = kFull || wbase + 32 * i < tile_n;
    const uint32_t dig = ((key[i] ^ flip) >> shift) & 255u;
    if (v) atomicOr(&wm[dig], me);
    __syncwarp();
    const uint32_t peers = wm[dig];
    const uint32_t old = wh[dig];
    __syncwarp();
    if (v && (peers & lt) == 0) {
      wh[dig] = (uint16_t)(old + __popc(peers));
      wm[dig] = 0u;
    }
    __syncwarp();
    const uint32_t r = old + __popc(peers & lt);
    if (i & 1) rank[i / 2] |= r << 16;
    else rank[i / 2] = r;
  }
}

// One stable pass over the 8-bit digit `digit` (digits 0-3 of the key column;
// 4-7: of the value column, the columns then change roles).  A CTA takes one
// tile, in order from a ticket.  Indices are 32-bit: the pair count is below
// 2^31 (the C ABI's int sizes).
template <int kThreads, int kIpt, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
    sweep_kernel(int digit, SortCols cols, int64_t n64, uint64_t* __restrict__ status,
                 SortCtrl* __restrict__ ctrl)
{
  using L = SweepSmem<kThreads, kIpt>;
  constexpr int kTile = L::kTile;
  constexpr int kWarps = L::kWarps;
  static_assert(kThreads >= kBins, "one thread per bin");
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  uint32_t* s_key = (uint32_t*)(sweep_smem + L::kKeys);
  uint32_t* s_val = (uint32_t*)(sweep_smem + L::kVals);
  uint16_t* s_whist = (uint16_t*)(sweep_smem + L::kHist);
  int* s_gbase = (int*)(sweep_smem + L::kGbase);
  int* s_wsum = (int*)(sweep_smem + L::kWsum);
  __shared__ int s_tile, s_stop;

  chain_wait();
  const int active = ctrl->active;
  if (!((active >> digit) & 1)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    s_tile = atomicAdd(&ctrl->tile_ctr[digit], 1);
    s_stop = ld_relaxed_i32(&ctrl->error) != 0;  // an earlier pass (or tile) gave up: its output is not whole
  }
  // counters and, behind them, masks
  for (int i = tid; i < kWarps * kBins * 3 / 2; i += kThreads) ((uint32_t*)s_whist)[i] = 0;
  const int step = __popc(active & ((1 << digit) - 1));  // active passes before this one
  const bool last = (active >> (digit + 1)) == 0;
  const int src = cols.src(step), dst = cols.dst(step, last);
  const bool swap = digit >= 4;
  const bool make_vals = step == 0 && cols.make_values;
  const bool drop_keys = last && cols.drop_keys;
  const int shift = 8 * (digit & 3);
  const uint32_t flip = cols.flip;
  const int n = (int)n64;
  const uint32_t* __restrict__ src_k = swap ? cols.vals(src) : cols.keys(src);
  const uint32_t* __restrict__ src_v = swap ? cols.keys(src) : cols.vals(src);
  uint32_t* __restrict__ dst_k = swap ? cols.vals(dst) : cols.keys(dst);
  uint32_t* __restrict__ dst_v = swap ? cols.keys(dst) : cols.vals(dst);
  const int bucket = tid < kBins ? ctrl->bucket_start[digit * kBins + tid] : 0;
  const int wbase = warp * 32 * kIpt + lane;  // this lane's first item in a tile
  uint16_t* wh = s_whist + warp * kBins;
  uint32_t* wm = (uint32_t*)(sweep_smem + L::kMask) + warp * kBins;
  __syncthreads();
  if (s_stop) return;
  const int tile = s_tile;
  const int base = tile * kTile;
  const int tile_n = min(kTile, n - base);
  const bool full = tile_n == kTile;

  // keys (warp-striped: item i of a lane is wbase + 32 i), their ranks, and
  // the values on their way while the bins are scanned
  uint32_t key[kIpt], rank[kIpt / 2], val[kIpt];
  if (full) {
#pragma unroll
    for (int i = 0; i < kIpt; i++) key[i] = src_k[base + wbase + 32 * i];
    rank_keys<true, kIpt>(key, rank, wh, wm, wbase, tile_n, shift, flip);
#pragma unroll
    for (int i = 0; i < kIpt; i++)
      val[i] = make_vals ? (uint32_t)(base + wbase + 32 * i) : src_v[base + wbase + 32 * i];
  } else {
#pragma unroll
    for (int i = 0; i < kIpt; i++) {
      const int j = wbase + 32 * i;
      key[i] = j < tile_n ? src_k[base + j] : 0u;
    }
    rank_keys<false, kIpt>(key, rank, wh, wm, wbase, tile_n, shift, flip);
#pragma unroll
    for (int i = 0; i < kIpt; i++) {
      const int j = wbase + 32 * i;
      val[i] = make_vals ? (uint32_t)(base + j) : (j < tile_n ? src_v[base + j] : 0u);
    }
  }
  __syncthreads();
  // bin b = tid: counts of every warp, the tile's count, exclusive scan over
  // the bins; the tile's aggregate is published before anything waits
  uint32_t cnt[kWarps / 2];  // two 16-bit counts per word
  int total = 0, x = 0;
  if (tid < kBins) {
#pragma unroll
    for (int w = 0; w < kWarps; w += 2) {
      const uint32_t a = s_whist[w * kBins + tid], b = s_whist[(w + 1) * kBins + tid];
      cnt[w / 2] = a | b << 16;
      total += (int)(a + b);
    }
    st_relaxed_u64(&status[(int64_t)tile * kBins + tid],
                   (tile == 0 ? kFlagIncl : kFlagAgg) | (uint32_t)total);
    x = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_wsum[warp] = x;
  }
  __syncthreads();
  int binstart = x - total;
  if (tid < kBins) {
    for (int w = 0; w < warp; w++) binstart += s_wsum[w];
    int off = binstart;
#pragma unroll
    for (int w = 0; w < kWarps; w += 2) {
      s_whist[w * kBins + tid] = (uint16_t)off;
      off += (int)(cnt[w / 2] & 0xFFFFu);
      s_whist[(w + 1) * kBins + tid] = (uint16_t)off;
      off += (int)(cnt[w / 2] >> 16);
    }
  }
  __syncthreads();
  // stage the pairs in the order of their destination (a permutation of the
  // tile: counters and ranks come from these same registers)
#pragma unroll
  for (int i = 0; i < kIpt; i++) {
    const uint32_t r = i & 1 ? rank[i / 2] >> 16 : rank[i / 2] & 0xFFFFu;
    const int pos = (int)(wh[((key[i] ^ flip) >> shift) & 255u] + r);
    if ((full || wbase + 32 * i < tile_n)) {
      s_key[pos] = key[i];
      s_val[pos] = val[i];
    }
  }
  // decoupled look-back for bin b = tid, kLook predecessors per round trip
  if (tid < kBins) {
    int excl = 0;
    if (tile > 0) {
      int t = tile - 1;
      uint32_t spins = 0;
      bool found = false;
      while (!found) {
        uint64_t v[kLook];
#pragma unroll
        for (int u = 0; u < kLook; u++)
          v[u] = t - u >= 0 ? ld_relaxed_u64(&status[(int64_t)(t - u) * kBins + tid]) : kFlagIncl;
        int used = 0;
        bool open = true;
#pragma unroll
        for (int u = 0; u < kLook; u++) {
          open = open && (v[u] & kFlagMask) != 0;
          if (open) {
            excl += (int)(uint32_t)v[u];
            used++;
            if ((v[u] & kFlagMask) == kFlagIncl) {
              found = true;
              open = false;
            }
          }
        }
        t -= used;
        if (!found && used == 0) {
          if (++spins > kSpinLimit || ld_relaxed_i32(&ctrl->error) != 0) {
            raise_error(&ctrl->error, CRT_ERR_DEVICE_TIMEOUT);
            s_stop = 1;  // nothing of this tile is written
            break;
          }
          if (spins > 64) __nanosleep(64);
        }
      }
      if (found)
        st_relaxed_u64(&status[(int64_t)tile * kBins + tid], kFlagIncl | (uint32_t)(excl + total));
    }
    // The bin's pairs go to [bucket + excl, + total): out of range only where the
    // keys are not the ones the histograms were made from (a caller's columns that
    // change during the call).  One test per bin: one per pair took 2% of a pass.
    if (total > 0 && (uint32_t)(bucket + excl) > (uint32_t)(n - total)) s_stop = 1;
    s_gbase[tid] = bucket + excl - binstart;
  }
  __syncthreads();
  chain_next();
  if (s_stop) return;
#pragma unroll
  for (int i = 0; i < kIpt; i++) {
    const int j = tid + i * kThreads;
    if (full || j < tile_n) {
      const uint32_t k = s_key[j];
      const int d = s_gbase[((k ^ flip) >> shift) & 255u] + j;
      // evict-first: a pass's output is read once, by the next pass, and
      // the look-back status words and the next tiles' runs want L2
      if (!drop_keys) __stcs(dst_k + d, k);
      __stcs(dst_v + d, s_val[j]);
    }
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct SweepShape {
  int threads;
  int tile;
  size_t smem;
  void (*fn)(int, SortCols, int64_t, uint64_t*, SortCtrl*);
};

#define CRT_SHAPE(T, I, B) {T, (T) * (I), SweepSmem<T, I>::kBytes, sweep_kernel<T, I, B>}
// Tile shapes by pair count: {most pairs, shape}.  A tile's fixed cost (ticket,
// bin scan, look-back) is a few microseconds whatever its size, so large sorts
// want large tiles, as large as the registers hold without spills (512 threads
// x 14; x 16 spills); small ones want enough tiles to use the SMs, and CTAs per
// SM (256 x 8 at six: 40 registers, 28 bytes of them spilled).  Sort of a
// build (four passes, us with event overhead), by threads x keys:
//   pairs   256x4  256x8  256x16  384x16  512x14  512x16  512x20
//    20k       37     43      43      49      49      52      57
//   200k       49     45      50      51      52      58      59
//     1M        -     73      67      65      59      64      65
//     3M        -    133     123     110     112     112     100
//    10M        -    346     291     270     260     272     274
//   100M        -   3192    2619    2394    2241    2279    2369
static const struct {
  int64_t most;
  SweepShape shape;
} kShapes[] = {
    {1 << 16, CRT_SHAPE(256, 4, 4)},
    {400'000, CRT_SHAPE(256, 8, 6)},
    {INT64_MAX, CRT_SHAPE(512, 14, 2)},
};

static const SweepShape& shape_for(int64_t n)
{
  int i = 0;
  while (n > kShapes[i].most) i++;
  return kShapes[i].shape;
}

static int64_t sort_tiles(int64_t n) { return std::max<int64_t>(1, cdiv(n, shape_for(n).tile)); }

size_t sort_zero_bytes(int64_t n, int digits)
{
  return sizeof(SortCtrl) + (size_t)digits * sort_tiles(n) * kBins * sizeof(uint64_t);
}

void sort_passes(const SortCols& cols, int64_t n, int digits, void* zero_block, cudaStream_t stream)
{
  const SweepShape& S = shape_for(n);
  const int64_t tiles = sort_tiles(n);
  SortCtrl* ctrl = sort_ctrl(zero_block);
  // a pass of at most one tile per SM asks for more than half of an SM's shared
  // memory: started while the pass before drains, its CTAs would otherwise share
  // the first SMs that fall free
  const size_t smem = tiles <= sm_count() ? std::max<size_t>(S.smem, 116 * 1024) : S.smem;
  allow_smem(S.fn, 1024);
  for (int d = 0; d < digits; d++) {
    ProfScope ps("sort_pass", stream);
    uint64_t* status = (uint64_t*)(ctrl + 1) + (size_t)d * tiles * kBins;
    launch_after(S.fn, (unsigned)tiles, S.threads, smem, stream, d, cols, n, status, ctrl);
  }
  CRT_LAUNCHED(digits);
}

}  // namespace crt
