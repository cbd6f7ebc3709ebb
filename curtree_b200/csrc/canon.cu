// Canonical pair order on the GPU: (window, box id) ascending, the order the
// reference's drivers produce on the host with two stable sorts, first by box
// id and then by window (src/rtree_test_frontier.cu:102-105).  Two stable
// radix sorts do the same here: by box id carrying the window, then by window
// carrying the box id.  Both keys are compared as signed ints, as the
// reference's int ids are.
#include <cuda_runtime.h>

#include "internal.h"

namespace crt {

// Digit histograms of both columns (signed order: the top digit's sign bit
// flipped), four of the box ids and four of the windows; the last CTA plans
// the passes.  The histograms do not depend on the order of the pairs, so one
// read serves all eight passes.
__global__ void __launch_bounds__(256)
    canon_hist_kernel(const int32_t* __restrict__ fid, const int32_t* __restrict__ tid, int64_t n,
                      SortCtrl* __restrict__ ctrl)
{
  __shared__ uint32_t sh[2 * kDigits][kBins];
  for (int i = threadIdx.x; i < 2 * kDigits * kBins; i += blockDim.x) (&sh[0][0])[i] = 0;
  __syncthreads();
  constexpr int kPer = 4;  // pairs in flight per thread
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += kPer * stride) {
    uint32_t k[kPer], w[kPer];
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      const int64_t i = min(i0 + u * stride, n - 1);
      k[u] = (uint32_t)fid[i] ^ 0x80000000u;
      w[u] = (uint32_t)tid[i] ^ 0x80000000u;
    }
#pragma unroll
    for (int u = 0; u < kPer; u++) {
      if (i0 + u * stride < n) {
#pragma unroll
        for (int d = 0; d < kDigits; d++) {
          atomicAdd(&sh[d][key_digit(k[u], d)], 1u);
          atomicAdd(&sh[kDigits + d][key_digit(w[u], d)], 1u);
        }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * kDigits * kBins; i += blockDim.x) {
    const uint32_t v = (&sh[0][0])[i];
    if (v) atomicAdd(&ctrl->hist[i], v);
  }
  sort_plan(ctrl, n, 2 * kDigits);
}

// Short lists: one CTA sorts the pairs in shared memory as 64-bit keys (window
// above, box id below, sign bits flipped) with a bitonic network (Batcher,
// "Sorting networks and their applications", 1968).  Equal keys are equal
// pairs, so stability does not matter.  Thread t compares elements i and i + j
// with i = 2t - (t mod j): for j <= 32 a warp stays inside its own 64
// elements and needs no block barrier.  A call with 244 pairs takes 20 us;
// its eight radix passes, nearly all launch latency, took 64 us.
constexpr int kCanonSmall = 8192;

__global__ void __launch_bounds__(1024)
    canon_small_kernel(int32_t* __restrict__ fid, int32_t* __restrict__ tid, int n, int size)
{
  extern __shared__ unsigned long long s_pair[];
  for (int i = threadIdx.x; i < size; i += blockDim.x)
    s_pair[i] = i < n ? (unsigned long long)((uint32_t)tid[i] ^ 0x80000000u) << 32 |
                            ((uint32_t)fid[i] ^ 0x80000000u)
                      : ~0ull;
  __syncthreads();
  for (int k = 2; k <= size; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = threadIdx.x; t < size / 2; t += blockDim.x) {
        const int i = 2 * t - (t & (j - 1));
        const unsigned long long a = s_pair[i], b = s_pair[i + j];
        if ((a > b) == ((i & k) == 0)) {
          s_pair[i] = b;
          s_pair[i + j] = a;
        }
      }
      // the next step's elements: this warp's own (j <= 32), or any warp's
      if (j > 32 || (j == 1 && k >= 64)) __syncthreads();
      else __syncwarp();
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const unsigned long long v = s_pair[i];
    tid[i] = (int32_t)((uint32_t)(v >> 32) ^ 0x80000000u);
    fid[i] = (int32_t)((uint32_t)v ^ 0x80000000u);
  }
}

// A sort of one pass ends in the scratch buffer: back to the caller's arrays.
__global__ void canon_copy_kernel(const SortCtrl* __restrict__ ctrl, int64_t n,
                                  const uint32_t* __restrict__ sf, const uint32_t* __restrict__ st,
                                  uint32_t* __restrict__ fid, uint32_t* __restrict__ tid)
{
  chain_wait();
  if (ctrl->n_active != 1) return;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    fid[i] = sf[i];
    tid[i] = st[i];
  }
}

int pairs_canonicalize(int32_t* fid, int32_t* tid, int64_t n, cudaStream_t stream)
{
  if (n < 0 || (n > 0 && (!fid || !tid))) return fail(CRT_ERR_INVALID_ARG, "canonicalize: bad arguments");
  if (n <= 1) return CRT_OK;
  if (n > INT32_MAX)
    return fail(CRT_ERR_NOT_SUPPORTED, "canonicalize: at most INT32_MAX pairs per call");
  if (n <= kCanonSmall) {
    int size = 64;
    while (size < n) size <<= 1;
    const size_t smem = sizeof(unsigned long long) * (size_t)size;
    cudaFuncSetAttribute(canon_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(sizeof(unsigned long long) * kCanonSmall));
    canon_small_kernel<<<1, std::min(1024, size / 2), smem, stream>>>(fid, tid, (int)n, size);
    CRT_LAUNCHED(1);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    return e == cudaSuccess ? CRT_OK : cuda_fail(e, "canonicalize");
  }
  const size_t zero = (sort_zero_bytes(n, 2 * kDigits) + 255) / 256 * 256;
  const size_t kv = ((size_t)n * 4 + 255) / 256 * 256;
  char* scr = nullptr;
  if (cudaMallocAsync((void**)&scr, zero + 4 * kv, stream) != cudaSuccess) {
    cudaGetLastError();
    return fail(CRT_ERR_OOM, "canonicalize: scratch allocation failed");
  }
  // by box id (carrying the window), then stably by window (carrying the box
  // id): passes 4-7 take the other column's digits.  The first pass reads the
  // caller's arrays and the last one writes them.
  SortCols cols{};
  cols.key[0] = (uint32_t*)fid;
  cols.val[0] = (uint32_t*)tid;
  for (int b = 0; b < 2; b++) {
    cols.key[1 + b] = (uint32_t*)(scr + zero + 2 * b * kv);
    cols.val[1 + b] = (uint32_t*)(scr + zero + (2 * b + 1) * kv);
  }
  cols.flip = 0x80000000u;
  cols.home = true;
  SortCtrl* ctrl = sort_ctrl(scr);
  const int grid = (int)std::min<int64_t>(cdiv(n, 256), (int64_t)sm_count() * 8);
  cudaMemsetAsync(scr, 0, sort_zero_bytes(n, 2 * kDigits), stream);
  // at least 2048 pairs per CTA: each adds up to 2048 bins to the global
  // histograms (384k pairs with one CTA per 325: 16 us instead of 5)
  const int hist_grid = (int)std::min<int64_t>(cdiv(n, 2048), (int64_t)sm_count() * 8);
  canon_hist_kernel<<<hist_grid, 256, 0, stream>>>(fid, tid, n, ctrl);
  sort_passes(cols, n, 2 * kDigits, scr, stream);
  launch_after(canon_copy_kernel, (unsigned)grid, 256, 0, stream, ctrl, n, cols.key[1], cols.val[1],
               cols.key[0], cols.val[0]);
  CRT_LAUNCHED(2);
  int dev_err = 0;
  cudaMemcpyAsync(&dev_err, &ctrl->error, sizeof(int), cudaMemcpyDeviceToHost, stream);
  cudaFreeAsync(scr, stream);
  cudaError_t e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_fail(e, "canonicalize");
  if (dev_err) return fail(dev_err, "canonicalize: device-side wait timed out in the radix sort");
  return CRT_OK;
}

// ---------------------------------------------------------------------------
// Per-window counts and order-independent digests of a pair list.  The
// reference's drivers check a result by sorting both pair vectors and
// comparing them (src/rtree_test_frontier.cu:102-123); at billions of pairs
// the same check is a per-window count plus a per-window sum (mod 2^64) of a
// 64-bit mix of each (window, box id) pair, which any pair order gives alike.
// The mix is the splitmix64 finaliser (Steele, Lea and Flood, "Fast
// splittable pseudorandom number generators", OOPSLA 2014).
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long pair_mix(unsigned long long z)
{
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Each warp takes spans of kDigestSpan consecutive pairs, 256 per step: a lane
// holds eight consecutive pairs (two 16-byte loads per column, so a warp's
// loads are whole lines; one thread walking a run of 64 pairs on its own
// touched 32 lines per load).  Bound by the read of the pairs: 1.35e9 pairs of
// a mixed window batch took 10.7 ms that way (1.0 TB/s), about 1.9 ms now.  A result comes window by
// window, in runs longer than a step for all but the smallest windows: while
// every pair of a step belongs to the warp's open window, the lanes only add
// to their own sums, and the warp adds them up (two 64-bit atomics) when the
// window changes.  A step that meets several windows adds up runs of equal
// windows over neighbouring lanes first, so a run costs one pair of atomics
// however many lanes hold it.  Pairs are read through L2 only (ld.global.cg):
// they may come from a kernel still running on another stream, such as the
// serving loop, whose completed requests this checks.
constexpr int kDigestPer = 8;
constexpr int kDigestStep = 32 * kDigestPer;
constexpr int kDigestSpan = 16 * kDigestStep;

struct DigestOut {
  unsigned long long* __restrict__ counts;
  unsigned long long* __restrict__ hashes;
  __device__ __forceinline__ void add(long long w, unsigned c, unsigned long long h) const
  {
    if (w < 0 || c == 0) return;  // -1: pairs outside [0, nq), counted apart
    atomicAdd(&counts[w], (unsigned long long)c);
    atomicAdd(&hashes[w], h);
  }
};

__device__ __forceinline__ void flush_window(const DigestOut& o, long long w, unsigned c,
                                             unsigned long long h)
{
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) h += __shfl_down_sync(0xffffffffu, h, s);
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) o.add(w, c, h);
}

// kVec: fid and tid are 16-byte aligned.
template <bool kVec>
__global__ void __launch_bounds__(256)
    digest_kernel(const int32_t* __restrict__ fid, const int32_t* __restrict__ tid, int64_t n,
                  int64_t base, int64_t nq, DigestOut out, unsigned long long* __restrict__ bad)
{
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  unsigned nbad = 0;
  for (int64_t s0 = warp * kDigestSpan; s0 < n; s0 += nwarps * kDigestSpan) {
    const int64_t s1 = min(n, s0 + kDigestSpan);
    long long open = -1;  // the warp's open window (the same in every lane)
    unsigned oc = 0;      // this lane's share of it
    unsigned long long oh = 0;
    for (int64_t i0 = s0; i0 < s1; i0 += kDigestStep) {
      const int64_t i = i0 + lane * kDigestPer;
      int t[kDigestPer], f[kDigestPer];
      const int m = (int)max((int64_t)0, min((int64_t)kDigestPer, s1 - i));  // pairs of this lane
      if (kVec && m == kDigestPer) {
#pragma unroll
        for (int v = 0; v < kDigestPer / 4; v++) {
          const int4 a = __ldcg(reinterpret_cast<const int4*>(tid + i) + v);
          const int4 b = __ldcg(reinterpret_cast<const int4*>(fid + i) + v);
          t[4 * v] = a.x; t[4 * v + 1] = a.y; t[4 * v + 2] = a.z; t[4 * v + 3] = a.w;
          f[4 * v] = b.x; f[4 * v + 1] = b.y; f[4 * v + 2] = b.z; f[4 * v + 3] = b.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < kDigestPer; k++) {
          t[k] = k < m ? __ldcg(tid + i + k) : 0;
          f[k] = k < m ? __ldcg(fid + i + k) : 0;
        }
      }
      // one window over the whole step?
      const int t0 = __shfl_sync(0xffffffffu, t[0], 0);
      bool same = m == kDigestPer;
#pragma unroll
      for (int k = 0; k < kDigestPer; k++) same = same && t[k] == t0;
      if (__all_sync(0xffffffffu, same)) {
        const long long w = (long long)t0 + base;
        if (w < 0 || w >= nq) {
          nbad += kDigestPer;
          continue;
        }
        if (w != open) {
          if (open >= 0) flush_window(out, open, oc, oh);
          open = w;
          oc = 0;
          oh = 0;
        }
        oc += kDigestPer;
#pragma unroll
        for (int k = 0; k < kDigestPer; k++)
          oh += pair_mix(((unsigned long long)(uint32_t)w << 32) | (uint32_t)f[k]);
        continue;
      }
      // Several windows: this lane's first run (window w0) and last run (w1),
      // added up with its neighbours'; runs between them are its own.
      long long w0 = -1, w1 = -1, cur = -1;
      unsigned c0 = 0, c1 = 0, c = 0;
      unsigned long long h0 = 0, h1 = 0, h = 0;
      int runs = 0;
#pragma unroll
      for (int k = 0; k < kDigestPer; k++) {
        if (k < m) {
          long long w = (long long)t[k] + base;
          if (w < 0 || w >= nq) {
            nbad++;
            w = -1;
          }
          if (runs == 0 || w != cur) {
            if (runs == 1) {
              w0 = cur; c0 = c; h0 = h;
            } else if (runs > 1) {
              out.add(cur, c, h);
            }
            runs++;
            cur = w;
            c = 0;
            h = 0;
          }
          c++;
          if (w >= 0) h += pair_mix(((unsigned long long)(uint32_t)w << 32) | (uint32_t)f[k]);
        }
      }
      w1 = cur; c1 = c; h1 = h;
      // a lane with several runs gives its first run to the lane before it
      // when that lane's last run is of the same window
      const long long pw = __shfl_up_sync(0xffffffffu, w1, 1);
      const bool give = runs > 1 && lane > 0 && w0 == pw;
      if (runs > 1 && !give) out.add(w0, c0, h0);
      const unsigned gc = __shfl_down_sync(0xffffffffu, give ? c0 : 0u, 1);
      const unsigned long long gh = __shfl_down_sync(0xffffffffu, give ? h0 : 0ull, 1);
      if (lane < 31) {
        c1 += gc;
        h1 += gh;
      }
      // runs of equal last windows over lanes: a lane of one run joins the
      // lane before it; sums flow to the run's first lane
      const bool join = runs == 1 && lane > 0 && w1 == pw;
      const uint32_t heads = ~__ballot_sync(0xffffffffu, join);  // bit 0 is always set
      const uint32_t above = lane == 31 ? 0u : heads & (0xfffffffeu << lane);
      const int end = above ? __ffs(above) - 1 : 32;  // one past the run's last lane
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const unsigned yc = __shfl_down_sync(0xffffffffu, c1, s);
        const unsigned long long yh = __shfl_down_sync(0xffffffffu, h1, s);
        if (lane + s < end) {
          c1 += yc;
          h1 += yh;
        }
      }
      if ((heads >> lane) & 1u) out.add(runs ? w1 : -1, c1, h1);
    }
    if (open >= 0) flush_window(out, open, oc, oh);
  }
  nbad = __reduce_add_sync(0xffffffffu, nbad);
  if (nbad && bad && lane == 0) atomicAdd(bad, (unsigned long long)nbad);
}

int pairs_digest(const int32_t* fid, const int32_t* tid, int64_t n, int64_t window_base,
                 int64_t nq, int64_t* d_counts, uint64_t* d_hashes, int64_t* d_bad,
                 cudaStream_t stream)
{
  if (n < 0 || nq < 0 || (n > 0 && (!fid || !tid)) || (nq > 0 && (!d_counts || !d_hashes)))
    return fail(CRT_ERR_INVALID_ARG, "pairs_digest: bad arguments");
  if (n == 0) return CRT_OK;
  const int64_t spans = cdiv(n, kDigestSpan);
  const int grid = (int)std::min<int64_t>(cdiv(spans, 8), (int64_t)sm_count() * 8);
  const DigestOut out{(unsigned long long*)d_counts, (unsigned long long*)d_hashes};
  unsigned long long* bad = (unsigned long long*)d_bad;
  if (((((uintptr_t)fid) | ((uintptr_t)tid)) & 15) == 0)
    digest_kernel<true><<<grid, 256, 0, stream>>>(fid, tid, n, window_base, nq, out, bad);
  else
    digest_kernel<false><<<grid, 256, 0, stream>>>(fid, tid, n, window_base, nq, out, bad);
  CRT_LAUNCHED(1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "pairs_digest");
  return CRT_OK;
}

}  // namespace crt
