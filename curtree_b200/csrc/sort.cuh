// Interface of the radix sort (sort.cu) to the kernels that make its keys.
#pragma once

#include "common.cuh"

namespace crt {

// Radix digits: four of eight bits per 32-bit column.  8-bit digits (four
// passes, uniform digits skipped) measured faster on a B200 than 10 + 10 + 10
// + 2 (three passes for 30-bit Morton keys): 2.74 against 3.43 ms for 100M
// keys, the 1024-bin passes paying more for ranking, bin scans and look-back
// than the fourth pass costs.
constexpr int kBins = 256;
constexpr int kDigits = 4;

__device__ __forceinline__ uint32_t key_digit(uint32_t k, int d) { return (k >> (8 * d)) & 255u; }

// Control block of one sort, zeroed by the caller together with the look-back
// status words behind it (sort_zero_bytes).
struct SortCtrl {
  int tile_ctr[2 * kDigits];  // per pass: next tile index
  int error;                  // first device error
  int active;                 // bit d: digit d is not uniform
  int n_active;               // number of active passes
  int done;                   // CTAs of the key kernel that have added their histograms
  int level_done[12];         // a build's level launches: CTAs finished
  uint32_t hist[2 * kDigits * kBins];     // digit histograms, filled by the key kernel
  int bucket_start[2 * kDigits * kBins];  // exclusive prefix of each digit's histogram
};
static_assert(sizeof(SortCtrl) % 16 == 0, "status words follow");

// Where the pairs of a sort lie.  Ping-pong (home == false): pass k reads
// buffer k & 1 and writes the other; the result is in buffer n_active & 1.
// Home: the first pass reads buffer 0 and the last one writes it back, the
// passes between use buffers 1 and 2; a sort of a single pass ends in buffer 1
// (sort_home_copy moves it).
struct SortCols {
  uint32_t* key[3];
  uint32_t* val[3];
  uint32_t flip;     // xor on every key before its digits are taken (0x80000000: signed order)
  bool home;
  bool make_values;  // ping-pong: the first pass makes the values (positions 0..n-1)
  bool drop_keys;    // ping-pong: the last pass writes values only
  __device__ __forceinline__ int src(int step) const
  {
    return home ? (step == 0 ? 0 : 1 + ((step - 1) & 1)) : (step & 1);
  }
  __device__ __forceinline__ int dst(int step, bool last) const
  {
    return home ? (last && step > 0 ? 0 : 1 + (step & 1)) : ((step & 1) ^ 1);
  }
  // selects instead of an indexed parameter array, which would live in local memory
  __device__ __forceinline__ uint32_t* keys(int b) const { return b == 0 ? key[0] : b == 1 ? key[1] : key[2]; }
  __device__ __forceinline__ uint32_t* vals(int b) const { return b == 0 ? val[0] : b == 1 ? val[1] : val[2]; }
};

// Bytes of the zeroed block of a sort of n pairs over `digits` digits.
size_t sort_zero_bytes(int64_t n, int digits = kDigits);
inline SortCtrl* sort_ctrl(void* zero_block) { return (SortCtrl*)zero_block; }
// Enqueues the passes (histograms filled, passes planned).  digits == 8: by
// the key column's four digits, then by the value column's.
void sort_passes(const SortCols& cols, int64_t n, int digits, void* zero_block, cudaStream_t stream);

// Called by every CTA of a key kernel once its histograms are added: the last
// CTA to arrive plans the passes.  A digit with all keys in one bin is uniform
// and its pass is skipped (a stable pass over it leaves the order unchanged);
// the exclusive prefix of a digit's bins is each bucket's start.  Needs at
// least 32 threads per digit.
__device__ __forceinline__ void sort_plan(SortCtrl* ctrl, int64_t n, int digits)
{
  __shared__ int s_last;
  __shared__ int s_active;
  __threadfence();  // this thread's histogram additions before the count
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(&ctrl->done, 1) == (int)gridDim.x - 1;
    s_active = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int d = warp; d < digits; d += blockDim.x >> 5) {
    uint32_t v[kBins / 32];
    bool uniform = false;
#pragma unroll
    for (int c = 0; c < kBins / 32; c++) {
      v[c] = __ldcg(&ctrl->hist[d * kBins + 32 * c + lane]);
      uniform |= (int64_t)v[c] == n;
    }
    uint32_t carry = 0;
#pragma unroll
    for (int c = 0; c < kBins / 32; c++) {
      uint32_t x = v[c];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      ctrl->bucket_start[d * kBins + 32 * c + lane] = (int)(carry + x - v[c]);
      carry += __shfl_sync(0xffffffffu, x, 31);
    }
    if (!__any_sync(0xffffffffu, uniform) && lane == 0) atomicOr(&s_active, 1 << d);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ctrl->active = s_active;
    ctrl->n_active = __popc((unsigned)s_active);
  }
}

}  // namespace crt
