// Whether the 16-bit screen of srgemm_screened.cuh can help with the operands of a product, from a sample of them.
//
// The screen cannot hold values of the sign that improves most (negative ones under min, negative ones under max too: its fixed
// point starts at zero), and its 16 bits cannot tell sums apart that lie far below the largest operand.  On such data it does nearly
// every block exactly and loses to the kernel that does nothing else (4096^3, signed values: 18.4 ms against 12.3).  Only the
// operands know, and a flag in memory would have to live somewhere between two launches.  So the host launches both kernels, and
// every CTA of either looks at the same sample and comes to the same answer: one of the two launches returns at once.  The sample
// decides about speed alone: whichever kernel runs is exact.
// 12288 elements of each operand, as 384 stretches of 32 spread over the storage lines: values that occur once in 5000 are found with
// 99 %, once in 30 000 with 56 %.
#pragma once

#include "ptx.cuh"

namespace cuasr_b200 {

constexpr int kSampleThreads = 384;
constexpr int kSampleStretches = 32;               // of 32 elements, per warp and operand
constexpr float kSampleFine = 1.0f / 512;          // of the largest value: 32 steps of the fixed point

// Called by all threads of a CTA before anything else uses the named barriers or shared memory; element (r, k) of an operand is at
// base[r * ld + k] (along k) or base[r + k * ld].  True where the screen should help; the same for all threads.
template <bool kMax>
__device__ __forceinline__ bool screen_helps(const double* a, long long lda, bool a_along_k, int M, const double* b, long long ldb,
                                             bool b_along_k, int N, int K) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  // All loads at once, and every CTA begins elsewhere in the list, so that they do not all wait for the same lines.
  constexpr uint32_t kParts = kSampleThreads / 32 * kSampleStretches;
  const uint32_t first_part = blockIdx.x * 97u;
  float x[2][kSampleStretches];
#pragma unroll
  for (int s = 0; s < 2 * kSampleStretches; ++s) {
    const bool first = s < kSampleStretches;
    const double* base = first ? a : b;
    const bool along_k = first ? a_along_k : b_along_k;
    const int rows = first ? M : N, extent = along_k ? K : rows, lines = along_k ? rows : K;
    // line and place on it: multiples of the golden section and of another irrational number, modulo one
    const uint32_t part = (first_part + warp * kSampleStretches + s % kSampleStretches) % kParts + 1;
    const int line = (int)__umulhi(part * 2654435769u, (uint32_t)lines);
    const int room = extent > 32 ? extent - 31 : 1;
    const int at = min((int)__umulhi(part * 1779033704u, (uint32_t)room) + lane, extent - 1);
    const double v = __ldg(base + (long long)line * (first ? lda : ldb) + at);
    x[s / kSampleStretches][s % kSampleStretches] = kMax ? __double2float_ru(v) : __double2float_rd(v);
  }
  float largest = 0.0f;
  bool unfit = false;
#pragma unroll
  for (int s = 0; s < 2 * kSampleStretches; ++s) {
    const float v = x[s / kSampleStretches][s % kSampleStretches];
    const bool finite = fabsf(v) < INFINITY;
    unfit |= kMax ? v == INFINITY || (finite && v < 0.0f) : v < 0.0f;
    if (finite) largest = fmaxf(largest, v);
  }
  // the largest value of the CTA: floats that are not negative compare like integers
  __shared__ unsigned int tops[kSampleThreads / 32];
  const unsigned int top = __reduce_max_sync(~0u, __float_as_uint(largest));
  if (lane == 0) tops[warp] = top;
  if (__syncthreads_or(unfit)) return false;
  if (kMax) return true;                 // large sums are what it keeps; small values do not matter to it
  unsigned int all = 0;
#pragma unroll
  for (int w = 0; w < kSampleThreads / 32; ++w) all = max(all, tops[w]);
  const float fine_below = __uint_as_float(all) * kSampleFine;
  int fine_a = 0, fine_b = 0;
#pragma unroll
  for (int s = 0; s < kSampleStretches; ++s) {
    fine_a += x[0][s] > 0.0f && x[0][s] < fine_below;
    fine_b += x[1][s] > 0.0f && x[1][s] < fine_below;
  }
  // Expected number of k for which both terms of a sum are that small.  With a few of them the minima are sums the fixed point
  // cannot tell apart.
  __shared__ int fine[2][kSampleThreads / 32];
  const int wa = __reduce_add_sync(~0u, fine_a), wb = __reduce_add_sync(~0u, fine_b);
  if (lane == 0) { fine[0][warp] = wa; fine[1][warp] = wb; }
  __syncthreads();
  int na = 0, nb = 0;
#pragma unroll
  for (int w = 0; w < kSampleThreads / 32; ++w) { na += fine[0][w]; nb += fine[1][w]; }
  __syncthreads();
  constexpr float kSamples = kSampleThreads * kSampleStretches;
  return (na / kSamples) * (nb / kSamples) * (float)K < 4.0f;
}

// The same as a call, which leaves the code behind it other registers.
template <bool kMax>
__device__ __noinline__ bool screen_helps_called(const double* a, long long lda, bool a_along_k, int M, const double* b, long long ldb,
                                                 bool b_along_k, int N, int K) {
  return screen_helps<kMax>(a, lda, a_along_k, M, b, ldb, b_along_k, N, K);
}

}  // namespace cuasr_b200
