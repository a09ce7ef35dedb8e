// Screened tropical SRGEMM: D = min(A + B, beta + C) (or max) with most products looked at in 16 bits only.
//
// What bounds the ordinary kernel: a product of the fp64 min-plus ring costs 6.6 clocks per scheduler (add, compare, two
// selects: 12 register words at two a clock are 6).  But a product
// matters only if it IMPROVES its element, and the n-th product of an element does so with probability about 1/n.  So
// each operand tile is also kept as 16-bit fixed-point numbers rounded towards "better" (down for min, up for max): the
// sum of two such numbers is never worse than the exact sum, and one fused packed add-min instruction handles two
// products in 2 clocks (measured 1.08 per product with its shared-memory reads).  A block of k whose 16-bit sums
// cannot beat the element's current value cannot contain an improvement and is done; the few (element, block) pairs
// that might improve are recomputed exactly, by four lanes each, from the exact tile in shared memory.  The result is
// bit for bit that of the exact computation: the screen only ever lets too much through.  That includes the sign of zeros:
// alpha and beta are not negative zeros here, so no term of D is one, and every product gets the + 0 that alpha stands for.
//
// Fixed point: q(x) = floor(x * 2^e) (ceil for max), finite values at most 16382, +inf (-inf for max) = 32767 (-16384),
// so sums of finite values and sums with an infinity do not overlap.  2^e comes from the largest finite value of the
// tiles seen so far.  A stage with a negative or too large finite value is "unfit" and done exactly; a larger 2^-e
// follows for the next.
//
// What the screen saves depends on the data (4096^3, 12.3 ms with the exact kernel of srgemm_tma.cuh): sparse edges 7.1 ms,
// uniform values 7.3, small whole numbers 4.6, sums that improve along k 7.5.  Values it cannot hold, negative ones or
// magnitudes over hundreds of decades, are done exactly in runs of blocks, 15.8 ms; a sample of the operands sends such data to the
// exact kernel (screen_sample.cuh), and the runs are for what the sample does not show.
//
// The running result lives in D itself: an element is written when it improves, by the lane that found it.  Elements
// and blocks are independent of order, so K may be cut into pieces for different CTAs, which then meet in D by
// compare-and-swap (pieces > 1; D initialised by an earlier launch).
//
// Structure: one persistent CTA per SM.  Warps 8..11 bring exact tiles in (TMA or gather), turn them into 16-bit tiles;
// warps 0..7 own 64 x 32 blocks of the 128 x 128 tile, 8 x 8 elements per lane.  A stage is a block of 32 k, two stages.
#pragma once

#include "srgemm_tma.cuh"

namespace cuasr_b200 {

struct ScreenParams {
  using T = double;
  int M, N, K;
  const T* A;  long long lda;      // gathered operands only
  const T* B;  long long ldb;
  int a_mode, b_mode;              // LoadMode
  const T* C;  long long ldc;      // row-major; may alias D
  T* D;        long long ldd;      // row-major
  T beta, add_identity;
  int read_c;
  int n_extra;
  T* extra_d[kMaxDestinations - 1];
  int tiles_m, tiles_n, pieces, blocks_per_piece;
  int if_it_helps;                 // return at once where screen_helps says no (the exact kernel's launch follows)
  unsigned int* status;
};

constexpr int kScreenExactBytes = 65536;      // 2 operands x 128 rows x 256 bytes
constexpr int kScreenBlock = 32;                // k per block: 256 bytes of an exact row
constexpr int kScreenStageBytes = kScreenExactBytes + 2 * 128 * kScreenBlock * 2;
constexpr int kScreenStages = 2;
constexpr int kScreenBoundBytes = 8 * 64 * 32 * 2;   // per warp, element and lane: the value a 16-bit sum has to beat
constexpr int kListGroups = 4;                       // groups of eight elements that a warp recomputes at a time
constexpr int kListed = 96;                          // elements to recompute that a warp lists at a time
constexpr int kScreenListBytes = 8 * kListed * 2;
constexpr int kScreenRowBytes = kConsumerThreads * 8 * (int)sizeof(double);   // eight accumulators of every lane, on their way to D
constexpr int kScreenSmemBytes = kScreenStages * kScreenStageBytes + kScreenBoundBytes + kScreenListBytes + kScreenRowBytes + 512 + 1024;
static_assert(kScreenSmemBytes <= kMaxSmemBytes, "one CTA's shared memory");

__device__ __forceinline__ void sts16(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 lds16u(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds2(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts2(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"((uint16_t)v) : "memory");
}

// True where `ok` holds for all producer threads.
__device__ __forceinline__ bool producers_agree(bool ok) {
  uint32_t all;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, 2, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(all) : "r"((uint32_t)ok), "n"(kProducerWarps * 32) : "memory");
  return all != 0;
}

template <bool kMax>
struct Screen {
  static constexpr float kFiniteLimit = 16382.0f;
  // scaled fp32 image of an element, rounded towards "better" in both steps (the scaling is inexact where it underflows:
  // rounded to nearest, a tiny negative value would come out as a zero and a tiny maximum would lose its upper bound)
  static __device__ __forceinline__ float scaled(double x, float scale) {
    return kMax ? __fmul_ru(__double2float_ru(x), scale) : __fmul_rd(__double2float_rd(x), scale);
  }
  static constexpr uint32_t kNever = kMax ? 0x8000u : 0x7FFFu;       // the infinity no sum improves with
  static constexpr uint32_t kNothing = kMax ? 0x7FFFu : 0u;          // bound no sum beats (elements outside the matrix)
  // Widens [smallest, largest] by two scaled values.  The infinity that never improves (+inf for min) is legal and
  // becomes NaN here, which min and max ignore; the other one stays and makes the stage unfit.
  static __device__ __forceinline__ void survey(float y0, float y1, float& largest, float& smallest) {
    const float z0 = fmaf(y0, 0.0f, y0), z1 = fmaf(y1, 0.0f, y1);
    largest = kMax ? max3(largest, y0, y1) : max3(largest, z0, z1);
    smallest = kMax ? min3(smallest, z0, z1) : min3(smallest, y0, y1);
  }
  // 16-bit bound of a scaled operand element: saturating, so that infinities land on the ends of the range
  static __device__ __forceinline__ uint32_t quantise(float y) {
    int16_t q;
    if (kMax) asm("cvt.rpi.sat.s16.f32 %0, %1;" : "=h"(q) : "f"(y));
    else      asm("cvt.rmi.sat.s16.f32 %0, %1;" : "=h"(q) : "f"(y));
    return (uint16_t)q;
  }
  static __device__ __forceinline__ uint32_t fold(uint32_t a, uint32_t b, uint32_t acc) {
    return kMax ? __viaddmax_s16x2(a, b, acc) : __viaddmin_u16x2(a, b, acc);
  }
  // The bound of an element with current value v: a 16-bit sum may stand for an improvement only if it is below
  // (min) or above (max) it.  min: exact sum < v implies (sum of floors) < v * s, i.e. < ceil(v * s); the product is
  // rounded up, so that it only ever gets larger where it is inexact.
  static __device__ __forceinline__ uint32_t bound(double v, float scale) {
    const double y = kMax ? __dmul_rd(v, (double)scale) : __dmul_ru(v, (double)scale);
    if (y != y) return kNothing;                                        // a NaN (from C) stays: nothing is better than it
    if (kMax) {
      if (!(y >= 0.0)) return (uint32_t)(uint16_t)-1;                  // any sum of finite values
      if (y >= 32766.0) return 32766u;
      return (uint32_t)(int)y;
    }
    if (!(y < 32766.0)) return 32767u;                                 // any sum of finite values
    if (y < 0.0) return 0u;                                             // nothing: no negative values in a fit stage
    return (uint32_t)(int)ceil(y);
  }
  static __device__ __forceinline__ bool sooner(uint32_t a, uint32_t b) { return kMax ? (int16_t)a > (int16_t)b : a < b; }
  static __device__ __forceinline__ bool better(double candidate, double current) { return kMax ? candidate > current : candidate < current; }
};

// current = better(value, current) in memory other CTAs write too; returns the value that is there afterwards.
template <bool kMax>
__device__ __forceinline__ double improve_shared(double* at, double value, double seen) {
  while (Screen<kMax>::better(value, seen)) {
    const unsigned long long got = atomicCAS(reinterpret_cast<unsigned long long*>(at), (unsigned long long)__double_as_longlong(seen), (unsigned long long)__double_as_longlong(value));
    if (got == (unsigned long long)__double_as_longlong(seen)) return value;
    seen = __longlong_as_double((long long)got);
  }
  return seen;
}

// *at = better(*at, value) without reading it back.  `value` is not negative, and then the bit patterns of any double
// compare with it like signed integers; adding zero makes a negative zero a positive one, whose pattern does.
template <bool kMax>
__device__ __forceinline__ void merge_into(double* at, double value) {
  value += 0.0;
  if (kMax) atomicMax(reinterpret_cast<long long*>(at), __double_as_longlong(value));
  else      atomicMin(reinterpret_cast<long long*>(at), __double_as_longlong(value));
}

template <bool kMax>
__global__ void __launch_bounds__(kTmaThreads, 1)
srgemm_screened_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                       const __grid_constant__ ScreenParams p) {
  using T = double;
  using S = Screen<kMax>;
  using RingT = Ring<kMax ? CUASR_OP_MAXIMUM : CUASR_OP_MINIMUM, CUASR_OP_PLUS, T>;
  constexpr int EV = 16 / (int)sizeof(T);
  constexpr int TK = 128 / (int)sizeof(T);          // k per 128-byte column
  constexpr int KB = kScreenBlock;                  // k per stage
  static_assert(KB == 2 * TK, "two 128-byte columns");
  constexpr int kCoarseRow = KB * 2;                // bytes of a 16-bit row: 64
  constexpr int kCoarseChunks = kCoarseRow / 16;    // 4 chunks of 8 k
  constexpr int kExactOperand = 32768, kColumn = 16384;
  constexpr int kCoarseOperand = 128 * kCoarseRow;
  // Elements of a warp (of 2048) above which recomputing them one by one costs more than doing the block exactly, and how
  // many blocks are then done exactly: two, and twice as many each time the next block screened is no better.
  // (4096^3: 8.15 ms with 350 elements on uniform data and 8.25 on sparse edges, 7.98 and 7.68 with 600, 8.21 and 7.66 with 1000)
  constexpr int kExactAbove = 600, kPatience = 2, kMaxPatience = 256;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* bounds_smem = smem + kScreenStages * kScreenStageBytes;
  uint8_t* list_smem = bounds_smem + kScreenBoundBytes;
  uint8_t* rows_smem = list_smem + kScreenListBytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(rows_smem + kScreenRowBytes);   // exact tile landed
  uint64_t* ready_bar = full_bar + kScreenStages;                                     // 16-bit tile written
  uint64_t* empty_bar = ready_bar + kScreenStages;
  // per stage: largest and smallest finite scaled value seen by each producer warp, and the exponent
  volatile float* range = reinterpret_cast<volatile float*>(empty_bar + kScreenStages);   // [stage][warp][2]
  volatile int* stage_exp = reinterpret_cast<volatile int*>(range + kScreenStages * kProducerWarps * 2);
  // per consumer warp: it does the blocks before this one (counted over the CTA's whole work) exactly
  volatile int* exact_until = stage_exp + kScreenStages;
  volatile unsigned int* abandoned = reinterpret_cast<volatile unsigned int*>(exact_until + kConsumerWarps);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const bool gathers = p.a_mode != kLoadTma || p.b_mode != kLoadTma;
  const bool tmas = p.a_mode == kLoadTma || p.b_mode == kLoadTma;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kScreenStages; ++s) {
      mbar_init(&full_bar[s], (tmas ? 1 : 0) + (gathers ? kProducerWarps * 32 : 0));
      mbar_init(&ready_bar[s], kProducerWarps * 32);
      mbar_init(&empty_bar[s], kConsumerWarps);
    }
    *abandoned = 0;
    for (int v = 0; v < kConsumerWarps; ++v) exact_until[v] = 0;
    fence_barrier_init();
  }
  __syncthreads();
  grid_dependency_wait();
  grid_dependency_launch();
  if (p.if_it_helps && !screen_helps<kMax>(p.A, p.lda, p.a_mode != kLoadGatherMN, p.M, p.B, p.ldb, p.b_mode != kLoadGatherMN, p.N, p.K))
    return;

  const int blocks_total = (p.K + KB - 1) / KB;
  const int num_work = p.tiles_m * p.tiles_n * p.pieces;
  const int tiles = p.tiles_m * p.tiles_n;
  // A piece walks its blocks in a scattered order (stride near the golden section, coprime to the count), so that data
  // whose products improve steadily along k does not let an element improve in every block.
  auto stride_of = [&](int count) {
    if (count < 8) return 1;
    int st = (int)(count * 0.618f) | 1;
    auto gcd = [](int a, int b) { while (b) { const int t = a % b; a = b; b = t; } return a; };
    while (gcd(count, st) != 1) st += 2;
    return st % count;
  };

  if (warp >= kConsumerWarps) {
    // ---------------------------------------------------------------- producers
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kProducerRegs));
    const int pw = warp - kConsumerWarps;
    const bool issuer = pw == 0 && lane == 0;
    if (issuer && tmas) {
      prefetch_tensormap(&map_a);
      prefetch_tensormap(&map_b);
    }
    // loads of the next block in this CTA's sequence; (w, b) walk one block ahead of the conversions
    int lw = blockIdx.x, lb = 0, lpos = 0, lcount = 0, lbegin = 0, lstride = 1, lm0 = 0, ln0 = 0;
    auto open_work = [&]() {
      const int piece = lw / tiles, tile = lw - piece * tiles;
      int tm, tn;
      tile_coords(tile, p.tiles_m, p.tiles_n, tm, tn);
      lm0 = tm * 128; ln0 = tn * 128;
      lbegin = piece * p.blocks_per_piece;
      lcount = min(blocks_total - lbegin, p.blocks_per_piece);
      lstride = stride_of(lcount);
      lb = 0; lpos = 0;
    };
    uint32_t lit = 0;
    int k0_even = 0, k0_odd = 0;      // first k of the blocks in the two stages
    bool alive = true;
    auto load_next = [&]() {          // returns after issuing the copies of one block into stage lit % 2
      const int s = lit % kScreenStages;
      const uint32_t round = lit / kScreenStages;
      if (alive && round > 0) alive = mbar_wait(&empty_bar[s], (round - 1) & 1, p.status, kDeviceTimeoutEmpty);
      uint8_t* sa = smem + s * kScreenStageBytes;
      uint8_t* sb = sa + kExactOperand;
      const int k0 = (lbegin + lpos) * KB;
      if (s == 0) k0_even = k0;
      else        k0_odd = k0;
      if (alive && issuer && tmas) {
        mbar_arrive_expect_tx(&full_bar[s], (p.a_mode == kLoadTma ? kExactOperand : 0) + (p.b_mode == kLoadTma ? kExactOperand : 0));
#pragma unroll
        for (int sub = 0; sub < 2; ++sub) {
          if (p.a_mode == kLoadTma) tma_load_2d(sa + sub * kColumn, &map_a, &full_bar[s], k0 + sub * TK, lm0);
          if (p.b_mode == kLoadTma) tma_load_2d(sb + sub * kColumn, &map_b, &full_bar[s], k0 + sub * TK, ln0);
        }
      }
      if (alive && gathers) {
        // beyond K: infinities of the kind that never improves
        const T pad = kMax ? -static_cast<T>(INFINITY) : static_cast<T>(INFINITY);
        if (p.a_mode != kLoadTma) gather_tile<T, 128, 2, true>(smem_u32(sa), p.A, p.lda, p.a_mode, lm0, p.M, k0, p.K, pad, false, pw, lane);
        if (p.b_mode != kLoadTma) gather_tile<T, 128, 2, true>(smem_u32(sb), p.B, p.ldb, p.b_mode, ln0, p.N, k0, p.K, pad, false, pw, lane);
        if (k0 + KB > p.K) {
          cp_async_wait_all();
          mbar_arrive(&full_bar[s]);
        } else {
          cp_async_arrive_noinc(&full_bar[s]);
        }
      }
      ++lit;
      lpos += lstride;
      if (lpos >= lcount) lpos -= lcount;
      if (++lb == lcount) {
        lw += gridDim.x;
        if (lw < num_work) open_work();
      }
    };
    if (lw < num_work) { open_work(); load_next(); }

    int exponent = 0;                 // scale of the 16-bit tiles: 2^exponent
    bool have_exponent = false;
    uint32_t it = 0;
    for (; it < lit; ++it) {
      const int s = it % kScreenStages;
      // the producers meet at named barriers below: they go on, or leave, together
      if (alive) alive = mbar_wait(&full_bar[s], (it / kScreenStages) & 1, p.status, kDeviceTimeoutFull);
      alive = producers_agree(alive);
      if (!alive) break;
      const uint32_t exact = smem_u32(smem + s * kScreenStageBytes);
      const uint32_t coarse = exact + kScreenExactBytes;
      const int k_left = p.K - (s == 0 ? k0_even : k0_odd);          // below KB in the block that reaches beyond K
      // No 16-bit tile for a block that all consumers do exactly (what they promise, they keep).
      bool wanted = false;
#pragma unroll
      for (int v = 0; v < kConsumerWarps; ++v) wanted |= exact_until[v] <= (int)it;
      if (producers_agree(!wanted)) {
        if (lane == 0) {
          range[(s * kProducerWarps + pw) * 2] = INFINITY;            // unfit
          if (pw == 0) stage_exp[s] = exponent;
        }
        mbar_arrive(&ready_bar[s]);
        if (lw < num_work) load_next();
        continue;
      }
      // Two passes where the scale has to be found first (the first stage of the CTA), one otherwise.
      for (int pass = have_exponent ? 1 : 0; pass < 2; ++pass) {     // (uniform: all producers saw the same ranges)
        const float scale = __int_as_float((exponent + 127) << 23);
        float largest = -INFINITY, smallest = INFINITY;
        // a task: 8 k of one row.  8 lanes = 8 rows, so that neither the reads nor the writes of a swizzled chunk conflict
#pragma unroll 2
        for (int task = threadIdx.x - kConsumerThreads; task < 256 * kCoarseChunks; task += kProducerWarps * 32) {
          const int r8 = task & 7, c = (task >> 3) % kCoarseChunks, block = (task >> 3) / kCoarseChunks;   // 32 blocks of 8 rows
          const int row = block * 8 + r8;                             // 0..127: A, 128..255: B
          const uint32_t src = exact + (row >> 7) * kExactOperand + (row & 127) * 128;
          uint32_t words[4];
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            double x[2];
            const int chunk = 4 * c + w;                            // 2 k
            lds16(src + (chunk >> 3) * kColumn + (((chunk & 7) ^ r8) << 4), x);
            const float y0 = S::scaled(x[0], scale), y1 = S::scaled(x[1], scale);
            S::survey(y0, y1, largest, smallest);
            words[w] = S::quantise(y0) | (S::quantise(y1) << 16);
          }
          if (k_left < KB) {
            // TMA fills NaN beyond K; the screen shall see the infinity that never improves
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              if (c * 8 + 2 * w >= k_left) words[w] = (words[w] & 0xFFFF0000u) | S::kNever;
              if (c * 8 + 2 * w + 1 >= k_left) words[w] = (words[w] & 0xFFFFu) | (S::kNever << 16);
            }
          }
          if (kMax) {
#pragma unroll
            for (int w = 0; w < 4; ++w) words[w] = __vmaxs2(words[w], 0xC000C000u);    // -inf + -inf must not wrap
          }
          const uint32_t dst = coarse + (row >> 7) * kCoarseOperand + (row & 127) * kCoarseRow +
                               ((c ^ ((r8 >> 1) & 3)) << 4);
          sts16(dst, make_uint4(words[0], words[1], words[2], words[3]));
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
          largest = fmaxf(largest, __shfl_xor_sync(~0u, largest, d));
          smallest = fminf(smallest, __shfl_xor_sync(~0u, smallest, d));
        }
        if (lane == 0) {
          range[(s * kProducerWarps + pw) * 2] = largest;
          range[(s * kProducerWarps + pw) * 2 + 1] = smallest;
          if (pw == 0) stage_exp[s] = exponent;
        }
        asm volatile("bar.sync 2, %0;" ::"n"(kProducerWarps * 32) : "memory");
        float top = -INFINITY;
#pragma unroll
        for (int w = 0; w < kProducerWarps; ++w) top = fmaxf(top, range[(s * kProducerWarps + w) * 2]);
        // a new scale: room for values twice as large.  The stage it was found on stays unfit (pass 1) unless this is
        // the measuring pass.
        if (pass == 0 || top > S::kFiniteLimit) {
          if (top > 0.0f && top < INFINITY) {
            have_exponent = true;
            const int magnitude = ((__float_as_int(top) >> 23) & 255) - 127;     // floor(log2(top)) at the old scale
            exponent = max(-126, min(126, exponent + 12 - magnitude));
          }
        }
        if (pass == 0) asm volatile("bar.sync 2, %0;" ::"n"(kProducerWarps * 32) : "memory");   // range is written again
      }
      mbar_arrive(&ready_bar[s]);
      // the next block's loads go into the other stage, which the consumers finish while they work on this one
      if (lw < num_work) load_next();
    }
    if (gathers) cp_async_wait_all();
    return;
  }

  // ------------------------------------------------------------------ consumers
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kConsumerRegs));
  const int wm = warp / 4, wn = warp % 4;
  const int lr = lane / 4, lc = lane % 4;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t my_bounds = smem_u32(bounds_smem) + warp * (64 * 32 * 2) + lane * 16;   // row i: + i * 512, element j: + 2 j
  const uint32_t warp_bounds = smem_u32(bounds_smem) + warp * (64 * 32 * 2);
  const uint32_t list = smem_u32(list_smem) + warp * (kListed * 2);
  const uint32_t my_row = smem_u32(rows_smem) + warp * (32 * 8 * (int)sizeof(T)) + lane * 16;   // elements j .. j + EV - 1 of a row: + j * 512 / EV
  const bool shared_d = p.pieces > 1;

  uint32_t it = 0;
  int until = 0, patience = kPatience;      // blocks before `until` are done exactly; length of the next such run
  auto do_exactly = [&](uint32_t from, int blocks) {
    until = max(until, (int)from + blocks);
    if (lane == 0) exact_until[warp] = until;
  };
  for (int w = blockIdx.x; w < num_work; w += gridDim.x) {
    const int piece = w / tiles, tile = w - piece * tiles;
    int tm, tn;
    tile_coords(tile, p.tiles_m, p.tiles_n, tm, tn);
    const int begin = piece * p.blocks_per_piece;
    const int count = min(blocks_total - begin, p.blocks_per_piece);
    const int m_base = tm * 128 + wm * 64, n_base = tn * 128 + wn * 32;
    int my_exp = 1 << 30;             // exponent the bounds were made with
    bool opened = false;              // D holds the running values of this tile
    do_exactly(it, 1);                // the first block has nothing to be screened against

    for (int b = 0; b < count;) {
      const int s = it % kScreenStages;
      // In this order: an exact run below passes blocks without looking at ready_bar, and a parity wait is only sound if
      // the phase before its own is complete.  The loads of block `it` are issued after all producers met in block it - 1,
      // hence after each of them arrived for block it - 2; so once block `it` has landed, that phase is complete.
      mbar_wait_or_abandon(&full_bar[s], (it / kScreenStages) & 1, p.status, kDeviceTimeoutFull, abandoned);
      mbar_wait_or_abandon(&ready_bar[s], (it / kScreenStages) & 1, p.status, kDeviceTimeoutFull, abandoned);
      float top = -INFINITY, low = INFINITY;
#pragma unroll
      for (int v = 0; v < kProducerWarps; ++v) {
        top = fmaxf(top, range[(s * kProducerWarps + v) * 2]);
        low = fminf(low, range[(s * kProducerWarps + v) * 2 + 1]);
      }
      const int exponent = stage_exp[s];
      const float scale = __int_as_float((exponent + 127) << 23);
      const bool unfit = top > S::kFiniteLimit || low < 0.0f;

      if (unfit || (int)it < until) {
        if (unfit && (int)it >= until) {
          do_exactly(it, patience);
          patience = min(2 * patience, kMaxPatience);
        }
        // ---- a run of whole blocks exactly, for all 64 elements of the lane; then merged into D
        T acc[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[i][j] = p.add_identity;
        for (;;) {
          const int sx = it % kScreenStages;
          const uint32_t exact = smem_base + sx * kScreenStageBytes;
          const uint32_t a_base = exact + (wm * 64 + lr) * 128, b_base = exact + kExactOperand + (wn * 32 + lc) * 128;
#pragma unroll 1
          for (int chunk = 0; chunk < 16; ++chunk) {
            const uint32_t at = (chunk >> 3) * kColumn;
            const uint32_t ab = a_base + at + (((chunk ^ lr) & 7) << 4);
            const uint32_t b0 = b_base + at + (((chunk ^ lc) & 7) << 4), b1 = b_base + at + (((chunk ^ (lc + 4)) & 7) << 4);
            T a[8][EV];
#pragma unroll
            for (int i = 0; i < 8; ++i) lds16(ab + i * 1024, a[i]);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              T bj[EV];
              lds16(((j & 1) ? b1 : b0) + j * 512, bj);
#pragma unroll
              for (int e = 0; e < EV; ++e)               // kByColumn of srgemm_tma.cuh
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = RingT::add(a[i][e] + bj[e], acc[i][j]);
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty_bar[sx]);
          ++it;
          if (++b == count || (int)it >= until) break;
          // (the 16-bit tile of the next block is not waited for)
          mbar_wait_or_abandon(&full_bar[it % kScreenStages], (it / kScreenStages) & 1, p.status, kDeviceTimeoutFull, abandoned);
        }
        // Row by row through the lane's own 64 bytes of shared memory, four elements at a time in a loop that is not unrolled: with
        // the accumulators in registers the 64 copies of this code spill all of them.
#pragma unroll
        for (int i = 0; i < 8; ++i) {
#pragma unroll
          for (int j = 0; j < 8; j += EV) sts16(my_row + j * (512 / EV), *reinterpret_cast<const uint4*>(&acc[i][j]));
          const int m = m_base + lr + 8 * i;
#pragma unroll 1
          for (int half = 0; half < 2; ++half) {
            const int n0 = n_base + lc + 16 * half;
            T v[4], cur[4];                // loads together: none of them can pass a store
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (m >= p.M || n0 + 4 * j >= p.N) continue;
              if (shared_d || opened) cur[j] = __ldcg(p.D + (long long)m * p.ldd + n0 + 4 * j);   // improved at the L2 by other lanes
              else if (p.read_c) cur[j] = p.C[(long long)m * p.ldc + n0 + 4 * j];
            }
#pragma unroll
            for (int j = 0; j < 4; j += EV) lds16(my_row + (4 * half + j) * (512 / EV), *reinterpret_cast<T(*)[EV]>(&v[j]));
            uint32_t q[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              v[j] += T(0);                                  // alpha (x) product
              const bool inside = m < p.M && n0 + 4 * j < p.N;
              if (inside) {
                T* at = p.D + (long long)m * p.ldd + n0 + 4 * j;
                if (shared_d) {
                  if (!S::better(v[j], cur[j])) v[j] = cur[j];
                  else if (v[j] >= T(0)) merge_into<kMax>(at, v[j]);       // without waiting for the answer
                  else v[j] = improve_shared<kMax>(at, v[j], cur[j]);
                } else if (opened) {
                  if (S::better(v[j], cur[j])) *at = v[j];
                  else v[j] = cur[j];
                } else {
                  if (p.read_c) v[j] = RingT::add(v[j], RingT::mul(p.beta, cur[j]));
                  *at = v[j];
                }
              }
              q[j] = inside ? S::bound(v[j], scale) : S::kNothing;
            }
            asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(my_bounds + i * 512 + half * 8), "r"(q[0] | (q[1] << 16)), "r"(q[2] | (q[3] << 16)) : "memory");
          }
        }
        opened = true;
        my_exp = exponent;
        __syncwarp();
        continue;
      }
      const uint32_t exact = smem_base + s * kScreenStageBytes;
      const uint32_t coarse = exact + kScreenExactBytes;

      if (my_exp != exponent) {
        // bounds at this stage's scale, from the running values
#pragma unroll 1
        for (int i = 0; i < 8; ++i) {
          const int m = m_base + lr + 8 * i;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int n = n_base + lc + 4 * j;
            uint32_t q = S::kNothing;
            if (m < p.M && n < p.N) q = S::bound(__ldcg(p.D + (long long)m * p.ldd + n), scale);
            sts2(my_bounds + i * 512 + j * 2, q);
          }
        }
        my_exp = exponent;
        __syncwarp();
      }

      uint32_t mask_lo = 0, mask_hi = 0;              // bit 8 i + j: element (i, j) might improve in this block
      {
        // ---- the screen: two products per instruction
        uint32_t q[8][8];
        // row i of the lane's bounds, each in both halves of a word; read again after the contraction, which has no
        // registers for them
        auto bounds = [&](int i, uint32_t (&v)[8]) {
          const uint4 x = lds16u(my_bounds + i * 512);
          const uint32_t packed[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = __byte_perm(packed[j >> 1], 0, (j & 1) ? 0x3232 : 0x1010);
        };
#pragma unroll
        for (int i = 0; i < 8; ++i) bounds(i, q[i]);
        const uint32_t qa = coarse + (wm * 64 + lr) * kCoarseRow, qb = coarse + kCoarseOperand + (wn * 32 + lc) * kCoarseRow;
#pragma unroll 2
        for (int c = 0; c < kCoarseChunks; ++c) {
          const uint32_t ab = qa + ((c ^ (lr >> 1)) << 4);            // rows lr + 8 i: (row >> 1) & 3 == lr >> 1
          const uint32_t b0 = qb + ((c ^ (lc >> 1)) << 4), b1 = qb + ((c ^ ((lc + 4) >> 1)) << 4);   // rows lc + 4 j
          uint4 a[8], bv[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) a[i] = lds16u(ab + i * (8 * kCoarseRow));
#pragma unroll
          for (int j = 0; j < 8; ++j) bv[j] = lds16u(((j & 1) ? b1 : b0) + j * (4 * kCoarseRow));
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              q[i][j] = S::fold(a[i].x, bv[j].x, q[i][j]);
              q[i][j] = S::fold(a[i].y, bv[j].y, q[i][j]);
              q[i][j] = S::fold(a[i].z, bv[j].z, q[i][j]);
              q[i][j] = S::fold(a[i].w, bv[j].w, q[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          uint32_t bound[8];
          bounds(i, bound);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (q[i][j] != bound[j]) {
              if (i < 4) mask_lo |= 1u << (8 * i + j);
              else       mask_hi |= 1u << (8 * (i - 4) + j);
            }
        }
      }
      // ---- exact values of the elements that might improve, four lanes each, listed kListed at a time
      const int mine = __popc(mask_lo) + __popc(mask_hi);
      int slot_of_next = mine;                        // exclusive prefix sum over the lanes
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int below = __shfl_up_sync(~0u, slot_of_next, d);
        if (lane >= d) slot_of_next += below;
      }
      const int total = __shfl_sync(~0u, slot_of_next, 31);
      slot_of_next -= mine;
      if (total > kExactAbove) {        // this block and the next ones exactly
        do_exactly(it, patience);
        patience = min(2 * patience, kMaxPatience);
        continue;
      }
      patience = kPatience;
      for (int first = 0; first < total; first += kListed) {
        while (slot_of_next < first + kListed && (mask_lo | mask_hi) != 0) {
          int bit;
          if (mask_lo != 0) { bit = __ffs(mask_lo) - 1; mask_lo &= mask_lo - 1; }
          else              { bit = 31 + __ffs(mask_hi); mask_hi &= mask_hi - 1; }
          sts2(list + 2 * (slot_of_next - first), (lane << 6) | bit);
          ++slot_of_next;
        }
        __syncwarp();
        const int listed = min(kListed, total - first);
        const int t = lane & 3;
        for (int base = 0; base < listed; base += 8 * kListGroups) {
          // groups of eight elements, so that their loads and exchanges overlap
          T best[kListGroups];
          int code[kListGroups];
#pragma unroll
          for (int u = 0; u < kListGroups; ++u) {
            const int slot = base + u * 8 + (lane >> 2);
            code[u] = lds2(list + 2 * (slot < listed ? slot : base));
            const int el = code[u] >> 6, i = (code[u] >> 3) & 7, j = code[u] & 7;
            const int row = wm * 64 + (el >> 2) + 8 * i, col = wn * 32 + (el & 3) + 4 * j;
            const uint32_t ra = exact + row * 128 + ((t ^ (row & 3)) << 4), rb = exact + kExactOperand + col * 128 + ((t ^ (col & 3)) << 4);
            // the lane's chunks of 16 bytes: t and t + 4 of both 128-byte columns
            const uint32_t fa = (row & 4) << 4, fb = (col & 4) << 4;
            best[u] = kMax ? -static_cast<T>(INFINITY) : static_cast<T>(INFINITY);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              T a[EV], bb[EV];
              lds16(ra + (h >> 1) * kColumn + (((h & 1) << 6) ^ fa), a);
              lds16(rb + (h >> 1) * kColumn + (((h & 1) << 6) ^ fb), bb);
              best[u] = RingT::mac2(best[u], a[0], bb[0], a[1], bb[1]);
            }
          }
#pragma unroll
          for (int d = 2; d > 0; d >>= 1) {
#pragma unroll
            for (int u = 0; u < kListGroups; ++u) {
              const T other = __shfl_xor_sync(~0u, best[u], d);
              best[u] = RingT::add(other, best[u]);
            }
          }
#pragma unroll
          for (int u = 0; u < kListGroups; ++u) {
            const int el = code[u] >> 6, i = (code[u] >> 3) & 7, j = code[u] & 7;
            const int m = m_base + (el >> 2) + 8 * i, n = n_base + (el & 3) + 4 * j;
            if (t == u && base + u * 8 + (lane >> 2) < listed && m < p.M && n < p.N) {
              T* at = p.D + (long long)m * p.ldd + n;
              const uint32_t where = warp_bounds + i * 512 + el * 16 + j * 2;
              const uint32_t was = lds2(where), now = S::bound(best[u], scale);
              // Which of two values with the same 16-bit bound is better only D can tell; there a minimum (maximum) in
              // memory does, without waiting for its answer.
              const bool improved = S::sooner(now, was);
              if (improved || now == was) {
                if (best[u] >= T(0)) merge_into<kMax>(at, best[u]);
                else improve_shared<kMax>(at, best[u], __ldcg(at));   // max only: sums of values that round up to zero
              }
              if (improved) sts2(where, now);
            }
          }
        }
        __syncwarp();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_bar[s]);
      ++b; ++it;
    }
    // further copies of the finished tile (pieces == 1)
    if (p.n_extra > 0) {
      __syncwarp();
#pragma unroll 1
      for (int i = 0; i < 64; ++i) {
        const int m = m_base + i, n = n_base + lane;
        if (m < p.M && n < p.N) {
          const long long off = (long long)m * p.ldd + n;
          const T v = __ldcg(p.D + off);
          for (int x = 0; x < p.n_extra; ++x) p.extra_d[x][off] = v;
        }
      }
    }
  }
}

// D = the start values of a product whose pieces meet in D: the additive identity, folded with beta (x) C.
template <typename RingT>
__global__ void __launch_bounds__(kSampleThreads)
screened_init_kernel(const __grid_constant__ ScreenParams p) {
  using T = typename RingT::Element;
  grid_dependency_wait();
  grid_dependency_launch();
  // (start values are written for nothing where C is another matrix)
  if (p.if_it_helps && p.read_c && p.C == p.D && !screen_helps<RingT::kAdd == CUASR_OP_MAXIMUM>(p.A, p.lda, p.a_mode != kLoadGatherMN, p.M, p.B, p.ldb,
                                                                       p.b_mode != kLoadGatherMN, p.N, p.K))
    return;
  const long long total = (long long)p.M * p.N;
  for (long long idx = (long long)blockIdx.x * kSampleThreads + threadIdx.x; idx < total; idx += (long long)gridDim.x * kSampleThreads) {
    const int m = static_cast<int>(idx / p.N), n = static_cast<int>(idx - (long long)m * p.N);
    T v = p.add_identity + T(0);                             // alpha (x) identity
    if (p.read_c) v = RingT::add(v, RingT::mul(p.beta, p.C[(long long)m * p.ldc + n]));
    p.D[(long long)m * p.ldd + n] = v;
  }
}

// Launches srgemm_screened_kernel on `grid` persistent CTAs, and the kernel that prepares D where its pieces share it.
cudaError_t launch_screened(bool maximize, const CUtensorMap& map_a, const CUtensorMap& map_b, const ScreenParams& params, int grid,
                            cudaStream_t stream);
cudaError_t launch_screened_init(bool maximize, const ScreenParams& params, int sms, cudaStream_t stream);

}  // namespace cuasr_b200
