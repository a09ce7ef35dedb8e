// Operand staging by ordinary loads: copies a tile of an operand with ANY leading dimension, alignment and layout
// into the shared-memory layout the contraction reads, [rows][128 bytes of k] with TMA's 128-byte swizzle.
//
// TMA describes an operand only if its address and leading dimension are multiples of 16 bytes, cannot transpose,
// and fills out-of-range elements with zero or NaN only.  The four producer warps of a CTA have nothing to do while
// TMA works, so where TMA cannot deliver the K-contiguous layout they bring the elements themselves with 4- or 8-byte
// cp.async, transposing on the way, and write any padding value a ring needs past the end of K.
// Cost: 128 threads issue 64 cp.async each per 32 KiB stage, about 1000 of the 8500 clocks that stage's arithmetic takes.
#pragma once

#include "ring.cuh"

namespace cuasr_b200 {

// How an operand reaches shared memory.
enum LoadMode : int {
  kLoadTma = 0,          // contiguous along k, 16-byte aligned storage lines: TMA
  kLoadGatherK = 1,      // contiguous along k, any alignment: lanes along k
  kLoadGatherMN = 2,     // contiguous along rows, any alignment: 8 rows x 4 k per warp instruction
  kLoadTmaRows = 3,      // contiguous along rows, 16-byte aligned storage lines: TMA, as it lies (large tile, see LargeRowsTile)
};

template <int kBytes>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(kBytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// The barrier receives this thread's arrival when all cp.async the thread has issued so far have landed.
__device__ __forceinline__ void cp_async_arrive_noinc(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void sts(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void sts(uint32_t addr, int32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void sts(uint32_t addr, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
__device__ __forceinline__ void sts(uint32_t addr, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory"); }

// Stages rows [r0, r0 + kRows) x k [k0, k0 + kSub * 128 bytes) of an operand whose element (r, k) is base[r * ld + k]
// (kLoadGatherK) or base[r + k * ld] (kLoadGatherMN).  Rows at or beyond `rows` are left as they are (their results are
// never stored) or, where the kernel looks at the whole stage (kRepeatRow), repeat the last row, which takes more
// instructions.
// k at or beyond K repeats the last k where `repeat_k` is set (rings whose (+) is idempotent: a product
// twice changes nothing) and is else set to `pad` by plain stores, so a stage that reaches beyond K must not be announced
// with cp_async_arrive_noinc alone.  Called by all 128 producer threads; `pw` is the producer warp (0..3).
// Inside the matrix a copy is one cp.async and at most one addition: with the bounds tested element by element a
// 1024 x 768 x 1536 product of odd storage lines took 186 us, against 97 us with TMA.
template <typename T, int kRows, int kSub, bool kRepeatRow = false>
__device__ __forceinline__ void gather_tile(uint32_t dst, const T* __restrict__ base, long long ld, int mode, int r0,
                                            int rows, int k0, int K, T pad, bool repeat_k, int pw, int lane) {
  constexpr int TK = 128 / (int)sizeof(T);         // k per 128-byte row
  constexpr int ES = (int)sizeof(T);
  // opaque: the lane's offsets are computed here, per stage, instead of being held in the producers' few registers
  asm volatile("" : "+r"(lane), "+r"(pw));
  const int last = rows - 1 - r0;                  // last row, relative to the tile's first
  if (mode == kLoadGatherMN) {
    // A warp instruction covers 8 rows x 4 k: four 32-byte (64-byte for 8-byte elements) pieces of global memory, and
    // (row & 7) spreads the 8 rows over the 8 swizzled chunks, so the shared-memory writes do not conflict.
    const int r8 = lane & 7, kq = lane >> 3;
#pragma unroll 1
    for (int sub = 0; sub < kSub; ++sub) {
#pragma unroll 1
      for (int step = 0; step < TK / 16; ++step) {
        const int kk = step * 16 + pw * 4 + kq;
        const int k = repeat_k ? min(k0 + sub * TK + kk, K - 1) : k0 + sub * TK + kk;
        const uint32_t d = dst + sub * (kRows * 128) + r8 * 128 + ((((kk * ES) >> 4) ^ r8) << 4) + ((kk * ES) & 15);
        const T* line = base + (long long)k * ld + r0;
        if (k0 + sub * TK + TK <= K && last >= kRows - 1) {          // uniform over the warp
          const T* s = line + r8;
#pragma unroll
          for (int i = 0; i < kRows / 8; ++i) cp_async<ES>(d + i * 1024, s + 8 * i);
        } else if (k < K) {
          if constexpr (kRepeatRow) {
#pragma unroll 1
            for (int i = 0; i < kRows / 8; ++i) cp_async<ES>(d + i * 1024, line + min(r8 + 8 * i, last));
          } else {
            const T* s = line + r8;
#pragma unroll
            for (int i = 0; i < kRows / 8; ++i)
              if (8 * i <= last - r8) cp_async<ES>(d + i * 1024, s + 8 * i);
          }
        } else {
#pragma unroll 1
          for (int i = 0; i < kRows / 8; ++i) sts(d + i * 1024, pad);
        }
      }
    }
  } else {
    constexpr int kRowsPerInstr = ES == 8 ? 2 : 1;
    constexpr int kRowStep = 4 * kRowsPerInstr;
    const int kk = ES == 8 ? (lane & 15) : lane;
    const int rr = ES == 8 ? pw * 2 + (lane >> 4) : pw;
    // swizzled chunk of row rr + kRowStep i: the row's low three bits alternate for 4-byte elements
    const uint32_t c0 = (((kk * ES) >> 4) ^ (rr & 7)) << 4;
    const uint32_t c1 = ES == 8 ? c0 : c0 ^ 64;
#pragma unroll 1
    for (int sub = 0; sub < kSub; ++sub) {
      const int k = repeat_k ? min(k0 + sub * TK + kk, K - 1) : k0 + sub * TK + kk;
      const uint32_t d = dst + sub * (kRows * 128) + rr * 128 + ((kk * ES) & 15);
      const T* column = base + (long long)r0 * ld + k;
      if (k0 + sub * TK + TK <= K && last >= kRows - 1) {            // uniform over the warp
        const T* s = column + (long long)rr * ld;
#pragma unroll 4
        for (int i = 0; i < kRows / kRowStep; ++i) {
          cp_async<ES>(d + i * (kRowStep * 128) + ((i & 1) ? c1 : c0), s);
          s += (long long)kRowStep * ld;
        }
      } else if (k < K) {
        if constexpr (kRepeatRow) {
#pragma unroll 1
          for (int i = 0; i < kRows / kRowStep; ++i)
            cp_async<ES>(d + i * (kRowStep * 128) + ((i & 1) ? c1 : c0), column + (long long)min(rr + kRowStep * i, last) * ld);
        } else {
          const T* s = column + (long long)rr * ld;
#pragma unroll 4
          for (int i = 0; i < kRows / kRowStep; ++i) {
            if (kRowStep * i <= last - rr) cp_async<ES>(d + i * (kRowStep * 128) + ((i & 1) ? c1 : c0), s);
            s += (long long)kRowStep * ld;
          }
        }
      } else {
#pragma unroll 1
        for (int i = 0; i < kRows / kRowStep; ++i) sts(d + i * (kRowStep * 128) + ((i & 1) ? c1 : c0), pad);
      }
    }
  }
}

}  // namespace cuasr_b200
