// Closure of one diagonal block of the blocked Floyd-Warshall solve: all shortest paths inside at most 128 vertices.
//
// The block is the serial part of every step of the solve, so what counts is the length of its chain.  Squaring it
// repeatedly takes log2(n) launches; here one CTA keeps the whole 128 x 128 block in registers (16 x 16 threads, 8 x 8
// elements each) and runs the Floyd-Warshall recurrence on it, two vertices per step: rows and columns k and k + 1 go
// round through shared memory (double-buffered, one barrier per step), every thread brings its part of row and
// column k + 1 up to date with vertex k by itself, and an element is d = min3(d, d(i,k) + d(k,j), d(i,k+1) + d(k+1,j)).
// 64 steps of about 450 clocks: 15 us for 128 vertices against 7 squarings of 5 us, bound by the three-input minima
// of one SM.
#pragma once

#include "ring.cuh"

namespace cuasr_b200 {

constexpr int kClosureBlock = 128;
constexpr int kClosureThreads = 256;

template <typename T>
__device__ __forceinline__ T closure_min(T a, T b) { return b < a ? b : a; }
__device__ __forceinline__ float closure_min(float a, float b) { return fminf(a, b); }

// dst = closure of src: element (i, j) at [i * ld + j] of both (of the transposes: the same for both storage orders).
// `infinity` stands for vertices beyond n.  src and dst may be the same.
template <typename T>
__global__ void __launch_bounds__(kClosureThreads, 1)
fw_closure_kernel(const T* src, long long ld_src, T* dst, long long ld_dst, int n, T infinity) {
  // [buffer][row k, row k + 1, column k, column k + 1][vertex]
  __shared__ __align__(16) T line[2][4][kClosureBlock];
  using R = Ring<CUASR_OP_MINIMUM, CUASR_OP_PLUS, T>;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  // element (i, j) of a thread: row ty * 4 + i % 4 + 64 (i / 4), column tx * 4 + j % 4 + 64 (j / 4)
  grid_dependency_wait();
  grid_dependency_launch();
  T d[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int r = ty * 4 + i % 4 + 64 * (i / 4), c = tx * 4 + j % 4 + 64 * (j / 4);
      d[i][j] = r < n && c < n ? src[(long long)r * ld_src + c] : infinity;
    }
  int buffer = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll 1
    for (int t = 0; t < 16; ++t) {
      if (64 * h + 4 * t >= n) break;
#pragma unroll
      for (int r = 0; r < 4; r += 2, buffer ^= 1) {
        constexpr int kVec = 16 / (int)sizeof(T);
        const int k = 64 * h + 4 * t + r;          // rows and columns k, k + 1 are elements 4 h + r and 4 h + r + 1 of their owners
        T(*l)[kClosureBlock] = line[buffer];
        if (ty == t) {
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int j = 0; j < 8; ++j) l[q][tx * 4 + j % 4 + 64 * (j / 4)] = d[4 * h + r + q][j];
        }
        if (tx == t) {
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int i = 0; i < 8; ++i) l[2 + q][ty * 4 + i % 4 + 64 * (i / 4)] = d[i][4 * h + r + q];
        }
        __syncthreads();
        T row[2][8], col[2][8];
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int v = 0; v < 4; v += kVec) {
              alignas(16) T x[kVec], y[kVec];
              *reinterpret_cast<uint4*>(x) = *reinterpret_cast<const uint4*>(&l[q][tx * 4 + 64 * g + v]);
              *reinterpret_cast<uint4*>(y) = *reinterpret_cast<const uint4*>(&l[2 + q][ty * 4 + 64 * g + v]);
#pragma unroll
              for (int e = 0; e < kVec; ++e) { row[q][4 * g + v + e] = x[e]; col[q][4 * g + v + e] = y[e]; }
            }
        const T forth = l[0][k + 1], back = l[1][k];        // d(k, k + 1), d(k + 1, k)
#pragma unroll
        for (int j = 0; j < 8; ++j) row[1][j] = closure_min(row[1][j], back + row[0][j]);
#pragma unroll
        for (int i = 0; i < 8; ++i) col[1][i] = closure_min(col[1][i], col[0][i] + forth);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) d[i][j] = R::mac2(d[i][j], col[0][i], row[0][j], col[1][i], row[1][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int r = ty * 4 + i % 4 + 64 * (i / 4), c = tx * 4 + j % 4 + 64 * (j / 4);
      if (r < n && c < n) dst[(long long)r * ld_dst + c] = d[i][j];
    }
}

}  // namespace cuasr_b200
