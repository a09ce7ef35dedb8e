// Operand copies into K-contiguous, 16-byte aligned storage.
#pragma once

#include "ptx.cuh"

namespace cuasr_b200 {

// One operand to copy: rows x K elements (r, k) at src[r * ld_src + k] (kcontig: a copy, for addresses and leading
// dimensions TMA cannot use) or src[r + k * ld_src] (a transposition), to dst[r * ld_dst + k]; columns K .. K_out - 1 of
// the copy repeat column K - 1 (for an idempotent (+) a product taken twice changes nothing).
template <typename W>
struct RepackOperand {
  const W* src;
  long long ld_src;
  int kcontig, rows, K, K_out;
  W* dst;
  long long ld_dst;
  int tiles_r, tiles;
};

// Copies up to two operands through 32 x 32 shared-memory tiles, reads and writes both coalesced.  One launch for both
// (and its set-up under the kernel before it): the copies in front of a small product are all launch latency.
// W is an unsigned integer of the element's width: the data is only moved.  Tiles are numbered along grid.x
// (rows fastest), so neither extent is limited by the 65535 of the other grid dimensions.
template <typename W>
__global__ void __launch_bounds__(256)
repack_to_kcontig_kernel(const RepackOperand<W> first, const RepackOperand<W> second) {
  __shared__ W tile[32][33];
  grid_dependency_wait();
  grid_dependency_launch();
  const bool is_first = blockIdx.x < first.tiles;
  const RepackOperand<W>& o = is_first ? first : second;
  const int block = is_first ? blockIdx.x : blockIdx.x - first.tiles;
  const int r0 = (block % o.tiles_r) * 32, k0 = (block / o.tiles_r) * 32;
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;   // 32 x 8
  if (!o.kcontig) {
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
      const int r = r0 + tx, k = k0 + ty + i;
      if (r < o.rows && k < o.K_out) tile[ty + i][tx] = o.src[r + (long long)min(k, o.K - 1) * o.ld_src];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 32; i += 8) {
    const int r = r0 + ty + i, k = k0 + tx;
    if (r < o.rows && k < o.K_out)
      o.dst[(long long)r * o.ld_dst + k] = o.kcontig ? o.src[(long long)r * o.ld_src + min(k, o.K - 1)] : tile[tx][ty + i];
  }
}

}  // namespace cuasr_b200
