// Definitions of the launchers declared in srgemm_launch.h; included only by the inst_*.cu files.
#pragma once

#include <atomic>

#include "srgemm_launch.h"

namespace cuasr_b200 {

// More than 48 KiB of dynamic shared memory has to be opted into, once per kernel and device.  `done` has one bit
// per device.
template <typename Kernel>
cudaError_t opt_in_shared_memory(Kernel kernel, int bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  const unsigned long long bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (err == cudaSuccess) done.fetch_or(bit);
  return err;
}

template <typename RingT, typename Tile, bool kAsks>
cudaError_t launch_tma_kernel(const CUtensorMap& map_a, const CUtensorMap& map_b,
                              const TmaParams<typename RingT::Element>& params, int grid, int cluster,
                              cudaStream_t stream) {
  using T = typename RingT::Element;
  auto kernel = srgemm_tma_kernel<RingT, Tile, kAsks>;
  static std::atomic<unsigned long long> done{0};
  const cudaError_t err = opt_in_shared_memory(kernel, Tile::template kSmemBytes<T>, done);
  if (err != cudaSuccess) return err;
  return launch_overlapped(kernel, grid, kTmaThreads, Tile::template kSmemBytes<T>, cluster, stream, map_a, map_b, params);
}

template <typename RingT, typename Tile>
cudaError_t launch_tma_variant(const CUtensorMap& map_a, const CUtensorMap& map_b,
                               const TmaParams<typename RingT::Element>& params, int grid, int cluster,
                               cudaStream_t stream) {
  if constexpr (std::is_same<typename RingT::Element, double>::value && RingT::kMul == CUASR_OP_PLUS &&
                (RingT::kAdd == CUASR_OP_MINIMUM || RingT::kAdd == CUASR_OP_MAXIMUM)) {
    if (params.unless_screened) return launch_tma_kernel<RingT, Tile, true>(map_a, map_b, params, grid, cluster, stream);
  }
  return launch_tma_kernel<RingT, Tile, false>(map_a, map_b, params, grid, cluster, stream);
}

template <int ADD, int MUL, typename T>
cudaError_t launch_tma(int tile, const CUtensorMap& map_a, const CUtensorMap& map_b, const TmaParams<T>& params,
                       int grid, int cluster, cudaStream_t stream) {
  using R = Ring<ADD, MUL, T>;
  if constexpr (all_tiles_instantiated<ADD, MUL, T>()) {
    constexpr bool rows = !R::kPackedPairs && (sizeof(T) == 4 || ADD == CUASR_OP_PLUS || (MUL != CUASR_OP_PLUS && MUL != CUASR_OP_MULTIPLIES));
    if constexpr (rows) {                // takes_rows
      const bool rows_a = params.a_mode == kLoadTmaRows, rows_b = params.b_mode == kLoadTmaRows;
      if (rows_a && rows_b) return launch_tma_variant<R, LargeRowsTile<true, true>>(map_a, map_b, params, grid, cluster, stream);
      if (rows_a) return launch_tma_variant<R, LargeRowsTile<true, false>>(map_a, map_b, params, grid, cluster, stream);
      if (rows_b) return launch_tma_variant<R, LargeRowsTile<false, true>>(map_a, map_b, params, grid, cluster, stream);
    }
    if (tile == kLargeTile)
      return params.a_mode == kLoadTma && params.b_mode == kLoadTma
                 ? launch_tma_variant<R, LargeTmaTile>(map_a, map_b, params, grid, cluster, stream)
                 : launch_tma_variant<R, LargeTile>(map_a, map_b, params, grid, cluster, stream);
    if (tile == kMediumTile) return launch_tma_variant<R, MediumTile>(map_a, map_b, params, grid, cluster, stream);
  }
  if (tile == kTinyTile) {
    constexpr bool dmma = std::is_same<T, double>::value && ADD == CUASR_OP_PLUS && MUL == CUASR_OP_MULTIPLIES;
    return launch_tma_variant<R, std::conditional_t<dmma, TinyTileDeep, TinyTile>>(map_a, map_b, params, grid, cluster, stream);
  }
  return launch_tma_variant<R, SmallTile>(map_a, map_b, params, grid, cluster, stream);
}

#define CUASR_INSTANTIATE_TMA(ADD, MUL, T)                                                             \
  template cudaError_t launch_tma<ADD, MUL, T>(int, const CUtensorMap&, const CUtensorMap&,            \
                                               const TmaParams<T>&, int, int, cudaStream_t);

}  // namespace cuasr_b200
