// Host-side launchers of the SRGEMM kernel.  The definitions live in srgemm_launch_impl.cuh and are instantiated
// explicitly, ring by ring, in the inst_*.cu files so that the rings compile in parallel; abi.cu only sees these
// declarations.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "srgemm_tma.cuh"

namespace cuasr_b200 {

enum TileKind : int { kLargeTile = 0, kMediumTile = 1, kSmallTile = 2, kTinyTile = 3 };

// Launches srgemm_tma_kernel<Ring<ADD, MUL, T>, tile> on `grid` CTAs in clusters of `cluster`.
template <int ADD, int MUL, typename T>
cudaError_t launch_tma(int tile, const CUtensorMap& map_a, const CUtensorMap& map_b, const TmaParams<T>& params,
                       int grid, int cluster, cudaStream_t stream);

// (ring, element type) pairs that have every tile shape compiled in; the others run on the two smallest alone.
template <int ADD, int MUL, typename T>
constexpr bool all_tiles_instantiated() {
  constexpr bool tropical = (ADD == CUASR_OP_MINIMUM || ADD == CUASR_OP_MAXIMUM) && MUL == CUASR_OP_PLUS;
  constexpr bool minmax = (ADD == CUASR_OP_MINIMUM && MUL == CUASR_OP_MAXIMUM) ||
                          (ADD == CUASR_OP_MAXIMUM && MUL == CUASR_OP_MINIMUM);
  constexpr bool times = (ADD == CUASR_OP_MINIMUM || ADD == CUASR_OP_MAXIMUM || ADD == CUASR_OP_PLUS) &&
                         MUL == CUASR_OP_MULTIPLIES;
  constexpr bool bits = (ADD == CUASR_OP_BIT_XOR || ADD == CUASR_OP_BIT_OR) &&
                        (MUL == CUASR_OP_BIT_AND || MUL == CUASR_OP_BINARY_AND) &&
                        !(ADD == CUASR_OP_BIT_OR && MUL == CUASR_OP_BINARY_AND);
  if (std::is_floating_point<T>::value) return tropical || minmax || times;
  return bits || tropical || minmax;  // int32_t, uint32_t
}

// Copies of up to two operands of 4- or 8-byte elements into K-contiguous storage, in one launch (see repack.cuh).
struct RepackRequest {
  const void* src;
  long long ld_src;
  bool kcontig;
  int rows, K, K_out;
  void* dst;
  long long ld_dst;
};
cudaError_t launch_repack(const RepackRequest* requests, int count, size_t element_bytes, cudaStream_t stream);

// Closure of a diagonal block of n <= 128 vertices (see fw_closure.cuh); 4- or 8-byte floating-point elements.
cudaError_t launch_fw_closure(const void* src, long long ld_src, void* dst, long long ld_dst, int n, size_t element_bytes,
                              cudaStream_t stream);

// Kernel launch that lets the kernel's set-up overlap the end of the kernel before it in the stream (the kernel must
// call grid_dependency_wait() before it touches global memory).
template <typename... Params, typename... Args>
cudaError_t launch_overlapped(void (*kernel)(Params...), int grid, int block, int smem_bytes, int cluster,
                              cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(grid));
  config.blockDim = dim3(static_cast<unsigned>(block));
  config.dynamicSmemBytes = static_cast<size_t>(smem_bytes);
  config.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  config.attrs = attr;
  config.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
}

}  // namespace cuasr_b200
