// Path-tracking kernels: fp32 and fp64, min-plus and max-plus.
#include "srgemm_launch_impl.cuh"
#include "srgemm_path.cuh"
namespace cuasr_b200 {
template <typename T, bool kMaximize, typename Tile>
static cudaError_t launch_variant(const CUtensorMap& map_a, const CUtensorMap& map_b, const PathParams<T>& params, int grid,
                                  cudaStream_t stream) {
  auto kernel = srgemm_path_kernel<T, kMaximize, Tile>;
  static std::atomic<unsigned long long> done{0};
  const cudaError_t err = opt_in_shared_memory(kernel, kPathSmemBytes<T, Tile>, done);
  if (err != cudaSuccess) return err;
  return launch_overlapped(kernel, grid, kTmaThreads, kPathSmemBytes<T, Tile>, params.cluster, stream, map_a, map_b, params);
}
template <typename T>
cudaError_t launch_path(bool maximize, bool small_tile, const CUtensorMap& map_a, const CUtensorMap& map_b,
                        const PathParams<T>& params, int grid, cudaStream_t stream) {
  using Small = std::conditional_t<sizeof(T) == 4, SmallTile, TinyTile>;
  if (small_tile)
    return maximize ? launch_variant<T, true, Small>(map_a, map_b, params, grid, stream)
                    : launch_variant<T, false, Small>(map_a, map_b, params, grid, stream);
  return maximize ? launch_variant<T, true, LargeTile>(map_a, map_b, params, grid, stream)
                  : launch_variant<T, false, LargeTile>(map_a, map_b, params, grid, stream);
}
template cudaError_t launch_path<float>(bool, bool, const CUtensorMap&, const CUtensorMap&, const PathParams<float>&, int, cudaStream_t);
template cudaError_t launch_path<double>(bool, bool, const CUtensorMap&, const CUtensorMap&, const PathParams<double>&, int, cudaStream_t);
}  // namespace cuasr_b200
