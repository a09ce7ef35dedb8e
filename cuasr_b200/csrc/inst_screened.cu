// Screened tropical kernels: fp64 min-plus and max-plus.
#include "srgemm_launch_impl.cuh"
#include "srgemm_screened.cuh"
namespace cuasr_b200 {
template <typename T, bool kMax>
static cudaError_t launch_variant(const CUtensorMap& map_a, const CUtensorMap& map_b, const ScreenParams<T>& params, int grid,
                                  cudaStream_t stream) {
  auto kernel = srgemm_screened_kernel<T, kMax>;
  static std::atomic<unsigned long long> done{0};
  const cudaError_t err = opt_in_shared_memory(kernel, kScreenSmemBytes<T>, done);
  if (err != cudaSuccess) return err;
  return launch_overlapped(kernel, grid, kTmaThreads, kScreenSmemBytes<T>, 1, stream, map_a, map_b, params);
}
template <typename T>
cudaError_t launch_screened(bool maximize, const CUtensorMap& map_a, const CUtensorMap& map_b, const ScreenParams<T>& params,
                            int grid, cudaStream_t stream) {
  return maximize ? launch_variant<T, true>(map_a, map_b, params, grid, stream)
                  : launch_variant<T, false>(map_a, map_b, params, grid, stream);
}
template <typename T>
cudaError_t launch_screened_init(bool maximize, const ScreenParams<T>& params, int sms, cudaStream_t stream) {
  const long long blocks = (static_cast<long long>(params.M) * params.N + 255) / 256;
  const int grid = static_cast<int>(blocks < 8LL * sms ? blocks : 8LL * sms);
  return maximize ? launch_overlapped(screened_init_kernel<Ring<CUASR_OP_MAXIMUM, CUASR_OP_PLUS, T>>, grid, 256, 0, 1, stream, params)
                  : launch_overlapped(screened_init_kernel<Ring<CUASR_OP_MINIMUM, CUASR_OP_PLUS, T>>, grid, 256, 0, 1, stream, params);
}
template cudaError_t launch_screened<double>(bool, const CUtensorMap&, const CUtensorMap&, const ScreenParams<double>&, int, cudaStream_t);
template cudaError_t launch_screened_init<double>(bool, const ScreenParams<double>&, int, cudaStream_t);
}  // namespace cuasr_b200
