// Screened tropical kernels: fp64 min-plus and max-plus.
#include "srgemm_launch_impl.cuh"
#include "srgemm_screened.cuh"
namespace cuasr_b200 {
template <bool kMax>
static cudaError_t launch_variant(const CUtensorMap& map_a, const CUtensorMap& map_b, const ScreenParams& params, int grid,
                                  cudaStream_t stream) {
  auto kernel = srgemm_screened_kernel<kMax>;
  static std::atomic<unsigned long long> done{0};
  const cudaError_t err = opt_in_shared_memory(kernel, kScreenSmemBytes, done);
  if (err != cudaSuccess) return err;
  return launch_overlapped(kernel, grid, kTmaThreads, kScreenSmemBytes, 1, stream, map_a, map_b, params);
}
cudaError_t launch_screened(bool maximize, const CUtensorMap& map_a, const CUtensorMap& map_b, const ScreenParams& params, int grid,
                            cudaStream_t stream) {
  return maximize ? launch_variant<true>(map_a, map_b, params, grid, stream) : launch_variant<false>(map_a, map_b, params, grid, stream);
}
cudaError_t launch_screened_init(bool maximize, const ScreenParams& params, int sms, cudaStream_t stream) {
  const long long blocks = (static_cast<long long>(params.M) * params.N + kSampleThreads - 1) / kSampleThreads;
  const int grid = static_cast<int>(blocks < 2LL * sms ? blocks : 2LL * sms);
  return maximize ? launch_overlapped(screened_init_kernel<Ring<CUASR_OP_MAXIMUM, CUASR_OP_PLUS, double>>, grid, kSampleThreads, 0, 1, stream, params)
                  : launch_overlapped(screened_init_kernel<Ring<CUASR_OP_MINIMUM, CUASR_OP_PLUS, double>>, grid, kSampleThreads, 0, 1, stream, params);
}
}  // namespace cuasr_b200
