// Launcher of the diagonal-block closure.
#include <limits>

#include "fw_closure.cuh"
#include "srgemm_launch.h"
namespace cuasr_b200 {
cudaError_t launch_fw_closure(const void* src, long long ld_src, void* dst, long long ld_dst, int n, size_t element_bytes,
                              cudaStream_t stream) {
  if (n < 1 || n > kClosureBlock) return cudaErrorInvalidValue;
  if (element_bytes == 8)
    return launch_overlapped(fw_closure_kernel<double>, 1, kClosureThreads, 0, 1, stream, static_cast<const double*>(src), ld_src,
                             static_cast<double*>(dst), ld_dst, n, std::numeric_limits<double>::infinity());
  return launch_overlapped(fw_closure_kernel<float>, 1, kClosureThreads, 0, 1, stream, static_cast<const float*>(src), ld_src,
                           static_cast<float*>(dst), ld_dst, n, std::numeric_limits<float>::infinity());
}
}  // namespace cuasr_b200
