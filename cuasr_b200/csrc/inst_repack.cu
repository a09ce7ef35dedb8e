// Launcher of the operand copies.
#include "repack.cuh"
#include "srgemm_launch.h"
namespace cuasr_b200 {
template <typename W>
static cudaError_t launch(const RepackRequest* requests, int count, cudaStream_t stream) {
  RepackOperand<W> op[2] = {};
  long long grid = 0;
  for (int i = 0; i < count; ++i) {
    const RepackRequest& q = requests[i];
    const long long tiles_r = (q.rows + 31) / 32, tiles_k = (q.K_out + 31) / 32;
    grid += tiles_r * tiles_k;
    if (grid > 2147483647LL) return cudaErrorInvalidValue;
    op[i] = {static_cast<const W*>(q.src), q.ld_src, q.kcontig, q.rows, q.K, q.K_out,
             static_cast<W*>(q.dst), q.ld_dst, static_cast<int>(tiles_r), static_cast<int>(tiles_r * tiles_k)};
  }
  return launch_overlapped(repack_to_kcontig_kernel<W>, static_cast<int>(grid), 256, 0, 1, stream, op[0], op[1]);
}
cudaError_t launch_repack(const RepackRequest* requests, int count, size_t element_bytes, cudaStream_t stream) {
  return element_bytes == 8 ? launch<unsigned long long>(requests, count, stream) : launch<unsigned int>(requests, count, stream);
}
}  // namespace cuasr_b200
