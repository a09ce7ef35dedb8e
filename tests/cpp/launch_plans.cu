// Launch plans on the CPU: the planning functions of the library's boundary, called for other SM counts than this GPU's.
#include "../../cuasr_b200/csrc/abi.cu"

#include <cstdio>

using namespace cuasr_b200;

namespace {
int failures = 0;
cuasr_b200_desc_t desc_of(int add, int mul, int dtype) {
  cuasr_b200_desc_t d = {};
  d.add_op = add; d.mul_op = mul; d.dtype = dtype;
  d.layout_a = CUASR_ROW_MAJOR; d.layout_b = CUASR_COLUMN_MAJOR; d.layout_c = CUASR_ROW_MAJOR;
  return d;
}
cuasr_b200_args_t args_of(int m, int n, int k) {
  cuasr_b200_args_t a = {};
  a.m = m; a.n = n; a.k = k; a.split_k_slices = 1;
  a.lda = a.ldb = k; a.ldc = a.ldd = n;
  return a;
}

// How K is shared for a given SM count, as one number.
long long k_sharing(const cuasr_b200_desc_t& d, const cuasr_b200_args_t& a, int gpu_sms) {
  const int sms = planning_sms(d, gpu_sms);
  const LaunchPlan plan = plan_without_workspace(d, a.m, a.n, a.k, sms, has_all_tiles(d), Gathers());
  const BalancePlan balance = balance_plan(static_cast<long long>(tile_count(a)), sms, (a.k + 31) / 32);
  return ((plan.tile * 64LL + plan.cluster) * 64 + balance.pieces) * 1000000 + balance.whole_tiles;
}

void sums_do_not_depend_on_the_sm_count() {
  bool other_ring_does = false;
  for (int m : {40, 256, 500, 1024, 2000})
    for (int n : {64, 300, 1500})
      for (int k : {64, 512, 5000})
        for (int dtype : {CUASR_F32, CUASR_F64}) {
          const cuasr_b200_args_t a = args_of(m, n, k);
          const cuasr_b200_desc_t sum = desc_of(CUASR_OP_PLUS, CUASR_OP_MULTIPLIES, dtype), min = desc_of(CUASR_OP_MINIMUM, CUASR_OP_PLUS, dtype);
          for (int sms : {20, 74, 132, 160}) {
            if (k_sharing(sum, a, sms) != k_sharing(sum, a, 148)) {
              std::printf("FAILED: %d x %d x %d, type %d: another sum on %d SMs\n", m, n, k, dtype, sms);
              ++failures;
            }
            other_ring_does |= k_sharing(min, a, sms) != k_sharing(min, a, 148);
          }
        }
  if (!other_ring_does) { std::printf("FAILED: no plan depends on the SM count\n"); ++failures; }
}
}  // namespace

int main() {
  sums_do_not_depend_on_the_sm_count();
  std::printf(failures ? "%d failed\n" : "launch plans ok\n", failures);
  return failures != 0;
}
