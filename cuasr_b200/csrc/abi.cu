// extern "C" boundary of the library: validation, layout normalisation, kernel choice and launch.
//
// Host-side counterpart of the reference's device::Srgemm (include/cuasr/gemm/device/srgemm.h:85-357 and
// its column-major specialisation :398-567) and device::SrgemmSplitKParallel
// (include/cuasr/gemm/device/srgemm_splitk_parallel.h:101-378, :424-607).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/cuasr_b200.h"
#include "../../include/cuasr_b200_apsp.h"
#include "srgemm_launch.h"
#include "srgemm_path.cuh"
#include "srgemm_screened.cuh"

namespace cuasr_b200 {
namespace {

std::atomic<uint64_t> g_launches{0};
thread_local const char* t_last_kernel = "none";

// What the last call on this thread launched, for cuasr_b200_last_route: kept as numbers, written out when asked for.
struct Route {
  const char* kernel = "none";
  int tile_m = 0, tile_n = 0, cluster = 1, pieces = 1;
  const char* load_a = "";
  const char* load_b = "";
  bool tickets = false, copied_a = false, copied_b = false;
  int screened_pieces = 0;          // > 0: the screened kernel too, and the operands decided which of the two did the product
};
thread_local Route t_route;
thread_local char t_route_text[160];

const char* load_name(int mode) {
  static const char* const names[4] = {"tma", "gather", "gather", "tma-rows"};      // LoadMode
  return names[mode];
}

// ---- per-device state: SM count and the device status word --------------------------------------
__device__ unsigned int g_status_word;  // zero-initialised when the module loads

struct DeviceState {
  bool ready = false;
  int sms = 0;
  unsigned int* status = nullptr;
};
constexpr int kMaxDevices = 64;
DeviceState g_devices[kMaxDevices];
std::mutex g_device_mutex;

// First call on a device looks up the SM count and the address of the status word; no allocation.
bool device_state(DeviceState** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
  std::lock_guard<std::mutex> lock(g_device_mutex);
  DeviceState& st = g_devices[dev];
  if (!st.ready) {
    if (cudaDeviceGetAttribute(&st.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
    void* addr = nullptr;
    if (cudaGetSymbolAddress(&addr, g_status_word) != cudaSuccess) return false;
    st.status = static_cast<unsigned int*>(addr);
    st.ready = true;
  }
  *out = &st;
  return true;
}

// ---- cuTensorMapEncodeTiled through the runtime, so that the library does not link libcuda --------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

template <typename T> struct TmaType;
template <> struct TmaType<float>    { static constexpr CUtensorMapDataType v = CU_TENSOR_MAP_DATA_TYPE_FLOAT32; };
template <> struct TmaType<double>   { static constexpr CUtensorMapDataType v = CU_TENSOR_MAP_DATA_TYPE_FLOAT64; };
template <> struct TmaType<int32_t>  { static constexpr CUtensorMapDataType v = CU_TENSOR_MAP_DATA_TYPE_INT32; };
template <> struct TmaType<uint32_t> { static constexpr CUtensorMapDataType v = CU_TENSOR_MAP_DATA_TYPE_UINT32; };

// Describes one operand of `rows` x K elements to TMA.
//   K-contiguous:  tensor {K, rows}, box {128 bytes of k, box_rows rows}, 128-byte swizzle
//   MN-contiguous: tensor {rows, K}, box {128 rows, 128 bytes worth of k}, no swizzle
template <typename T>
bool make_operand_map(CUtensorMap* map, const T* ptr, long long ld, int rows, int K, bool kcontig, bool nan_fill,
                      int box_rows = kTileM) {
  EncodeTiledFn encode = encode_tiled_fn();
  if (encode == nullptr) return false;
  const cuuint32_t tk = kTileKBytes / sizeof(T);
  cuuint64_t dims[2];
  cuuint32_t box[2];
  if (kcontig) { dims[0] = K; dims[1] = rows; box[0] = tk; box[1] = box_rows; }
  else         { dims[0] = rows; dims[1] = K; box[0] = box_rows; box[1] = tk; }
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * sizeof(T)};
  const cuuint32_t elem_strides[2] = {1, 1};
  const CUresult r = encode(map, TmaType<T>::v, 2, const_cast<T*>(ptr), dims, strides, box, elem_strides,
                            CU_TENSOR_MAP_INTERLEAVE_NONE,
                            kcontig ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            nan_fill ? CU_TENSOR_MAP_FLOAT_OOB_FILL_NAN_REQUEST_ZERO_FMA
                                     : CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// ---- host evaluation of ring operators (only for the "is C needed" decision) ----------------------
template <typename T>
T host_op(int op, T l, T r) {
  switch (op) {
    case CUASR_OP_PLUS: return l + r;
    case CUASR_OP_MULTIPLIES: return l * r;
    case CUASR_OP_MINIMUM: return r < l ? r : l;
    case CUASR_OP_MAXIMUM: return l < r ? r : l;
    case CUASR_OP_BINARY_AND: return static_cast<T>(l && r);
    case CUASR_OP_BINARY_OR: return static_cast<T>(l || r);
    default: break;
  }
  if constexpr (std::is_integral<T>::value) {
    switch (op) {
      case CUASR_OP_BIT_AND: return l & r;
      case CUASR_OP_BIT_OR: return l | r;
      case CUASR_OP_BIT_XOR: return l ^ r;
      default: break;
    }
  }
  return l;
}

template <typename T>
T load_scalar(const cuasr_b200_scalar_t& s) {
  T v;
  std::memcpy(&v, s.bytes, sizeof(T));
  return v;
}

bool ring_supported(int add, int mul, int dtype) {
  const bool is_int = (dtype == CUASR_S32 || dtype == CUASR_U32);
  auto is = [&](int a, int m) { return add == a && mul == m; };
  if (is(CUASR_OP_PLUS, CUASR_OP_MULTIPLIES) || is(CUASR_OP_MINIMUM, CUASR_OP_PLUS) ||
      is(CUASR_OP_MAXIMUM, CUASR_OP_PLUS) || is(CUASR_OP_MINIMUM, CUASR_OP_MAXIMUM) ||
      is(CUASR_OP_MAXIMUM, CUASR_OP_MINIMUM) || is(CUASR_OP_MINIMUM, CUASR_OP_MULTIPLIES) ||
      is(CUASR_OP_MAXIMUM, CUASR_OP_MULTIPLIES) || is(CUASR_OP_BINARY_OR, CUASR_OP_BINARY_AND))
    return true;
  if (is_int && (is(CUASR_OP_BIT_XOR, CUASR_OP_BIT_AND) || is(CUASR_OP_BIT_OR, CUASR_OP_BIT_AND) ||
                 is(CUASR_OP_BIT_XOR, CUASR_OP_BINARY_AND)))
    return true;
  return false;
}

// The problem after the column-major-C transposition of device/srgemm.h:432-453, :513-523: always a
// row-major D (m x n), A' (m x k) and B' (k x n), each operand either K-contiguous or MN-contiguous.
struct Normalised {
  int m, n, k;
  const void* a; long long lda; bool a_kcontig;
  const void* b; long long ldb; bool b_kcontig;
  const void* c; long long ldc;
  void* d;       long long ldd;
};

Normalised normalise(const cuasr_b200_desc_t& desc, const cuasr_b200_args_t& args) {
  Normalised p;
  p.k = args.k;
  p.c = args.C; p.ldc = args.ldc; p.d = args.D; p.ldd = args.ldd;
  if (desc.layout_c == CUASR_ROW_MAJOR) {
    p.m = args.m; p.n = args.n;
    p.a = args.A; p.lda = args.lda; p.a_kcontig = (desc.layout_a == CUASR_ROW_MAJOR);
    p.b = args.B; p.ldb = args.ldb; p.b_kcontig = (desc.layout_b == CUASR_COLUMN_MAJOR);
  } else {
    // D^T = B^T (x)(+) A^T; a column-major matrix is the row-major storage of its transpose
    p.m = args.n; p.n = args.m;
    p.a = args.B; p.lda = args.ldb; p.a_kcontig = (desc.layout_b == CUASR_COLUMN_MAJOR);
    p.b = args.A; p.ldb = args.lda; p.b_kcontig = (desc.layout_a == CUASR_ROW_MAJOR);
  }
  return p;
}

int validate(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args) {
  if (desc == nullptr || args == nullptr) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  if (desc->dtype < CUASR_F32 || desc->dtype > CUASR_U32) return CUASR_STATUS_ERROR_INVALID_DATA_TYPE;
  for (int l : {desc->layout_a, desc->layout_b, desc->layout_c})
    if (l != CUASR_ROW_MAJOR && l != CUASR_COLUMN_MAJOR) return CUASR_STATUS_ERROR_INVALID_LAYOUT;
  if (!ring_supported(desc->add_op, desc->mul_op, desc->dtype)) return CUASR_STATUS_ERROR_NOT_SUPPORTED;
  if (args->m <= 0 || args->n <= 0 || args->k <= 0) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  if (args->split_k_slices < 1) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  if (args->A == nullptr || args->B == nullptr || args->D == nullptr) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  // A leading dimension shorter than the contiguous extent makes storage lines overlap.  For D (and C, which may
  // alias it) that would be a race, so it is refused.  A and B are only read: the reference never looks at their
  // leading dimensions (its own examples/02_splitk_srgemm/splitk_srgemm.cu:247-248 passes 128 for a row-major
  // 128 x 4096 operand), and an overlapping view is well defined, so any positive value is accepted; such views
  // are gathered.
  const long long c_min = desc->layout_c == CUASR_ROW_MAJOR ? args->n : args->m;
  if (args->lda < 1 || args->ldb < 1 || args->ldd < c_min) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  if (args->C != nullptr && args->ldc < c_min) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  const size_t es = desc->dtype == CUASR_F64 ? 8 : 4;
  for (const void* ptr : {args->A, args->B, args->C, static_cast<const void*>(args->D)})
    if (reinterpret_cast<uintptr_t>(ptr) % es != 0) return CUASR_STATUS_ERROR_MISALIGNED_OPERAND;
  return CUASR_STATUS_SUCCESS;
}

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

size_t tile_count(const cuasr_b200_args_t& args) {
  return static_cast<size_t>((args.m + kTileM - 1) / kTileM) * ((args.n + kTileN - 1) / kTileN);
}
size_t ticket_bytes_for(const cuasr_b200_args_t& args) { return align_up(tile_count(args) * sizeof(unsigned int), 256); }

// Scratch layout: [tickets: one u32 per 128 x 128 tile, padded to 256 B][partials: one full 128 x 128 block per
// (split tile, slice)].  With every tile split (explicit split-K) that is tiles * slices blocks.
size_t splitk_bytes_for_pieces(const cuasr_b200_desc_t& desc, const cuasr_b200_args_t& args, long long pieces) {
  const size_t es = desc.dtype == CUASR_F64 ? 8 : 4;
  return ticket_bytes_for(args) + es * tile_count(args) * kTileM * kTileN * static_cast<size_t>(pieces);
}

// Explicit split-K: into how many pieces of consecutive K tiles every output tile is really cut.  The reference
// launches exactly tiles x slices CTAs (include/cuasr/gemm/kernel/srgemm_splitk_parallel.h:86-89), whatever the GPU;
// here a slice count that leaves SMs idle (4 tiles x 16 slices = 64 work items on 148 SMs, or 4 x 32 = 128) is
// refined to the piece count in [slices, 8 x slices] that the cost model likes best (4 x 37 = 148).  That is only
// done where (+) is exact and order-independent (everything but floating-point plus): the pieces are folded in K
// order and the result cannot depend on how K was cut, hence not on the SM count either.  The cost model counts K
// tiles: waves x (K tiles per piece) for the contraction, plus half a K tile per piece for parking and folding a
// 128 x 128 partial.
bool splitk_order_independent(const cuasr_b200_desc_t& desc) {
  return !(desc.add_op == CUASR_OP_PLUS && (desc.dtype == CUASR_F32 || desc.dtype == CUASR_F64));
}
// The SM count a launch is planned for.  How K is shared decides the order of a floating-point sum and with it the last bits,
// so sums are planned for a B200's 148 SMs wherever they run (in a partition of the GPU with fewer they run in more waves).
int planning_sms(const cuasr_b200_desc_t& desc, int sms) { return splitk_order_independent(desc) ? sms : 148; }
long long splitk_pieces(const cuasr_b200_desc_t& desc, const cuasr_b200_args_t& args, int sms, long long max_pieces) {
  const long long slices = args.split_k_slices;
  if (sms <= 0 || slices <= 1 || !splitk_order_independent(desc)) return slices;
  const int tk = kTileKBytes / (desc.dtype == CUASR_F64 ? 8 : 4);
  const long long k_tiles = (args.k + tk - 1) / tk;
  const long long tiles = static_cast<long long>(tile_count(args));
  auto cost = [&](long long pieces) {
    const long long waves = (tiles * pieces + sms - 1) / sms;
    return static_cast<double>(waves * ((k_tiles + pieces - 1) / pieces)) + 0.5 * static_cast<double>(pieces);
  };
  long long best = slices;
  double best_cost = cost(slices);
  const long long limit = std::min<long long>(std::min<long long>(8 * slices, max_pieces), k_tiles / 4);
  for (long long pieces = slices + 1; pieces <= limit; ++pieces) {
    const double c = cost(pieces);
    if (c < 0.97 * best_cost) { best = pieces; best_cost = c; }
  }
  return best;
}

// Workspace the split-K entry points ask for: room for the refined plan on the current GPU (the plain
// tiles x slices layout where no GPU is visible).  A smaller workspace, down to the plain layout, is accepted at run
// time and simply limits the refinement.
size_t splitk_workspace_bytes(const cuasr_b200_desc_t& desc, const cuasr_b200_args_t& args) {
  if (args.split_k_slices <= 1) return 0;
  return splitk_bytes_for_pieces(desc, args, args.split_k_slices);
}
size_t splitk_workspace_bytes_refined(const cuasr_b200_desc_t& desc, const cuasr_b200_args_t& args) {
  if (args.split_k_slices <= 1) return 0;
  DeviceState* dev = nullptr;
  const long long pieces = device_state(&dev) ? splitk_pieces(desc, args, dev->sms, 1LL << 30) : args.split_k_slices;
  return splitk_bytes_for_pieces(desc, args, pieces);
}

// Load balancing of a launch that was not asked to split K: the tiles of the last, partial wave are cut along K
// so that their pieces fill the SMs.  Returns the number of pieces (1 = leave the launch alone) and the number of
// tiles that stay whole.
struct BalancePlan {
  int whole_tiles;
  int pieces;
};
BalancePlan balance_plan(long long tiles, int sms, int k_tiles) {
  BalancePlan plan{static_cast<int>(tiles), 1};
  if (sms <= 0 || tiles <= 0) return plan;
  const long long rem = tiles % sms;
  if (rem == 0) return plan;
  double best = 1.0;    // time of the last wave in units of one whole tile
  const int max_pieces = k_tiles / 4 < 16 ? k_tiles / 4 : 16;
  for (int s = 2; s <= max_pieces; ++s) {
    const double t = static_cast<double>((rem * s + sms - 1) / sms) / s + 0.02 * s;   // + a little per piece for the fold
    if (t < best - 0.05) { best = t; plan.pieces = s; }
  }
  if (plan.pieces > 1) plan.whole_tiles = static_cast<int>(tiles - rem);
  return plan;
}
size_t balance_workspace_bytes(const cuasr_b200_desc_t& desc, const cuasr_b200_args_t& args, int sms) {
  const size_t es = desc.dtype == CUASR_F64 ? 8 : 4;
  const int tk = kTileKBytes / static_cast<int>(es);
  const BalancePlan plan = balance_plan(static_cast<long long>(tile_count(args)), sms, (args.k + tk - 1) / tk);
  if (plan.pieces <= 1) return 0;
  return ticket_bytes_for(args) + es * (tile_count(args) - plan.whole_tiles) * kTileM * kTileN * plan.pieces;
}

// Dispatch over rings.  X(ADD, MUL) is expanded for each ring the element type supports.
#define CUASR_FLOAT_RINGS(X)                   \
  X(CUASR_OP_PLUS, CUASR_OP_MULTIPLIES)        \
  X(CUASR_OP_MINIMUM, CUASR_OP_PLUS)           \
  X(CUASR_OP_MAXIMUM, CUASR_OP_PLUS)           \
  X(CUASR_OP_MINIMUM, CUASR_OP_MAXIMUM)        \
  X(CUASR_OP_MAXIMUM, CUASR_OP_MINIMUM)        \
  X(CUASR_OP_MINIMUM, CUASR_OP_MULTIPLIES)     \
  X(CUASR_OP_MAXIMUM, CUASR_OP_MULTIPLIES)     \
  X(CUASR_OP_BINARY_OR, CUASR_OP_BINARY_AND)
#define CUASR_BIT_RINGS(X)                     \
  X(CUASR_OP_BIT_XOR, CUASR_OP_BIT_AND)        \
  X(CUASR_OP_BIT_OR, CUASR_OP_BIT_AND)         \
  X(CUASR_OP_BIT_XOR, CUASR_OP_BINARY_AND)

// Further destinations of the output (cuasr_b200_srgemm_push); empty for the ordinary entry points.
struct ExtraOutputs {
  int count = 0;
  void* ptr[kMaxDestinations - 1] = {};
};

// Which operands a launch with an optional workspace copies into K-contiguous, 16-byte aligned scratch, so that TMA
// brings them in: an operand TMA cannot describe (its address or its leading dimension is not a multiple of 16 bytes;
// the reference accepts alignment 1, include/cuasr/gemm/device/default_srgemm_configuration.h:88-89).  Without the
// workspace the kernel gathers such an operand itself.  Rows are padded to a multiple of 16 bytes; the padding is never
// read (the tensor map ends at K).
struct RepackPlan {
  bool a = false, b = false;
  bool faster_a = false, faster_b = false;   // copied although TMA could bring in the operand's lines as they are
  int k_padded = 0;      // > 0: both copies are extended along K to this length (a multiple of the kernel's K step)
  size_t bytes = 0;
};
bool tma_describable(const void* ptr, long long ld, size_t es) {
  return reinterpret_cast<uintptr_t>(ptr) % 16 == 0 && (ld * static_cast<long long>(es)) % 16 == 0;
}
size_t repack_operand_bytes(int rows, int k, size_t es) {
  return align_up(static_cast<size_t>(rows) * align_up(static_cast<size_t>(k), 16 / es) * es, 256);
}
// Rings whose ragged last K step the TMA kernel pads by itself: floating min/max rings (out-of-range elements are
// filled with NaN, which min and max ignore) and rings where 0 (x) 0 is neutral (zero fill).
bool ring_pads_itself(const cuasr_b200_desc_t& desc, const cuasr_b200_args_t& args) {
  const bool is_float = desc.dtype == CUASR_F32 || desc.dtype == CUASR_F64;
  if (is_float && (desc.add_op == CUASR_OP_MINIMUM || desc.add_op == CUASR_OP_MAXIMUM)) return true;
  if (desc.add_op == CUASR_OP_PLUS && desc.mul_op == CUASR_OP_MULTIPLIES) return true;
  if ((desc.add_op == CUASR_OP_BIT_OR || desc.add_op == CUASR_OP_BIT_XOR) &&
      (desc.mul_op == CUASR_OP_BINARY_AND || desc.mul_op == CUASR_OP_BIT_AND))
    return true;
  if (desc.add_op == CUASR_OP_BINARY_OR && desc.mul_op == CUASR_OP_BINARY_AND) {
    // zero fill is neutral when the accumulator starts at 0 or 1
    switch (desc.dtype) {
      case CUASR_F32: { const float v = load_scalar<float>(args.add_identity); return v == 0.0f || v == 1.0f; }
      case CUASR_F64: { const double v = load_scalar<double>(args.add_identity); return v == 0.0 || v == 1.0; }
      default:        { const uint32_t v = load_scalar<uint32_t>(args.add_identity); return v == 0u || v == 1u; }
    }
  }
  return false;
}

// ---- which tile, and how K is shared ---------------------------------------------------------------------------
// Clocks the 8 consumer warps of a CTA (two per scheduler, 64 products per lane and k) take for one k: measured per
// product and scheduler 2.15 (fp32 with a packed add and a three-input minimum, fused integer add-min, one logic
// instruction), 3.0 (two-instruction bottleneck products), 1.55 (fp32 sums), 2.1 (fp64 sums on the tensor cores), and for fp64
// minima by tile (4096^3 on the large tile, 1000^3 on 128 x 64, 2048^3 on 64 x 64).
double clocks_per_k(const cuasr_b200_desc_t& desc, int tile) {
  static constexpr double f64_min[4] = {6.6, 7.1, 7.2, 7.3}, f64_bottleneck[4] = {9.1, 9.6, 9.5, 9.7};
  const bool sum = desc.add_op == CUASR_OP_PLUS, logical = desc.add_op == CUASR_OP_BINARY_OR;
  const bool bottleneck = desc.mul_op == CUASR_OP_MINIMUM || desc.mul_op == CUASR_OP_MAXIMUM;
  double per_product = 2.15;
  if (logical) per_product = 3.1;
  else if (desc.dtype == CUASR_F64) per_product = sum ? 2.1 : bottleneck ? f64_bottleneck[tile] : f64_min[tile];
  else if (desc.dtype == CUASR_F32 && sum) per_product = 1.55;
  else if (bottleneck) per_product = 3.0;
  // the shorter runs of chunks of the smaller tiles: 2048^3 on 64 x 64 522 us where 2.15 a product would be 504
  return 2 * 64 * per_product * (desc.dtype != CUASR_F64 && tile != kLargeTile ? 1.06 : 1.0);
}

struct LaunchPlan {
  int tile = kSmallTile;
  int cluster = 1;                 // CTAs that share a tile's K range through a cluster
  int whole_tiles = 0, pieces = 1; // ticket pieces (cluster == 1)
  double cost = 1e300;             // modelled clocks
};
constexpr int kTileRows[4] = {LargeTile::kM, MediumTile::kM, SmallTile::kM, TinyTile::kM};
constexpr int kTileCols[4] = {LargeTile::kN, MediumTile::kN, SmallTile::kN, TinyTile::kN};
constexpr int kTileWk[4] = {LargeTile::WK, MediumTile::WK, SmallTile::WK, TinyTile::WK};
// k columns per stage; fp64 sums use the deep form of the tiny tile
int tile_sub(int tile, const cuasr_b200_desc_t& desc) {
  constexpr int sub[4] = {LargeTile::kSub, MediumTile::kSub, SmallTile::kSub, TinyTile::kSub};
  const bool dmma = desc.dtype == CUASR_F64 && desc.add_op == CUASR_OP_PLUS && desc.mul_op == CUASR_OP_MULTIPLIES;
  return tile == kTinyTile && dmma ? TinyTileDeep::kSub : sub[tile];
}

// The fastest of the launches that need no workspace, by a model in clocks: start of the launch and first tile of
// operands 3000, then per wave of CTAs the contraction (above) and the tile's end (8000 for the large tile, 1500 for the
// fold of the small ones, twice that for 8-byte elements), 2500 for the exchange inside a cluster.  Clusters of four
// and eight do not fill every SM (a cluster lives in one GPC): 144 and 128 of the 148.
// A cluster launch is not persistent: each further wave starts its CTAs anew, 4000, and 30000 where eight have to find room in one
// GPC together (77 x 3001 x 2999 in fp64 as three waves of such clusters: 262 to 434 us where 266 were modelled).  The 64 x 32 tile hands a stage over
// for every chunk of a warp: 250 clocks a stage, twice that for 8-byte elements (a 512 x 4096 x 4096 product as seven waves of it took 635 us instead of
// the 514 modelled without; the 128 x 128 tile takes 580).
// A gathered element costs 0.17 clocks on the small tiles where the contraction is bound by register reads (2048^3
// min-plus with one operand transposed on 64 x 64 tiles: 589 us against 522 with TMA) and in fp32 sums (457 against 373), 0.08
// in the other rings (max-min: 795 against 765), and 0.07, 0.155 and 0.02 on the large one (4096^3 min-plus: 3998 against 3969,
// both operands 4096; fp32 sums 3240 against 2950).
bool packs_pairs(const cuasr_b200_desc_t& desc) {          // Ring::kPackedPairs
  return desc.dtype == CUASR_F32 && (desc.add_op == CUASR_OP_MINIMUM || desc.add_op == CUASR_OP_MAXIMUM) &&
         (desc.mul_op == CUASR_OP_PLUS || desc.mul_op == CUASR_OP_MULTIPLIES);
}
// Rings whose large tile has variants for operands along their rows (LargeRowsTile).
bool takes_rows(const cuasr_b200_desc_t& desc) {
  if (desc.dtype == CUASR_F64 && desc.add_op != CUASR_OP_PLUS) return desc.mul_op != CUASR_OP_PLUS && desc.mul_op != CUASR_OP_MULTIPLIES;
  return !packs_pairs(desc);
}
double gather_clocks(const cuasr_b200_desc_t& desc, bool large) {
  if (desc.dtype == CUASR_F32 && desc.add_op == CUASR_OP_PLUS) return large ? 0.155 : 0.18;
  return packs_pairs(desc) ? (large ? 0.07 : 0.17) : (large ? 0.02 : 0.08);
}

// Which operands a launch has to gather, given which ones are copied first.  The large tile takes operands that lie along
// their rows as they are where TMA can bring in both (rows_a, rows_b) and the ring gains nothing from pairs of k.
struct Gathers {
  bool a = false, b = false;                 // the smaller tiles
  bool large_a = false, large_b = false;
  bool rows_a = false, rows_b = false;       // large tile: along its rows, by TMA
};
Gathers gathers_of(const cuasr_b200_desc_t& desc, const cuasr_b200_args_t& args, const Normalised& p, bool copied_a, bool copied_b) {
  const size_t es = desc.dtype == CUASR_F64 ? 8 : 4;
  const int tk = kTileKBytes / static_cast<int>(es);
  const bool by_tma_a = copied_a || tma_describable(p.a, p.lda, es), by_tma_b = copied_b || tma_describable(p.b, p.ldb, es);
  const bool along_k_a = copied_a || p.a_kcontig, along_k_b = copied_b || p.b_kcontig;
  Gathers g;
  g.a = g.large_a = !along_k_a || !by_tma_a;
  g.b = g.large_b = !along_k_b || !by_tma_b;
  const bool dense = p.lda >= (p.a_kcontig ? p.k : p.m) && p.ldb >= (p.b_kcontig ? p.k : p.n);
  if (takes_rows(desc) && by_tma_a && by_tma_b && dense && (p.k % tk == 0 || ring_pads_itself(desc, args))) {
    g.rows_a = !along_k_a; g.rows_b = !along_k_b;
    g.large_a = g.large_b = false;
  }
  return g;
}

LaunchPlan plan_without_workspace(const cuasr_b200_desc_t& desc, int m, int n, int k, int sms, bool all_tiles, const Gathers& g,
                                  bool asks = false) {
  const int tk = kTileKBytes / (desc.dtype == CUASR_F64 ? 8 : 4);
  const double wide = desc.dtype == CUASR_F64 ? 2.0 : 1.0;
  LaunchPlan best;
  for (int tile = all_tiles ? kLargeTile : kSmallTile; tile <= kTinyTile; ++tile) {
    const long long tiles = static_cast<long long>((m + kTileRows[tile] - 1) / kTileRows[tile]) * ((n + kTileCols[tile] - 1) / kTileCols[tile]);
    if (asks && tile == kMediumTile && best.whole_tiles >= sms) break;  // (the variants that ask are slower on smaller tiles: 2048^3 1921 us on 64 x 64)
    const int step = tk * tile_sub(tile, desc);
    const int k_steps = (k + step - 1) / step;
    for (int z = 1; z <= (tile == kLargeTile ? 1 : 8); z *= 2) {
      const int per_piece = (k_steps + z - 1) / z;
      if ((z - 1) * per_piece >= k_steps) break;                        // every CTA of a cluster has work
      const long long room = z <= 2 ? sms : z == 4 ? sms * 36LL / 37 : sms * 32LL / 37;
      const long long waves = (tiles * z + room - 1) / room;
      if (asks && z > 1 && waves > 1) break;                            // every CTA looks at the sample: once
      const double end = (tile == kLargeTile ? 8000 : 1500) * wide + (z > 1 ? 2500 + (waves > 1 ? (z == 8 ? 30000 : 4000) : 0) : 0);
      const bool gather_a = tile == kLargeTile ? g.large_a : g.a, gather_b = tile == kLargeTile ? g.large_b : g.b;
      const double gathered = gather_clocks(desc, tile == kLargeTile) * step * ((gather_a ? kTileRows[tile] : 0) + (gather_b ? kTileCols[tile] : 0));
      const double per_stage = clocks_per_k(desc, tile) * step / kTileWk[tile] + gathered + (tile == kTinyTile ? 250 * wide : 0);
      const double cost = 3000 + static_cast<double>(waves) * (per_stage * per_piece + end);
      if (cost < best.cost) {
        best.tile = tile; best.cluster = z; best.cost = cost;
        best.whole_tiles = z > 1 ? 0 : static_cast<int>(tiles); best.pieces = z;
      }
    }
  }
  return best;
}
template <typename T>
bool ring_has_all_tiles(const cuasr_b200_desc_t& desc) {
#define X(ADD, MUL) if (desc.add_op == ADD && desc.mul_op == MUL) return all_tiles_instantiated<ADD, MUL, T>();
  CUASR_FLOAT_RINGS(X)
  if constexpr (std::is_integral<T>::value) { CUASR_BIT_RINGS(X) }
#undef X
  return false;
}

bool has_all_tiles(const cuasr_b200_desc_t& desc) {
  switch (desc.dtype) {
    case CUASR_F32: return ring_has_all_tiles<float>(desc);
    case CUASR_F64: return ring_has_all_tiles<double>(desc);
    case CUASR_S32: return ring_has_all_tiles<int32_t>(desc);
    default:        return ring_has_all_tiles<uint32_t>(desc);
  }
}

// ---- the screened kernel (srgemm_screened.cuh) -------------------------------------------------------------------
struct ScreenPlan {
  int pieces = 1, blocks_per_piece = 0;
  double cost = 1e300;
};
// Modelled clocks: 3.7 per product and scheduler with the tests, the conversions and the usual number of recomputed
// elements (1000 x 1000 x 3000 takes 250 us more than 1000^3 with 31 blocks more per CTA), and 400000 per tile or piece for
// its first blocks, which are done exactly or with many recomputed elements; 40000 for the two launches and their samples.  So
// 2048^3 is screened (1.37 - 1.43 ms against 1.72 exact) and 1000^3 is not (334 - 379 us against 237).
// An operand that is gathered costs it 4.5 % (4096^3 7760 -> 8066 us with one, 2048^3 1397 -> 1475).
ScreenPlan screen_plan(int m, int n, int k, int sms, bool may_split, const Gathers& g) {
  const int blocks = (k + kScreenBlock - 1) / kScreenBlock;
  const long long tiles = static_cast<long long>((m + kTileM - 1) / kTileM) * ((n + kTileN - 1) / kTileN);
  const double per_block = 128.0 * kScreenBlock * 3.7;
  const double first = 400000;
  ScreenPlan best;
  for (int pieces = 1; pieces <= (may_split ? 128 : 1) && pieces <= blocks; ++pieces) {
    const int per_piece = (blocks + pieces - 1) / pieces;
    if ((pieces - 1) * per_piece >= blocks) continue;                     // every piece has work
    const long long waves = (tiles * pieces + sms - 1) / sms;
    const double cost = 40000 + (pieces > 1 ? 4000 : 0) + static_cast<double>(waves) * (per_block * per_piece + first + 2000);
    if (cost < best.cost) { best.cost = cost; best.pieces = pieces; best.blocks_per_piece = per_piece; }
  }
  best.cost *= 1 + 0.045 * (g.a + g.b);
  return best;
}
// The products the screened kernel can do: no factor (alpha is the identity of +) and a start value that compares, so that the running
// minimum can live in D; and no negative zeros among the factors, so that D holds none and values that compare equal are the same.
bool can_screen(const cuasr_b200_desc_t& desc, const cuasr_b200_args_t& args) {
  if (desc.dtype != CUASR_F64 || desc.mul_op != CUASR_OP_PLUS || (desc.add_op != CUASR_OP_MINIMUM && desc.add_op != CUASR_OP_MAXIMUM)) return false;
  const double alpha = load_scalar<double>(args.alpha), beta = load_scalar<double>(args.beta), id = load_scalar<double>(args.add_identity);
  return id == id && alpha == 0.0 && !std::signbit(alpha) && !(beta == 0.0 && std::signbit(beta));
}

// Every other ring (the integer min/max rings) has no value TMA could fill in.  With the optional workspace both
// operands are copied and their K range is extended to a whole number of K steps by repeating the last k, as the gather
// does without the workspace: these rings are idempotent, and nothing depends on the caller's identities.
// An operand that lies along its rows is copied, transposed, where that makes the modelled launch faster by more than the
// copy takes (12000 clocks for its launch and the tail of its stores, 2200 bytes per clock): 2048^3 min-plus with one such
// operand 589 us gathered, 538 copied; 4096^3 3998 and 4007.
size_t copies_bytes(const RepackPlan& plan, const Normalised& p, size_t es) {
  const int k = plan.k_padded > 0 ? plan.k_padded : p.k;
  return (plan.a ? repack_operand_bytes(p.m, k, es) : 0) + (plan.b ? repack_operand_bytes(p.n, k, es) : 0);
}
double copies_clocks(const RepackPlan& plan, const Normalised& p, size_t es) {
  if (!plan.a && !plan.b) return 0;
  return 12000.0 + 2.0 * es * p.k * ((plan.a ? p.m : 0.0) + (plan.b ? p.n : 0.0)) / 2200;
}
RepackPlan repack_plan(const cuasr_b200_desc_t& desc, const cuasr_b200_args_t& args, const Normalised& p, int sms) {
  RepackPlan plan;
  const size_t es = desc.dtype == CUASR_F64 ? 8 : 4;
  // not for storage lines that overlap, nor for small products: up to about 128^3 the copy's launch costs as much as
  // the product itself, which gathers its operands just as well
  if (static_cast<double>(p.m) * p.n * p.k < 128.0 * 128 * 128 || static_cast<long long>(p.m) * p.n < 64 * 64) return plan;
  if (p.lda < (p.a_kcontig ? p.k : p.m) || p.ldb < (p.b_kcontig ? p.k : p.n)) return plan;
  const int tk = kTileKBytes / static_cast<int>(es);
  if (p.k % tk != 0 && !ring_pads_itself(desc, args)) {
    plan.a = plan.b = true;
    plan.k_padded = (p.k + 2 * tk - 1) / (2 * tk) * (2 * tk);     // the longest K step of a tile (rings without padding)
  } else {
    plan.a = !tma_describable(p.a, p.lda, es);
    plan.b = !tma_describable(p.b, p.ldb, es);
    const bool all_tiles = has_all_tiles(desc);
    const bool screens = can_screen(desc, args);
    auto cost = [&](bool copy_a, bool copy_b) {
      const Gathers g = gathers_of(desc, args, p, copy_a, copy_b);
      const double exact = plan_without_workspace(desc, p.m, p.n, p.k, sms, all_tiles, g).cost;
      return screens ? std::min(exact, screen_plan(p.m, p.n, p.k, sms, true, g).cost) : exact;
    };
    for (const bool first : {true, false}) {
      RepackPlan more = plan;
      bool& copied = first ? more.a : more.b;
      if (copied || (first ? p.a_kcontig : p.b_kcontig)) continue;
      copied = (first ? more.faster_a : more.faster_b) = true;
      if (cost(more.a, more.b) + copies_clocks(more, p, es) < cost(plan.a, plan.b) + copies_clocks(plan, p, es)) plan = more;
    }
  }
  plan.bytes = copies_bytes(plan, p, es);
  return plan;
}

// Modelled clocks of a launch of large tiles whose pieces meet through tickets in a workspace.
double ticket_plan_cost(const cuasr_b200_desc_t& desc, long long tiles, int whole_tiles, int pieces, int k, int sms, int gathered) {
  const int tk = kTileKBytes / (desc.dtype == CUASR_F64 ? 8 : 4);
  const double wide = desc.dtype == CUASR_F64 ? 2.0 : 1.0;
  const int k_steps = (k + tk - 1) / tk, per_piece = (k_steps + pieces - 1) / pieces;
  const double per_step = (clocks_per_k(desc, kLargeTile) + gather_clocks(desc, true) * kTileM * gathered) * tk;
  const long long waves = whole_tiles / sms, tail = ((tiles - whole_tiles) * pieces + sms - 1) / sms;
  // the tickets are cleared by a memset in front of the launch; a piece is parked and read back by the last one, 20000 clocks a
  // wave (1000^3 in two pieces 88 us, 2048^3 in four of its last wave 527)
  const double parked = 10000 * (1 + wide);
  return 3000 + 4000 + waves * (per_step * k_steps + 8000 * wide) + tail * (per_step * per_piece + parked) + 1000 * wide * pieces;
}

// How the kernels that can fill in NaN or an infinity bring in one operand, and its tensor map if that is TMA.
template <typename T>
int operand_mode(CUtensorMap* map, const void* ptr, long long ld, bool kcontig, int rows, int k, int box_rows) {
  if (!kcontig) return kLoadGatherMN;
  if (encode_tiled_fn() != nullptr && ld >= k && tma_describable(ptr, ld, sizeof(T)) &&
      make_operand_map<T>(map, static_cast<const T*>(ptr), ld, rows, k, true, true, box_rows))
    return kLoadTma;
  return kLoadGatherK;
}

// The screened kernel reads D back and updates it with atomics: only where D lies in this GPU's memory (or migrates there).
// In host memory or on a peer every one of these crosses a link, where the exact kernel writes each element once.
bool in_device_memory(const void* ptr) {
  cudaPointerAttributes at = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaPointerGetAttributes(&at, ptr) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeManaged || (at.type == cudaMemoryTypeDevice && at.device == dev);
}

// Launches the screened kernel on a normalised problem (row-major D).
int run_screened(bool maximize, const Normalised& p, double beta, double add_id, bool read_c, const ScreenPlan& plan, bool if_it_helps,
                 const ExtraOutputs& extra, DeviceState* dev, cudaStream_t stream) {
  ScreenParams sp = {};
  sp.M = p.m; sp.N = p.n; sp.K = p.k;
  sp.A = static_cast<const double*>(p.a); sp.lda = p.lda;
  sp.B = static_cast<const double*>(p.b); sp.ldb = p.ldb;
  CUtensorMap map_a = {}, map_b = {};
  sp.a_mode = operand_mode<double>(&map_a, p.a, p.lda, p.a_kcontig, p.m, p.k, kTileM);
  sp.b_mode = operand_mode<double>(&map_b, p.b, p.ldb, p.b_kcontig, p.n, p.k, kTileN);
  sp.C = static_cast<const double*>(p.c); sp.ldc = p.ldc;
  sp.D = static_cast<double*>(p.d); sp.ldd = p.ldd;
  sp.beta = beta; sp.add_identity = add_id; sp.read_c = read_c;
  sp.n_extra = extra.count;
  for (int x = 0; x < extra.count; ++x) sp.extra_d[x] = static_cast<double*>(extra.ptr[x]);
  sp.tiles_m = (p.m + kTileM - 1) / kTileM; sp.tiles_n = (p.n + kTileN - 1) / kTileN;
  sp.if_it_helps = if_it_helps;
  sp.pieces = plan.pieces; sp.blocks_per_piece = plan.blocks_per_piece;
  sp.status = dev->status;
  const long long work = static_cast<long long>(sp.tiles_m) * sp.tiles_n * sp.pieces;
  if (work > 2147483647LL) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  if (plan.pieces > 1) {
    if (launch_screened_init(maximize, sp, dev->sms, stream) != cudaSuccess) return CUASR_STATUS_ERROR_INTERNAL;
    g_launches.fetch_add(1);
  }
  const int grid = static_cast<int>(work < dev->sms ? work : dev->sms);
  if (launch_screened(maximize, map_a, map_b, sp, grid, stream) != cudaSuccess) return CUASR_STATUS_ERROR_INTERNAL;
  g_launches.fetch_add(1);
  t_route = {"screened", kTileM, kTileN, 1, plan.pieces, load_name(sp.a_mode), load_name(sp.b_mode)};
  t_route.screened_pieces = plan.pieces;
  return CUASR_STATUS_SUCCESS;
}

// ---- the path-tracking kernel (srgemm_path.cuh) -------------------------------------------------------------------
// Its launch by the model of plan_without_workspace, with the work that comes on top of the contraction: per stage a
// test of 64 elements (256 clocks per warp), and the look-ups, about 64 / t + 1.5 per lane after stage t of cold data, of
// 60 clocks per four chunks of the stage that a warp works on.
template <typename T>
int run_path(bool maximize, const Normalised& p, int32_t* parent, long long ld_parent, int k_offset, DeviceState* dev,
             cudaStream_t stream) {
  constexpr int TK = kTileKBytes / sizeof(T);
  constexpr int small = sizeof(T) == 4 ? kSmallTile : kTinyTile;
  double best = 1e300;
  int tile = kLargeTile, cluster = 1;
  for (int candidate : {(int)kLargeTile, small}) {
    const bool large = candidate == kLargeTile;
    const long long tiles = static_cast<long long>((p.m + kTileRows[candidate] - 1) / kTileRows[candidate]) * ((p.n + kTileCols[candidate] - 1) / kTileCols[candidate]);
    const int step = candidate == kSmallTile ? 2 * TK : TK;
    const double per_k = 2 * 64 * (sizeof(T) == 4 ? 2.1 : large ? 6.6 : 9.1);
    const double chunks = large ? 2 : candidate == kSmallTile ? 1 : 0.25;           // in fours, of a warp and stage
    const int k_steps = (p.k + step - 1) / step;
    for (int z = 1; z <= (large ? 1 : 8); z *= 2) {
      const int per_piece = (k_steps + z - 1) / z;
      if ((z - 1) * per_piece >= k_steps) break;
      const long long room = z <= 2 ? dev->sms : z == 4 ? dev->sms * 36LL / 37 : dev->sms * 32LL / 37;
      const long long waves = (tiles * z + room - 1) / room;
      const double per_stage = per_k * step / kTileWk[candidate] + (sizeof(T) == 8 && !large ? 250 : 2 * 256 + 2 * 1.5 * 60 * chunks);
      // fp64: 300 clocks on the large tile for each look-up of the slowest lane, half of them counted (cold and settled distances are
      // as common); none on the small one, whose index follows every product
      const double lookups = sizeof(T) == 4 ? 2 * 64 * 60 * chunks * std::log(1.0 + per_piece)
                             : large ? (96 * std::log(1.0 + per_piece) + 4 * per_piece) * 300 : 0;
      const double cost = 3000 + static_cast<double>(waves) * (per_stage * per_piece + lookups + 3000 + (z > 1 ? 3000 + (waves > 1 ? 8000 : 0) : 0));
      if (cost < best) { best = cost; tile = candidate; cluster = z; }
    }
  }
  PathParams<T> pp = {};
  pp.M = p.m; pp.N = p.n; pp.K = p.k;
  pp.A = static_cast<const T*>(p.a); pp.lda = p.lda;
  pp.B = static_cast<const T*>(p.b); pp.ldb = p.ldb;
  CUtensorMap map_a = {}, map_b = {};
  pp.a_mode = operand_mode<T>(&map_a, p.a, p.lda, p.a_kcontig, p.m, p.k, kTileRows[tile]);
  pp.b_mode = operand_mode<T>(&map_b, p.b, p.ldb, p.b_kcontig, p.n, p.k, kTileCols[tile]);
  pp.pad = static_cast<T>(NAN);
  pp.dist = static_cast<T*>(p.d); pp.ldd = p.ldd;
  pp.parent = parent; pp.ld_parent = ld_parent; pp.k_offset = k_offset;
  pp.tiles_m = (p.m + kTileRows[tile] - 1) / kTileRows[tile]; pp.tiles_n = (p.n + kTileCols[tile] - 1) / kTileCols[tile];
  const int step = tile == kSmallTile ? 2 * TK : TK;
  const int k_steps = (p.k + step - 1) / step;
  pp.cluster = cluster; pp.k_tiles_per_slice = (k_steps + cluster - 1) / cluster;
  pp.status = dev->status;
  const long long work = static_cast<long long>(pp.tiles_m) * pp.tiles_n * cluster;
  if (work > 2147483647LL) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  const int grid = static_cast<int>(cluster > 1 || work < dev->sms ? work : dev->sms);
  if (launch_path<T>(maximize, tile != kLargeTile, map_a, map_b, pp, grid, stream) != cudaSuccess) return CUASR_STATUS_ERROR_INTERNAL;
  g_launches.fetch_add(1);
  t_route = {"path", kTileRows[tile], kTileCols[tile], cluster, cluster, load_name(pp.a_mode), load_name(pp.b_mode)};
  return CUASR_STATUS_SUCCESS;
}

template <typename T>
int run_typed(const cuasr_b200_desc_t& desc, const cuasr_b200_args_t& args, int slices, const ExtraOutputs& extra, int screen_pieces) {
  DeviceState* dev = nullptr;
  if (!device_state(&dev)) return CUASR_STATUS_ERROR_INTERNAL;
  cudaStream_t stream = static_cast<cudaStream_t>(args.stream);
  Normalised p = normalise(desc, args);

  const int plan_sms = planning_sms(desc, dev->sms);

  const T alpha = load_scalar<T>(args.alpha), beta = load_scalar<T>(args.beta);
  const T add_id = load_scalar<T>(args.add_identity), mul_id = load_scalar<T>(args.mul_identity);
  // semiring_linear_combination.h:118-125: C is read unless mult(beta, mult-identity) is the add-identity
  const bool read_c = !(host_op<T>(desc.mul_op, beta, mul_id) == add_id);

  if (slices > 1 && args.workspace == nullptr) return CUASR_STATUS_ERROR_WORKSPACE_NULL;
  if (read_c && p.c == nullptr) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  // partials are moved 16 bytes at a time and re-packed operands are read by TMA: a workspace that does not start
  // on a 16-byte boundary is an error where it is required and is left unused where it is optional
  const bool workspace_aligned = reinterpret_cast<uintptr_t>(args.workspace) % 16 == 0;
  constexpr int TK = kTileKBytes / sizeof(T);
  const long long tiles = static_cast<long long>(tile_count(args));
  const bool all_tiles = ring_has_all_tiles<T>(desc);
  // an optional workspace buys load balancing and, behind its scratch, copies of operands, as far as it has room for them
  BalancePlan balance{0, 1};
  bool balanced = false;
  size_t copies_at = 0;
  RepackPlan copies;
  if (slices == 1 && args.workspace != nullptr && workspace_aligned) {
    const size_t balance_bytes = balance_workspace_bytes(desc, args, plan_sms);
    balanced = all_tiles && balance_bytes > 0 && args.workspace_bytes >= balance_bytes;
    if (balanced) balance = balance_plan(tiles, plan_sms, (args.k + TK - 1) / TK);
    copies_at = align_up(balance_bytes, 256);
    copies = repack_plan(desc, args, p, plan_sms);
    if (copies.bytes == 0 || args.workspace_bytes < copies_at + copies.bytes) copies = RepackPlan();
  }
  long long pieces = 1;
  if (slices > 1) {
    const size_t need = splitk_workspace_bytes(desc, args);
    if (args.workspace_bytes < need) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
    if (!workspace_aligned) return CUASR_STATUS_ERROR_MISALIGNED_OPERAND;
    if (all_tiles) {
      // as many pieces as the workspace at hand has room for (it always has room for `slices`)
      const size_t per_piece = splitk_bytes_for_pieces(desc, args, 1) - splitk_bytes_for_pieces(desc, args, 0);
      const long long room = static_cast<long long>((args.workspace_bytes - splitk_bytes_for_pieces(desc, args, 0)) / per_piece);
      pieces = splitk_pieces(desc, args, plan_sms, room);
    }
  }
  // the fastest launch with a given set of copies: without the workspace, or in pieces that meet through tickets in it
  Gathers gathers;
  bool tickets_used = false;
  auto plan_with = [&](const RepackPlan& c, Gathers& g, bool& tickets, bool asks = false) {
    g = gathers_of(desc, args, p, c.a, c.b);
    LaunchPlan best = plan_without_workspace(desc, p.m, p.n, p.k, plan_sms, all_tiles, g, asks);
    tickets = false;
    auto in_pieces = [&](int whole_tiles, int count, bool always) {
      const double cost = ticket_plan_cost(desc, tiles, whole_tiles, count, p.k, plan_sms, g.large_a + g.large_b);
      if (cost >= best.cost && !always) return;
      best.tile = kLargeTile; best.cluster = 1; best.whole_tiles = whole_tiles; best.pieces = count; best.cost = cost;
      tickets = true;
    };
    // floating-point sums keep the cutting that was asked for
    if (slices > 1 && all_tiles) in_pieces(0, static_cast<int>(pieces), !splitk_order_independent(desc));
    if (balanced) in_pieces(balance.whole_tiles, balance.pieces, false);
    best.cost += copies_clocks(c, p, sizeof(T));
    return best;
  };
  // The screened kernel, where it is modelled faster, if the operands are what it helps with: it is launched in front of the exact one,
  // and a sample of the operands tells either of them whether the product is its own.
  const bool may_screen = can_screen(desc, args) && !(read_c && std::signbit(beta) && beta == T(0));
  auto screened_with = [&](const RepackPlan& c, const Gathers& g) {
    ScreenPlan best;
    if (may_screen) best = screen_plan(p.m, p.n, p.k, dev->sms, extra.count == 0, g);
    best.cost += copies_clocks(c, p, sizeof(T));
    return best;
  };
  LaunchPlan plan = plan_with(copies, gathers, tickets_used);
  ScreenPlan screened = screened_with(copies, gathers);
  if (copies.faster_a || copies.faster_b) {          // in pieces the large tile may do as well on the operands as they are
    RepackPlan fewer = copies;
    fewer.a = copies.a && !copies.faster_a; fewer.b = copies.b && !copies.faster_b;
    fewer.faster_a = fewer.faster_b = false;
    fewer.bytes = copies_bytes(fewer, p, sizeof(T));
    Gathers g;
    bool tickets;
    const LaunchPlan other = plan_with(fewer, g, tickets);
    const ScreenPlan other_screened = screened_with(fewer, g);
    if (std::min(other.cost, other_screened.cost) < std::min(plan.cost, screened.cost)) {
      plan = other; screened = other_screened; copies = fewer; gathers = g; tickets_used = tickets;
    }
  }
  const bool use_screen = screen_pieces < 0 && screened.cost < plan.cost && in_device_memory(p.d);
  if (use_screen) plan = plan_with(copies, gathers, tickets_used, true);
  const bool pads_itself = ring_pads_itself(desc, args);
  // operands whose storage lines overlap (leading dimension below the contiguous extent) stay off the TMA path
  const bool dense = p.lda >= (p.a_kcontig ? p.k : p.m) && p.ldb >= (p.b_kcontig ? p.k : p.n);
  const bool small = static_cast<long long>(p.m) * p.n < 64 * 64;
  // the rest of an optional workspace holds K-contiguous, aligned copies of operands (see RepackPlan)
  const bool repacked = copies.bytes > 0;
  int k_map = p.k;              // K extent the tensor maps describe
  if (repacked) {
    char* cursor = static_cast<char*>(args.workspace) + copies_at;
    k_map = copies.k_padded > 0 ? copies.k_padded : p.k;
    const long long ldt = static_cast<long long>(align_up(static_cast<size_t>(k_map), 16 / sizeof(T)));
    RepackRequest requests[2];
    int count = 0;
    if (copies.a) {
      requests[count++] = {p.a, p.lda, p.a_kcontig, p.m, p.k, k_map, cursor, ldt};
      p.a = cursor; p.lda = ldt; p.a_kcontig = true;
      cursor += repack_operand_bytes(p.m, k_map, sizeof(T));
    }
    if (copies.b) {
      requests[count++] = {p.b, p.ldb, p.b_kcontig, p.n, p.k, k_map, cursor, ldt};
      p.b = cursor; p.ldb = ldt; p.b_kcontig = true;
    }
    if (launch_repack(requests, count, sizeof(T), stream) != cudaSuccess) return CUASR_STATUS_ERROR_INTERNAL;
    g_launches.fetch_add(1);
  }

  const bool describable = tma_describable(p.a, p.lda, sizeof(T)) && tma_describable(p.b, p.ldb, sizeof(T));
  // the name a caller sees: "tma..." where the storage lines are what TMA could describe
  const bool aligned_name = (pads_itself || k_map % TK == 0) && !small && dense && describable;
  const char* const name = !aligned_name ? (slices > 1 ? "generic_splitk" : "generic")
                           : slices > 1 ? "tma_splitk" : balanced ? "tma_balanced" : repacked ? "tma_repacked" : "tma";
  if constexpr (std::is_same<T, double>::value) {
    const bool maximize = desc.add_op == CUASR_OP_MAXIMUM;
    if (screen_pieces >= 0) {          // cuasr_b200_srgemm_screened
      if (!may_screen) return CUASR_STATUS_ERROR_NOT_SUPPORTED;
      if (screen_pieces > 0) {
        const int blocks = (p.k + kScreenBlock - 1) / kScreenBlock;
        screened.pieces = screen_pieces; screened.blocks_per_piece = (blocks + screen_pieces - 1) / screen_pieces;
        if ((screened.pieces - 1LL) * screened.blocks_per_piece >= blocks) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
      }
    }
    if (screen_pieces >= 0 || use_screen) {
      const int st = run_screened(maximize, p, beta, add_id, read_c, screened, use_screen, extra, dev, stream);
      if (st != CUASR_STATUS_SUCCESS) return st;
      t_last_kernel = name;
      t_route.copied_a = copies.a; t_route.copied_b = copies.b;
      if (!use_screen) return st;
    }
  }
  const int step = TK * tile_sub(plan.tile, desc);
  const bool nan_pad = std::is_floating_point<T>::value && (desc.add_op == CUASR_OP_MINIMUM || desc.add_op == CUASR_OP_MAXIMUM);
  // TMA brings in what lies along k on aligned lines, unless a ragged last step needs padding it cannot write
  const bool fill_ok = encode_tiled_fn() != nullptr && dense && (pads_itself || k_map % step == 0);
  TmaParams<T> tp;
  tp.M = p.m; tp.N = p.n; tp.K = p.k;
  tp.A = static_cast<const T*>(p.a); tp.lda = p.lda;
  tp.B = static_cast<const T*>(p.b); tp.ldb = p.ldb;
  tp.a_mode = p.a_kcontig ? (fill_ok && tma_describable(p.a, p.lda, sizeof(T)) ? kLoadTma : kLoadGatherK) : kLoadGatherMN;
  tp.b_mode = p.b_kcontig ? (fill_ok && tma_describable(p.b, p.ldb, sizeof(T)) ? kLoadTma : kLoadGatherK) : kLoadGatherMN;
  CUtensorMap map_a = {}, map_b = {};
  if (plan.tile == kLargeTile && (gathers.rows_a || gathers.rows_b) && encode_tiled_fn() != nullptr &&
      make_operand_map<T>(&map_a, tp.A, p.lda, p.m, k_map, !gathers.rows_a, nan_pad) &&
      make_operand_map<T>(&map_b, tp.B, p.ldb, p.n, k_map, !gathers.rows_b, nan_pad)) {
    tp.a_mode = gathers.rows_a ? kLoadTmaRows : kLoadTma;
    tp.b_mode = gathers.rows_b ? kLoadTmaRows : kLoadTma;
  }
  if (tp.a_mode == kLoadTma &&
      !make_operand_map<T>(&map_a, tp.A, p.lda, p.m, k_map, true, nan_pad, kTileRows[plan.tile])) tp.a_mode = kLoadGatherK;
  if (tp.b_mode == kLoadTma &&
      !make_operand_map<T>(&map_b, tp.B, p.ldb, p.n, k_map, true, nan_pad, kTileCols[plan.tile])) tp.b_mode = kLoadGatherK;
  if (k_map != p.k && (tp.a_mode != kLoadTma || tp.b_mode != kLoadTma)) tp.K = k_map;   // copies that hold their own padding
  tp.pad = nan_pad ? static_cast<T>(NAN) : T(0);
  // the other rings (integer minima and maxima, logical or from an odd start value) are idempotent
  tp.repeat_k = !pads_itself;
  tp.C = static_cast<const T*>(p.c); tp.ldc = p.ldc;
  tp.D = static_cast<T*>(p.d); tp.ldd = p.ldd;
  tp.alpha = alpha; tp.beta = beta; tp.add_identity = add_id; tp.read_c = read_c;
  tp.part_identity = desc.add_op == CUASR_OP_PLUS || desc.add_op == CUASR_OP_BIT_XOR ? T(0) : add_id;
  tp.n_extra = extra.count;
  bool vec = tma_describable(p.d, p.ldd, sizeof(T)) && (!read_c || tma_describable(p.c, p.ldc, sizeof(T))) && p.n % (16 / (int)sizeof(T)) == 0;
  for (int x = 0; x < extra.count; ++x) {
    tp.extra_d[x] = static_cast<T*>(extra.ptr[x]);
    vec = vec && reinterpret_cast<uintptr_t>(extra.ptr[x]) % 16 == 0;
  }
  tp.vector_epilogue = vec;
  tp.tiles_m = (p.m + kTileRows[plan.tile] - 1) / kTileRows[plan.tile];
  tp.tiles_n = (p.n + kTileCols[plan.tile] - 1) / kTileCols[plan.tile];
  tp.status = dev->status;
  tp.whole_tiles = plan.whole_tiles;
  tp.slices = plan.pieces;
  tp.cluster = plan.cluster > 1;
  tp.unless_screened = use_screen;
  const int k_steps = (p.k + step - 1) / step;
  tp.k_tiles_per_slice = (k_steps + plan.pieces - 1) / plan.pieces;
  tp.partial = nullptr; tp.tickets = nullptr;
  if (tickets_used && plan.pieces > 1) {
    const size_t ticket_bytes = ticket_bytes_for(args);
    tp.tickets = static_cast<unsigned int*>(args.workspace);
    tp.partial = reinterpret_cast<T*>(static_cast<char*>(args.workspace) + ticket_bytes);
    // same role as the semaphore memset of device/srgemm.h:253-259
    if (cudaMemsetAsync(tp.tickets, 0, ticket_bytes, stream) != cudaSuccess) return CUASR_STATUS_ERROR_INTERNAL;
  }
  const long long all = static_cast<long long>(tp.tiles_m) * tp.tiles_n;
  const long long work = plan.whole_tiles + (all - plan.whole_tiles) * plan.pieces;
  if (work > 2147483647LL) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  const int grid = static_cast<int>(plan.cluster > 1 || work < dev->sms ? work : dev->sms);
  cudaError_t err = cudaErrorInvalidValue;
  bool launched = false;
#define X(ADD, MUL)                                                                                    \
  if (!launched && desc.add_op == ADD && desc.mul_op == MUL) {                                         \
    err = launch_tma<ADD, MUL, T>(plan.tile, map_a, map_b, tp, grid, plan.cluster, stream);            \
    launched = true;                                                                                   \
  }
  CUASR_FLOAT_RINGS(X)
  if constexpr (std::is_integral<T>::value) { CUASR_BIT_RINGS(X) }
#undef X
  if (!launched) return CUASR_STATUS_ERROR_NOT_SUPPORTED;
  if (err != cudaSuccess) return CUASR_STATUS_ERROR_INTERNAL;
  t_last_kernel = name;
  t_route = {"product", kTileRows[plan.tile], kTileCols[plan.tile], plan.cluster, plan.pieces, load_name(tp.a_mode), load_name(tp.b_mode),
             tickets_used && plan.pieces > 1, copies.a, copies.b, use_screen ? screened.pieces : 0};
  g_launches.fetch_add(1);
  return CUASR_STATUS_SUCCESS;
}

int run(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args, int slices,
        const ExtraOutputs& extra = ExtraOutputs(), int screen_pieces = -1) {
  switch (desc->dtype) {
    case CUASR_F32: return run_typed<float>(*desc, *args, slices, extra, screen_pieces);
    case CUASR_F64: return run_typed<double>(*desc, *args, slices, extra, screen_pieces);
    case CUASR_S32: return run_typed<int32_t>(*desc, *args, slices, extra, screen_pieces);
    case CUASR_U32: return run_typed<uint32_t>(*desc, *args, slices, extra, screen_pieces);
    default: return CUASR_STATUS_ERROR_INVALID_DATA_TYPE;
  }
}

// ---- one-sided flags between GPUs --------------------------------------------------------------------------
// A producer raises a word in every consumer's memory after the kernel whose peer stores it announces; a consumer
// waits for its own copy of the word on its own stream.  Neither side ever waits for the other to ARRIVE at a
// collective, which is what lets the owner of a panel run ahead of the ranks that only consume it.
constexpr int kMaxFlagTargets = 8;
constexpr int kMaxFlagWords = 64;
struct FlagTargets {
  unsigned int* ptr[kMaxFlagTargets];
};

// Stream order puts this kernel after the stores it announces; the fence makes them visible system-wide first.
// atomicMax keeps the word monotonic when several producers raise it in turn.
__global__ void flag_raise_kernel(FlagTargets targets, int count, unsigned int value) {
  const int i = threadIdx.x;
  if (i < count) {
    __threadfence_system();
    atomicMax_system(targets.ptr[i], value);
  }
}

// Thread i waits until word i is at least `value`.  The wait is bounded twice (wall time and iterations); when it
// runs out the kernel records kDeviceTimeoutPeerFlag in the status word and returns, so the stream keeps moving and
// the host finds the code with cuasr_b200_device_status.
__global__ void flag_wait_kernel(const unsigned int* words, int count, unsigned int value, unsigned long long limit_ns,
                                 unsigned int* status) {
  const int i = threadIdx.x;
  if (i >= count) return;
  unsigned long long start, now;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(start));
  for (unsigned int spin = 0; spin < (1u << 26); ++spin) {
    unsigned int v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(words + i) : "memory");
    if (v >= value) return;
    __nanosleep(256);
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (now - start > limit_ns) break;
  }
  report_device_error(status, kDeviceTimeoutPeerFlag);
}

// ---- built-in scratch for cuasr_b200_srgemm_splitk_static --------------------------------------------
// The array is device memory that belongs to the loaded module.  Its name is only a host-side handle: a
// kernel must be given the address cudaGetSymbolAddress returns for the CURRENT device, never the name.
static __device__ __align__(256) unsigned char g_static_scratch[CUASR_B200_STATIC_SCRATCH_BYTES];
void* g_static_scratch_ptr[kMaxDevices] = {};
std::mutex g_static_scratch_mutex;

// Device address of the static scratch on the current device; looked up once per device.
cudaError_t static_scratch_address(void** out) {
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return err;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
  if (g_static_scratch_ptr[dev] == nullptr) {
    void* ptr = nullptr;
    err = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_static_scratch);
    if (err != cudaSuccess) return err;
    g_static_scratch_ptr[dev] = ptr;
  }
  *out = g_static_scratch_ptr[dev];
  return cudaSuccess;
}

}  // namespace
}  // namespace cuasr_b200

using namespace cuasr_b200;

extern "C" {

int cuasr_b200_srgemm_can_implement(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args) {
  const int st = validate(desc, args);
  if (st != CUASR_STATUS_SUCCESS) return st;
  // device/srgemm.h:198-200
  if (!desc->split_k_serial && args->split_k_slices > 1) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  return CUASR_STATUS_SUCCESS;
}

size_t cuasr_b200_srgemm_workspace_size(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args) {
  if (desc == nullptr || args == nullptr) return 0;
  if (desc->split_k_serial && args->split_k_slices > 1) return splitk_workspace_bytes_refined(*desc, *args);
  return 0;
}

size_t cuasr_b200_srgemm_optional_workspace_size(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args) {
  if (desc == nullptr || args == nullptr || validate(desc, args) != CUASR_STATUS_SUCCESS) return 0;
  if (args->split_k_slices > 1) return 0;
  DeviceState* dev = nullptr;
  if (!device_state(&dev)) return 0;
  const int sms = planning_sms(*desc, dev->sms);
  const size_t repack = repack_plan(*desc, *args, normalise(*desc, *args), sms).bytes;
  const size_t balance = balance_workspace_bytes(*desc, *args, sms);
  return repack > 0 ? align_up(balance, 256) + repack : balance;
}

int cuasr_b200_srgemm(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args) {
  const int st = cuasr_b200_srgemm_can_implement(desc, args);
  if (st != CUASR_STATUS_SUCCESS) return st;
  return run(desc, args, args->split_k_slices);
}

int cuasr_b200_srgemm_push(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args, int n_extra,
                           void* const* extra_d) {
  const int st = cuasr_b200_srgemm_can_implement(desc, args);
  if (st != CUASR_STATUS_SUCCESS) return st;
  if (n_extra < 0 || n_extra > kMaxDestinations - 1 || (n_extra > 0 && extra_d == nullptr))
    return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  ExtraOutputs extra;
  extra.count = n_extra;
  const size_t es = desc->dtype == CUASR_F64 ? 8 : 4;
  for (int x = 0; x < n_extra; ++x) {
    if (extra_d[x] == nullptr) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
    if (reinterpret_cast<uintptr_t>(extra_d[x]) % es != 0) return CUASR_STATUS_ERROR_MISALIGNED_OPERAND;
    extra.ptr[x] = extra_d[x];
  }
  return run(desc, args, args->split_k_slices, extra);
}

int cuasr_b200_srgemm_screened(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args, int pieces) {
  const int st = cuasr_b200_srgemm_can_implement(desc, args);
  if (st != CUASR_STATUS_SUCCESS) return st;
  if (desc->dtype != CUASR_F64 || args->split_k_slices != 1) return CUASR_STATUS_ERROR_NOT_SUPPORTED;
  if (pieces < 0) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  return run(desc, args, 1, ExtraOutputs(), pieces);
}

int cuasr_b200_srgemm_splitk_can_implement(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args) {
  return validate(desc, args);
}

size_t cuasr_b200_srgemm_splitk_workspace_size(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args) {
  if (desc == nullptr || args == nullptr) return 0;
  return splitk_workspace_bytes_refined(*desc, *args);
}

int cuasr_b200_srgemm_splitk(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args) {
  const int st = validate(desc, args);
  if (st != CUASR_STATUS_SUCCESS) return st;
  // device/srgemm_splitk_parallel.h:247-249
  if (args->split_k_slices > 1 && args->workspace == nullptr) return CUASR_STATUS_ERROR_WORKSPACE_NULL;
  return run(desc, args, args->split_k_slices);
}

int cuasr_b200_srgemm_splitk_static(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args) {
  const int st = validate(desc, args);
  if (st != CUASR_STATUS_SUCCESS) return st;
  if (splitk_workspace_bytes(*desc, *args) > CUASR_B200_STATIC_SCRATCH_BYTES)
    return CUASR_STATUS_ERROR_STATIC_SCRATCH_TOO_SMALL;
  void* scratch = nullptr;
  if (static_scratch_address(&scratch) != cudaSuccess) return CUASR_STATUS_ERROR_INTERNAL;
  cuasr_b200_args_t with_scratch = *args;
  with_scratch.workspace = scratch;
  with_scratch.workspace_bytes = CUASR_B200_STATIC_SCRATCH_BYTES;
  return run(desc, &with_scratch, with_scratch.split_k_slices);
}

int cuasr_b200_srgemm_path(const cuasr_b200_desc_t* desc, const cuasr_b200_args_t* args, int32_t* parent,
                           int64_t ld_parent, int32_t k_offset) {
  const int st = validate(desc, args);
  if (st != CUASR_STATUS_SUCCESS) return st;
  const bool minimize = desc->add_op == CUASR_OP_MINIMUM, maximize = desc->add_op == CUASR_OP_MAXIMUM;
  if (!(minimize || maximize) || desc->mul_op != CUASR_OP_PLUS) return CUASR_STATUS_ERROR_NOT_SUPPORTED;
  if (desc->dtype != CUASR_F32 && desc->dtype != CUASR_F64) return CUASR_STATUS_ERROR_INVALID_DATA_TYPE;
  if (args->split_k_slices != 1) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  if (parent == nullptr || reinterpret_cast<uintptr_t>(parent) % 4 != 0) return CUASR_STATUS_ERROR_MISALIGNED_OPERAND;
  const bool row_c = desc->layout_c == CUASR_ROW_MAJOR;
  if (ld_parent < (row_c ? args->n : args->m)) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  DeviceState* dev = nullptr;
  if (!device_state(&dev)) return CUASR_STATUS_ERROR_INTERNAL;
  // the normalised problem has a row-major D: element (m, n) at D[m * ldd + n], whatever the caller's layout
  const Normalised p = normalise(*desc, *args);
  cudaStream_t stream = static_cast<cudaStream_t>(args->stream);
  const bool f32 = desc->dtype == CUASR_F32;
  const size_t es = f32 ? 4 : 8;
  const bool dense = p.lda >= (p.a_kcontig ? p.k : p.m) && p.ldb >= (p.b_kcontig ? p.k : p.n);
  const bool pipelined = f32 && dense && static_cast<long long>(args->m) * args->n >= 64 * 64 &&
                         tma_describable(p.a, p.lda, es) && tma_describable(p.b, p.ldb, es);
  const int done = f32 ? run_path<float>(maximize, p, parent, ld_parent, k_offset, dev, stream)
                       : run_path<double>(maximize, p, parent, ld_parent, k_offset, dev, stream);
  if (done == CUASR_STATUS_SUCCESS) t_last_kernel = pipelined ? "path_tma" : "path";
  return done;
}

int cuasr_b200_pack_k_contiguous(int32_t dtype, const void* src, int64_t ld_src, int32_t src_k_contiguous, int32_t rows,
                                 int32_t k, void* dst, int64_t ld_dst, void* stream) {
  if (dtype != CUASR_F32 && dtype != CUASR_F64 && dtype != CUASR_S32 && dtype != CUASR_U32)
    return CUASR_STATUS_ERROR_INVALID_DATA_TYPE;
  if (src == nullptr || dst == nullptr || rows <= 0 || k <= 0 || ld_dst < k) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  if (ld_src < (src_k_contiguous ? k : rows)) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  const size_t es = dtype == CUASR_F64 ? 8 : 4;
  if (reinterpret_cast<uintptr_t>(src) % es != 0 || reinterpret_cast<uintptr_t>(dst) % es != 0)
    return CUASR_STATUS_ERROR_MISALIGNED_OPERAND;
  const RepackRequest request = {src, ld_src, src_k_contiguous != 0, rows, k, k, dst, ld_dst};
  if (launch_repack(&request, 1, es, static_cast<cudaStream_t>(stream)) != cudaSuccess)
    return CUASR_STATUS_ERROR_INTERNAL;
  g_launches.fetch_add(1);
  t_last_kernel = "pack";
  t_route = Route();
  t_route.kernel = "pack";
  return CUASR_STATUS_SUCCESS;
}

int cuasr_b200_device_status(void* stream) {
  DeviceState* dev = nullptr;
  if (!device_state(&dev)) return -1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  unsigned int host = 0;
  if (cudaMemcpyAsync(&host, dev->status, sizeof(host), cudaMemcpyDeviceToHost, s) != cudaSuccess) return -1;
  if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
  if (host != 0) cudaMemsetAsync(dev->status, 0, sizeof(unsigned int), s);
  return static_cast<int>(host);
}

int cuasr_b200_flag_raise(void* const* words, int count, uint32_t value, void* stream) {
  if (words == nullptr || count < 1 || count > kMaxFlagTargets) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  FlagTargets targets = {};
  for (int i = 0; i < count; ++i) {
    if (words[i] == nullptr) return CUASR_STATUS_ERROR_INVALID_PROBLEM;
    if (reinterpret_cast<uintptr_t>(words[i]) % 4 != 0) return CUASR_STATUS_ERROR_MISALIGNED_OPERAND;
    targets.ptr[i] = static_cast<unsigned int*>(words[i]);
  }
  flag_raise_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(targets, count, value);
  if (cudaGetLastError() != cudaSuccess) return CUASR_STATUS_ERROR_INTERNAL;
  g_launches.fetch_add(1);
  return CUASR_STATUS_SUCCESS;
}

int cuasr_b200_flag_wait(const void* words, int count, uint32_t value, uint32_t timeout_ms, void* stream) {
  if (words == nullptr || count < 1 || count > kMaxFlagWords || timeout_ms == 0 || timeout_ms > 10000)
    return CUASR_STATUS_ERROR_INVALID_PROBLEM;
  if (reinterpret_cast<uintptr_t>(words) % 4 != 0) return CUASR_STATUS_ERROR_MISALIGNED_OPERAND;
  DeviceState* dev = nullptr;
  if (!device_state(&dev)) return CUASR_STATUS_ERROR_INTERNAL;
  flag_wait_kernel<<<1, kMaxFlagWords, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const unsigned int*>(words), count, value, 1000000ull * timeout_ms, dev->status);
  if (cudaGetLastError() != cudaSuccess) return CUASR_STATUS_ERROR_INTERNAL;
  g_launches.fetch_add(1);
  return CUASR_STATUS_SUCCESS;
}

const char* cuasr_b200_last_kernel(void) { return t_last_kernel; }

const char* cuasr_b200_last_route(void) {
  const Route& r = t_route;
  if (r.tile_m == 0) return r.kernel;
  char screened[32] = "";
  if (r.screened_pieces > 0 && std::strcmp(r.kernel, "product") == 0)
    std::snprintf(screened, sizeof(screened), "screened pieces=%d or ", r.screened_pieces);
  std::snprintf(t_route_text, sizeof(t_route_text), "%s%s tile=%dx%d cluster=%d pieces=%d tickets=%d a=%s%s b=%s%s", screened, r.kernel, r.tile_m,
                r.tile_n, r.cluster, r.pieces, (int)r.tickets, r.copied_a ? "copy+" : "", r.load_a, r.copied_b ? "copy+" : "", r.load_b);
  return t_route_text;
}

uint64_t cuasr_b200_launch_count(void) { return g_launches.load(); }

const char* cuasr_b200_status_string(int status) {
  switch (status) {
    case CUASR_STATUS_SUCCESS: return "success";
    case CUASR_STATUS_ERROR_MISALIGNED_OPERAND: return "misaligned operand";
    case CUASR_STATUS_ERROR_INVALID_DATA_TYPE: return "invalid data type";
    case CUASR_STATUS_ERROR_INVALID_LAYOUT: return "invalid layout";
    case CUASR_STATUS_ERROR_INVALID_PROBLEM: return "invalid problem";
    case CUASR_STATUS_ERROR_NOT_SUPPORTED: return "not supported";
    case CUASR_STATUS_ERROR_WORKSPACE_NULL: return "workspace null";
    case CUASR_STATUS_ERROR_INTERNAL: return "internal error";
    case CUASR_STATUS_ERROR_STATIC_SCRATCH_TOO_SMALL:
      return "problem needs more scratch than the library's static scratch array holds";
    default: return "unknown status";
  }
}

const char* cuasr_b200_version(void) { return "cuasr_b200 0.1 (sm_100a)"; }

}  // extern "C"
