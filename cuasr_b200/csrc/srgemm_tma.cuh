// The B200 SRGEMM kernel: D = (alpha (x) (A (x)(+) B)) (+) (beta (x) C), row-major D.
//
// It replaces, as one kernel, the reference's kernel::Srgemm (include/cuasr/gemm/kernel/srgemm.h:156-321),
// its threadblock mainloop SrmmaPipelined (include/cuasr/gemm/threadblock/srmma_pipelined.h:153-288),
// the warp/thread level (include/cuasr/gemm/warp/srmma_simt.h:139-199,
// include/cuasr/gemm/thread/srmma_sm50.h:118-146) and the epilogue functor
// (include/cuasr/gemm/epilogue/thread/semiring_linear_combination.h:118-183); with split tiles it is
// also kernel::SrgemmSplitKParallel (include/cuasr/gemm/kernel/srgemm_splitk_parallel.h:86-219).
//
// Structure (one CTA per SM, 12 warps = 2 consumer warpgroups + 1 producer warpgroup that hands most of its
// registers to the consumers with setmaxnreg):
//   warps 8..11         producers: for every K step of every output tile this CTA owns, wait for a free stage and
//                       fill it: operands that lie contiguous along k on 16-byte storage lines by TMA (one lane),
//                       all others by the cp.async gather of gather.cuh (all 128 threads).  Either way the stage
//                       holds [rows][128 bytes of k] with the 128-byte swizzle, so there is one contraction loop; only
//                       its loads differ where the large tile takes an operand along its rows as it lies (LargeRowsTile).
//   warps 0..7          consumers: WM x WN x WK warps.  A warp owns a 64 x 32 block of the tile (8 x 4 lanes, an
//                       8 x 8 register micro-tile per lane) and every WK-th part of each stage's k range.
//                       They wait for a stage, read 16-byte vectors and run the contraction two k steps at a time:
//                       acc = add(acc, a0 (x) b0, a1 (x) b1)  — for fp32 min/max rings one packed add for both
//                       products plus ONE three-input min/max.
// Tiles: WM x WN x WK = 2 x 4 x 1 is a 128 x 128 tile, for outputs with enough of them to fill the GPU.  Smaller
// outputs leave most SMs idle with it, and a smaller micro-tile would be bound by shared-memory reads, so the smaller
// tiles keep the 8 x 8 micro-tile and put the spare warps on other parts of k: 2 x 2 x 2 (128 x 64) and 1 x 2 x 4
// (64 x 64).  Their partial results meet in shared memory, in a fixed order, on the way to the output.
// Clusters: where even the 64 x 64 tiles are fewer than the SMs, the CTAs of a thread-block cluster share a tile's k
// range and fold their partial tiles through distributed shared memory: no workspace, no second launch.
#pragma once

#include "gather.cuh"
#include "screen_sample.cuh"

namespace cuasr_b200 {

constexpr int kTileM = 128;                       // the large tile; also the unit of the split-K scratch
constexpr int kTileN = 128;
constexpr int kTileKBytes = 128;                 // bytes of k per swizzled shared-memory row
constexpr int kConsumerWarps = 8;
constexpr int kProducerWarps = 4;                 // one warpgroup
constexpr int kConsumerThreads = kConsumerWarps * 32;
constexpr int kTmaThreads = (kConsumerWarps + kProducerWarps) * 32;
// Registers per thread after the warpgroups re-balance with setmaxnreg: 256 x 224 + 128 x 56 = the 64512 registers
// the CTA is launched with (384 x 168).
constexpr int kConsumerRegs = 224;
constexpr int kProducerRegs = 56;
constexpr int kEpilogueWarpBytes = 8192;          // per consumer warp: staging for coalesced output rows
constexpr int kMaxDestinations = 8;               // output copies one launch can write (this GPU + peers)
constexpr int kMaxSmemBytes = 232448;             // 227 KiB: what one CTA may have

// Tile shape of a kernel variant.  kRowsA / kRowsB: the operand lies along its rows and TMA brings it in as it lies.
template <int WM_, int WN_, int WK_, int kSub_ = WK_ == 4 ? 2 : 1, bool kGathers_ = true, bool kRowsA_ = false, bool kRowsB_ = false>
struct TileShape {
  static constexpr bool kRowsA = kRowsA_, kRowsB = kRowsB_;
  // Without the gather the producers need no more than 40 registers, and the consumers of the 128 x 128 tile get the 232
  // that hold their fragments and tables without spilling (see LargeTmaTile).
  static constexpr bool kGathers = kGathers_;
  static constexpr int kConsumerRegisters = kGathers ? kConsumerRegs : 232, kProducerRegisters = kGathers ? kProducerRegs : 40;
  static_assert(2 * kConsumerRegisters + kProducerRegisters <= 3 * 168, "the registers the CTA is launched with");
  static constexpr int WM = WM_, WN = WN_, WK = WK_;
  static_assert(WM * WN * WK == kConsumerWarps, "eight consumer warps");
  static constexpr int kM = 64 * WM, kN = 32 * WN;
  // 128-byte k columns per stage: two where the k range is shared by four warps, so that each warp gets four of the
  // 16-byte chunks of a stage (one unrolled pass of the contraction loop)
  static constexpr int kSub = kSub_;
  static constexpr int kABytes = kM * kTileKBytes * kSub;
  static constexpr int kBBytes = kN * kTileKBytes * kSub;
  static constexpr int kStageBytes = kABytes + kBBytes;
  // WK > 1: every warp's 64 x 32 partial block, for the fold; WK = 1: 8 KiB of staging per warp
  template <typename T>
  static constexpr int kFoldBytes = WK > 1 ? kConsumerWarps * 64 * 32 * (int)sizeof(T) : kConsumerWarps * kEpilogueWarpBytes;
  template <typename T>
  static constexpr int kStages = (kMaxSmemBytes - 1024 - 512 - kFoldBytes<T>) / kStageBytes;
  template <typename T>
  static constexpr int kSmemBytes = kStages<T> * kStageBytes + kFoldBytes<T> + 1024 /* alignment */ + 512 /* barriers */;
};
using LargeTile = TileShape<2, 4, 1>;    // 128 x 128
// The same where TMA brings in both operands.  With the gather compiled in (224 registers) the fp32 tropical contraction
// spills 64 bytes: 256 x 256 x 262144 split along K takes 1049 us with it and 1036 without, 8192^3 31.38 and 31.20 ms.
using LargeTmaTile = TileShape<2, 4, 1, 1, false>;
// The same with operands that lie along their rows, which TMA then brings in as they lie: a stage of such an operand is
// [k][128 rows], a 16-byte vector holds rows of one k.  Not for the rings that need pairs of k in a register
// (Ring::kPackedPairs), nor for fp64 products that are sums or products, which run as fast on gathered stages (see order_of).
// 4096^3, operand B along its rows, gathered and as it lies: max-min fp32 5975 and 5871 us, s32 min-plus 4130 and 4017, fp32 sums
// 3240 and 2935, fp64 max-min 17333 and 16581.
template <bool kRowsA, bool kRowsB>
using LargeRowsTile = TileShape<2, 4, 1, 1, false, kRowsA, kRowsB>;
using MediumTile = TileShape<2, 2, 2>;   // 128 x 64
using SmallTile = TileShape<1, 2, 4>;    // 64 x 64
// 64 x 32, one 16-byte chunk of k per warp and stage: the shortest chain for the smallest products, and the finest
// pieces of k for a cluster (fp64 sums take their chunks in fours, so their stage is four columns deep)
using TinyTile = TileShape<1, 1, 8>;
using TinyTileDeep = TileShape<1, 1, 8, 4>;

template <typename T>
struct TmaParams {
  int M, N, K;
  const T* A;  long long lda;   // gathered operands only
  const T* B;  long long ldb;
  int a_mode, b_mode;           // LoadMode
  T pad;                        // what a gather writes for k >= K ...
  int repeat_k;                 // ... unless it repeats the last k there: (+) is idempotent and there is no such value
  const T* C;  long long ldc;   // row-major; may alias D; may be null when !read_c
  T* D;        long long ldd;   // row-major
  // Extra copies of the output: when n_extra > 0 every element of D is also stored to extra_d[i] (same
  // leading dimension).  The pointers may be peer-GPU memory; this is how the sharded squaring step pushes
  // its block of the result into every rank's next-iteration matrix while the tile is still in registers.
  int n_extra;
  T* extra_d[kMaxDestinations - 1];
  T alpha, beta, add_identity;
  // start value of accumulators beyond the first of an element whose k range is shared (by warps, CTAs or pieces):
  // the additive identity where (+) is idempotent, the neutral 0 for sums and exclusive ors
  T part_identity;
  int read_c;
  int vector_epilogue;          // D, C and every extra_d are 16-byte aligned, ld * sizeof(T) % 16 == 0, N % EV == 0
  int tiles_m, tiles_n;
  unsigned int* status;         // device status word (see DeviceStatus)
  // Work decomposition.  Tiles [0, whole_tiles) are computed whole by one CTA each.  Every later tile is cut
  // along K into `slices` pieces: piece z handles K steps [z * k_tiles_per_slice, ...), the last piece takes the
  // rest.
  //  * cluster == 0 (large tile only): a piece writes its raw accumulators to partial +
  //    ((tile - whole_tiles) * slices + z) * 128 * 128.  tickets[tile - whole_tiles] counts the pieces written; the
  //    CTA that draws the last ticket folds the pieces in slice order and runs the epilogue, so nobody ever waits
  //    and the result does not depend on which CTA finishes last.  tickets must be zero at launch; the kernel leaves
  //    them zero.  Explicit split-K is whole_tiles = 0; a balanced launch splits only the tiles of the last wave.
  //  * cluster == 1 (WK > 1 only): whole_tiles = 0 and the `slices` CTAs of a cluster hold the pieces of one tile;
  //    CTA r of the cluster folds and writes the r-th part of the tile.
  int whole_tiles, slices, k_tiles_per_slice, cluster;
  int unless_screened;          // behind the screened kernel: the variant that asks
  T* partial;
  unsigned int* tickets;
};

// One 16-byte shared-memory load into EV = 16 / sizeof(T) elements.
__device__ __forceinline__ void lds16(uint32_t addr, float (&v)[4]) {
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(addr));
}
__device__ __forceinline__ void lds16(uint32_t addr, uint32_t (&v)[4]) {
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}
__device__ __forceinline__ void lds16(uint32_t addr, int32_t (&v)[4]) {
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr));
}
__device__ __forceinline__ void lds16(uint32_t addr, double (&v)[2]) {
  asm volatile("ld.shared.v2.f64 {%0,%1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(addr));
}
// The same from the shared memory of CTA `rank` of the cluster (own-CTA address).
__device__ __forceinline__ uint4 lds16_cluster(uint32_t addr, int rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  uint4 v;
  asm volatile("ld.shared::cluster.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void consumer_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kConsumerThreads) : "memory");
}

// Tile rasterisation: bands of kBand tile columns, rows fastest inside a band, so that the CTAs that
// run at the same time share A row-panels and B column-panels in L2.
constexpr int kBand = 16;
__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int& tm, int& tn) {
  const int per_band = kBand * tiles_m;
  const int band = t / per_band;
  const int in_band = t - band * per_band;
  const int width = min(kBand, tiles_n - band * kBand);
  tm = in_band / width;
  tn = band * kBand + in_band % width;
}

// Work item w of a launch -> (tile, K piece z, number of pieces of that tile).
template <typename T>
__device__ __forceinline__ void decode_work(const TmaParams<T>& p, int w, int num_tiles, int& tile, int& z, int& pieces) {
  if (p.cluster) {                       // the CTAs of a cluster are consecutive
    tile = w / p.slices; z = w - tile * p.slices; pieces = p.slices;
  } else if (w < p.whole_tiles) {
    tile = w; z = 0; pieces = 1;
  } else {
    const int tail = num_tiles - p.whole_tiles;
    const int v = w - p.whole_tiles;
    z = v / tail;
    tile = p.whole_tiles + (v - z * tail);
    pieces = p.slices;
  }
}

// Order of the 128 updates of a lane for one 16-byte chunk (two k) of 8-byte elements: column by column with k outside the
// rows or inside, by half tiles, or k outermost.  us at 4096^3 on 128 x 128 tiles / 1000^3 on 128 x 64 / 2048^3 on 64 x 64,
// both operands K-contiguous:
//   min-plus  by column 12255 / 258 / 1767, by element 12239 / 255 / 1689, by half 12390 / 237 / 1828, by k 12774 / 237 / 1977,
//             rows outside columns 13770 - 14360 / 242 - 273 / 1750 - 1860; with one operand gathered by column 12295, by element 13145;
//   max-min   by column 17500 / 323 / 2310, by half 17290 / 321 / 2233, by k 17315 / 322 / 2290; with operands along rows by k 16581
//             (one) and 16843 (both), by half 17192 and 16971.
enum UpdateOrder : int { kByColumn, kByElement, kByHalf, kByK };
template <typename RingT, typename Tile>
__host__ __device__ constexpr int order_of() {
  constexpr bool compares_only = RingT::kMul != CUASR_OP_PLUS && RingT::kMul != CUASR_OP_MULTIPLIES;
  if (Tile::WK == 1) return compares_only ? kByK : kByColumn;
  return compares_only || Tile::WK == 2 ? kByHalf : kByElement;
}

// kAsks: launched behind the screened kernel; returns at once where screen_helps says that that one has done the product.  A variant of
// its own, because code in front of it takes the fp64 contraction from 12.3 to 14.5 or 15.5 ms at 4096^3, and in the form that
// the registers of either ring come off best with: 3000^3 on signed data, both operands by TMA / one gathered, min-plus 5130 / 5312 us
// called and 5173 / 6260 inlined, max-plus 5192 / 6896 called and 5157 / 5160 inlined.
template <typename RingT, typename Tile, bool kAsks>
__global__ void __launch_bounds__(kTmaThreads, 1)
srgemm_tma_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ TmaParams<typename RingT::Element> p) {
  using T = typename RingT::Element;
  constexpr int WM = Tile::WM, WN = Tile::WN, WK = Tile::WK, kSub = Tile::kSub;
  constexpr bool kRowsA = Tile::kRowsA, kRowsB = Tile::kRowsB;
  constexpr bool kSums = RingT::kAdd == CUASR_OP_PLUS || RingT::kAdd == CUASR_OP_BIT_XOR;     // (+) is not idempotent
  static_assert(!(kRowsA || kRowsB) || (WK == 1 && kSub == 1 && !Tile::kGathers), "operands along rows: the large tile, by TMA");
  constexpr int kStages = Tile::template kStages<T>;
  static_assert(kStages >= 2, "at least double-buffered");
  constexpr int EV = 16 / sizeof(T);              // elements per 16-byte vector: 4 (fp32/int32) or 2 (fp64)
  constexpr int TK = kTileKBytes / sizeof(T);     // k per 128-byte column: 32 or 16
  constexpr int kStep = TK * kSub;                // k per stage
  constexpr int kChunks = 8 * kSub / WK;          // 16-byte k chunks of a stage that one warp works on

  if constexpr (kAsks) {
    static_assert(kTmaThreads == kSampleThreads, "the sample is spread over the CTA");
    grid_dependency_wait();
    const bool a_along_k = p.a_mode != kLoadGatherMN, b_along_k = p.b_mode != kLoadGatherMN;
    if constexpr (RingT::kAdd == CUASR_OP_MAXIMUM) {
      if (screen_helps<true>(p.A, p.lda, a_along_k, p.M, p.B, p.ldb, b_along_k, p.N, p.K)) return;
    } else {
      if (screen_helps_called<false>(p.A, p.lda, a_along_k, p.M, p.B, p.ldb, b_along_k, p.N, p.K)) return;
    }
  }

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi_smem = smem + kStages * Tile::kStageBytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(epi_smem + Tile::template kFoldBytes<T>);
  uint64_t* empty_bar = full_bar + kStages;
  unsigned int* ticket_smem = reinterpret_cast<unsigned int*>(empty_bar + kStages);
  volatile unsigned int* abandoned = ticket_smem + 1;     // raised when a consumer's wait ran out (see ptx.cuh)

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const bool a_tma = !Tile::kGathers || p.a_mode == kLoadTma, b_tma = !Tile::kGathers || p.b_mode == kLoadTma;
  const bool gathers = !a_tma || !b_tma, tmas = a_tma || b_tma;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], (tmas ? 1 : 0) + (gathers ? kProducerWarps * 32 : 0));
      mbar_init(&empty_bar[s], kConsumerWarps);
    }
    *abandoned = 0;
    fence_barrier_init();
  }
  __syncthreads();
  // Launched with programmatic stream serialisation: everything above overlaps the end of the kernel before this one;
  // nothing below touches global memory before that kernel's results are there.
  grid_dependency_wait();
  grid_dependency_launch();

  const int k_tiles_total = (p.K + kStep - 1) / kStep;
  const int num_tiles = p.tiles_m * p.tiles_n;
  const int num_work = p.whole_tiles + (num_tiles - p.whole_tiles) * p.slices;

  if (warp >= kConsumerWarps) {
    // ---------------------------------------------------------------- producers
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Tile::kProducerRegisters));
    const int pw = warp - kConsumerWarps;
    const bool issuer = pw == 0 && lane == 0;
    bool working = gathers || issuer;
    if (issuer && tmas) {
      prefetch_tensormap(&map_a);
      prefetch_tensormap(&map_b);
    }
    uint32_t it = 0;  // running K-step counter across all work items: stage = it % kStages
    for (int w = blockIdx.x; working && w < num_work; w += gridDim.x) {
      int tile, z, pieces, tm, tn;
      decode_work(p, w, num_tiles, tile, z, pieces);
      tile_coords(tile, p.tiles_m, p.tiles_n, tm, tn);
      const int m0 = tm * Tile::kM, n0 = tn * Tile::kN;
      const int kt_begin = pieces == 1 ? 0 : z * p.k_tiles_per_slice;
      const int kt_end = (z == pieces - 1) ? k_tiles_total : min(k_tiles_total, kt_begin + p.k_tiles_per_slice);
      for (int kt = kt_begin; kt < kt_end; ++kt, ++it) {
        const int s = it % kStages;
        const uint32_t round = it / kStages;
        if (round > 0 && !mbar_wait(&empty_bar[s], (round - 1) & 1, p.status, kDeviceTimeoutEmpty)) { working = false; break; }
        uint8_t* sa = smem + s * Tile::kStageBytes;
        uint8_t* sb = sa + Tile::kABytes;
        const int k0 = kt * kStep;
        if (issuer && tmas) {
          mbar_arrive_expect_tx(&full_bar[s], (a_tma ? Tile::kABytes : 0) + (b_tma ? Tile::kBBytes : 0));
#pragma unroll
          for (int sub = 0; sub < kSub; ++sub) {
            if (kRowsA)     tma_load_2d(sa, &map_a, &full_bar[s], m0, k0);
            else if (a_tma) tma_load_2d(sa + sub * (Tile::kM * 128), &map_a, &full_bar[s], k0 + sub * TK, m0);
            if (kRowsB)     tma_load_2d(sb, &map_b, &full_bar[s], n0, k0);
            else if (b_tma) tma_load_2d(sb + sub * (Tile::kN * 128), &map_b, &full_bar[s], k0 + sub * TK, n0);
          }
        }
        if (gathers) {
          if (!a_tma)
            gather_tile<T, Tile::kM, kSub>(smem_u32(sa), p.A, p.lda, p.a_mode, m0, p.M, k0, p.K, p.pad, p.repeat_k, pw, lane);
          if (!b_tma)
            gather_tile<T, Tile::kN, kSub>(smem_u32(sb), p.B, p.ldb, p.b_mode, n0, p.N, k0, p.K, p.pad, p.repeat_k, pw, lane);
          if (k0 + kStep > p.K) {         // padding was written by ordinary stores: announce with an ordinary arrival
            cp_async_wait_all();
            mbar_arrive(&full_bar[s]);
          } else {
            cp_async_arrive_noinc(&full_bar[s]);
          }
        }
      }
    }
    // every copy has landed before the thread goes away
    if (gathers) cp_async_wait_all();
    if (p.cluster) {                       // the two barriers of the consumers' fold are for all threads of the cluster
      __syncwarp();
      cluster_sync();
      cluster_sync();
    }
    return;
  }

  // ------------------------------------------------------------------ consumers
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Tile::kConsumerRegisters));
  const int wk = warp / (WM * WN), wm = (warp / WN) % WM, wn = warp % WN;
  const int lr = lane / 4, lc = lane % 4;        // 8 x 4 lanes
  // Row i (0..7) of this lane inside the warp's 64 rows; column j (0..7) inside the warp's 32 columns.
  // Plus-times fp64 runs on the tensor cores (DMMA): acc[mb][2 nb + e] is then element e of the lane's
  // accumulator pair of the 8 x 8 block (mb, nb) of the warp tile; its row inside the block is lr, its column
  // 2 lc + e.  Blocks fed from an operand along its rows are interleaved in pairs (see the loaders below).
  constexpr bool kDmma = std::is_same<T, double>::value && RingT::kAdd == CUASR_OP_PLUS &&
                         RingT::kMul == CUASR_OP_MULTIPLIES;
  auto row_of = [&](int i) {
    if (!kRowsA) return 8 * i + lr;
    return kDmma ? 16 * (i / 2) + 2 * lr + (i % 2) : EV * lr + (i % EV) + 8 * EV * (i / EV);
  };
  auto col_of = [&](int j) {
    if (kDmma) return kRowsB ? 16 * (j / 4) + 4 * lc + 2 * (j % 2) + ((j / 2) % 2) : 8 * (j / 2) + 2 * lc + (j % 2);
    return kRowsB ? EV * lc + (j % EV) + 4 * EV * (j / EV) : lc + 4 * j;
  };

  // Byte offset of this lane's first operand vector inside a stage; every other vector of the lane is a
  // compile-time constant away from it:  row * 128 + ((chunk ^ (row & 7)) * 16)
  //   A rows are lr + 8 i  -> + i * 1024 bytes, row & 7 == lr for every i
  //   B rows are lc + 4 j  -> + j * 512 bytes,  row & 7 == lc + 4 (j & 1)
  // An operand along its rows: k * (128 * sizeof(T)) + first row of the group * sizeof(T); the groups of EV rows are
  // 8 EV (A) or 4 EV (B) rows apart -> + g * 128 or + g * 64 bytes.
  // The warp's first chunk of a stage: column wk * kChunks / 8, chunk wk * kChunks % 8 of it.
  constexpr int kChunksPerColumn = 8;
  const int first_chunk = WK == 1 ? 0 : (wk * kChunks) % kChunksPerColumn;
  const int column = WK == 1 ? 0 : (wk * kChunks) / kChunksPerColumn;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t a_base = kRowsA ? (wm * 64 + EV * lr) * (int)sizeof(T) : column * (Tile::kM * 128) + (wm * 64 + lr) * 128;
  const uint32_t b_base = Tile::kABytes + (kRowsB ? (wn * 32 + EV * lc) * (int)sizeof(T) : column * (Tile::kN * 128) + (wn * 32 + lc) * 128);

  T acc[8][8];

  // Per-lane byte offsets of the 16-byte k chunks of an operand row, swizzle applied: computed once, so that inside
  // the contraction an operand vector is addressed as (stage base + one of these + a constant).
  // Only for 4-byte elements: with 8-byte elements the accumulators leave no registers for the table, and the
  // offsets are computed where they are used.
  constexpr bool kOffsetTable = sizeof(T) == 4;
  // Chunks unrolled in the contraction loop; the table holds the offsets of that many chunks.  Chunk c + kUnroll of a
  // stage differs in bit 6 of the offset (bit 2 of the chunk index), and so do the B rows of odd j.  That bit is the same
  // for all entries of a lane's table, so the flip is an addition of 64 or -64 that goes into the stage's base once:
  // 4096^3 max-min 5952 -> 5920 us.  The packed rings with the gather compiled in have no registers for it (4096^3
  // min-plus, one operand gathered: 3998 -> 4090 us) and flip the bit of each offset.
  constexpr bool kFlipBase = !Tile::kGathers || !RingT::kPackedPairs;
  // (four chunks keep the loop body near 16 KiB of instructions; unrolling all eight measured the same on min-plus
  // and 25 % slower on max-min, whose body is half as large again)
  constexpr int kUnroll = kChunks < 4 ? kChunks : 4;
  uint32_t a_off[kOffsetTable ? kUnroll : 1], b_off[kOffsetTable ? kUnroll : 1];
  const int a_flip = ((first_chunk ^ lr) & 4) ? -64 : 64, b_flip = ((first_chunk ^ lc) & 4) ? -64 : 64;
  if constexpr (kOffsetTable) {
#pragma unroll
    for (int c = 0; c < kUnroll; ++c) {
      a_off[c] = a_base + ((((c + first_chunk) ^ lr) & 7) << 4);
      b_off[c] = b_base + ((((c + first_chunk) ^ lc) & 7) << 4);       // rows lc + 4 j with even j
    }
  }

  uint32_t it = 0;
  for (int w = blockIdx.x; w < num_work; w += gridDim.x) {
    int tile, z, pieces, tm, tn;
    decode_work(p, w, num_tiles, tile, z, pieces);
    tile_coords(tile, p.tiles_m, p.tiles_n, tm, tn);
    const int kt_begin = pieces == 1 ? 0 : z * p.k_tiles_per_slice;
    const int kt_end = (z == pieces - 1) ? k_tiles_total : min(k_tiles_total, kt_begin + p.k_tiles_per_slice);

    // The two are the same for an idempotent (+).  Not choosing brings max-min fp32 4096^3 from 5913 to 5877 us; the packed rings (512^3
    // 16.15 -> 16.36 us) and fp64 have better registers with the choice.
    T start = p.add_identity;
    if constexpr (kSums || sizeof(T) == 8 || RingT::kPackedPairs) start = (wk == 0 && z == 0) ? p.add_identity : p.part_identity;
    if constexpr (RingT::kLogical) start = static_cast<T>(start != T(0));      // as the first product makes it
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = start;

    for (int kt = kt_begin; kt < kt_end; ++kt, ++it) {
      const int s = it % kStages;
      mbar_wait_or_abandon(&full_bar[s], (it / kStages) & 1, p.status, kDeviceTimeoutFull, abandoned);
      const uint32_t st = smem_base + s * Tile::kStageBytes;

      // fragment loaders for one 16-byte k chunk: a[i][e] = A(row i, k = chunk * EV + e).  With the offset table the
      // chunk is given as (c, h): chunk = h * kUnroll + c with c a compile-time constant; without it h is 0.
      auto load_a = [&](T (&a)[8][EV], int c, int h = 0) {
        if constexpr (kRowsA) {
          const uint32_t base = st + a_base + (kOffsetTable ? h * kUnroll + c : c) * (EV * Tile::kM * (int)sizeof(T));
#pragma unroll
          for (int e = 0; e < EV; ++e)
#pragma unroll
            for (int g = 0; g < 8 / EV; ++g) {
              T v[EV];
              lds16(base + e * (Tile::kM * (int)sizeof(T)) + g * 128, v);
#pragma unroll
              for (int t = 0; t < EV; ++t) a[g * EV + t][e] = v[t];
            }
          return;
        }
        uint32_t base;
        if constexpr (kOffsetTable) base = kFlipBase ? st + h * a_flip + a_off[c] : st + (a_off[c] ^ (h << 6));
        else base = st + a_base + ((((c + first_chunk) ^ lr) & 7) << 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) lds16(base + i * 1024, a[i]);
      };
      auto load_b = [&](T (&b)[8][EV], int c, int h = 0) {
        if constexpr (kRowsB) {
          const uint32_t base = st + b_base + (kOffsetTable ? h * kUnroll + c : c) * (EV * Tile::kN * (int)sizeof(T));
#pragma unroll
          for (int e = 0; e < EV; ++e)
#pragma unroll
            for (int g = 0; g < 8 / EV; ++g) {
              T v[EV];
              lds16(base + e * (Tile::kN * (int)sizeof(T)) + g * 64, v);
#pragma unroll
              for (int t = 0; t < EV; ++t) b[g * EV + t][e] = v[t];
            }
          return;
        }
        uint32_t base0, base1;
        if constexpr (kOffsetTable) {
          base0 = kFlipBase ? st + h * b_flip + b_off[c] : st + (b_off[c] ^ (h << 6));
          base1 = kFlipBase ? st + (1 - h) * b_flip + b_off[c] : st + (b_off[c] ^ ((h << 6) ^ 64));
        } else {
          base0 = st + b_base + ((((c + first_chunk) ^ lc) & 7) << 4);
          base1 = st + b_base + ((((c + first_chunk) ^ (lc + 4)) & 7) << 4);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) lds16(((j & 1) ? base1 : base0) + j * 512, b[j]);
      };
      auto compute = [&](const T (&a)[8][EV], const T (&b)[8][EV]) {
        if constexpr (RingT::kPackedPairs) {
          // both fragments came from 16-byte loads along k: (k, k+1) are adjacent registers, so the pairs below
          // are register renames, not moves
#pragma unroll
          for (int e = 0; e < EV; e += 2) {
            uint64_t pa[8], pb[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) { pa[i] = pack2(a[i][e], a[i][e + 1]); pb[i] = pack2(b[i][e], b[i][e + 1]); }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
              for (int j = 0; j < 8; ++j) acc[i][j] = RingT::mac_packed(acc[i][j], pa[i], pb[j]);
          }
          return;
        }
        if constexpr (RingT::kLogical) {
#pragma unroll
          for (int e = 0; e < EV; ++e) {
            uint32_t ma[8], mb[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) { ma[i] = RingT::mask(a[i][e]); mb[i] = RingT::mask(b[i][e]); }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
              for (int j = 0; j < 8; ++j) acc[i][j] = RingT::or_mask(acc[i][j], ma[i] & mb[j]);
          }
          return;
        }
        if constexpr (sizeof(T) == 8) {
          // An instruction's operands have to come from both register banks, so the rate depends on the order of the updates,
          // which the compiler's register assignment follows (see order_of).
#pragma unroll
          for (int x = 0; x < 128; ++x) {
            constexpr int kOrder = order_of<RingT, Tile>();
            const int e = kOrder == kByColumn ? (x / 8) % 2 : kOrder == kByElement ? x % 2 : x / 64;
            const int i = kOrder == kByHalf ? (x / 32) % 2 * 4 + x % 4 : kOrder == kByElement ? (x / 2) % 8 : x % 8;
            const int j = kOrder == kByHalf ? (x / 4) % 8 : kOrder == kByK ? (x / 8) % 8 : x / 16;
            acc[i][j] = RingT::add(RingT::mul(a[i][e], b[j][e]), acc[i][j]);
          }
          return;
        }
#pragma unroll
        for (int e = 0; e < EV; e += 2)
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j)
              acc[i][j] = RingT::mac2(acc[i][j], a[i][e], b[j][e], a[i][e + 1], b[j][e + 1]);
      };

      if constexpr (kDmma) {
        // Tensor-core path.  The fp64 mma takes, per lane, A(row lr [+8], k slot lc [+4]) and B(k slot lc [+4], column lr).
        // The contraction index may be permuted freely as long as A and B agree: within a group of 8 k (four
        // chunks) the slot lc of step s (s = 0, 1) stands for k = 2 lc + s, so one 16-byte load delivers both steps
        // of a block.  An operand along its rows delivers two adjacent rows with one 16-byte load; they feed the two
        // blocks of an interleaved pair (block rows 2 lr and 2 lr + 1).
        constexpr int kGroups = kChunks / 4;
        static_assert(kGroups == 1 || kGroups == 2, "one or two groups of 8 k per warp and stage");
        auto load_group = [&](double (&a)[8][2], double (&b)[4][2], int group) {
          const uint32_t chunk = ((((group * 4 + first_chunk + lc) ^ lr) & 7) << 4);
          if constexpr (kRowsA) {
#pragma unroll
            for (int step = 0; step < 2; ++step)
#pragma unroll
              for (int pair = 0; pair < 4; ++pair) {
                double v[2];
                lds16(st + (group * 8 + 2 * lc + step) * (Tile::kM * 8) + (wm * 64 + 2 * lr) * 8 + pair * 128, v);
                a[2 * pair][step] = v[0];
                a[2 * pair + 1][step] = v[1];
              }
          } else {
            const uint32_t abase = st + a_base + chunk;
#pragma unroll
            for (int mb = 0; mb < 8; ++mb) lds16(abase + mb * 1024, a[mb]);
          }
          // B rows (columns of the product) of this path are lr + 8 nb
          if constexpr (kRowsB) {
#pragma unroll
            for (int step = 0; step < 2; ++step)
#pragma unroll
              for (int pair = 0; pair < 2; ++pair) {
                double v[2];
                lds16(st + Tile::kABytes + (group * 8 + 2 * lc + step) * (Tile::kN * 8) + (wn * 32 + 2 * lr) * 8 + pair * 128, v);
                b[2 * pair][step] = v[0];
                b[2 * pair + 1][step] = v[1];
              }
          } else {
            const uint32_t bbase = st + Tile::kABytes + column * (Tile::kN * 128) + (wn * 32 + lr) * 128 + chunk;
#pragma unroll
            for (int nb = 0; nb < 4; ++nb) lds16(bbase + nb * 1024, b[nb]);
          }
        };
        auto mma_group = [&](const double (&a)[8][2], const double (&b)[4][2]) {
          // m16n8k8: rows lr and lr + 8 of the instruction are the two 8-row blocks 2 h and 2 h + 1, k slots lc and
          // lc + 4 are the two steps of this group
#pragma unroll
          for (int h = 0; h < 4; ++h)
#pragma unroll
            for (int nb = 0; nb < 4; ++nb)
              asm volatile(
                  "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                  "{%0, %1, %2, %3};"
                  : "+d"(acc[2 * h][2 * nb]), "+d"(acc[2 * h][2 * nb + 1]), "+d"(acc[2 * h + 1][2 * nb]),
                    "+d"(acc[2 * h + 1][2 * nb + 1])
                  : "d"(a[2 * h][0]), "d"(a[2 * h + 1][0]), "d"(a[2 * h][1]), "d"(a[2 * h + 1][1]), "d"(b[nb][0]),
                    "d"(b[nb][1]));
        };
        double a0[8][2], b0[4][2], a1[8][2], b1[4][2];
        load_group(a0, b0, 0);
        if constexpr (kGroups == 2) load_group(a1, b1, 1);
        mma_group(a0, b0);
        if constexpr (kGroups == 2) mma_group(a1, b1);
      } else if constexpr (sizeof(T) == 4) {
        // 4-byte elements: operand fragments are double-buffered in registers (64 + 4 x 32 registers)
        T a0[8][EV], b0[8][EV], a1[8][EV], b1[8][EV];
        load_a(a0, 0, 0);
        load_b(b0, 0, 0);
        if constexpr (kChunks == 1) {
          compute(a0, b0);
        } else {
          // kUnroll chunks at a time with compile-time chunk indices, so that the only integer work left per chunk is
          // combining the stage base with a table entry (integer instructions share the half-rate pipe with the
          // three-input min: each one costs as much as a product pair)
#pragma unroll 1
          for (int h = 0; h < kChunks / kUnroll; ++h) {
#pragma unroll
            for (int c = 0; c < kUnroll; c += 2) {
              load_a(a1, c + 1, h);
              load_b(b1, c + 1, h);
              compute(a0, b0);
              if (c + 2 < kUnroll) {
                load_a(a0, c + 2, h);
                load_b(b0, c + 2, h);
              } else if (h + 1 < kChunks / kUnroll) {
                load_a(a0, 0, h + 1);
                load_b(b0, 0, h + 1);
              }
              compute(a1, b1);
            }
          }
        }
      } else {
        // 8-byte elements: the 8 x 8 accumulators alone take 128 registers, so one fragment set is live
        T a0[8][EV], b0[8][EV];
#pragma unroll 1
        for (int chunk = 0; chunk < kChunks; ++chunk) {
          load_a(a0, chunk);
          load_b(b0, chunk);
          compute(a0, b0);
        }
      }
      // Release the stage only after the math that consumed its last fragments: every value loaded from it is
      // then in registers for certain (a release placed right after the loads leaves the compiler free to sink
      // not-yet-needed loads below it, and the refill would race with them).
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_bar[s]);
    }

    // ---------------------------------------------------------------- epilogue
    // 16 bytes of an output row: C is read, the epilogue applied and the vector stored to D and to every extra copy;
    // element by element where the row is not 16-byte aligned or the vector crosses N.
    auto store_vector = [&](T (&v)[EV], int m, int n) {
      if (m >= p.M || n >= p.N) return;
#pragma unroll
      for (int e = 0; e < EV; ++e) v[e] = RingT::mul(p.alpha, v[e]);
      const long long off = (long long)m * p.ldd + n;
      if (p.vector_epilogue) {
        if (p.read_c) {
          alignas(16) T c[EV];
          *reinterpret_cast<uint4*>(c) = *reinterpret_cast<const uint4*>(p.C + (long long)m * p.ldc + n);
#pragma unroll
          for (int e = 0; e < EV; ++e) v[e] = RingT::add(v[e], RingT::mul(p.beta, c[e]));
        }
        *reinterpret_cast<uint4*>(p.D + off) = *reinterpret_cast<const uint4*>(v);
        for (int x = 0; x < p.n_extra; ++x) *reinterpret_cast<uint4*>(p.extra_d[x] + off) = *reinterpret_cast<const uint4*>(v);
      } else {
        T c[EV];
        if (p.read_c) {
#pragma unroll
          for (int e = 0; e < EV; ++e) c[e] = n + e < p.N ? p.C[(long long)m * p.ldc + n + e] : p.add_identity;
        }
#pragma unroll
        for (int e = 0; e < EV; ++e) {
          if (p.read_c) v[e] = RingT::add(v[e], RingT::mul(p.beta, c[e]));
          if (n + e < p.N) {
            p.D[off + e] = v[e];
            for (int x = 0; x < p.n_extra; ++x) p.extra_d[x][off + e] = v[e];
          }
        }
      }
    };

    if constexpr (WK > 1) {
      // Every warp leaves its block in shared memory ([wk][row][column], the 16-byte column groups XOR-swizzled by
      // row & 7); then the 256 threads fold the WK partial values of an output vector in k-group order and store it,
      // one vector per thread at a time.
      constexpr int kRowGroups = Tile::kN / EV;                      // 16-byte groups per tile row
      constexpr int kVectors = Tile::kM * kRowGroups;
      T* fold = reinterpret_cast<T*>(epi_smem);
      consumer_sync();                                               // the previous tile's fold has been read
      {
        T* mine = fold + wk * (Tile::kM * Tile::kN);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = wm * 64 + row_of(i);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int c = wn * 32 + col_of(j);
            mine[r * Tile::kN + (((c / EV) ^ (r & 7)) * EV) + (c % EV)] = acc[i][j];
          }
        }
      }
      consumer_sync();
      auto folded = [&](int r, int g, T (&v)[EV]) {
        const int at = r * Tile::kN + ((g ^ (r & 7)) * EV);
        *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(fold + at);
#pragma unroll
        for (int q = 1; q < WK; ++q) {
          alignas(16) T t[EV];
          *reinterpret_cast<uint4*>(t) = *reinterpret_cast<const uint4*>(fold + q * (Tile::kM * Tile::kN) + at);
#pragma unroll
          for (int e = 0; e < EV; ++e) v[e] = RingT::add(t[e], v[e]);
        }
        return at;
      };
      if (!p.cluster) {
#pragma unroll 4
        for (int idx = threadIdx.x; idx < kVectors; idx += kConsumerThreads) {
          const int r = idx / kRowGroups, g = idx % kRowGroups;
          alignas(16) T v[EV];
          folded(r, g, v);
          store_vector(v, tm * Tile::kM + r, tn * Tile::kN + g * EV);
        }
      } else {
        // fold this CTA's k groups into block 0, then the cluster's blocks, CTA by CTA in k order; CTA z of the cluster
        // finishes the z-th part of the tile.  The hardware barriers also keep every CTA's memory in place until
        // all of them have read it.
#pragma unroll 4
        for (int idx = threadIdx.x; idx < kVectors; idx += kConsumerThreads) {
          const int r = idx / kRowGroups, g = idx % kRowGroups;
          alignas(16) T v[EV];
          const int at = folded(r, g, v);
          *reinterpret_cast<uint4*>(fold + at) = *reinterpret_cast<const uint4*>(v);
        }
        cluster_sync();
        const int share = kVectors / p.slices;
        for (int idx = z * share + threadIdx.x; idx < (z + 1) * share; idx += kConsumerThreads) {
          const int r = idx / kRowGroups, g = idx % kRowGroups;
          const uint32_t at = smem_u32(fold + r * Tile::kN + ((g ^ (r & 7)) * EV));
          alignas(16) T v[EV];
          *reinterpret_cast<uint4*>(v) = lds16_cluster(at, 0);
          for (int q = 1; q < p.slices; ++q) {
            alignas(16) T t[EV];
            *reinterpret_cast<uint4*>(t) = lds16_cluster(at, q);
#pragma unroll
            for (int e = 0; e < EV; ++e) v[e] = RingT::add(t[e], v[e]);
          }
          store_vector(v, tm * Tile::kM + r, tn * Tile::kN + g * EV);
        }
        cluster_sync();
      }
    } else {
      const int m_base = tm * Tile::kM + wm * 64, n_base = tn * Tile::kN + wn * 32;
      if (pieces > 1) {
        // A piece of a split tile: park the raw accumulators in the tile's scratch block, in "fragment order"
        // ([16 vectors][256 consumer threads][16 bytes], so that every access is a coalesced 16-byte vector and the
        // thread that folds reads exactly the layout it would have written), then take a ticket.
        constexpr int kVecPerThread = 64 / EV;
        const int split = tile - p.whole_tiles;                     // index among the split tiles
        T* block = p.partial + (long long)split * pieces * (kTileM * kTileN);
        uint4* mine = reinterpret_cast<uint4*>(block + (long long)z * (kTileM * kTileN)) + threadIdx.x;
#pragma unroll
        for (int v = 0; v < kVecPerThread; ++v) {
          alignas(16) T tmp[EV];
#pragma unroll
          for (int e = 0; e < EV; ++e) tmp[e] = acc[(v * EV + e) / 8][(v * EV + e) % 8];
          mine[v * kConsumerThreads] = *reinterpret_cast<const uint4*>(tmp);
        }
        __threadfence();
        consumer_sync();
        if (threadIdx.x == 0) *ticket_smem = atomicAdd(&p.tickets[split], 1u);
        consumer_sync();
        const bool last = (*ticket_smem == (unsigned)pieces - 1);
        consumer_sync();
        if (!last) continue;
        // This CTA completed the tile: fold all pieces in slice order (a fixed order, whoever comes last), then
        // fall through to the ordinary epilogue with the folded accumulators.  An idempotent (+) folds them onto this
        // CTA's own piece, which is one of them; sums start over.  (A test for the first piece inside the fold costs the
        // fp64 contraction, which needs every register, 76 bytes of spills.)
        __threadfence();
        if (threadIdx.x == 0) p.tickets[split] = 0;
        if constexpr (kSums) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = T(0);
        }
        for (int zz = 0; zz < pieces; ++zz) {
          const uint4* theirs = reinterpret_cast<const uint4*>(block + (long long)zz * (kTileM * kTileN)) + threadIdx.x;
          uint4 raw[kVecPerThread];
#pragma unroll
          for (int v = 0; v < kVecPerThread; ++v) raw[v] = __ldcg(theirs + v * kConsumerThreads);
#pragma unroll
          for (int v = 0; v < kVecPerThread; ++v) {
            alignas(16) T tmp[EV];
            *reinterpret_cast<uint4*>(tmp) = raw[v];
#pragma unroll
            for (int e = 0; e < EV; ++e) {
              T& a = acc[(v * EV + e) / 8][(v * EV + e) % 8];
              a = RingT::add(tmp[e], a);
            }
          }
        }
      }
      // The warp's 64 x 32 block goes through its private staging area (rows of 32 elements, the 16-byte column
      // groups XOR-swizzled by row & 7), then every lane handles 16 bytes of a row.
      constexpr int kRowsPerPass = kEpilogueWarpBytes / (32 * (int)sizeof(T));   // 64 (4-byte) or 32 (8-byte)
      constexpr int kGroups = 32 / EV;                                            // 16-byte groups per row
      T* stage = reinterpret_cast<T*>(epi_smem + warp * kEpilogueWarpBytes);
#pragma unroll
      for (int pass = 0; pass < 64 / kRowsPerPass; ++pass) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = row_of(i) - pass * kRowsPerPass;
          if (r < 0 || r >= kRowsPerPass) continue;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int c = col_of(j);
            const int group = ((c / EV) ^ (r & 7)) & (kGroups - 1);
            stage[r * 32 + group * EV + (c % EV)] = acc[i][j];
          }
        }
        __syncwarp();
        if constexpr (kDmma) {
          // C may be D, so a load of C after a store to D cannot be moved in front of it: one by one, the 32 vectors of a
          // lane are as many memory latencies in a row.  Here they are loaded four at a time (every element is read and
          // written by one thread only): 1500^3 230 -> 219 us, 4096^3 3991 -> 3901.  The rings with more registers in
          // use lose as much in the contraction as they gain (8192^3 min-plus 31.2 -> 31.9 ms).
          if (p.vector_epilogue && p.read_c) {
            constexpr int kBatch = 4;
#pragma unroll 1
            for (int at = lane; at < kRowsPerPass * kGroups; at += kBatch * 32) {
              alignas(16) T c[kBatch][EV];
#pragma unroll
              for (int u = 0; u < kBatch; ++u) {
                const int m = m_base + pass * kRowsPerPass + (at + u * 32) / kGroups, n = n_base + (at + u * 32) % kGroups * EV;
                if (m < p.M && n < p.N)
                  *reinterpret_cast<uint4*>(c[u]) = *reinterpret_cast<const uint4*>(p.C + (long long)m * p.ldc + n);
              }
#pragma unroll
              for (int u = 0; u < kBatch; ++u) {
                const int r = (at + u * 32) / kGroups, g = (at + u * 32) % kGroups;
                const int m = m_base + pass * kRowsPerPass + r, n = n_base + g * EV;
                if (m >= p.M || n >= p.N) continue;
                alignas(16) T v[EV];
                *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(stage + r * 32 + ((g ^ (r & 7)) & (kGroups - 1)) * EV);
#pragma unroll
                for (int e = 0; e < EV; ++e) v[e] = RingT::add(RingT::mul(p.alpha, v[e]), RingT::mul(p.beta, c[u][e]));
                const long long off = (long long)m * p.ldd + n;
                *reinterpret_cast<uint4*>(p.D + off) = *reinterpret_cast<const uint4*>(v);
                for (int x = 0; x < p.n_extra; ++x) *reinterpret_cast<uint4*>(p.extra_d[x] + off) = *reinterpret_cast<const uint4*>(v);
              }
            }
            continue;
          }
        }
#pragma unroll 4
        for (int idx = lane; idx < kRowsPerPass * kGroups; idx += 32) {
          const int r = idx / kGroups, g = idx % kGroups;
          const int group = (g ^ (r & 7)) & (kGroups - 1);
          alignas(16) T v[EV];
          *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(stage + r * 32 + group * EV);
          store_vector(v, m_base + pass * kRowsPerPass + r, n_base + g * EV);
        }
      }
    }
  }
}

}  // namespace cuasr_b200
