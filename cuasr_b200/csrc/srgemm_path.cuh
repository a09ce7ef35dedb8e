// Path-tracking tropical SRGEMM: dist <- min/max(dist, A (x) B) in place, and for every element that improved the first
// contraction index k that attains its new value (parent).
//
// Device counterpart of the reference's legacy CPU routine cpu_fwgemm_naive
// (test/regress/include/fwgpu/cpu_srgemm.hpp:20-48): "strictly better, first such k; untouched when nothing improved".
//
// The staging and the contraction are srgemm_tma_kernel's (any layout and alignment, packed adds and three-input
// minima); the accumulators start from dist, and nothing per product is spent on the index.  After every stage (32 or
// 64 k) each lane compares its accumulators with what they were before it, kept in shared memory, and notes the elements
// that changed in a 64-bit mask: 2 instructions per element and stage.  One pass per noted element then finds the k:
// it reads the operand rows again from the stage, which is still there, and takes the first sum that equals the new
// value.  The n-th product of random data is a new minimum with probability 1/n, so late stages note next to nothing.
// With a test every four k and an index per improvement among those, 2048^3 from +inf took 1.69 ms and 0.96 once nothing
// improves; now 1.36 and 0.65 (the plain product: 0.52).
// Tiles: 128 x 128 with whole k ranges per warp (the index then goes straight to `parent`: a lane meets its k in
// ascending order), and for outputs too small to fill the GPU with those, 64 x 64 (fp32) or 64 x 32 (fp64, whose partial
// values leave no room for a pipeline beside the larger one) with the k range shared by four or eight warps and, beyond
// that, by the CTAs of a cluster; their (value, k) candidates meet in shared memory, the smaller k
// winning ties.  On the fp64 one the index follows every product (improve below): 1000^3 from +inf 757 us on the large tile, 370.
#pragma once

#include "srgemm_tma.cuh"

namespace cuasr_b200 {

template <typename T>
struct PathParams {
  int M, N, K;
  const T* A;  long long lda;   // gathered operands only
  const T* B;  long long ldb;
  int a_mode, b_mode;           // LoadMode
  T pad;                        // what a gather writes for k >= K: NaN, which never improves anything
  T* dist;          long long ldd;          // row-major, read and written
  int32_t* parent;  long long ld_parent;    // row-major, written where an element improves
  int k_offset;                             // added to every recorded k
  int tiles_m, tiles_n;
  int cluster, k_tiles_per_slice;           // CTAs that share a tile's k range (64 x 64 tiles), K steps of each
  unsigned int* status;
};

// Shared memory: stages, the accumulators of the stage before (later the partial values of the fold), and where the
// k range is shared the k of every partial value.
template <typename T, typename Tile>
constexpr int kPathKeptBytes = kConsumerThreads * 64 * (int)sizeof(T);
template <typename Tile>
constexpr int kPathIndexBytes = Tile::WK > 1 ? kConsumerThreads * 64 * 4 : 0;
template <typename T, typename Tile>
constexpr int kPathStages = (kMaxSmemBytes - 1024 - 512 - kPathKeptBytes<T, Tile> - kPathIndexBytes<Tile>) / Tile::kStageBytes;
template <typename T, typename Tile>
constexpr int kPathSmemBytes = kPathStages<T, Tile> * Tile::kStageBytes + kPathKeptBytes<T, Tile> + kPathIndexBytes<Tile> + 1024 + 512;

__device__ __forceinline__ void ld_cluster(uint32_t addr, int rank, float& v) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
}
__device__ __forceinline__ void ld_cluster(uint32_t addr, int rank, double& v) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote) : "memory");
}
__device__ __forceinline__ uint32_t ld4_cluster(uint32_t addr, int rank) {
  uint32_t remote, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.b32 %0, [%1];" : "=r"(v) : "r"(remote) : "memory");
  return v;
}

// If t is better than acc: acc = t, and k to the element's word of shared memory.  Five instructions per product where the product
// alone takes four, but no test and no look-up per stage: for the fp64 tile whose warps have two k of a stage, where a test costs a
// quarter of the products and, from a cold start, some lane has an element to look up in nearly every stage.
template <bool kMaximize>
__device__ __forceinline__ void improve(double& acc, double t, uint32_t word, int k) {
  if (kMaximize)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.f64 p, %1, %0;\n\t@p st.shared.b32 [%2], %3;\n\tselp.f64 %0, %1, %0, p;\n\t}"
                 : "+d"(acc) : "d"(t), "r"(word), "r"(k) : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.f64 p, %1, %0;\n\t@p st.shared.b32 [%2], %3;\n\tselp.f64 %0, %1, %0, p;\n\t}"
                 : "+d"(acc) : "d"(t), "r"(word), "r"(k) : "memory");
}

template <typename T, bool kMaximize, typename Tile>
__global__ void __launch_bounds__(kTmaThreads, 1)
srgemm_path_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                   const __grid_constant__ PathParams<T> p) {
  using R = Ring<kMaximize ? CUASR_OP_MAXIMUM : CUASR_OP_MINIMUM, CUASR_OP_PLUS, T>;
  constexpr int WM = Tile::WM, WN = Tile::WN, WK = Tile::WK, kSub = Tile::kSub;
  constexpr int kStages = kPathStages<T, Tile>;
  static_assert(kStages >= 2, "at least double-buffered");
  constexpr int EV = 16 / (int)sizeof(T);
  constexpr int TK = kTileKBytes / (int)sizeof(T);
  constexpr int kStep = TK * kSub;
  constexpr int kChunks = 8 * kSub / WK;          // 16-byte k chunks of a stage that one warp works on
  constexpr bool kDirect = sizeof(T) == 8 && WK > 1;    // the index follows every product (see improve)
  auto better = [](T candidate, T current) { return kMaximize ? candidate > current : candidate < current; };

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* kept_smem = smem + kStages * Tile::kStageBytes;
  uint8_t* index_smem = kept_smem + kPathKeptBytes<T, Tile>;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(index_smem + kPathIndexBytes<Tile>);
  uint64_t* empty_bar = full_bar + kStages;
  volatile unsigned int* abandoned = reinterpret_cast<unsigned int*>(empty_bar + kStages);   // see ptx.cuh

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const bool gathers = p.a_mode != kLoadTma || p.b_mode != kLoadTma;
  const bool tmas = p.a_mode == kLoadTma || p.b_mode == kLoadTma;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], (tmas ? 1 : 0) + (gathers ? kProducerWarps * 32 : 0));
      mbar_init(&empty_bar[s], kConsumerWarps);
    }
    *abandoned = 0;
    fence_barrier_init();
  }
  __syncthreads();
  grid_dependency_wait();
  grid_dependency_launch();

  const int k_tiles_total = (p.K + kStep - 1) / kStep;
  const int num_work = p.tiles_m * p.tiles_n * p.cluster;
  // the CTAs of a cluster are consecutive and hold consecutive parts of a tile's k range
  auto decode = [&](int w, int& tm, int& tn, int& z, int& kt_begin, int& kt_end) {
    const int tile = w / p.cluster;
    z = w - tile * p.cluster;
    tile_coords(tile, p.tiles_m, p.tiles_n, tm, tn);
    kt_begin = p.cluster == 1 ? 0 : z * p.k_tiles_per_slice;
    kt_end = z == p.cluster - 1 ? k_tiles_total : min(k_tiles_total, kt_begin + p.k_tiles_per_slice);
  };

  if (warp >= kConsumerWarps) {
    // ---------------------------------------------------------------- producers
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kProducerRegs));
    const int pw = warp - kConsumerWarps;
    const bool issuer = pw == 0 && lane == 0;
    bool working = gathers || issuer;
    if (issuer && tmas) {
      prefetch_tensormap(&map_a);
      prefetch_tensormap(&map_b);
    }
    uint32_t it = 0;
    for (int w = blockIdx.x; working && w < num_work; w += gridDim.x) {
      int tm, tn, z, kt_begin, kt_end;
      decode(w, tm, tn, z, kt_begin, kt_end);
      const int m0 = tm * Tile::kM, n0 = tn * Tile::kN;
      for (int kt = kt_begin; kt < kt_end; ++kt, ++it) {
        const int s = it % kStages;
        const uint32_t round = it / kStages;
        if (round > 0 && !mbar_wait(&empty_bar[s], (round - 1) & 1, p.status, kDeviceTimeoutEmpty)) { working = false; break; }
        uint8_t* sa = smem + s * Tile::kStageBytes;
        uint8_t* sb = sa + Tile::kABytes;
        const int k0 = kt * kStep;
        if (issuer && tmas) {
          mbar_arrive_expect_tx(&full_bar[s], (p.a_mode == kLoadTma ? Tile::kABytes : 0) + (p.b_mode == kLoadTma ? Tile::kBBytes : 0));
#pragma unroll
          for (int sub = 0; sub < kSub; ++sub) {
            if (p.a_mode == kLoadTma) tma_load_2d(sa + sub * (Tile::kM * 128), &map_a, &full_bar[s], k0 + sub * TK, m0);
            if (p.b_mode == kLoadTma) tma_load_2d(sb + sub * (Tile::kN * 128), &map_b, &full_bar[s], k0 + sub * TK, n0);
          }
        }
        if (gathers) {
          if (p.a_mode != kLoadTma)
            gather_tile<T, Tile::kM, kSub>(smem_u32(sa), p.A, p.lda, p.a_mode, m0, p.M, k0, p.K, p.pad, false, pw, lane);
          if (p.b_mode != kLoadTma)
            gather_tile<T, Tile::kN, kSub>(smem_u32(sb), p.B, p.ldb, p.b_mode, n0, p.N, k0, p.K, p.pad, false, pw, lane);
          if (k0 + kStep > p.K) {
            cp_async_wait_all();
            mbar_arrive(&full_bar[s]);
          } else {
            cp_async_arrive_noinc(&full_bar[s]);
          }
        }
      }
    }
    if (gathers) cp_async_wait_all();
    if (p.cluster > 1) {
      __syncwarp();
      cluster_sync();
      cluster_sync();
    }
    return;
  }

  // ------------------------------------------------------------------ consumers
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kConsumerRegs));
  const int wk = warp / (WM * WN), wm = (warp / WN) % WM, wn = warp % WN;
  const int lr = lane / 4, lc = lane % 4;
  constexpr int kChunksPerColumn = 8;
  const int first_chunk = WK == 1 ? 0 : (wk * kChunks) % kChunksPerColumn;
  const int column = WK == 1 ? 0 : (wk * kChunks) / kChunksPerColumn;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t a_base = column * (Tile::kM * 128) + (wm * 64 + lr) * 128;
  const uint32_t b_base = Tile::kABytes + column * (Tile::kN * 128) + (wn * 32 + lc) * 128;
  // element e = 8 i + j of this thread, accumulators of the stage before: vector e / EV at + (e / EV) * 256 * 16
  const uint32_t kept = smem_u32(kept_smem) + threadIdx.x * 16;
  const uint32_t index = smem_u32(index_smem) + threadIdx.x * 4;      // + e * 256 * 4

  T acc[8][8];
  auto keep = [&]() {
#pragma unroll
    for (int v = 0; v < 64 / EV; ++v) {
      alignas(16) T x[EV];
#pragma unroll
      for (int e = 0; e < EV; ++e) x[e] = acc[(v * EV + e) / 8][(v * EV + e) % 8];
      const uint4 u = *reinterpret_cast<const uint4*>(x);
      asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(kept + v * (kConsumerThreads * 16)), "r"(u.x), "r"(u.y), "r"(u.z), "r"(u.w) : "memory");
    }
  };

  uint32_t it = 0;
  for (int w = blockIdx.x; w < num_work; w += gridDim.x) {
    int tm, tn, z, kt_begin, kt_end;
    decode(w, tm, tn, z, kt_begin, kt_end);
    const int m_base = tm * Tile::kM + wm * 64, n_base = tn * Tile::kN + wn * 32;

    // the running best starts from what is stored
    if (WK > 1) consumer_sync();                  // the previous tile's fold has been read
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int m = m_base + lr + 8 * i, n = n_base + lc + 4 * j;
        const T x = (m < p.M && n < p.N) ? p.dist[(long long)m * p.ldd + n] : T(0);
        // nothing is better than a NaN; the minimum instruction would drop it for the first product
        acc[i][j] = x == x ? x : kMaximize ? static_cast<T>(INFINITY) : -static_cast<T>(INFINITY);
      }
    if (!kDirect) keep();

    for (int kt = kt_begin; kt < kt_end; ++kt, ++it) {
      const int s = it % kStages;
      mbar_wait_or_abandon(&full_bar[s], (it / kStages) & 1, p.status, kDeviceTimeoutFull, abandoned);
      const uint32_t st = smem_base + s * Tile::kStageBytes;
#pragma unroll(sizeof(T) == 4 ? 4 : 1)
      for (int c = 0; c < kChunks; ++c) {
        T a[8][EV], b[8][EV];
        const int chunk = c + first_chunk;
        const uint32_t base = st + a_base + (((chunk ^ lr) & 7) << 4);
        const uint32_t base0 = st + b_base + (((chunk ^ lc) & 7) << 4), base1 = st + b_base + (((chunk ^ (lc + 4)) & 7) << 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) lds16(base + i * 1024, a[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) lds16(((j & 1) ? base1 : base0) + j * 512, b[j]);
        if constexpr (kDirect) {
          // k stays ascending for every element
          const int k = kt * kStep + column * TK + first_chunk * EV;
#pragma unroll
          for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int e = 0; e < EV; ++e)
#pragma unroll
              for (int i = 0; i < 8; ++i) improve<kMaximize>(acc[i][j], a[i][e] + b[j][e], index + (8 * i + j) * (kConsumerThreads * 4), k + e);
        } else if constexpr (R::kPackedPairs) {
#pragma unroll
          for (int e = 0; e < EV; e += 2)
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
              for (int j = 0; j < 8; ++j) acc[i][j] = R::mac_packed(acc[i][j], pack2(a[i][e], a[i][e + 1]), pack2(b[j][e], b[j][e + 1]));
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)                          // kByColumn of srgemm_tma.cuh
#pragma unroll
            for (int e = 0; e < EV; ++e)
#pragma unroll
              for (int i = 0; i < 8; ++i) acc[i][j] = R::add(a[i][e] + b[j][e], acc[i][j]);
        }
      }
      // which elements improved in this stage?  (a minimum only ever moves one way)
      if constexpr (!kDirect) {
        uint32_t mask_lo = 0, mask_hi = 0;
#pragma unroll
        for (int v = 0; v < 64 / EV; ++v) {
          T x[EV];
          lds16(kept + v * (kConsumerThreads * 16), x);
#pragma unroll
          for (int e = 0; e < EV; ++e) {
            const int el = v * EV + e;
            if (better(acc[el / 8][el % 8], x[e])) {
              if (el < 32) mask_lo |= 1u << el;
              else         mask_hi |= 1u << (el - 32);
            }
          }
        }
        if ((mask_lo | mask_hi) != 0) keep();
        while ((mask_lo | mask_hi) != 0) {
          int el;
          if (mask_lo != 0) { el = __ffs(mask_lo) - 1; mask_lo &= mask_lo - 1; }
          else              { el = 31 + __ffs(mask_hi); mask_hi &= mask_hi - 1; }
          const int i = el >> 3, j = el & 7;
          T value;
          {
            const uint32_t at = kept + (el / EV) * (kConsumerThreads * 16) + (el % EV) * (int)sizeof(T);
            if constexpr (sizeof(T) == 4) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(value) : "r"(at));
            else                          asm volatile("ld.shared.f64 %0, [%1];" : "=d"(value) : "r"(at));
          }
          const uint32_t ra = st + a_base + i * 1024, rb = st + b_base + j * 512;
          const int bx = lc + 4 * (j & 1);
          int found = 0;
#pragma unroll 4
          for (int c = kChunks - 1; c >= 0; --c) {          // descending: the first k that attains the value stays
            const int chunk = c + first_chunk;
            T a[EV], b[EV];
            lds16(ra + (((chunk ^ lr) & 7) << 4), a);
            lds16(rb + (((chunk ^ bx) & 7) << 4), b);
#pragma unroll
            for (int e = EV - 1; e >= 0; --e)
              if (a[e] + b[e] == value) found = c * EV + e;
          }
          const int k = kt * kStep + column * TK + first_chunk * EV + found;
          if constexpr (WK == 1) {
            const int m = m_base + lr + 8 * i, n = n_base + lc + 4 * j;
            if (m < p.M && n < p.N) p.parent[(long long)m * p.ld_parent + n] = k + p.k_offset;
          } else {
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(index + el * (kConsumerThreads * 4)), "r"(k) : "memory");
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_bar[s]);
    }

    if constexpr (WK == 1) {
      // (the opaque zero: the addresses are computed here again instead of being carried through the loop above)
      int zero;
      asm volatile("mov.s32 %0, 0;" : "=r"(zero));
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int m = m_base + lr + 8 * i + zero;
        T cur[8];                      // a row's loads together: none of them can pass a store
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int n = n_base + lc + 4 * j + zero;
          cur[j] = m < p.M && n < p.N ? p.dist[(long long)m * p.ldd + n] : acc[i][j];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int n = n_base + lc + 4 * j + zero;
          if (better(acc[i][j], cur[j])) p.dist[(long long)m * p.ldd + n] = acc[i][j];
        }
      }
    } else {
      // Partial values to shared memory ([wk][row][column], column groups swizzled), then one element per thread at a
      // time: the best value, and among equal ones the smallest k.  A value that is not better than dist has no k.
      constexpr int kRowGroups = Tile::kN / EV;
      T* fold = reinterpret_cast<T*>(kept_smem);
      const int32_t* ks = reinterpret_cast<const int32_t*>(index_smem);
      consumer_sync();                                   // every thread is done with its kept values
      T* mine = fold + wk * (Tile::kM * Tile::kN);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int r = wm * 64 + lr + 8 * i, c = wn * 32 + lc + 4 * j;
          mine[r * Tile::kN + (((c / EV) ^ (r & 7)) * EV) + (c % EV)] = acc[i][j];
        }
      consumer_sync();
      int32_t* tile_k = reinterpret_cast<int32_t*>(smem);        // a stage that is not needed any more (cluster only)
      for (int idx = threadIdx.x; idx < Tile::kM * Tile::kN; idx += kConsumerThreads) {
        const int r = idx / Tile::kN, c = idx % Tile::kN;
        const int at = r * Tile::kN + (((c / EV) ^ (r & 7)) * EV) + (c % EV);
        T v[WK];
#pragma unroll
        for (int q = 0; q < WK; ++q) v[q] = fold[q * (Tile::kM * Tile::kN) + at];
        T best = v[0];
#pragma unroll
        for (int q = 1; q < WK; ++q) best = better(v[q], best) ? v[q] : best;
        const int m = tm * Tile::kM + r, n = tn * Tile::kN + c;
        const bool inside = m < p.M && n < p.N;
        const bool improved = inside && better(best, p.dist[(long long)m * p.ldd + n]);
        int k = 0x7FFFFFFF;
        if (improved) {
          // thread and element that hold (row, column) in k group q
          const int el = ((r % 64) / 8) * 8 + (c % 32) / 4;
          const int t = ((r / 64) * WN + c / 32) * 32 + (r % 8) * 4 + c % 4;
#pragma unroll
          for (int q = 0; q < WK; ++q)
            if (v[q] == best) k = min(k, ks[el * kConsumerThreads + q * (WM * WN * 32) + t]);
        }
        if (p.cluster == 1) {
          if (improved) {
            p.dist[(long long)m * p.ldd + n] = best;
            p.parent[(long long)m * p.ld_parent + n] = k + p.k_offset;
          }
        } else {
          fold[at] = best;
          tile_k[idx] = k;
        }
      }
      if (p.cluster > 1) {
        cluster_sync();
        const int share = Tile::kM * Tile::kN / p.cluster;
        for (int idx = z * share + threadIdx.x; idx < (z + 1) * share; idx += kConsumerThreads) {
          const int r = idx / Tile::kN, c = idx % Tile::kN;
          const uint32_t at = smem_u32(fold + r * Tile::kN + (((c / EV) ^ (r & 7)) * EV) + (c % EV));
          T best, v;
          ld_cluster(at, 0, best);
          int k = (int)ld4_cluster(smem_u32(tile_k + idx), 0);
          for (int q = 1; q < p.cluster; ++q) {
            ld_cluster(at, q, v);
            const int kq = (int)ld4_cluster(smem_u32(tile_k + idx), q);
            if (better(v, best) || (v == best && kq < k)) { best = v; k = kq; }
          }
          const int m = tm * Tile::kM + r, n = tn * Tile::kN + c;
          if (m < p.M && n < p.N && k != 0x7FFFFFFF) {
            p.dist[(long long)m * p.ldd + n] = best;
            p.parent[(long long)m * p.ld_parent + n] = k + p.k_offset;
          }
        }
        cluster_sync();
      }
    }
  }
}

// Launches srgemm_path_kernel on `grid` CTAs: the 128 x 128 tile, or the small one (fp32 64 x 64, fp64 64 x 32) in clusters of
// params.cluster.
template <typename T>
cudaError_t launch_path(bool maximize, bool small_tile, const CUtensorMap& map_a, const CUtensorMap& map_b,
                        const PathParams<T>& params, int grid, cudaStream_t stream);

}  // namespace cuasr_b200
