// SIMT GETT kernels: FP32 FFMA (packed pairs) on the CUDA cores, FP64 on the
// FP64 tensor pipe (mma.sync m16n8k8; the short-K kernel: DFMA).
//
// Operands come packed MN-major by pack_kernel (Ap[k][Mp], Bp[k][Np], zero
// padded), so the main loop is a dense 16-byte cp.async pipeline -- or, for
// bandwidth-bound contractions (short K), straight from the user's tensors
// through the offset tables with element-wise cp.async ("direct": one read of
// each operand instead of read + packed write + packed read). The
// epilogue writes C straight into its own (multi-index) layout through the
// offset tables: element (m, n) of the GETT view is C[c_m_off[m] + c_n_off[n]].
// That is GETT's defining property (TCCG's micro-kernel stores into C's
// original layout, tccg/gett.py:192-223) -- there is no C transposition.
//
// FP32 tiles come in three shapes (128x128, and 128x32 / 32x128 for a small
// N / M); simt_shortk_kernel is the K <= 32 variant that reads the tile's C
// block under the FMA phase (below).
//
// beta == 0 writes C without reading it (TCCG's update = 0 path,
// tccg/gett.py:516-525). With a k-split the CTAs of split z write raw partial
// sums to a workspace and simt_reduce_kernel adds them (in T: FP64 for the
// double path) and applies alpha/beta, like TCCG's k-split with one private C
// per k-group and a final sum (tccg/gett.py:755-781).
#pragma once
#include <cuda.h>
#include "common.cuh"

namespace tccg {

// Tile shapes S: 0 = the square tile; FP32 also 1 = 128 x 32 (small N) and
// 2 = 32 x 128 (small M), for contractions whose small extent would leave
// most of a 128 x 128 tile empty (4 x 4 per thread instead of 8 x 8).
enum SimtShape : int { SIMT_SQUARE = 0, SIMT_NARROW_N = 1, SIMT_NARROW_M = 2 };

template <typename T, int S = SIMT_SQUARE>
struct SimtCfg;

template <>
struct SimtCfg<float, SIMT_SQUARE> {
  static constexpr int BM = 128, BN = 128, BK = 16;
  static constexpr int WARPS_M = 2, WARPS_N = 4;
  static constexpr int TMG = 2, TNG = 2;  // 4-wide groups per thread along m / n
  static constexpr int STAGES = 4;
  static constexpr int EPN = 128;         // epilogue columns per pass (the whole tile)
  static constexpr int PAD = 4;
  static constexpr int MIN_BLOCKS = 2;    // CTAs per SM the register budget allows
  static constexpr int LDA = BM, LDB = BN;  // stage row strides (elements)
};

template <>
struct SimtCfg<float, SIMT_NARROW_N> {
  static constexpr int BM = 128, BN = 32, BK = 16;
  static constexpr int WARPS_M = 4, WARPS_N = 2;
  static constexpr int TMG = 1, TNG = 1;
  static constexpr int STAGES = 4;
  static constexpr int EPN = 32;
  static constexpr int PAD = 4;
  static constexpr int MIN_BLOCKS = 3;
  // padded stage rows: gathers along k (lanes 4 elements apart in k) spread
  // over the banks
  static constexpr int LDA = BM + 4, LDB = BN + 4;
};

template <>
struct SimtCfg<float, SIMT_NARROW_M> {
  static constexpr int BM = 32, BN = 128, BK = 16;
  static constexpr int WARPS_M = 1, WARPS_N = 8;
  static constexpr int TMG = 1, TNG = 1;
  static constexpr int STAGES = 4;
  static constexpr int EPN = 128;
  static constexpr int PAD = 4;
  static constexpr int MIN_BLOCKS = 3;
  static constexpr int LDA = BM + 4, LDB = BN + 4;
};

// FP64: mma.sync m16n8k8 (simt_fma_ktile), warp tiles of 32 x 32. The stage
// rows are padded by 32 bytes: a fragment load's 4 k x 4 (half warp) rows
// then cover all banks. Epilogue rows padded by 64 bytes: the 16-byte
// accumulator pairs of 2 columns x 4 lanes do.
template <>
struct SimtCfg<double, SIMT_SQUARE> {
  static constexpr int BM = 128, BN = 64, BK = 8;
  static constexpr int WARPS_M = 4, WARPS_N = 2;
  static constexpr int TMG = 2, TNG = 1;  // 8 m x 4 n per thread
  static constexpr int STAGES = 4;
  static constexpr int EPN = 64;
  static constexpr int PAD = 8;
  static constexpr int MIN_BLOCKS = 2;
  static constexpr int LDA = BM + 4, LDB = BN + 4;
};

template <typename T>
struct SimtArgs {
  const T* Ap;  // [Kp][Mp]
  const T* Bp;  // [Kp][Np]
  int64_t Mp, Np, M, N;
  int32_t ktiles;          // Kp / BK
  int32_t ktiles_per_split;
  T* C;
  const int64_t* c_m_off;
  const int64_t* c_n_off;
  T alpha, beta;
  T* partial;  // non-null: write raw sums to partial[z][n][Mp]
  // direct != 0: no packing pass; the stage loader gathers A[k][m] =
  // Asrc[a_m_off[m] + a_k_off[k]] and B[k][n] = Bsrc[b_n_off[n] + b_k_off[k]]
  // element by element (zeros beyond M, N, K)
  int32_t direct;
  // narrow tiles, direct: 1 = the operand is gathered along k (its unit
  // stride is a K mode)
  int32_t a_kfast, b_kfast;
  int64_t K;
  const T* Asrc;
  const T* Bsrc;
  const int64_t* a_m_off;
  const int64_t* a_k_off;
  const int64_t* b_n_off;
  const int64_t* b_k_off;
  int32_t* status;  // device error word (bounded waits of the short-K kernel)
  // C layout (as TcArgs::crun): e0 in [2, 31] = C's stride-one index is the
  // first M mode, of extent e0, directly followed in C by the first N mode;
  // the epilogue then stores runs of e0 m by 32 / e0 columns per warp
  // instruction (consecutive addresses); 0 = quads along m, or lanes along m
  int32_t crun;
  // every quad m % 4 == 0 .. + 3 of C is 4 consecutive, aligned elements in
  // every column: the epilogue moves 4 m per thread as a vector. Otherwise
  // its lanes run along m, one element each: a quad of scattered alignment
  // would write each 32-byte sector of C in 4 instructions of 4 bytes a lane
  int32_t c_vec;
  int64_t ldc;  // > 0: C(m, n) = C[m + ldc n] (short-K kernel, SHORTK_BULK)
};

template <typename T, int S = SIMT_SQUARE>
constexpr size_t simt_smem_bytes() {
  using Cfg = SimtCfg<T, S>;
  size_t pipe = (size_t)Cfg::STAGES * Cfg::BK * (Cfg::LDA + Cfg::LDB) * sizeof(T);
  // epilogue: the C tile (one pass of EPN columns), C offsets of the pass's
  // columns and of the tile's rows
  size_t epi = (size_t)Cfg::EPN * (Cfg::BM + Cfg::PAD) * sizeof(T) +
               (Cfg::EPN + Cfg::BM) * sizeof(int64_t);
  return pipe > epi ? pipe : epi;
}

template <typename T>
struct Vec4 {
  T v[4];
};

template <typename T>
__device__ __forceinline__ Vec4<T> lds4(const T* p) {
  Vec4<T> r;
  if constexpr (sizeof(T) == 4) {
    float4 x = *reinterpret_cast<const float4*>(p);
    r.v[0] = x.x; r.v[1] = x.y; r.v[2] = x.z; r.v[3] = x.w;
  } else {
    double2 x = *reinterpret_cast<const double2*>(p);
    double2 y = *reinterpret_cast<const double2*>(p + 2);
    r.v[0] = x.x; r.v[1] = x.y; r.v[2] = y.x; r.v[3] = y.y;
  }
  return r;
}

// Thread fragment geometry of the 256-thread tiles.
// FMA fragments (FP32, and FP64 in the short-K kernel): lanes 8 (m) x 4 (n),
// a thread has groups of 4 m of every 32 and groups of 4 n of every 16. FP32:
// warps WARPS_M x WARPS_N, m = 4 lm + i, one 16-byte load. FP64: warps 2 x 4,
// two 16-byte loads at m = 2 lm + {0, 1} and 16 + 2 lm + {0, 1}, so the 8 lane
// groups of each load read 128 contiguous bytes (4 consecutive doubles per
// lane would put lanes lm and lm + 4 on the same banks).
// MMA fragments (FP64): warp tiles of 32 x 32, computed as (n x k) (k x m)
// products of mma m16n8k8: a thread holds, per 16 n and 8 m, n = lane / 4 +
// {0, 8} and the pair m = 2 (lane % 4) + {0, 1} (consecutive in C's staged
// columns).
template <typename T, int S = SIMT_SQUARE, bool MMA = sizeof(T) == 8>
struct SimtFrag {
  using Cfg = SimtCfg<T, S>;
  static constexpr int TM = Cfg::TMG * 4, TN = Cfg::TNG * 4;
  static constexpr bool PAIRS = sizeof(T) == 8;
  // panel row strides: the FP64 FMA fragments read dense panels
  static constexpr int LDA = PAIRS && !MMA ? Cfg::BM : Cfg::LDA, LDB = PAIRS && !MMA ? Cfg::BN : Cfg::LDB;
  int a_off, b_off;  // this thread's first element of the A and B panels
  int m0, n0;        // its first m and n
  __device__ __forceinline__ explicit SimtFrag(int tid) {
    const int warp = tid >> 5, lane = tid & 31;
    if constexpr (MMA) {
      static_assert(Cfg::WARPS_M * 32 == Cfg::BM && Cfg::WARPS_N * 32 == Cfg::BN, "32 x 32 per warp");
      const int wm = warp % Cfg::WARPS_M, wn = warp / Cfg::WARPS_M;
      a_off = (lane & 3) * LDA + wm * 32 + (lane >> 2);
      b_off = (lane & 3) * LDB + wn * 32 + (lane >> 2);
      m0 = wm * 32 + 2 * (lane & 3);
      n0 = wn * 32 + (lane >> 2);
    } else {
      constexpr int WARPS_M = PAIRS ? 2 : Cfg::WARPS_M, WARPS_N = PAIRS ? 4 : Cfg::WARPS_N;
      static_assert(WARPS_M * Cfg::TMG * 32 == Cfg::BM && WARPS_N * Cfg::TNG * 16 == Cfg::BN,
                    "warps cover the tile");
      const int wm = warp % WARPS_M, wn = warp / WARPS_M;
      a_off = m0 = wm * (Cfg::TMG * 32) + (lane & 7) * (PAIRS ? 2 : 4);
      b_off = n0 = wn * (Cfg::TNG * 16) + (lane >> 3) * 4;
    }
  }
  // tile-local m of accumulator row i and n of accumulator column j
  __device__ __forceinline__ int m(int i) const {
    return MMA     ? m0 + (i / 2) * 8 + (i % 2)
           : PAIRS ? m0 + (i / 4) * 32 + ((i % 4) / 2) * 16 + (i % 2)
                   : m0 + (i / 4) * 32 + (i % 4);
  }
  __device__ __forceinline__ int n(int j) const {
    return MMA ? n0 + (j / 2) * 16 + (j % 2) * 8 : n0 + (j / 4) * 16 + (j % 4);
  }
};

// D (16 x 8) += A (16 x 8) B (8 x 8) in FP64. Lane l holds A(l / 4 + {0, 8},
// l % 4 + {0, 4}) as a0 a1 (k), a2 a3 (k + 4); B(l % 4 + {0, 4}, l / 4); D rows
// l / 4 (c0 c1) and l / 4 + 8 (c2 c3), columns 2 (l % 4) + {0, 1}.
__device__ __forceinline__ void mma_f64(double& c0, double& c1, double& c2, double& c3, double a0,
                                        double a1, double a2, double a3, double b0, double b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+d"(c0), "+d"(c1), "+d"(c2), "+d"(c3)
      : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// A thread's TM x TN sums.
// FP32: pairs for fma.rn.f32x2. A pair of m times a pair of n gives the two
// "diagonal" sums, times the swapped pair of n the other two, so no operand
// has to be duplicated: v[ip][j] = (sum of (2 ip, j), sum of (2 ip + 1, j ^ 1)).
// The FMA pipe takes a pair in two cycles: half the issue slots of the loop
// are left for its shared-memory loads and the swaps.
template <typename T, int S = SIMT_SQUARE, bool MMA = sizeof(T) == 8>
struct SimtAcc {
  static constexpr int TM = SimtFrag<T, S, MMA>::TM, TN = SimtFrag<T, S, MMA>::TN;
  T v[TM][TN];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) v[i][j] = T(0);
  }
  __device__ __forceinline__ T get(int i, int j) const { return v[i][j]; }
};
template <int S>
struct SimtAcc<float, S, false> {
  static constexpr int TM = SimtFrag<float, S, false>::TM, TN = SimtFrag<float, S, false>::TN;
  uint64_t v[TM / 2][TN];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) v[i][j] = 0;
  }
  __device__ __forceinline__ float get(int i, int j) const {
    return i % 2 == 0 ? f32x2_lo(v[i / 2][j]) : f32x2_hi(v[i / 2][j ^ 1]);
  }
};

// One k-tile: acc += A[k][m] * B[k][n] over the BK rows of the stage's
// A [BK][LDA] and B [BK][LDB] panels, k in increasing order.
// FP64 bound: the fp64 pipe. Fragments of DFMA (8 x 4 per thread) read 12
// doubles of shared memory per 32 FMAs -- 79 % of the shared-memory wavefronts
// at 64 % of the pipe; the mma fragments read 16 per 256 FMAs of a lane:
// 3825 x 4056 x 3080 in 3.04 ms against 4.25 (31.4 and 22.5 TFLOP/s). A K
// that ends after two steps is bound by C and keeps DFMA, whose short phases
// cost less (96^4 x 16 in the short-K kernel: 217 us, 238 with mma).
template <typename T, int S = SIMT_SQUARE, bool MMA = sizeof(T) == 8, int BK = SimtCfg<T, S>::BK>
__device__ __forceinline__ void simt_fma_ktile(
    const T* as, const T* bs, int a_off, int b_off, SimtAcc<T, S, MMA>& acc_) {
  using Cfg = SimtCfg<T, S>;
  using Frag = SimtFrag<T, S, MMA>;
  constexpr int TM = Frag::TM, TN = Frag::TN;
  auto& acc = acc_.v;
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      uint64_t av[TM / 2], bv[TN / 2];  // pairs of m, pairs of n
#pragma unroll
      for (int g = 0; g < Cfg::TMG; ++g) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(as + k * Frag::LDA + a_off + g * 32);
        av[2 * g] = x.x;
        av[2 * g + 1] = x.y;
      }
#pragma unroll
      for (int g = 0; g < Cfg::TNG; ++g) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(bs + k * Frag::LDB + b_off + g * 16);
        bv[2 * g] = x.x;
        bv[2 * g + 1] = x.y;
      }
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) {
        const uint64_t sw = f32x2_swap(bv[j]);
#pragma unroll
        for (int i = 0; i < TM / 2; ++i) {
          acc[i][2 * j] = fma_x2(av[i], bv[j], acc[i][2 * j]);
          acc[i][2 * j + 1] = fma_x2(av[i], sw, acc[i][2 * j + 1]);
        }
      }
    }
  } else if constexpr (MMA) {
    static_assert(BK == 8 && TM == 8 && TN == 4, "one mma k step per tile");
    double a[4][2], b[2][4];  // [8 m][k, k + 4], [16 n][(n, k), (n + 8, k), (n, k + 4), (n + 8, k + 4)]
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
      for (int h = 0; h < 2; ++h) a[mt][h] = as[a_off + 4 * h * Cfg::LDA + 8 * mt];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int h = 0; h < 4; ++h) b[nt][h] = bs[b_off + 4 * (h / 2) * Cfg::LDB + 16 * nt + 8 * (h % 2)];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int mt = 0; mt < 4; ++mt)
        mma_f64(acc[2 * mt][2 * nt], acc[2 * mt + 1][2 * nt], acc[2 * mt][2 * nt + 1],
                acc[2 * mt + 1][2 * nt + 1], b[nt][0], b[nt][1], b[nt][2], b[nt][3], a[mt][0], a[mt][1]);
  } else {
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      T av[TM], bv[TN];
#pragma unroll
      for (int g = 0; g < Cfg::TMG; ++g) {
        const double2 lo = *reinterpret_cast<const double2*>(as + k * Frag::LDA + a_off + g * 32);
        const double2 hi = *reinterpret_cast<const double2*>(as + k * Frag::LDA + a_off + g * 32 + 16);
        av[g * 4 + 0] = lo.x; av[g * 4 + 1] = lo.y; av[g * 4 + 2] = hi.x; av[g * 4 + 3] = hi.y;
      }
#pragma unroll
      for (int g = 0; g < Cfg::TNG; ++g) {
        const Vec4<T> x = lds4<T>(bs + k * Frag::LDB + b_off + g * 16);
        bv[g * 4 + 0] = x.v[0]; bv[g * 4 + 1] = x.v[1]; bv[g * 4 + 2] = x.v[2]; bv[g * 4 + 3] = x.v[3];
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fma(av[i], bv[j], acc[i][j]);
    }
  }
}

// One BM x BN tile (bx, by) of split bz; all 256 threads of the CTA take part.
// Operand loading of simt_gett_tile: packed operands only, direct gathers
// only, or either by a.direct at run time (the grouped kernel). The packed
// instantiation carries none of the gather code, so its register allocation
// and epilogue stay those of a pure packed kernel.
enum SimtLoad : int { SIMT_PACKED = 0, SIMT_DIRECT = 1, SIMT_EITHER = 2 };

template <typename T, int LOAD = SIMT_EITHER, int S = SIMT_SQUARE>
__device__ __forceinline__ void simt_gett_tile(const SimtArgs<T>& a, int bx, int by, int bz) {
  using Cfg = SimtCfg<T, S>;
  constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, STAGES = Cfg::STAGES;
  constexpr int LDA = Cfg::LDA, LDB = Cfg::LDB;
  constexpr int TM = Cfg::TMG * 4, TN = Cfg::TNG * 4;
  constexpr int VEC = 16 / sizeof(T);                 // elements per 16-byte chunk
  constexpr int A_CHUNKS = BK * BM / VEC, B_CHUNKS = BK * BN / VEC;
  constexpr int A_ROW_CHUNKS = BM / VEC, B_ROW_CHUNKS = BN / VEC;

  extern __shared__ __align__(16) uint8_t smem_raw[];
  T* As = reinterpret_cast<T*>(smem_raw);              // [STAGES][BK][LDA]
  T* Bs = As + (size_t)STAGES * BK * LDA;              // [STAGES][BK][LDB]

  const int tid = threadIdx.x;
  const int64_t m0 = (int64_t)bx * BM, n0 = (int64_t)by * BN;
  const int kt_begin = bz * a.ktiles_per_split;
  int kt_end = kt_begin + a.ktiles_per_split;
  if (kt_end > a.ktiles) kt_end = a.ktiles;

  // direct loads: thread tid always fills column tid % BM of A's stage and
  // tid % BN of B's (256 is a multiple of both), rows tid / BM + j * 256 / BM
  static_assert(256 % BM == 0 && 256 % BN == 0, "direct loader layout");
  const int dcol_a = tid % BM, drow_a = tid / BM;
  const int dcol_b = tid % BN, drow_b = tid / BN;
  constexpr int64_t NONE = INT64_MIN;  // offsets may be negative (negative strides)
  int64_t dm_off = NONE, dn_off = NONE;
  const bool direct = LOAD == SIMT_DIRECT || (LOAD == SIMT_EITHER && a.direct);
  if (direct) {
    if (m0 + dcol_a < a.M) dm_off = a.a_m_off[m0 + dcol_a];
    if (n0 + dcol_b < a.N) dn_off = a.b_n_off[n0 + dcol_b];
  }
  // Narrow tiles: an operand whose unit stride is along k (a_kfast /
  // b_kfast) is gathered with lanes along k instead -- thread tid fills
  // k = tid % BK of rows tid / BK + j * (256 / BK) -- so each warp reads two
  // 64-byte runs; the rows' offsets are loaded once per tile.
  constexpr bool KFAST = S != SIMT_SQUARE;
  constexpr int KR = 256 / BK;  // rows per pass of the k-fast gather
  constexpr int JAK = KFAST ? BM / KR : 1, JBK = KFAST ? BN / KR : 1;
  const int kk = tid % BK, kr = tid / BK;
  int64_t kfa[JAK], kfb[JBK];
  const bool kfast_a = KFAST && direct && a.a_kfast, kfast_b = KFAST && direct && a.b_kfast;
  if constexpr (KFAST) {
    static_assert(BM % KR == 0 && BN % KR == 0, "k-fast gather layout");
#pragma unroll
    for (int j = 0; j < JAK; ++j) {
      const int64_t m = m0 + kr + j * KR;
      kfa[j] = kfast_a && m < a.M ? a.a_m_off[m] : NONE;
    }
#pragma unroll
    for (int j = 0; j < JBK; ++j) {
      const int64_t n = n0 + kr + j * KR;
      kfb[j] = kfast_b && n < a.N ? a.b_n_off[n] : NONE;
    }
  }

  auto load_stage = [&](int stage, int kt) {
    T* as = As + (size_t)stage * BK * LDA;
    T* bs = Bs + (size_t)stage * BK * LDB;
    const int64_t krow = (int64_t)kt * BK;
    if (KFAST && (kfast_a || kfast_b)) {
      // one operand (or both) along k; the other, if any, along its rows
      const int64_t k = krow + kk;
      const int64_t koa = k < a.K ? __ldg(a.a_k_off + k) : NONE;
      const int64_t kob = k < a.K ? __ldg(a.b_k_off + k) : NONE;
      constexpr int JA = BK * BM / 256, JB = BK * BN / 256;
      if (kfast_a) {
#pragma unroll
        for (int j = 0; j < JAK; ++j) {
          T* dst = as + kk * LDA + kr + j * KR;
          const bool in = kfa[j] != NONE && koa != NONE;
          cp_async_elem_or_zero<sizeof(T)>(dst, a.Asrc + (in ? kfa[j] + koa : 0), in);
        }
      } else {
#pragma unroll
        for (int j = 0; j < JA; ++j) {
          const int64_t kj = krow + drow_a + j * (256 / BM);
          T* dst = as + (drow_a + j * (256 / BM)) * LDA + dcol_a;
          const bool in = dm_off != NONE && kj < a.K;
          cp_async_elem_or_zero<sizeof(T)>(dst, a.Asrc + (in ? dm_off + __ldg(a.a_k_off + kj) : 0), in);
        }
      }
      if (kfast_b) {
#pragma unroll
        for (int j = 0; j < JBK; ++j) {
          T* dst = bs + kk * LDB + kr + j * KR;
          const bool in = kfb[j] != NONE && kob != NONE;
          cp_async_elem_or_zero<sizeof(T)>(dst, a.Bsrc + (in ? kfb[j] + kob : 0), in);
        }
      } else {
#pragma unroll
        for (int j = 0; j < JB; ++j) {
          const int64_t kj = krow + drow_b + j * (256 / BN);
          T* dst = bs + (drow_b + j * (256 / BN)) * LDB + dcol_b;
          const bool in = dn_off != NONE && kj < a.K;
          cp_async_elem_or_zero<sizeof(T)>(dst, a.Bsrc + (in ? dn_off + __ldg(a.b_k_off + kj) : 0), in);
        }
      }
    } else if (direct) {
      // all k offsets first (independent loads), then the copies: an offset
      // load between two asynchronous copies would serialise them
      // Elements outside the operands are copies of no bytes, not branches
      // (2048^2 x 256 FP32 98.7 -> 89.4 us, FP64 512^3 31.3 -> 24.9 with the
      // mma.sync tiles, 20000 x 32 x 1000 90.1 -> 82.3).
      constexpr int JA = BK * BM / 256, JB = BK * BN / 256;
      int64_t koa[JA], kob[JB];
#pragma unroll
      for (int j = 0; j < JA; ++j) {
        const int64_t k = krow + drow_a + j * (256 / BM);
        koa[j] = k < a.K ? __ldg(a.a_k_off + k) : NONE;
      }
#pragma unroll
      for (int j = 0; j < JB; ++j) {
        const int64_t k = krow + drow_b + j * (256 / BN);
        kob[j] = k < a.K ? __ldg(a.b_k_off + k) : NONE;
      }
#pragma unroll
      for (int j = 0; j < JA; ++j) {
        T* dst = as + (drow_a + j * (256 / BM)) * LDA + dcol_a;
        const bool in = dm_off != NONE && koa[j] != NONE;
        cp_async_elem_or_zero<sizeof(T)>(dst, a.Asrc + (in ? dm_off + koa[j] : 0), in);
      }
#pragma unroll
      for (int j = 0; j < JB; ++j) {
        T* dst = bs + (drow_b + j * (256 / BN)) * LDB + dcol_b;
        const bool in = dn_off != NONE && kob[j] != NONE;
        cp_async_elem_or_zero<sizeof(T)>(dst, a.Bsrc + (in ? dn_off + kob[j] : 0), in);
      }
    } else if constexpr (LOAD != SIMT_DIRECT) {
#pragma unroll
      for (int c = tid; c < A_CHUNKS; c += 256) {
        const int row = c / A_ROW_CHUNKS, col = (c % A_ROW_CHUNKS) * VEC;
        cp_async_16(as + row * LDA + col, a.Ap + (krow + row) * a.Mp + m0 + col);
      }
#pragma unroll
      for (int c = tid; c < B_CHUNKS; c += 256) {
        const int row = c / B_ROW_CHUNKS, col = (c % B_ROW_CHUNKS) * VEC;
        cp_async_16(bs + row * LDB + col, a.Bp + (krow + row) * a.Np + n0 + col);
      }
    }
  };

  SimtAcc<T, S> acc;
  acc.zero();

#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (kt_begin + s < kt_end) load_stage(s, kt_begin + s);
    cp_async_commit();
  }

  const SimtFrag<T, S> frag(tid);
  const int a_off = frag.a_off, b_off = frag.b_off;
  for (int kt = kt_begin; kt < kt_end; ++kt) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    {
      const int nk = kt + STAGES - 1;
      if (nk < kt_end) load_stage((nk - kt_begin) % STAGES, nk);
      cp_async_commit();
    }
    const int stage = (kt - kt_begin) % STAGES;
    const T* as = As + (size_t)stage * BK * LDA;
    const T* bs = Bs + (size_t)stage * BK * LDB;
    simt_fma_ktile<T, S>(as, bs, a_off, b_off, acc);
  }
  cp_async_wait<0>();
  __syncthreads();

  auto mloc = [&](int i) { return frag.m(i); };
  auto nloc = [&](int j) { return frag.n(j); };

  if (a.partial != nullptr) {
    T* P = a.partial + (size_t)bz * a.Np * a.Mp;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int64_t n = n0 + nloc(j);
#pragma unroll
      for (int i = 0; i < TM; ++i) P[n * a.Mp + m0 + mloc(i)] = acc.get(i, j);
    }
    return;
  }

  // Epilogue through shared memory. Each thread owns 4 consecutive m of one
  // column at a time; where those 4 elements of C are contiguous and 16-byte
  // aligned (C's stride-one index is the first M mode) they move as one
  // vector, otherwise element by element. All C loads of a pass are issued
  // before its stores, so a thread keeps several loads in flight.
  constexpr int EPN = Cfg::EPN, LDC = BM + Cfg::PAD;
  constexpr int QPC = BM / 4;              // m quads per column
  constexpr int CPI = 256 / QPC;           // columns per iteration
  constexpr int ITER = EPN / CPI;
  T* Cs = reinterpret_cast<T*>(smem_raw);  // [EPN][LDC]
  // C offsets of the pass's columns, staged once: the C loads of a chunk then
  // depend on shared memory only, not on a table load from L2
  int64_t* Cn = reinterpret_cast<int64_t*>(smem_raw + (size_t)EPN * LDC * sizeof(T));
  int64_t* Cm = Cn + EPN;  // C offsets of the tile's rows (staged C stores)
  static_assert((EPN * LDC * sizeof(T)) % 8 == 0 && EPN <= 256, "column offset staging");
  if (a.crun > 0)
    for (int r = tid; r < BM; r += 256) Cm[r] = m0 + r < a.M ? a.c_m_off[m0 + r] : 0;
  const int q = tid % QPC, cl = tid / QPC;
  const int64_t mq = m0 + 4 * q;
  int64_t cmo[4];
  bool mok[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    mok[i] = mq + i < a.M;
    cmo[i] = mok[i] ? a.c_m_off[mq + i] : 0;
  }
  const bool vec_m = mok[3] && cmo[1] == cmo[0] + 1 && cmo[2] == cmo[0] + 2 && cmo[3] == cmo[0] + 3;
  const T alpha = a.alpha, beta = a.beta;
  for (int p = 0; p < BN / EPN; ++p) {
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int nl = nloc(j) - p * EPN;
      if (nl >= 0 && nl < EPN) {
        if constexpr (sizeof(T) == 8) {
#pragma unroll
          for (int i = 0; i < TM; i += 2)
            *reinterpret_cast<double2*>(Cs + nl * LDC + mloc(i)) = make_double2(acc.get(i, j), acc.get(i + 1, j));
        } else {
#pragma unroll
          for (int i = 0; i < TM; ++i) Cs[nl * LDC + mloc(i)] = acc.get(i, j);
        }
      }
    }
    if (tid < EPN) {
      const int64_t n = n0 + p * EPN + tid;
      Cn[tid] = n < a.N ? a.c_n_off[n] : 0;
    }
    __syncthreads();
    if (a.crun > 0) {
      // runs of e0 consecutive m (clipped to the tile and M, length L), one
      // per warp at a time: the run's L x ncols block is stored in C's
      // address order, element f = i + L * j (row ma + i, column j) by lane
      // f % 32, so a store instruction covers 32 consecutive positions of
      // one contiguous stretch of C; the C offsets of rows and columns come
      // from shared memory. Same arithmetic as the quad path (alpha * acc,
      // then fma with beta).
      const int e0 = a.crun;
      const int lane = tid & 31, w = tid >> 5;
      const int64_t rfirst = (m0 / e0) * e0;
      const int nruns = (int)((m0 + BM - rfirst + e0 - 1) / e0);
      const int64_t nleft = a.N - (n0 + p * EPN);
      const int ncols = nleft < EPN ? (int)nleft : EPN;
#pragma unroll 1
      for (int ri = w; ri < nruns; ri += 8) {
        const int64_t rs = rfirst + (int64_t)ri * e0;
        const int64_t ma = rs > m0 ? rs : m0;
        int64_t mb = rs + e0 < m0 + BM ? rs + e0 : m0 + BM;
        if (mb > a.M) mb = a.M;
        const int L = (int)(mb - ma);
        if (L <= 0 || ncols <= 0) continue;
        const int total = L * ncols;
        int i = lane % L, j = lane / L;
        const int di = 32 % L, dj = 32 / L;
        const int moff = (int)(ma - m0);
#pragma unroll 2
        for (int f = lane; f < total; f += 32) {
          T* d = a.C + Cm[moff + i] + Cn[j];
          T v = alpha * Cs[j * LDC + moff + i];
          if (beta != T(0)) v = fma(beta, *d, v);
          *d = v;
          i += di;
          j += dj;
          if (i >= L) {
            i -= L;
            ++j;
          }
        }
      }
    } else if (!a.c_vec) {
      // lanes along m, one element per thread and column
      constexpr int CS = 256 / BM, CH = 8;  // columns per step, steps whose C loads are in flight
      const int ml = tid % BM, c0 = tid / BM;
      const int64_t nleft = a.N - (n0 + p * EPN);
      const int ncols = nleft < EPN ? (int)nleft : EPN;
      if (m0 + ml < a.M) {
        T* const Cb = a.C + a.c_m_off[m0 + ml];
#pragma unroll 1
        for (int c1 = c0; c1 < ncols; c1 += CS * CH) {
          // shared memory is read before the stores (which may alias it as
          // far as the compiler knows): one wait per CH columns
          int64_t no[CH];
          T v[CH], old[CH];
#pragma unroll
          for (int u = 0; u < CH; ++u) {
            const int c = c1 + u * CS;
            no[u] = c < ncols ? Cn[c] : 0;
            v[u] = c < ncols ? Cs[c * LDC + ml] : T(0);
          }
          if (beta != T(0)) {
#pragma unroll
            for (int u = 0; u < CH; ++u)
              old[u] = c1 + u * CS < ncols ? Cb[no[u]] : T(0);
          }
#pragma unroll
          for (int u = 0; u < CH; ++u) {
            if (c1 + u * CS < ncols) {
              v[u] = alpha * v[u];
              if (beta != T(0)) v[u] = fma(beta, old[u], v[u]);
              Cb[no[u]] = v[u];
            }
          }
        }
      }
    } else if (mok[0]) {
      constexpr int CH = sizeof(T) == 8 ? 4 : 8;  // columns whose C loads are in flight together
#pragma unroll 1
      for (int it0 = 0; it0 < ITER; it0 += CH) {
        int64_t coff[CH];
        bool nok[CH];
#pragma unroll
        for (int u = 0; u < CH; ++u) {
          const int64_t n = n0 + p * EPN + (it0 + u) * CPI + cl;
          nok[u] = (it0 + u < ITER) && n < a.N;
          coff[u] = nok[u] ? Cn[(it0 + u) * CPI + cl] : 0;
        }
        T old[CH][4];
        if (beta != T(0)) {
#pragma unroll
          for (int u = 0; u < CH; ++u) {
            if (!nok[u]) continue;
            const T* d = a.C + cmo[0] + coff[u];
            if (vec_m && (reinterpret_cast<uintptr_t>(d) % (4 * sizeof(T))) == 0) {
              const Vec4<T> v = lds4<T>(d);  // 16/32-byte vector load
              old[u][0] = v.v[0]; old[u][1] = v.v[1]; old[u][2] = v.v[2]; old[u][3] = v.v[3];
            } else {
#pragma unroll
              for (int i = 0; i < 4; ++i) old[u][i] = mok[i] ? a.C[cmo[i] + coff[u]] : T(0);
            }
          }
        }
#pragma unroll
        for (int u = 0; u < CH; ++u) {
          if (!nok[u]) continue;
          const int nl = (it0 + u) * CPI + cl;
          T v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            v[i] = alpha * Cs[nl * LDC + 4 * q + i];
            if (beta != T(0)) v[i] = fma(beta, old[u][i], v[i]);
          }
          T* d = a.C + cmo[0] + coff[u];
          if (vec_m && (reinterpret_cast<uintptr_t>(d) % (4 * sizeof(T))) == 0) {
            if constexpr (sizeof(T) == 4) {
              *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
              reinterpret_cast<double2*>(d)[0] = make_double2(v[0], v[1]);
              reinterpret_cast<double2*>(d)[1] = make_double2(v[2], v[3]);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (mok[i]) a.C[cmo[i] + coff[u]] = v[i];
          }
        }
      }
    }
    __syncthreads();
  }
}

template <typename T, int LOAD, int S = SIMT_SQUARE>
__global__ void __launch_bounds__(256, SimtCfg<T, S>::MIN_BLOCKS) simt_gett_kernel(const SimtArgs<T> a) {
  grid_dep_wait();  // packed operands written by the kernel before
  simt_gett_tile<T, LOAD, S>(a, blockIdx.x, blockIdx.y, blockIdx.z);
}

// FP32 contractions that run as products of the operands' three-way bf16
// splits (TC_F32X6) but whose values the splits do not represent: the tile
// kernel on operands packed by the tensor-core kernel (f32_fallback_pack),
// with the k slices of the FFMA plan. Launched behind the tensor-core kernel;
// in the ordinary case the CTAs read the range words and leave at once.
struct F32FallbackItem {
  SimtArgs<float> args;
  SplitRange split;
  int32_t tiles_m;
  int64_t tiles, jobs;  // tiles x k slices
};

__device__ __forceinline__ void f32_fallback_job(const F32FallbackItem& it, int64_t j) {
  const int64_t t = j % it.tiles;
  simt_gett_tile<float, SIMT_PACKED>(it.args, (int)(t % it.tiles_m), (int)(t / it.tiles_m),
                                     (int)(j / it.tiles));
}

// One CTA per job: 1024 CTAs that leave cost 1 us; the same tiles by 296
// persistent CTAs take 15 % longer (they all store at the same time, and the
// loop spills). With one infinity, us, the FFMA plan / this path: 4096 x 4096 x
// 1024 673 / 716, 13824 x 13824 x 1024 7300 / 7235, 512 x 700 x 3000 70 / 101,
// 12648 x 85 x 4418 516 / 789 (three passes over the operands).
__global__ void __launch_bounds__(256, 2)
    f32_fallback_kernel(const __grid_constant__ F32FallbackItem it) {
  grid_dep_wait();  // range words of the packing pass; C written by nobody before this
  if (!f32_split_exact(it.split)) f32_fallback_job(it, blockIdx.x);
}

// Grouped: a persistent wave; the jobs of the items that need it, one item's
// after another's, go round the grid.
__global__ void __launch_bounds__(256, 2)
    f32_fallback_group_kernel(const F32FallbackItem* items, int n_items) {
  bool any = false;
  for (int i = threadIdx.x; i < n_items; i += blockDim.x) any |= !f32_split_exact(items[i].split);
  if (!__syncthreads_or(any)) return;
  const int64_t g = gridDim.x;
  int64_t first = 0;  // the CTA that takes the item's first job
  for (int i = 0; i < n_items; ++i) {
    const F32FallbackItem& it = items[i];
    if (f32_split_exact(it.split)) continue;
    for (int64_t j = (blockIdx.x + g - first) % g; j < it.jobs; j += g) f32_fallback_job(it, j);
    first = (first + it.jobs) % g;
  }
}

// ---------------------------------------------------------------------------
// Short-K kernel (packed operands, K <= KP, no k-split). For K = 16 a tile's
// FMA work (16 FMAs per C element) is short next to its C traffic, and
// simt_gett_tile reads C only in its epilogue, where the loads' latency
// stalls the CTA, then spends its own issue slots on the stores. Here the CTA
// brings its C block into shared memory right after the operand panels, so
// the read runs under the FMA phase; the epilogue combines in shared memory
// (alpha * acc + beta * C, 16-byte accesses at the fragment positions) and
// the block leaves as one bulk store.
//   SHORTK_TMA  (C is a 2-D matrix in the GETT view: unit M stride, one N
//               stride of 16-byte multiple): the C block comes in and goes
//               out by TMA -- one instruction each, the store draining while
//               the next CTA on the SM computes.
//   SHORTK_BULK (FP32, a 2-D C whose columns start off 16-byte boundaries):
//               one bulk copy per column each way. A column lies in shared
//               memory at its global offset modulo 16 bytes; it comes in as
//               the 16-byte-aligned range around it (where that is inside
//               C) and leaves as the aligned range inside it, its up to 3 + 3
//               edge elements by plain stores. In the combine step the 4 lanes
//               that share a bank group take their 4 m in rotated order.
//   SHORTK_ANY  (any layout): each thread has one m and every other column,
//               cp.async in and stores out with lanes along m.
// 6930 x 8585 x 19, FP32, beta = 1: 119 us; SHORTK_ANY 156 (bound by its
// per-element instructions), the tile kernel with 4-element quads per thread
// 181. HBM time of C in and out: 73 us; the FMA phase (its shared-memory loads
// at 60 TFLOP/s) and the C traffic share the shared-memory path and add up.
// The FMA loop stops at K rounded up to 4, not at the packed panel's end.
// Two CTAs per SM. Same k order and epilogue arithmetic as simt_gett_tile:
// the results are bitwise equal.
template <typename T>
struct SimtShortKCfg {
  using Cfg = SimtCfg<T>;
  static constexpr int KP = sizeof(T) == 4 ? 32 : 16;  // longest padded K it takes
  static constexpr int LDCB = Cfg::BM + 4;  // SHORTK_BULK: column pitch
  // [BN][BM], dense; FP32 also [BN][LDCB]
  static constexpr size_t C_BYTES = (size_t)Cfg::BN * (sizeof(T) == 4 ? LDCB : Cfg::BM) * sizeof(T);
  static constexpr size_t N_BYTES = (size_t)Cfg::BN * sizeof(int64_t);
  static constexpr size_t A_BYTES = (size_t)KP * Cfg::BM * sizeof(T);
  static constexpr size_t B_BYTES = (size_t)KP * Cfg::BN * sizeof(T);
  static constexpr size_t USED = C_BYTES + N_BYTES + A_BYTES + B_BYTES + 16;  // + mbarrier
  static constexpr size_t SMEM_BYTES = USED + 128;  // slack to align the C block to 128 bytes
  static_assert(C_BYTES % 128 == 0 && N_BYTES % 16 == 0 && A_BYTES % 16 == 0, "aligned panels");
  static_assert(2 * (SMEM_BYTES + 1024) <= 228 * 1024, "two CTAs per SM");
};

enum ShortKC : int { SHORTK_ANY = 0, SHORTK_TMA = 1, SHORTK_BULK = 2 };

// One column of a SHORTK_BULK block: g = its first element (len of them), at
// element `shift` of its shared-memory column; [lo, hi) = the aligned range
// around it, [in0, in1) the one inside it (empty when in1 <= in0).
struct ShortKCol {
  const char *g, *end, *lo, *hi, *in0, *in1;
  int shift;
  __device__ __forceinline__ ShortKCol(const float* first, int len) {
    g = reinterpret_cast<const char*>(first);
    end = g + 4 * (int64_t)len;
    const uintptr_t u = reinterpret_cast<uintptr_t>(g), e = reinterpret_cast<uintptr_t>(end);
    lo = g - (u & 15);
    hi = end + (-e & 15);
    in0 = g + (-u & 15);
    in1 = end - (e & 15);
    shift = (int)(u & 15) / 4;
  }
  // offset of p in the column's shared memory (bytes)
  __device__ __forceinline__ int at(const char* p) const { return (int)(p - lo); }
};

template <typename T, int MODE>
__global__ void __launch_bounds__(256, 2)
    simt_shortk_kernel(const SimtArgs<T> a, const __grid_constant__ CUtensorMap tmC) {
  constexpr bool TMA = MODE == SHORTK_TMA, BULK = MODE == SHORTK_BULK;
  static_assert(!BULK || sizeof(T) == 4, "bulk columns: FP32");
  using Cfg = SimtCfg<T>;
  using SC = SimtShortKCfg<T>;
  constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK;
  constexpr int VEC = 16 / sizeof(T);  // elements per 16-byte access
  constexpr int CPI = 256 / BM, CH = 16;  // element path: columns per step, steps at once
  static_assert(BN % (CPI * CH) == 0, "whole steps");
  using Frag = SimtFrag<T, SIMT_SQUARE, false>;
  constexpr int TM = Frag::TM, TN = Frag::TN;
  constexpr int64_t NONE = INT64_MIN;  // offsets may be negative (negative strides)
  static_assert(BN <= 256, "one column offset per thread");
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw_addr + 127u) & ~127u) - raw_addr);  // TMA: 128-byte aligned
  T* Cs = reinterpret_cast<T*>(smem);                                  // [BN][BM]
  int64_t* Cn = reinterpret_cast<int64_t*>(smem + SC::C_BYTES);        // [BN]
  T* As = reinterpret_cast<T*>(smem + SC::C_BYTES + SC::N_BYTES);      // [KP][BM]
  T* Bs = As + (size_t)SC::KP * BM;                                    // [KP][BN]
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + SC::USED - 16);
  const int tid = threadIdx.x;
  const Frag frag(tid);
  const int64_t m0 = (int64_t)blockIdx.x * BM, n0 = (int64_t)blockIdx.y * BN;
  const int kp = a.ktiles * BK;
  const T alpha = a.alpha, beta = a.beta;
  const bool read_c = beta != T(0);

  if constexpr (BULK) {
    if (tid == 0) {
      mbar_init(bar, BN);
      fence_mbar_init();
    }
    __syncthreads();
    if (read_c && tid < BN) {  // column tid; the packing kernel does not write C
      uint32_t bytes = 0;
      if (n0 + tid < a.N) {
        const float* first = a.C + m0 + a.ldc * (n0 + tid);
        const ShortKCol c(first, (int)(a.M - m0 < BM ? a.M - m0 : BM));
        char* dst = reinterpret_cast<char*>(Cs + tid * SC::LDCB);
        const char *b0 = c.lo, *b1 = c.hi;
        if (c.lo < reinterpret_cast<const char*>(a.C) ||
            c.hi > reinterpret_cast<const char*>(a.C + a.M + a.ldc * (a.N - 1))) {
          // an end of C: the aligned range inside the column, edges one by one
          b0 = c.in0;
          b1 = c.in1 > c.in0 ? c.in1 : c.in0;
          for (const char* p = c.g; p < c.end; p += 4)
            if (p < b0 || p >= b1)
              *reinterpret_cast<float*>(dst + c.at(p)) = *reinterpret_cast<const float*>(p);
        }
        bytes = (uint32_t)(b1 - b0);
        if (bytes) {
          mbar_arrive_expect_tx(bar, bytes);
          bulk_load_1d(dst + c.at(b0), b0, bytes, bar);
        }
      }
      if (!bytes) mbar_arrive(bar);
    }
  } else if constexpr (TMA) {
    if (tid == 0) {
      mbar_init(bar, 1);
      fence_mbar_init();
    }
    __syncthreads();
    // the packing kernel before this one does not write C: the block comes
    // in while that kernel may still run
    if (read_c && tid == 0) {
      mbar_arrive_expect_tx(bar, (uint32_t)(BN * BM * sizeof(T)));
      tma_load_2d(Cs, &tmC, (int32_t)m0, (int32_t)n0, bar);
    }
  }
  grid_dep_wait();  // packed operands written by the kernel before
  // operand panels first: their latency runs under the offset loads
  for (int c = tid; c < kp * (BM / VEC); c += 256) {
    const int row = c / (BM / VEC), col = (c % (BM / VEC)) * VEC;
    cp_async_16(As + row * BM + col, a.Ap + (int64_t)row * a.Mp + m0 + col);
  }
  for (int c = tid; c < kp * (BN / VEC); c += 256) {
    const int row = c / (BN / VEC), col = (c % (BN / VEC)) * VEC;
    cp_async_16(Bs + row * BN + col, a.Bp + (int64_t)row * a.Np + n0 + col);
  }
  cp_async_commit();
  // element path: the thread's m and its columns cl + u * CPI
  const int ml = tid % BM, cl = tid / BM;
  int64_t cmo = NONE;
  if constexpr (MODE == SHORTK_ANY) {
    if (tid < BN) Cn[tid] = n0 + tid < a.N ? __ldg(a.c_n_off + n0 + tid) : NONE;
    if (m0 + ml < a.M) cmo = __ldg(a.c_m_off + m0 + ml);
    __syncthreads();  // Cn staged
    if (read_c && cmo != NONE) {
      T* const Cb = a.C + cmo;
#pragma unroll 1
      for (int c1 = cl; c1 < BN; c1 += CPI * CH) {
        int64_t no[CH];  // read before the copies (each clobbers memory)
#pragma unroll
        for (int u = 0; u < CH; ++u) no[u] = Cn[c1 + u * CPI];
#pragma unroll
        for (int u = 0; u < CH; ++u)
          if (no[u] != NONE) cp_async_elem<sizeof(T)>(Cs + (c1 + u * CPI) * BM + ml, Cb + no[u]);
      }
    }
  }
  cp_async_commit();
  cp_async_wait<1>();  // operand panels in place; the C block may still be in flight
  __syncthreads();
  SimtAcc<T, SIMT_SQUARE, false> acc;
  acc.zero();
  for (int k = 0; k < (int)a.K; k += 4)  // the panels are padded with zeros past K
    simt_fma_ktile<T, SIMT_SQUARE, false, 4>(As + k * BM, Bs + k * BN, frag.a_off, frag.b_off, acc);
  if constexpr (TMA || BULK) {
    if (read_c && !mbar_wait(bar, 0)) {
      record_error(a.status, 4);
      return;  // nothing stored; the block's load never completed
    }
  } else {
    cp_async_wait<0>();
    __syncthreads();
  }
  if constexpr (BULK) {
    // element (n, m) at Cs[n LDCB + shift(n) + m]; a thread's 4 columns n, n +
    // 1, .. of a group are 4 lanes' worth apart (same shift, banks 16 apart):
    // lane group ln takes m = 4 lm + (i + ln) % 4
    const int ln = (tid & 31) >> 3;
    const uint32_t s0 = (uint32_t)(reinterpret_cast<uintptr_t>(a.C) / 4) + (uint32_t)m0 +
                        (uint32_t)a.ldc * (uint32_t)n0;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = frag.n(j);
      float* c = Cs + n * SC::LDCB + (int)((s0 + (uint32_t)n * (uint32_t)a.ldc) & 3u) + frag.m0;
#pragma unroll
      for (int g = 0; g < TM; g += 4) {
        float w[4], v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = alpha * acc.get(g + i, j);
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = ln & 1 ? v[(i + 1) & 3] : v[i];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = ln & 2 ? w[(i + 2) & 3] : w[i];
        float* cg = c + 8 * g;  // group g / 4: 32 m further
        if (read_c) {
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] = fma(beta, cg[(i + ln) & 3], v[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) cg[(i + ln) & 3] = v[i];
      }
    }
    fence_proxy_async_smem();
    __syncthreads();
    const int col = tid % BN;
    if (n0 + col >= a.N) return;
    const ShortKCol c(a.C + m0 + a.ldc * (n0 + col), (int)(a.M - m0 < BM ? a.M - m0 : BM));
    const char* src = reinterpret_cast<const char*>(Cs + col * SC::LDCB);
    if (tid < BN) {  // the aligned range inside the column
      if (c.in1 > c.in0) {
        bulk_store_1d(const_cast<char*>(c.in0), src + c.at(c.in0), (uint32_t)(c.in1 - c.in0));
        bulk_commit();
        bulk_wait_read_all();  // shared memory stays valid until the store has read it
      }
    } else {  // its edges: before in0, and from in1 on
      const char* e0 = c.in0 < c.end ? c.in0 : c.end;
      const char* e1 = c.in1 > e0 ? c.in1 : e0;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const char *p = c.g + 4 * i, *q = e1 + 4 * i;
        if (p < e0) *reinterpret_cast<float*>(const_cast<char*>(p)) = *reinterpret_cast<const float*>(src + c.at(p));
        if (q < c.end) *reinterpret_cast<float*>(const_cast<char*>(q)) = *reinterpret_cast<const float*>(src + c.at(q));
      }
    }
    return;
  }
  // combine at the fragment positions: runs of VEC consecutive m (16 bytes)
#pragma unroll
  for (int j = 0; j < TN; ++j)
#pragma unroll
    for (int i0 = 0; i0 < TM; i0 += VEC) {
      T* c = Cs + frag.n(j) * BM + frag.m(i0);
      T v[VEC];
#pragma unroll
      for (int e = 0; e < VEC; ++e) v[e] = alpha * acc.get(i0 + e, j);
      if (read_c) {
        if constexpr (sizeof(T) == 4) {
          const float4 o = *reinterpret_cast<const float4*>(c);
          v[0] = fma(beta, o.x, v[0]); v[1] = fma(beta, o.y, v[1]);
          v[2] = fma(beta, o.z, v[2]); v[3] = fma(beta, o.w, v[3]);
        } else {
          const double2 o = *reinterpret_cast<const double2*>(c);
          v[0] = fma(beta, o.x, v[0]); v[1] = fma(beta, o.y, v[1]);
        }
      }
      if constexpr (sizeof(T) == 4)
        *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
      else
        *reinterpret_cast<double2*>(c) = make_double2(v[0], v[1]);
    }
  if constexpr (TMA) {
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      tma_store_2d(&tmC, Cs, (int32_t)m0, (int32_t)n0);
      bulk_commit();
      bulk_wait_read_all();  // shared memory stays valid until the store has read it
    }
    return;
  }
  __syncthreads();
  if (cmo == NONE) return;
  T* const Cb = a.C + cmo;
#pragma unroll 1
  for (int c1 = cl; c1 < BN; c1 += CPI * CH) {
    int64_t no[CH];  // read before the stores (which may alias as far as the compiler knows)
    T v[CH];
#pragma unroll
    for (int u = 0; u < CH; ++u) {
      no[u] = Cn[c1 + u * CPI];
      v[u] = Cs[(c1 + u * CPI) * BM + ml];
    }
#pragma unroll
    for (int u = 0; u < CH; ++u)
      if (no[u] != NONE) Cb[no[u]] = v[u];
  }
}

// Grouped launch: item i owns CTAs [tile_begin[i], tile_begin[i+1]); the CTA
// finds its item by binary search and runs the same tile code.
template <typename T>
struct SimtGroupItem {
  SimtArgs<T> args;
  int64_t tile_begin;
  int32_t tiles_m, tiles_n;  // tiles of one k-split slice
  int32_t shape;             // SimtShape (FP32 items)
};

// Shared memory of the grouped kernel: the largest of its tile shapes.
template <typename T>
constexpr size_t simt_group_smem_bytes() {
  if constexpr (sizeof(T) == 4) {
    constexpr size_t a = simt_smem_bytes<T, SIMT_SQUARE>(), b = simt_smem_bytes<T, SIMT_NARROW_N>(),
                     c = simt_smem_bytes<T, SIMT_NARROW_M>();
    return a > b ? (a > c ? a : c) : (b > c ? b : c);
  } else {
    return simt_smem_bytes<T, SIMT_SQUARE>();
  }
}

template <typename T>
__global__ void __launch_bounds__(256, 2) simt_gett_group_kernel(const SimtGroupItem<T>* items,
                                                                  const int64_t* begin,
                                                                  int n_items) {
  const int64_t t = blockIdx.x;
  const SimtGroupItem<T>& it = items[find_segment(begin, n_items, t)];
  const int64_t local = t - it.tile_begin;
  const int64_t mn = (int64_t)it.tiles_m * it.tiles_n;
  const int64_t rem = local % mn;
  const int bx = (int)(rem % it.tiles_m), by = (int)(rem / it.tiles_m), bz = (int)(local / mn);
  if constexpr (sizeof(T) == 4) {  // the item's tile shape (uniform over the CTA)
    if (it.shape == SIMT_NARROW_N) {
      simt_gett_tile<T, SIMT_EITHER, SIMT_NARROW_N>(it.args, bx, by, bz);
      return;
    }
    if (it.shape == SIMT_NARROW_M) {
      simt_gett_tile<T, SIMT_EITHER, SIMT_NARROW_M>(it.args, bx, by, bz);
      return;
    }
  }
  simt_gett_tile<T>(it.args, bx, by, bz);
}

// C = alpha * sum_z partial[z] + beta * C.
// grid = (ceil(M/256), min(N, 65535)), block 256; n strides by gridDim.y.
template <typename T>
__global__ void __launch_bounds__(256) simt_reduce_kernel(const T* __restrict__ partial,
                                                          int splits, int64_t Mp, int64_t Np,
                                                          int64_t M, int64_t N, T* C,
                                                          const int64_t* c_m_off,
                                                          const int64_t* c_n_off, T alpha,
                                                          T beta, SplitRange split,
                                                          bool fallback) {
  grid_dep_wait();  // partial sums written by the GETT kernel before
  // an FP32 plan on the tensor cores: its slices, or the fallback's
  if (split.w && f32_split_exact(split) == fallback) return;
  const int64_t m = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (m >= M) return;
  const int64_t cmo = c_m_off[m];
  for (int64_t n = blockIdx.y; n < N; n += gridDim.y) {
    T s = T(0);
#pragma unroll 4
    for (int z = 0; z < splits; ++z) s += partial[(size_t)z * Np * Mp + n * Mp + m];
    T* dst = C + cmo + c_n_off[n];
    T v = alpha * s;
    if (beta != T(0)) v = fma(beta, *dst, v);
    *dst = v;
  }
}

// Grouped k-split reduction: job j (one contraction with a k-split) owns the
// CTAs [begin, begin + mblocks * nblocks); CTA (mb, nb) sums the slices of
// 256 rows over columns [ncols nb, ncols nb + ncols) in split order.
template <typename T>
struct ReduceJob {
  const T* partial;
  int64_t Mp, Np, M, N;
  T* C;
  const int64_t* c_m_off;
  const int64_t* c_n_off;
  T alpha, beta;
  int64_t begin;
  int32_t splits, mblocks;
  int32_t ncols;  // columns per CTA: fewer when there are many slices
  int32_t fallback;  // FP32 on the tensor cores: the fallback's slices, not the split products'
  SplitRange split;  // FP32 on the tensor cores: the item's ranges
};

template <typename T>
__global__ void __launch_bounds__(256) reduce_group_kernel(const ReduceJob<T>* jobs,
                                                           const int64_t* begin, int n_jobs) {
  const int64_t t = blockIdx.x;
  const ReduceJob<T> j = jobs[find_segment(begin, n_jobs, t)];  // fields loaded up front
  if (j.split.w && f32_split_exact(j.split) == (j.fallback != 0)) return;
  const int64_t local = t - j.begin;
  const int64_t m = (local % j.mblocks) * 256 + threadIdx.x;
  if (m >= j.M) return;
  const int64_t n0 = (local / j.mblocks) * j.ncols;
  const int64_t n1 = n0 + j.ncols < j.N ? n0 + j.ncols : j.N;
  const int64_t cmo = j.c_m_off[m];
  for (int64_t n = n0; n < n1; ++n) {
    T s = T(0);
#pragma unroll 4
    for (int z = 0; z < j.splits; ++z) s += j.partial[(size_t)z * j.Np * j.Mp + n * j.Mp + m];
    T* dst = j.C + cmo + j.c_n_off[n];
    T v = j.alpha * s;
    if (j.beta != T(0)) v = fma(j.beta, *dst, v);
    *dst = v;
  }
}

}  // namespace tccg
