// native.cu -- plain-precision GEMM kernels: FP64 on the DMMA tensor-core path
// (mma.sync f64) and FP32 on the FFMA pipes.  They compute
//     C = alpha * op(A) * op(B) + beta * C        (column-major, any ld)
// exactly as Eigen's GEBP store does it (R = alpha*acc + R after the BLAS shim's
// beta pre-scale, Eigen/src/Core/products/GeneralBlockPanelKernel.h:1446-1455,
// blas/level3_impl.h:80-87), with beta == 0 never reading C.  The FP64 kernel is
// the on-device correctness reference for the emulated DGEMM and its fallback for
// inputs with NaN/Inf.
//
// The tile loaders play the role of gemm_pack_lhs/gemm_pack_rhs
// (GeneralBlockPanelKernel.h:1879-2478): they read op(A)/op(B) through lda/ldb and
// the transpose flags and write one fixed shared-memory layout, so the inner
// product loop is the same for NN/NT/TN/TT.
#include <climits>
#include <utility>

#include "device_common.cuh"
#include "kernels.h"

namespace eb2 {

namespace {

// ------------------------------------------------------------------ FP64 DMMA
// BM x BN output tiles, K in tiles of 16 through a shared-memory ring, warp-specialised:
// producer warps copy the tiles with cp.async (any alignment and leading dimension; edges
// zero-filled) and hand each stage over with cp.async.mbarrier.arrive on its `full` barrier;
// consumer warps (WM x WN outputs each) wait on `full`, run DMMA m16n8k4 with K in steps of 4
// from 0 upward for every output, and release the stage on its `empty` barrier.  No block-wide
// barrier in the main loop: measured, the copy issue and the per-tile __syncthreads of a
// cooperative ring cost a fifth of the DMMA rate.  Shared memory follows each operand's
// contiguous direction in global memory ([k][m] when op(A) is stored column-major, [m][k] when
// transposed; likewise for op(B)), padded so that the 64-bit fragment loads of each half-warp
// hit distinct banks.  Every wait is bounded (kWaitLimitNs); one that runs out records
// EB2_DEV_ERR_TIMEOUT in *status and the roles leave.
//
// An output's sum does not depend on the tile it lies in (the same K order), so the tile size is
// chosen by the work per SM alone (dmma_tile).
constexpr int kDBK = 16;
constexpr int kDPadK = kDBK + 4;  // [m or n][k] row stride (doubles)

template <int BM_, int BN_, int WM_, int WN_, int PW_, int ST_, int BLOCKS_>
struct DTile {
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_;
  static constexpr int kProducerWarps = PW_, kStages = ST_, kBlocksPerSm = BLOCKS_;
  static constexpr int kWarpsM = BM / WM, kWarpsN = BN / WN;
  static constexpr int kConsumerWarps = kWarpsM * kWarpsN;
  static constexpr int kThreads = 32 * (kConsumerWarps + kProducerWarps);
  static constexpr int kPadM = BM + 4, kPadN = BN + 4;  // [k][m or n] row strides (doubles)
  static constexpr int kAElems = kDBK * kPadM > BM * kDPadK ? kDBK * kPadM : BM * kDPadK;
  static constexpr int kBElems = kDBK * kPadN > BN * kDPadK ? kDBK * kPadN : BN * kDPadK;
  static constexpr int kGroupM = 1024 / BM;  // tile rows per raster group
  struct Smem {
    double a[kStages][kAElems];
    double b[kStages][kBElems];
    uint64_t full[kStages], empty[kStages];
    int abort_flag;
  };
};
using DTile128 = DTile<128, 128, 64, 32, 4, 4, 1>;
using DTile64 = DTile<64, 64, 32, 16, 4, 4, 2>;
using DTile32 = DTile<32, 32, 16, 16, 2, 6, 3>;

// where a native-kernel wait that ran out is recorded when the caller passes no status word
__device__ uint32_t g_native_status;

__device__ __forceinline__ void dmma_16x8x4(double (&d)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// The producer warps' copies of one K tile (ROWS rows) of one operand (rows x k view at X,
// leading dimension ld).  MN_CONTIG: the operand's m (or n) index is the contiguous one in global
// memory (op(A) = A column-major, op(B) = B^T of a column-major B).  V = 2: 16-byte copies of
// two neighbours along the contiguous index (X 16-byte aligned, ld even); a pair that
// straddles the edge copies its first element and zero-fills the second.
template <int ROWS, int PRODUCERS, bool MN_CONTIG, int V>
__device__ __forceinline__ void dcopy_operand(double* st, const double* __restrict__ X, int64_t ld, int64_t rows,
                                              int64_t k, int64_t r0, int64_t k0, int pt) {
  constexpr int kPT = 32 * PRODUCERS, kPad = ROWS + 4;
  constexpr int kRowsV = MN_CONTIG ? ROWS / V : ROWS, kColsV = MN_CONTIG ? kDBK : kDBK / V;
  constexpr int kCopies = kRowsV * kColsV / kPT;
  // thread pt copies a fixed contiguous-direction offset and steps through the other index
  // (kStep columns of K, or kStep rows) from copy to copy
  constexpr int kStep = MN_CONTIG ? kPT / kRowsV : kPT / kColsV;
  static_assert(kPT % (MN_CONTIG ? kRowsV : kColsV) == 0 && kCopies * kPT == kRowsV * kColsV,
                "fixed contiguous offset per thread");
  const int c_off = (pt % (MN_CONTIG ? kRowsV : kColsV)) * V;  // along the contiguous index
  const int s_first = pt / (MN_CONTIG ? kRowsV : kColsV);      // first value of the stepped index
  const int64_t g_c = (MN_CONTIG ? r0 : k0) + c_off, g_s = (MN_CONTIG ? k0 : r0) + s_first;
  const int64_t lim_c = MN_CONTIG ? rows : k, lim_s = MN_CONTIG ? k : rows;
  // elements of the contiguous pair inside the matrix (0, 1 or V); the same for every copy
  const int in_c = g_c + V <= lim_c ? V : (g_c < lim_c ? int(lim_c - g_c) : 0);
  const double* src = X + g_c + g_s * ld;
  const int64_t src_step = int64_t(kStep) * ld;
  uint32_t dst = smem_u32(MN_CONTIG ? st + s_first * kPad + c_off : st + s_first * kDPadK + c_off);
  constexpr uint32_t kDstStep = uint32_t(kStep * (MN_CONTIG ? kPad : kDPadK) * 8);
#pragma unroll
  for (int i = 0; i < kCopies; ++i, src += src_step, dst += kDstStep) {
    const int in = (g_s + int64_t(i) * kStep < lim_s) ? in_c : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(dst), "l"(in ? src : X), "n"(8 * V),
                 "r"(8 * in)
                 : "memory");
  }
}

// Tile t of the grid in groups of `group` tile rows (column-major inside a group), so that
// the CTAs in flight share A panels in L2 as well as B panels.
__device__ __forceinline__ void dtile_coords(int64_t t, int group, int64_t tiles_m, int64_t tiles_n, int64_t& tm,
                                             int64_t& tn) {
  const int64_t per_group = int64_t(group) * tiles_n;
  const int64_t first_m = (t / per_group) * group;
  const int64_t gm = tiles_m - first_m < group ? tiles_m - first_m : group;
  const int64_t r = t % per_group;
  tm = first_m + r % gm;
  tn = r / gm;
}

template <class D, bool TA, bool TB, int VA, int VB>
__global__ void __launch_bounds__(D::kThreads, D::kBlocksPerSm)
    dgemm_dmma_kernel(int64_t m, int64_t n, int64_t k, double alpha, const double* __restrict__ A, int64_t lda,
                      const double* __restrict__ B, int64_t ldb, double beta, double* __restrict__ C, int64_t ldc,
                      const int* only_if_flag, uint32_t* status) {
  if (only_if_flag && *only_if_flag == 0) return;
  extern __shared__ __align__(16) uint8_t dsmem_raw[];
  typename D::Smem& s = *reinterpret_cast<typename D::Smem*>(dsmem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int64_t tm, tn;
  dtile_coords(blockIdx.x, D::kGroupM, (m + D::BM - 1) / D::BM, (n + D::BN - 1) / D::BN, tm, tn);
  const int64_t m0 = tm * D::BM, n0 = tn * D::BN;
  // op(A) m-contiguous unless transposed; op(B)'s n index is contiguous only when transposed
  constexpr bool kAmn = !TA, kBmn = TB;
  uint32_t* const st_word = status ? status : &g_native_status;
  volatile int* const abort_flag = &s.abort_flag;
  if (threadIdx.x == 0) {
    for (int i = 0; i < D::kStages; ++i) {
      mbar_init(&s.full[i], 32 * D::kProducerWarps);  // one cp.async arrival per producer thread
      mbar_init(&s.empty[i], D::kConsumerWarps);      // one arrival per consumer warp
    }
    s.abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();
  const int64_t nkt = (k + kDBK - 1) / kDBK;
  int stg = 0;          // stage of K tile kt
  uint32_t phase = 0u;  // its use count's parity

  if (warp >= D::kConsumerWarps) {
    // producers: tile kt into its stage once the consumers released the stage's previous use
    const int pt = int(threadIdx.x) - 32 * D::kConsumerWarps;
    for (int64_t kt = 0; kt < nkt; ++kt) {
      if (kt >= D::kStages && !mbar_wait(&s.empty[stg], phase ^ 1u, abort_flag, st_word)) break;
      dcopy_operand<D::BM, D::kProducerWarps, kAmn, VA>(s.a[stg], A, lda, m, k, m0, kt * kDBK, pt);
      dcopy_operand<D::BN, D::kProducerWarps, kBmn, VB>(s.b[stg], B, ldb, n, k, n0, kt * kDBK, pt);
      cp_async_mbar_arrive(&s.full[stg]);
      if (++stg == D::kStages) {
        stg = 0;
        phase ^= 1u;
      }
    }
    cp_async_wait_all();  // no copy outlives the block
    return;
  }

  constexpr int kMI = D::WM / 16, kNJ = D::WN / 8;
  const int wm = warp % D::kWarpsM, wn = warp / D::kWarpsM;
  const int g = lane >> 2, tig = lane & 3;
  double acc[kMI][kNJ][4];
#pragma unroll
  for (int i = 0; i < kMI; ++i)
#pragma unroll
    for (int j = 0; j < kNJ; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.0;

  bool ok = true;
  for (int64_t kt = 0; kt < nkt && ok; ++kt) {
    if (!mbar_wait(&s.full[stg], phase, abort_flag, st_word)) {
      ok = false;
      break;
    }
    const double* sa = s.a[stg];
    const double* sb = s.b[stg];
#pragma unroll
    for (int ks = 0; ks < kDBK / 4; ++ks) {
      const int kk = ks * 4 + tig;
      double af[kMI][2], bf[kNJ];
#pragma unroll
      for (int i = 0; i < kMI; ++i) {
        const int r = wm * D::WM + i * 16 + g;
        af[i][0] = kAmn ? sa[kk * D::kPadM + r] : sa[r * kDPadK + kk];
        af[i][1] = kAmn ? sa[kk * D::kPadM + r + 8] : sa[(r + 8) * kDPadK + kk];
      }
#pragma unroll
      for (int j = 0; j < kNJ; ++j) {
        const int c = wn * D::WN + j * 8 + g;
        bf[j] = kBmn ? sb[kk * D::kPadN + c] : sb[c * kDPadK + kk];
      }
#pragma unroll
      for (int i = 0; i < kMI; ++i)
#pragma unroll
        for (int j = 0; j < kNJ; ++j) dmma_16x8x4(acc[i][j], af[i][0], af[i][1], bf[j]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&s.empty[stg]);
    if (++stg == D::kStages) {
      stg = 0;
      phase ^= 1u;
    }
  }
  if (!ok) return;  // C is left as it was; the status word records the timeout

  // epilogue: C = alpha*acc + beta*C
#pragma unroll
  for (int i = 0; i < kMI; ++i)
#pragma unroll
    for (int j = 0; j < kNJ; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t row = m0 + wm * D::WM + i * 16 + g + h * 8;
        if (row >= m) continue;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int64_t col = n0 + wn * D::WN + j * 8 + tig * 2 + c;
          if (col >= n) continue;
          double* dst = C + row + col * ldc;
          const double v = __dmul_rn(alpha, acc[i][j][h * 2 + c]);
          *dst = (beta == 0.0) ? v : __fma_rn(beta, *dst, v);
        }
      }
}

// ------------------------------------------------------------------ FP32 FFMA
constexpr int kSBM = 128, kSBN = 128, kSBK = 8, kSThreads = 256;

template <bool TA, bool TB>
__global__ void __launch_bounds__(kSThreads)
    sgemm_ffma_kernel(int64_t m, int64_t n, int64_t k, float alpha, const float* __restrict__ A, int64_t lda,
                      const float* __restrict__ B, int64_t ldb, float beta, float* __restrict__ C, int64_t ldc,
                      const int* only_if_flag) {
  if (only_if_flag && *only_if_flag == 0) return;
  __shared__ float sa[2][kSBK][kSBM + 4];
  __shared__ float sb[2][kSBK][kSBN + 4];
  const int t = threadIdx.x;
  const int tx = t % 16, ty = t / 16;  // 16 x 16 threads, 8 x 8 outputs each
  const int64_t m0 = int64_t(blockIdx.x) * kSBM, n0 = int64_t(blockIdx.y) * kSBN;
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;

  float ra[4], rb[4];
  auto load = [&](int64_t k0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = t + kSThreads * i;
      int mm, kk;
      if (!TA) {
        mm = idx % kSBM;
        kk = idx / kSBM;
      } else {
        kk = idx % kSBK;
        mm = idx / kSBK;
      }
      const int64_t gm = m0 + mm, gk = k0 + kk;
      ra[i] = (gm < m && gk < k) ? (TA ? A[gk + gm * lda] : A[gm + gk * lda]) : 0.f;
      int nn;
      if (!TB) {
        kk = idx % kSBK;
        nn = idx / kSBK;
      } else {
        nn = idx % kSBN;
        kk = idx / kSBN;
      }
      const int64_t gn = n0 + nn, gk2 = k0 + kk;
      rb[i] = (gn < n && gk2 < k) ? (TB ? B[gn + gk2 * ldb] : B[gk2 + gn * ldb]) : 0.f;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = t + kSThreads * i;
      int mm, kk;
      if (!TA) {
        mm = idx % kSBM;
        kk = idx / kSBM;
      } else {
        kk = idx % kSBK;
        mm = idx / kSBK;
      }
      sa[buf][kk][mm] = ra[i];
      int nn;
      if (!TB) {
        kk = idx % kSBK;
        nn = idx / kSBK;
      } else {
        nn = idx % kSBN;
        kk = idx / kSBN;
      }
      sb[buf][kk][nn] = rb[i];
    }
  };
  const int64_t nkt = (k + kSBK - 1) / kSBK;
  load(0);
  store(0);
  __syncthreads();
  for (int64_t kt = 0; kt < nkt; ++kt) {
    const int buf = int(kt & 1);
    if (kt + 1 < nkt) load((kt + 1) * kSBK);
#pragma unroll
    for (int kk = 0; kk < kSBK; ++kk) {
      float av[8], bv[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        av[i] = sa[buf][kk][ty * 4 + i];
        av[i + 4] = sa[buf][kk][64 + ty * 4 + i];
        bv[i] = sb[buf][kk][tx * 4 + i];
        bv[i + 4] = sb[buf][kk][64 + tx * 4 + i];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    if (kt + 1 < nkt) store(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t row = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4);
    if (row >= m) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int64_t col = n0 + (j < 4 ? tx * 4 + j : 64 + tx * 4 + j - 4);
      if (col >= n) continue;
      float* dst = C + row + col * ldc;
      const float v = __fmul_rn(alpha, acc[i][j]);
      *dst = (beta == 0.f) ? v : __fmaf_rn(beta, *dst, v);
    }
  }
}

// ------------------------------------------------------------------ FP32, small products
// One launch with FP32 inputs and sums, for products too small to fill the tensor cores with
// split-BF16 pieces (a split, a GEMM whose K blocks follow one another on a few SMs, a sum of K
// ranges and a fallback launch: 23 us and more of device time).  The eight warps of a block share
// a 32 x 32 output tile and split K: each warp computes all 32 x 32 outputs (8 x 4 per lane) over
// its 8 of every K tile's 64.  K tiles arrive by cp.async in a ring of kFStages; shared memory is
// [k][row] for both operands, so a lane's rows and columns are 16-byte loads.  A lane adds its
// products 32 K steps at a time (FMA chains) into running sums, and the eight partial sums are
// added in a fixed order through shared memory, so rounding errors grow with sqrt(32) and
// sqrt(K / 256) instead of sqrt(K).  Bound by issue slots: 35 instructions per K step and warp for
// 1024 FMAs, plus the copies, so a copy is one address and one predicated instruction.
constexpr int kFTile = 32, kFWarps = 8, kFThreads = 32 * kFWarps;
constexpr int kFKW = 8, kFKT = kFWarps * kFKW;  // K per warp and per tile
constexpr int kFLd = kFTile + 4;                // [k] row stride (floats)
constexpr int kFStages = 4, kFChunk = 32;
constexpr int kFStage = 2 * kFKT * kFLd;        // floats
constexpr int kFSmem = 4 * kFStages * kFStage;
static_assert(kFWarps * kFTile * kFLd * 4 <= kFSmem, "the sums are staged in the ring");

// The copies of one operand (rows x k view at X, tile rows r0 .. r0+31), K tile after K tile:
// element (r, kk) of a tile to dst[kk * kFLd + r].  MN_CONTIG: the rows are contiguous in global
// memory, and a warp takes the 32 rows of a K offset; else the K index is, and a warp takes 8
// neighbours along K of 4 rows (distinct banks).  Rows outside the matrix are not copied (their
// outputs are not stored); the K tail is zero-filled.
template <bool MN_CONTIG>
struct FCopy {
  static constexpr int kCopies = kFTile * kFKT / kFThreads;  // K offsets kk, kk + 8, ... of one row
  const char* src;  // first copy of the next tile
  int64_t step;     // bytes from copy to copy
  int left;         // K elements from the thread's first one to the end
  uint32_t dst;
  int row_ok;
  __device__ __forceinline__ void start(const float* x, int64_t ld, int64_t rows, int64_t k, int64_t r0, int t) {
    const int r = MN_CONTIG ? t % 32 : ((t >> 3) & 3) + 4 * (t >> 5), kk = MN_CONTIG ? t / 32 : t & 7;
    row_ok = r0 + r < rows ? 1 : 0;
    left = int(k) - kk;
    step = MN_CONTIG ? 8 * ld * 4 : 32;
    src = reinterpret_cast<const char*>(MN_CONTIG ? x + (r0 + r) + kk * ld : x + kk + (r0 + r) * ld);
    dst = uint32_t((kk * kFLd + r) * 4);
  }
  template <int... q>
  __device__ __forceinline__ void whole(uint32_t d, std::integer_sequence<int, q...>) const {
    (cp_async_elem_if<4, q * 8 * kFLd * 4>(d, src + q * step, 0, row_ok), ...);
  }
  __device__ __forceinline__ void issue(uint32_t stage, const void* any) {
    const uint32_t d = stage + dst;
    if (left > (kCopies - 1) * 8) {  // every K offset of the tile inside
      whole(d, std::make_integer_sequence<int, kCopies>{});
    } else {
#pragma unroll
      for (int q = 0; q < kCopies; ++q) {
        const bool in = left > 8 * q;
        cp_async_fill_if<4>(d + uint32_t(q * 8 * kFLd * 4), in ? src + q * step : any, in ? 4 : 0, 0, row_ok);
      }
    }
    src += kCopies * step;
    left -= kFKT;
  }
};

template <bool TA, bool TB>
__global__ void __launch_bounds__(kFThreads, 2)
    sgemm_small_kernel(int64_t m, int64_t n, int64_t k, float alpha, const float* __restrict__ A, int64_t lda,
                       const float* __restrict__ B, int64_t ldb, float beta, float* __restrict__ C, int64_t ldc) {
  extern __shared__ __align__(16) float fsmem[];
  const int t = int(threadIdx.x), warp = t >> 5, lane = t & 31;
  const int ty = lane >> 3, tx = lane & 7;  // rows 4 ty .., 16 + 4 ty ..; columns 4 tx ..
  const int64_t m0 = int64_t(blockIdx.x) * kFTile, n0 = int64_t(blockIdx.y) * kFTile;
  const int nkt = int((k + kFKT - 1) / kFKT);
  FCopy<!TA> ca;
  FCopy<TB> cb;
  ca.start(A, lda, m, k, m0, t);
  cb.start(B, ldb, n, k, n0, t);
  const uint32_t ring = smem_u32(fsmem);
  auto copy = [&](int stage) {
    const uint32_t st = ring + uint32_t(stage * kFStage * 4);
    ca.issue(st, A);
    cb.issue(st + uint32_t(kFKT * kFLd * 4), B);
  };
#pragma unroll
  for (int s = 0; s < kFStages - 1; ++s) {
    if (s < nkt) copy(s);
    cp_async_commit();
  }
  float c[8][4], sum[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) c[i][j] = sum[i][j] = 0.f;
  auto flush = [&]() {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sum[i][j] += c[i][j];
        c[i][j] = 0.f;
      }
  };
  int stage = 0;
  for (int kt = 0; kt < nkt; ++kt) {
    cp_async_wait<kFStages - 2>();
    __syncthreads();  // tile kt has landed for everyone; the slot refilled below is free
    if (kt + kFStages - 1 < nkt) copy(stage == 0 ? kFStages - 1 : stage - 1);
    cp_async_commit();
    const float* sa = fsmem + stage * kFStage + warp * kFKW * kFLd + ty * 4;
    const float* sb = fsmem + stage * kFStage + (kFKT + warp * kFKW) * kFLd + tx * 4;
#pragma unroll
    for (int kk = 0; kk < kFKW; ++kk) {
      const float4 a0 = *reinterpret_cast<const float4*>(sa + kk * kFLd);
      const float4 a1 = *reinterpret_cast<const float4*>(sa + kk * kFLd + 16);
      const float4 b0 = *reinterpret_cast<const float4*>(sb + kk * kFLd);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, bv[4] = {b0.x, b0.y, b0.z, b0.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] = fmaf(av[i], bv[j], c[i][j]);
    }
    if ((kt + 1) % (kFChunk / kFKW) == 0) flush();
    stage = stage == kFStages - 1 ? 0 : stage + 1;
  }
  flush();
  cp_async_wait<0>();
  __syncthreads();  // the ring becomes the staging of the sums: [warp][column][row]
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float* p = fsmem + (warp * kFTile + tx * 4 + j) * kFLd + ty * 4;
    *reinterpret_cast<float4*>(p) = make_float4(sum[0][j], sum[1][j], sum[2][j], sum[3][j]);
    *reinterpret_cast<float4*>(p + 16) = make_float4(sum[4][j], sum[5][j], sum[6][j], sum[7][j]);
  }
  __syncthreads();
  constexpr int kOut = kFTile * kFTile / kFThreads;  // outputs of a thread: row r, columns c0, c0 + 8, ..
  const int r = t % kFTile, c0 = t / kFTile;
  float v[kOut];
  bool lost = false;  // an output of the product is not finite
#pragma unroll
  for (int q = 0; q < kOut; ++q) {
    const int cc = c0 + 8 * q;
    v[q] = fsmem[cc * kFLd + r];
#pragma unroll
    for (int w = 1; w < kFWarps; ++w) v[q] += fsmem[(w * kFTile + cc) * kFLd + r];
    lost |= m0 + r < m && n0 + cc < n && !isfinite(v[q]);
  }
  if (__any_sync(0xffffffffu, lost)) {
    // Partial sums that overflow with both signs add up to NaN.  One chain of FMAs keeps the infinity it
    // reaches first, as the FFMA kernel's does; where NaN and Inf come from the operands it gives the
    // same.  Rare, so a warp reads its operands again from global memory (edges clamped).
    const int64_t row = m0 + r < m ? m0 + r : m - 1;
    const float* ap = TA ? A + row * lda : A + row;
    const float* bp[kOut];
    float s[kOut];
#pragma unroll
    for (int q = 0; q < kOut; ++q) {
      const int64_t col = n0 + c0 + 8 * q < n ? n0 + c0 + 8 * q : n - 1;
      bp[q] = TB ? B + col : B + col * ldb;
      s[q] = 0.f;
    }
    const int64_t sa = TA ? 1 : lda, sb = TB ? ldb : 1;
#pragma unroll 8
    for (int64_t l = 0; l < k; ++l) {
      const float a = ap[l * sa];
#pragma unroll
      for (int q = 0; q < kOut; ++q) s[q] = fmaf(a, bp[q][l * sb], s[q]);
    }
#pragma unroll
    for (int q = 0; q < kOut; ++q)
      if (!isfinite(v[q])) v[q] = s[q];
  }
#pragma unroll
  for (int q = 0; q < kOut; ++q) {
    const int cc = c0 + 8 * q;
    if (m0 + r < m && n0 + cc < n) {
      float* dst = C + (m0 + r) + (n0 + cc) * ldc;
      const float x = __fmul_rn(alpha, v[q]);
      *dst = (beta == 0.f) ? x : __fmaf_rn(beta, *dst, x);
    }
  }
}

template <typename T>
__global__ void scale_matrix_kernel(int64_t m, int64_t n, T beta, T* C, int64_t ldc) {
  const int64_t total = m * n;
  for (int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += int64_t(gridDim.x) * blockDim.x) {
    const int64_t i = idx % m, j = idx / m;
    T* p = C + i + j * ldc;
    *p = (beta == T(0)) ? T(0) : T(beta * *p);
  }
}

}  // namespace

namespace {

// 16-byte copies where the operand allows them
bool dmma_wide(const double* X, int64_t ld) { return reinterpret_cast<uintptr_t>(X) % 16 == 0 && ld % 2 == 0; }

template <class D>
cudaError_t launch_dmma(bool transA, bool transB, int64_t m, int64_t n, int64_t k, double alpha, const double* A,
                        int64_t lda, const double* B, int64_t ldb, double beta, double* C, int64_t ldc,
                        const int* only_if_flag, cudaStream_t stream) {
  const int64_t tiles = ((m + D::BM - 1) / D::BM) * ((n + D::BN - 1) / D::BN);
  if (tiles > 0x7FFFFFFF) return cudaErrorInvalidConfiguration;
  const int smem = int(sizeof(typename D::Smem));
  auto pick = [&](auto kern) -> cudaError_t {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    kern<<<unsigned(tiles), D::kThreads, smem, stream>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, only_if_flag,
                                                         nullptr);
    return cudaGetLastError();
  };
  const bool va = dmma_wide(A, lda), vb = dmma_wide(B, ldb);
  auto by_vec = [&](auto k11, auto k12, auto k21, auto k22) -> cudaError_t {
    if (va) return vb ? pick(k22) : pick(k21);
    return vb ? pick(k12) : pick(k11);
  };
#define EB2_DMMA_VARIANTS(TA_, TB_)                                                                               \
  by_vec(dgemm_dmma_kernel<D, TA_, TB_, 1, 1>, dgemm_dmma_kernel<D, TA_, TB_, 1, 2>,                              \
         dgemm_dmma_kernel<D, TA_, TB_, 2, 1>, dgemm_dmma_kernel<D, TA_, TB_, 2, 2>)
  if (!transA && !transB) return EB2_DMMA_VARIANTS(false, false);
  if (transA && !transB) return EB2_DMMA_VARIANTS(true, false);
  if (!transA && transB) return EB2_DMMA_VARIANTS(false, true);
  return EB2_DMMA_VARIANTS(true, true);
#undef EB2_DMMA_VARIANTS
}

}  // namespace

int dmma_tile(int64_t m, int64_t n, int64_t k, bool wide) {
  // The side whose busiest SM has the least work, tiles per SM (rounded up) times the tile's area,
  // weighted by how far each size falls short of the DMMA rate when the chip is full (4096 x 4096 x
  // 1024: 1033, 1056 and 1209 us for sides 128, 64 and 32).  Measured with 128 / 64 / 32 (us): 128^3
  // 24.7 / 10.4 / 6.3; 512^3 78 / 24.7 / 16.5; 768^3 115 / 35.0 / 41.7; 1000 x 1531 x 777 117 / 95 /
  // 103; 1536 x 1536 x 256 43.1 / 44.1 / 53.3.
  constexpr int64_t kSms = 148;
  auto tiles = [&](int64_t side) { return ((m + side - 1) / side) * ((n + side - 1) / side); };
  auto cost = [&](int64_t side, double weight) {
    return double((tiles(side) + kSms - 1) / kSms) * double(side * side) * weight;
  };
  const double c128 = cost(128, 1.0), c64 = cost(64, 1.02), c32 = cost(32, 1.2);
  if (c32 < c64 && c32 < c128) return 32;
  if (c64 >= c128) return 128;
  // A shallow product is its tiles' fill, first copies and stores: a wave of 128 tiles takes 5 us and
  // 2.3 us per K tile, a wave of 64 tiles (two on an SM) 2.9 and 1.15 us (us, 128 / 64: 2048 x 2048 x
  // 32 19.0 / 20.2, 2500 x 2500 x 16 21.0 / 22.1, 3000 x 3000 x 20 36.8 / 39.0, but 1700 x 1700 x 32
  // 18.7 / 15.3, 1000 x 1000 x 16 7.7 / 4.9).  Many waves are bound by the copies and stores, where
  // 8-byte copies favour the smaller tile (7000 x 7000 x 4: 140 / 148 aligned, 173 / 165 not).
  if (k <= 64) {
    const double kt = double((k + kDBK - 1) / kDBK);
    const int64_t w128 = (tiles(128) + kSms - 1) / kSms, w64 = (tiles(64) + 2 * kSms - 1) / (2 * kSms);
    if ((wide || w128 <= 6) && double(w128) * (5.0 + 2.3 * kt) < double(w64) * (2.9 + 1.15 * kt)) return 128;
  }
  return 64;
}

cudaError_t launch_dgemm_native(bool transA, bool transB, int64_t m, int64_t n, int64_t k, double alpha,
                                const double* A, int64_t lda, const double* B, int64_t ldb, double beta, double* C,
                                int64_t ldc, const int* only_if_flag, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  // a launch that will usually leave at once (only_if_flag) takes the fewest blocks
  const int tile = only_if_flag ? 128 : dmma_tile(m, n, k, dmma_wide(A, lda) && dmma_wide(B, ldb));
  auto go = [&](auto d) {
    return launch_dmma<decltype(d)>(transA, transB, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, only_if_flag,
                                    stream);
  };
  if (tile == 32) return go(DTile32{});
  if (tile == 64) return go(DTile64{});
  return go(DTile128{});
}

cudaError_t launch_sgemm_native(bool transA, bool transB, int64_t m, int64_t n, int64_t k, float alpha,
                                const float* A, int64_t lda, const float* B, int64_t ldb, float beta, float* C,
                                int64_t ldc, const int* only_if_flag, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  dim3 grid(unsigned((m + kSBM - 1) / kSBM), unsigned((n + kSBN - 1) / kSBN));
  if (grid.y > 65535u) return cudaErrorInvalidConfiguration;
  if (!transA && !transB)
    sgemm_ffma_kernel<false, false><<<grid, kSThreads, 0, stream>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc,
                                                                     only_if_flag);
  else if (transA && !transB)
    sgemm_ffma_kernel<true, false><<<grid, kSThreads, 0, stream>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc,
                                                                    only_if_flag);
  else if (!transA && transB)
    sgemm_ffma_kernel<false, true><<<grid, kSThreads, 0, stream>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc,
                                                                    only_if_flag);
  else
    sgemm_ffma_kernel<true, true><<<grid, kSThreads, 0, stream>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc,
                                                                   only_if_flag);
  return cudaGetLastError();
}

bool sgemm_small_applies(int64_t m, int64_t n, int64_t k) {
  // Rounds of tiles over the SMs times K, up to where split-BF16 takes over (device time, us, this
  // kernel / split-BF16 or the FFMA kernel before): 64^3 2.9 / 11.6, 128^3 3.9 / 26.2, 256^3 5.7 /
  // 24.8, 384^3 7.4 / 23.3, 512^3 16.0 / 23.7, 32 x 4096 x 1024 16.1 / 27.7; past the line
  // 300 x 517 x 1100 33 / 26.9, 640^3 28.9 / 25.8.  And not too many rounds, since a round costs a
  // whole K tile and the sum of the shares (0.75 us each) however short K is, while the other
  // kernels' time steps up past K = 64 (a call, us): 1216^2 x 32 (10 rounds) 18.5 / 18.9, 1344^2 x 32
  // (12) 22.6 / 18.9, 3000^2 x 4 (60) 96 / 35, 6000^2 x 4 (239) 374 / 83; 1216^2 x 100 25.7 / 29.8,
  // 1344^2 x 100 30.8 / 29.9, 1536^2 x 75 (16) 39 / 32.
  const int64_t tiles = ((m + kFTile - 1) / kFTile) * ((n + kFTile - 1) / kFTile), rounds = (tiles + 147) / 148;
  return (n + kFTile - 1) / kFTile <= 65535 && rounds * k <= 1200 && rounds <= (k <= kFKT ? 10 : 11);
}

cudaError_t launch_sgemm_small(bool transA, bool transB, int64_t m, int64_t n, int64_t k, float alpha, const float* A,
                               int64_t lda, const float* B, int64_t ldb, float beta, float* C, int64_t ldc,
                               cudaStream_t stream) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  const dim3 grid(unsigned((m + kFTile - 1) / kFTile), unsigned((n + kFTile - 1) / kFTile));
  if (grid.y > 65535u || k > INT_MAX / 2) return cudaErrorInvalidConfiguration;
  auto pick = [&](auto kern) -> cudaError_t {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kFSmem);
    if (e != cudaSuccess) return e;
    kern<<<grid, kFThreads, kFSmem, stream>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    return cudaGetLastError();
  };
  if (!transA && !transB) return pick(sgemm_small_kernel<false, false>);
  if (transA && !transB) return pick(sgemm_small_kernel<true, false>);
  if (!transA) return pick(sgemm_small_kernel<false, true>);
  return pick(sgemm_small_kernel<true, true>);
}

cudaError_t launch_scale_matrix_d(int64_t m, int64_t n, double beta, double* C, int64_t ldc, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  const int64_t total = m * n;
  const int blocks = int(total / 256 + 1 < 148 * 16 ? total / 256 + 1 : 148 * 16);
  scale_matrix_kernel<double><<<blocks, 256, 0, stream>>>(m, n, beta, C, ldc);
  return cudaGetLastError();
}

cudaError_t launch_scale_matrix_s(int64_t m, int64_t n, float beta, float* C, int64_t ldc, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  const int64_t total = m * n;
  const int blocks = int(total / 256 + 1 < 148 * 16 ? total / 256 + 1 : 148 * 16);
  scale_matrix_kernel<float><<<blocks, 256, 0, stream>>>(m, n, beta, C, ldc);
  return cudaGetLastError();
}

}  // namespace eb2
