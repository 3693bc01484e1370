// split_bf16.cu -- SGEMM emulated on the BF16 tensor cores (split-BF16).
//
// Method (Henry, Tang & Heinecke, "Leveraging the bfloat16 Artificial Intelligence
// Datatype For Higher-Precision Computations", ARITH 2019): every FP32 input x is
// written exactly as the sum of three BF16 pieces
//     h = bf16(x),  m = bf16(x - h),  l = bf16(x - h - m),
// (each difference is exact in FP32).  The product keeps the pieces' cross products
// with p + q <= s + 1 (pieces numbered h = 1, m = 2, l = 3): s = 2 gives the three
// products hh + hm + mh ("bf16x3"), s = 3 adds mm + hl + lh ("bf16x6").  All of them
// accumulate in FP32 in one TMEM accumulator of the shared slice GEMM, smallest
// products first, and the epilogue applies C = alpha*acc + beta*C.
// The split is the GPU counterpart of Eigen's gemm_pack_lhs/gemm_pack_rhs
// (Eigen/src/Core/products/GeneralBlockPanelKernel.h:1879-2478): it reads op(A)/op(B)
// through ld and the transpose flags and writes K-major zero-padded panels.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "device_common.cuh"
#include "kernels.h"
#include "slice_gemm.cuh"
#include "tma_host.h"

namespace eb2 {

namespace {

constexpr int kBRows = 32;
constexpr int kBCols = 64;  // K elements per tile = 128 bytes of one BF16 piece

// Both operands of a product, walked by one launch: tile t belongs to operand `t >= tiles0`.
struct SplitOperand {
  const float* X;  // element (r, l) at X[r*sr + l*sl], rows x cols
  int64_t rows, cols, sr, sl, rows_pad, k_pad;
  __nv_bfloat16* pieces;
  unsigned tiles_l;  // tiles along K
  int vec;           // 16-byte loads along the contiguous index (X aligned, stride a multiple of 4)
};
struct SplitArgs {
  SplitOperand op[2];
  unsigned tiles0;
};

// The pieces of two values, packed as bf16x2 (first value in the low half).
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// A 32 x 64 tile per block, 8 neighbours along K per thread; each piece plane receives 128
// contiguous bytes per row.  An operand stored along K is read straight into registers, one stored
// along its rows through shared memory.  Bound by issue slots, so the pieces are formed two values
// to a conversion (11 instructions per pair, half of the scalar form) and the NaN/Inf test is one
// running maximum of packed exponents.  4096 x 4096 x 4096 with both splits: 767 -> 742 us a call.
__global__ void __launch_bounds__(256) bf16_split_kernel(const __grid_constant__ SplitArgs args, int* nonfinite) {
  __shared__ float tile[kBRows][kBCols + 1];
  const bool second = blockIdx.x >= args.tiles0;
  const SplitOperand& O = args.op[second ? 1 : 0];
  const unsigned bt = second ? blockIdx.x - args.tiles0 : blockIdx.x;
  const int64_t r0 = int64_t(bt / O.tiles_l) * kBRows, l0 = int64_t(bt % O.tiles_l) * kBCols;
  const int64_t rows = O.rows, cols = O.cols, sr = O.sr, sl = O.sl;
  const int t = int(threadIdx.x);
  const int rr = t >> 3;        // 32 rows
  const int cb = (t & 7) * 8;   // 8 consecutive K elements
  float x[8];
  if (sl == 1) {
    const int64_t r = r0 + rr, l = l0 + cb;
    const float* src = O.X + r * sr + l;
    if (r < rows && l + 8 <= cols && O.vec) {
      const float4 u = *reinterpret_cast<const float4*>(src), v = *reinterpret_cast<const float4*>(src + 4);
      x[0] = u.x, x[1] = u.y, x[2] = u.z, x[3] = u.w, x[4] = v.x, x[5] = v.y, x[6] = v.z, x[7] = v.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = (r < rows && l + j < cols) ? src[j] : 0.f;
    }
  } else {
    if (O.vec && r0 + kBRows <= rows) {
      // (sr == 1) four neighbouring rows of two columns per thread
      const int r4 = (t & 7) * 4;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int ll = (t >> 3) + 32 * q;
        const float4 u = l0 + ll < cols ? *reinterpret_cast<const float4*>(O.X + (r0 + r4) + (l0 + ll) * sl)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
        tile[r4][ll] = u.x;
        tile[r4 + 1][ll] = u.y;
        tile[r4 + 2][ll] = u.z;
        tile[r4 + 3][ll] = u.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int lr = t & 31, ll = (t >> 5) + 8 * q;
        const int64_t r = r0 + lr, l = l0 + ll;
        tile[lr][ll] = (r < rows && l < cols) ? O.X[r * sr + l * sl] : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = tile[rr][cb + j];
  }
  uint32_t h[4], m[4], l[4];
  uint32_t top = 0u;  // per half: the largest |h| seen (exponent 0xFF: Inf or NaN, x's or by rounding)
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float x0 = x[2 * j], x1 = x[2 * j + 1];
    h[j] = bf16_pair(x0, x1);
    const float a0 = __fsub_rn(x0, __uint_as_float(h[j] << 16));
    const float a1 = __fsub_rn(x1, __uint_as_float(h[j] & 0xFFFF0000u));
    m[j] = bf16_pair(a0, a1);
    l[j] = bf16_pair(__fsub_rn(a0, __uint_as_float(m[j] << 16)), __fsub_rn(a1, __uint_as_float(m[j] & 0xFFFF0000u)));
    top = __vmaxu2(top, h[j] & 0x7FFF7FFFu);
  }
  if ((top & 0xFFFFu) >= 0x7F80u || (top >> 16) >= 0x7F80u) *nonfinite = 1;
  const size_t plane = size_t(O.rows_pad) * size_t(O.k_pad);
  __nv_bfloat16* const dst = O.pieces + size_t(r0 + rr) * size_t(O.k_pad) + size_t(l0 + cb);
  *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<uint4*>(dst + plane) = make_uint4(m[0], m[1], m[2], m[3]);
  *reinterpret_cast<uint4*>(dst + 2 * plane) = make_uint4(l[0], l[1], l[2], l[3]);
}

// C = alpha sum_s partial_s + beta C on the split tiles, the K ranges in order with round-to-nearest
// adds; four rows of a column per thread.
template <int BN, int ROWS>
__global__ void __launch_bounds__(256) bf16_reduce_kernel(const SliceGemmParams P) {
  if (P.skip_if_flag && *P.skip_if_flag) return;
  const int rest = int(gridDim.y), t = int(blockIdx.y);
  int tm, tn;
  tile_coords(P.whole_tiles + t, P.tiles_m, P.tiles_n, P.group_m, tm, tn);
  constexpr int kQuads = ROWS / 4;
  for (int idx = int(threadIdx.x); idx < 32 * kQuads; idx += 256) {
    const int r = idx % kQuads * 4, c = int(blockIdx.x) * 32 + idx / kQuads;
    const int64_t i = int64_t(tm) * ROWS + r, j = int64_t(tn) * BN + c;
    if (i >= P.m || j >= P.n) continue;
    const float* p = P.partial + int64_t(t) * (BN * ROWS) + c * ROWS + r;
    float4 s = *reinterpret_cast<const float4*>(p);
    for (int q = 1; q < P.splits; ++q) {
      const float4 v = *reinterpret_cast<const float4*>(p + int64_t(q) * rest * (BN * ROWS));
      s.x = __fadd_rn(s.x, v.x);
      s.y = __fadd_rn(s.y, v.y);
      s.z = __fadd_rn(s.z, v.z);
      s.w = __fadd_rn(s.w, v.w);
    }
    const float sv[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (i + e >= P.m) break;
      float* dst = static_cast<float*>(P.C) + i + e + j * P.ldc;
      const float v = __fmul_rn(P.alpha_f, sv[e]);
      *dst = P.beta_f == 0.f ? v : __fmaf_rn(P.beta_f, *dst, v);
    }
  }
}

template <int BN, int STAGES, bool PAIR>
cudaError_t launch_config(const Bf16Operand& a, const Bf16Operand& b, const SgemmSplitArgs& args,
                          cudaStream_t stream) {
  constexpr int kRowsPerTile = PAIR ? 2 * kSliceBM : kSliceBM;
  if (a.rows_pad % kRowsPerTile != 0 || b.rows_pad % BN != 0) return cudaErrorInvalidValue;
  CUtensorMap tmA, tmB;
  if (!make_tensor_map_3d(&tmA, a.pieces, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, uint64_t(a.k_pad),
                          uint64_t(a.rows_pad), 3, kSliceKBytes / 2, kSliceBM))
    return cudaErrorInvalidValue;
  if (!make_tensor_map_3d(&tmB, b.pieces, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, uint64_t(b.k_pad),
                          uint64_t(b.rows_pad), 3, kSliceKBytes / 2, PAIR ? BN / 2 : BN))
    return cudaErrorInvalidValue;
  SliceGemmParams P{};
  P.m = args.m;
  P.n = args.n;
  P.num_kb = int(a.k_pad / (kSliceKBytes / 2));
  P.tiles_m = int(a.rows_pad / kRowsPerTile);
  P.tiles_n = int(b.rows_pad / BN);
  P.slices = args.pieces;
  P.diag_lo = 2;
  P.diag_hi = args.pieces + 1;
  P.first_writes = 1;
  P.alpha_f = args.alpha;
  P.beta_f = args.beta;
  P.C = args.C;
  P.ldc = args.ldc;
  P.skip_if_flag = args.skip_if_flag;
  P.status = args.status;
  P.group_m = tuning().group_m > 0 ? tuning().group_m : P.tiles_m;
  P.splits = args.split.ranges;
  P.whole_tiles = int(args.split.whole_tiles);
  const int tiles = P.tiles_m * P.tiles_n, chunks = (P.num_kb + kBf16ChunkKb - 1) / kBf16ChunkKb;
  if (P.splits < 1 || P.splits > chunks || P.whole_tiles < 0 || P.whole_tiles > tiles ||
      (P.whole_tiles < tiles && args.partial == nullptr))
    return cudaErrorInvalidValue;
  P.partial = args.partial;
  P.wait_limit_ns = tuning().wait_limit_ns ? tuning().wait_limit_ns : kWaitLimitNs;
  // 128 accumulator columns per epilogue thread: 4 epilogue warps for 128-wide tiles, 8 for 256
  const cudaError_t e = launch_slice_gemm<kModeSplitBF16, BN, STAGES, BN / 32, PAIR>(tmA, tmB, P, args.num_sms, stream);
  if (e != cudaSuccess || P.whole_tiles == tiles) return e;
  // 32 columns of a split tile per block
  const dim3 grid(unsigned(BN / 32), unsigned(tiles - P.whole_tiles));
  bf16_reduce_kernel<BN, kRowsPerTile><<<grid, 256, 0, stream>>>(P);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_bf16_split(const StridedView<float>& xa, const Bf16Operand& oa, const StridedView<float>& xb,
                              const Bf16Operand& ob, int* nonfinite, cudaStream_t stream) {
  SplitArgs A;
  int64_t total = 0;
  for (int i = 0; i < 2; ++i) {
    const StridedView<float>& x = i ? xb : xa;
    const Bf16Operand& op = i ? ob : oa;
    if (op.k_pad % kBCols != 0 || op.rows_pad % kBRows != 0) return cudaErrorInvalidValue;
    const int64_t tl = op.k_pad / kBCols, tr = op.rows_pad / kBRows;
    const int64_t ld = x.sl == 1 ? x.sr : x.sl;
    const int vec = (x.sl == 1 || x.sr == 1) && ld % 4 == 0 && reinterpret_cast<uintptr_t>(x.ptr) % 16 == 0;
    A.op[i] = SplitOperand{x.ptr, x.rows, x.cols, x.sr, x.sl, op.rows_pad, op.k_pad,
                           static_cast<__nv_bfloat16*>(op.pieces), unsigned(tl), vec};
    total += tr * tl;
    if (i == 0) A.tiles0 = unsigned(total);
    if (tr > 65535 || tl > 0x7FFFFFFF || total > 0x7FFFFFFF) return cudaErrorInvalidConfiguration;
  }
  bf16_split_kernel<<<unsigned(total), 256, 0, stream>>>(A, nonfinite);
  return cudaGetLastError();
}

cudaError_t launch_sgemm_split_bf16(const Bf16Operand& a, const Bf16Operand& b, const SgemmSplitArgs& args,
                                    cudaStream_t stream) {
  if (args.pieces < 1 || args.pieces > 3) return cudaErrorInvalidValue;
  if (a.k_pad != b.k_pad || a.k_pad % (kSliceKBytes / 2) != 0) return cudaErrorInvalidValue;
  if (args.tile_n == kTilePair) return launch_config<256, 6, true>(a, b, args, stream);
  if (args.tile_n == 256) return launch_config<256, 4, false>(a, b, args, stream);
  if (args.tile_n == 128) return launch_config<128, 6, false>(a, b, args, stream);
  return cudaErrorInvalidValue;
}

// Measured without / with K ranges (us of device time): 300 x 517 x 1100 (9 tiles of 148) 52.6 / 26.9,
// 1024^3 (32 tiles) 49.3 / 29.2, 100 x 100 x 4000 (1 tile) 136 / 29.5, 4096^3 (3.46 rounds, two
// ranges of the last 68 tiles) 659 / 617.
Bf16Split bf16_split_rule(int64_t tiles, int64_t k_pad, int ctas) {
  const int64_t chunk = kBf16ChunkKb * (kSliceKBytes / 2), chunks = (k_pad + chunk - 1) / chunk;
  const int64_t rest = tiles % ctas;
  Bf16Split best{tiles, 1};
  double best_cost = double(chunks);
  for (int64_t s = 2; rest > 0 && s <= std::min<int64_t>(chunks, 16); ++s) {
    // rounds of CTAs times the longest range, and the second launch with its traffic (a chunk is
    // about 10 us; a tile's sum takes 0.07 us to write and read)
    const double cost = double((rest * s + ctas - 1) / ctas * ((chunks + s - 1) / s)) + 0.4 + 0.007 * double(rest * s);
    if (cost < best_cost) {
      best_cost = cost;
      best = Bf16Split{tiles - rest, int(s)};
    }
  }
  return best;
}

}  // namespace eb2
