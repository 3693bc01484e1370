// grouped.cu -- one persistent launch for thousands of independent small products.
//
// Eigen has no batch entry point: fixed-size products (3x3 ... 8x8) never reach GEBP
// but are unrolled coefficient-based products (Eigen/src/Core/GeneralProduct.h:76-80,
// Eigen/src/Core/ProductEvaluators.h:703-880), and dynamic ones each go through
// general_matrix_matrix_product.  Here a whole batch is one launch:
//   * the host cuts the batch into work items of three classes: class 32 = one 32 x 32
//     output tile of a product; class 16 = two whole products of at most 16 x 16; class 8 =
//     four whole products of at most 8 x 8 (Eigen's fixed-size range), so that small
//     products share a warp instead of each filling a 32 x 32 tile;
//   * an FP32 item is computed by ONE warp, an FP64 item by a block of TWO (half of the fragments and
//     one operand's copies each: half the FP64 sums per lane leaves registers for 24 warps per SM
//     instead of 16).  Its operands arrive in K-chunks ("stages") of two
//     32-line panels (rows of op(A), columns of op(B)) copied by cp.async into a
//     shared-memory ring.  The copies of the next stages -- of the next item too -- are in
//     flight while the current stage computes, which hides the latency of these short,
//     scattered products' loads;
//   * bound by the L1 data pipe (66 % busy for FP64: element-wise copies in, fragments out) and issue
//     slots (60 %; DMMA pipe 50 %), so a stage carries no work for padding: lines outside the product are
//     not copied (their outputs are not stored), only the K tail is zero-filled, and the fragments
//     computed are those the item has (FP32: column fragments in pairs, four variants of the stage
//     instead of eight, which the instruction cache holds: 262 -> 249 us).  10,000 products of sides
//     3 .. 256: FP64 313.9 -> 240.7 us, FP32 286.6 -> 230.2 us against one warp per item with padded
//     fragments and longer rings for both;
//   * FP64: mma.sync m16n8k4 (DMMA), K in steps of 4 from 0 upward for every output, the
//     same sequence as the native DGEMM kernel, so each product equals one plain native call
//     bit for bit (m16n8k8 takes the same two steps in one instruction);
//   * FP32: split-BF16 on the tensor cores (x = h + m + l in bf16 pieces; the six products hl, lh, mm,
//     hm, mh, hh of every 8-deep chunk, mma.sync m16n8k8 with FP32 accumulation, added to the FP32
//     result with round-to-nearest);
//   * items are ordered longest-K first by the host and strided over the persistent warps;
//   * C = alpha*op(A)op(B) + beta*C per problem with the BLAS rules (beta == 0 never reads
//     C, alpha == 0 or k == 0 leaves beta*C and reads neither A nor B).
#include <cuda_bf16.h>

#include <climits>
#include <cstdint>
#include <utility>

#include "device_common.cuh"
#include "grouped.h"

namespace eb2 {

namespace {

constexpr int kLineStride = 36;  // a panel's k-row: 32 lines (rows of op(A) / columns of op(B)), padded
constexpr int kKc = 8;           // K per stage: two m16n8k4 steps (FP64) or one m16n8k8 step (FP32)
constexpr int kWarpsPerBlock = 2;

// FP64: a block of two warps shares an item and its ring; FP32: an item per warp.  Short rings leave
// more of the SM's memory to L1, where the copies find the sectors that neighbouring stages share
// (us for 10,000 products of sides 3 .. 256, stages x blocks: FP64 5 x 9 332, 4 x 10 252, 3 x 12 253,
// 3 x 14 270, 2 x 12 243, 2 x 16 312; FP32 6 x 8 249, 5 x 8 233, 4 x 8 231, 3 x 8 230).
constexpr int kStages64 = 2;  // 9.2 KB per block
constexpr int kStages32 = 3;  // 6.9 KB per warp
constexpr int kBlocks64 = 12, kBlocks32 = 8;  // per SM
// A launch of few items is the latency of one item's chain of stages, and memory for longer rings and
// registers for more copies in flight are free: FP64 takes a longer ring (us, 2 stages / 4: 100
// products of 32 x 32 x 2048 184 / 119, 30 of 64 x 64 x 4096 372 / 246; 1184 items, eight per SM, 69 /
// 69), and both unroll the copies of small products, FP32 in a kernel without the code of tiles where
// all are small (500 products of 8 x 8 x 4000 361 / 257, 100 of 16 x 16 x 4000 343 / 247; 343 and 287
// in the kernel that knows tiles too).  Unrolled, FP32 is slower from 1184 items on (62.8 / 67.7).
constexpr int kDeepStages64 = 4;
constexpr int64_t kDeepK = 128;  // the longest item's K, at least (at 32 the ring only takes longer to fill)
constexpr int kDeepBlocks64 = 6, kDeepBlocks32 = 2;  // per SM, at most
constexpr int kPanelElems = kKc * kLineStride;
// K rows 4 .. 7 of an FP64 panel start two elements later: the 8-byte copies of a half-warp, 8 K
// offsets of two lines, then hit distinct banks, and so do its fragment reads (307.5 -> 299.3 us).
template <typename T>
constexpr int kRowGap = sizeof(T) == 8 ? 2 : 0;
constexpr int kStageElems = 2 * kPanelElems;

__device__ __forceinline__ void dmma_16x8x8_g(double (&d)[4], double a0, double a1, double a2, double a3, double b0,
                                              double b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

__device__ __forceinline__ void mma_bf16_1688(float (&d)[4], const uint32_t (&a)[2], uint32_t b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(b));
}
// the same from a zero accumulator
__device__ __forceinline__ void mma_bf16_1688_fresh(float (&d)[4], const uint32_t (&a)[2], uint32_t b) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(b), "f"(0.f));
}

// two values as one bf16x2 register (first value in the low half: the smaller k)
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
// x = h + m + l for two values, each piece packed as bf16x2: h, m exact bf16 values, l the rest
// rounded to bf16; each difference is exact in FP32 (Henry, Tang & Heinecke, ARITH 2019)
__device__ __forceinline__ void split_pair(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  auto low = [](uint32_t v) { return __uint_as_float(v << 16); };
  auto high = [](uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); };
  h = pack_bf16(x0, x1);
  const float r0 = __fsub_rn(x0, low(h)), r1 = __fsub_rn(x1, high(h));
  m = pack_bf16(r0, r1);
  l = pack_bf16(__fsub_rn(r0, low(m)), __fsub_rn(r1, high(m)));
}

// The items of a launch: the plan's list (grouped launch), or the 32 x 32 tiles of one
// product passed by value (the per-product launches of the same arithmetic).
struct PlanItems {
  const GroupedProblem* problems;
  const GroupedItem* items;
  int64_t count;
  __device__ __forceinline__ GroupedItem item(int64_t i) const { return items[i]; }
  __device__ __forceinline__ const GroupedProblem& problem(uint32_t p) const { return problems[p]; }
  __device__ __forceinline__ const void* dummy() const { return problems; }
  // the first problem of item i, and that problem's descriptor on its way to L1
  __device__ __forceinline__ uint32_t first_problem(int64_t i) const { return i < count ? items[i].problem[0] : 0u; }
  __device__ __forceinline__ void prefetch(uint32_t p) const {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(problems + p));
  }
};
struct OneProduct {
  GroupedProblem pr;
  int tiles_m;
  int64_t count;
  __device__ __forceinline__ GroupedItem item(int64_t i) const {
    GroupedItem it{};
    it.problem[0] = 0;
    it.problem[1] = it.problem[2] = it.problem[3] = kNoProblem;
    it.k = int32_t(pr.k);
    it.tile_m = uint16_t(i % tiles_m);
    it.tile_n = uint16_t(i / tiles_m);
    it.cls = 32;
    it.frags = grouped_frags(pr.m, pr.n, it.tile_m, it.tile_n);
    return it;
  }
  __device__ __forceinline__ const GroupedProblem& problem(uint32_t) const { return pr; }
  __device__ __forceinline__ const void* dummy() const { return pr.c; }
  __device__ __forceinline__ uint32_t first_problem(int64_t) const { return 0u; }
  __device__ __forceinline__ void prefetch(uint32_t) const {}
};

__device__ __forceinline__ uint32_t slot_problem(const GroupedItem& it, int q) {
  // (a select chain: an indexed read of the item would put it in local memory)
  return q == 0 ? it.problem[0] : (q == 1 ? it.problem[1] : (q == 2 ? it.problem[2] : it.problem[3]));
}

// One panel's copies for one lane: the lanes of problem slot q are lanes q*R .. q*R+R-1 (R =
// the item's class: lines per problem).  Along the panel's contiguous direction consecutive
// lanes take consecutive elements: if the lines are contiguous (op(A) not transposed, op(B)
// transposed) lane ls takes line ls and element t is K offset t; otherwise lane ls takes K
// offset ls % 8 of lines ls / 8 + t R/8.  Either way the address and the shared-memory slot of
// element t are affine in t.  A line outside the product is not copied: what its slot holds
// reaches only outputs that are not stored.  The K tail is zero-filled.
template <typename T>
struct PanelCopy {
  static constexpr int kSize = int(sizeof(T));
  const char* ptr;  // element t = 0 of the next stage
  int64_t step;     // bytes from element t to t + 1
  uint32_t dst0;    // shared-memory byte offset of element t = 0 within the panel
  int valid;        // the elements t < valid lie on lines of the product

  __device__ __forceinline__ void set(const T* base, int64_t ldx, bool contig, int first_line, int slot_off, int ls,
                                      int r, int64_t extent) {
    if (contig) {  // X(line, kk) = base[line + kk * ld]
      const int line0 = first_line + ls;
      ptr = reinterpret_cast<const char*>(base + line0);
      step = ldx * kSize;
      dst0 = uint32_t((slot_off + ls) * kSize);
      valid = line0 < extent ? kKc : 0;
    } else {  // X(line, kk) = base[kk + line * ld]
      const int line0 = first_line + ls / kKc, dline = r / kKc, kk0 = ls % kKc;
      ptr = reinterpret_cast<const char*>(base + kk0 + int64_t(line0) * ldx);
      step = int64_t(dline) * ldx * kSize;
      dst0 = uint32_t((kk0 * kLineStride + (kk0 >> 2) * kRowGap<T> + slot_off + ls / kKc) * kSize);
      const int64_t rest = extent - line0;
      valid = rest <= 0 ? 0 : (rest > (kKc - 1) * dline ? kKc : (int(rest) + dline - 1) / dline);
    }
  }

  // byte offset of element t from element 0 in the panel of a class-32 item
  template <bool CONTIG>
  static constexpr int place(int t) {
    return (CONTIG ? t * kLineStride + (t >> 2) * kRowGap<T> : t * (32 / kKc)) * kSize;
  }
  // A stage of a class-32 item: one address and one predicated copy per element.  CONTIG: the first
  // `left` elements lie inside K (all lanes alike); else a lane's K offset is inside or not.  What
  // lies past K is zeroed.
  template <bool CONTIG, int... t>
  __device__ __forceinline__ void issue_wide(uint32_t d, int left, std::integer_sequence<int, t...>) const {
    const uint32_t st = uint32_t(step);
    if (left >= kKc) {
      (cp_async_elem_if<kSize, place<CONTIG>(t)>(d, ptr + uint64_t(st) * uint32_t(t), t, valid), ...);
    } else if constexpr (CONTIG) {
      ((t < left ? cp_async_elem_if<kSize, place<CONTIG>(t)>(d, ptr + uint64_t(st) * uint32_t(t), t, valid)
                 : zero_elem_if<kSize, place<CONTIG>(t)>(d, t, valid)),
       ...);
    } else {
      const bool in = int(threadIdx.x) % kKc < left;
      const int copied = in ? valid : 0, zeroed = in ? 0 : valid;
      (cp_async_elem_if<kSize, place<CONTIG>(t)>(d, ptr + uint64_t(st) * uint32_t(t), t, copied), ...);
      (zero_elem_if<kSize, place<CONTIG>(t)>(d, t, zeroed), ...);
    }
  }

  // `contig`: the lines are contiguous (element t is K offset t); `left`: K from the stage's start to
  // the end; `wide`: class 32 and the step fits 32 bits (`left` and `contig` are then the warp's).
  // SMALL: no item of class 32.
  template <bool DEEP, bool SMALL>
  __device__ __forceinline__ void issue(uint32_t panel, const void* dummy, bool contig, int left, int r, bool wide) {
    constexpr int kUnroll = DEEP ? kKc : 16 / kSize;
    const uint32_t d = panel + dst0;
    if (!SMALL && wide) {
      using Seq = std::make_integer_sequence<int, kKc>;
      if (contig)
        issue_wide<true>(d, left, Seq{});
      else
        issue_wide<false>(d, left, Seq{});
    } else {
      const char* p = ptr;
      uint32_t dt = d;
      const uint32_t dstep = uint32_t((contig ? kLineStride : r / kKc) * kSize);
      const int kk0 = contig ? 0 : int(threadIdx.x) % kKc;  // ls % kKc: R is a multiple of kKc
      if (SMALL && __all_sync(0xffffffffu, left >= kKc)) {
#pragma unroll
        for (int t = 0; t < kKc; ++t, p += step, dt += dstep)
          cp_async_elem_if<kSize, 0>(dt + (contig && t >= 4 ? kRowGap<T> * kSize : 0), p, t, valid);
        ptr += contig ? kKc * step : int64_t(kKc * kSize);
        return;
      }
#pragma unroll kUnroll
      for (int t = 0; t < kKc; ++t, p += step, dt += dstep) {
        const bool in = kk0 + (contig ? t : 0) < left;
        const uint32_t gap = contig && t >= 4 ? kRowGap<T> * kSize : 0;
        cp_async_fill_if<kSize>(dt + gap, in ? static_cast<const void*>(p) : dummy, in ? kSize : 0, t, valid);
      }
    }
    ptr += contig ? kKc * step : int64_t(kKc * kSize);
  }
};

// The copies of an item's stages for one lane: its slot's rows of op(A) and / or columns of op(B).
template <typename T>
struct ItemCopy {
  int left;      // K of the lane's product from the next stage on
  uint32_t how;  // the item's class, | 64: op(A)'s lines contiguous, | 128: op(B)'s, | 256: wide

  // the lane's lines of op(A) (rhs = false) or op(B) into p
  template <class Src>
  __device__ __forceinline__ void open(const Src& src, const GroupedItem& it, int lane, bool rhs, PanelCopy<T>& p) {
    const int r = it.cls;
    const int log_r = r == 8 ? 3 : (r == 16 ? 4 : 5);
    const int q = lane >> log_r;
    const int ls = lane & (r - 1);
    const uint32_t pid = slot_problem(it, q);
    const bool ok = pid != kNoProblem;
    const GroupedProblem& pr = src.problem(ok ? pid : it.problem[0]);
    left = ok ? int(pr.k < INT_MAX ? pr.k : INT_MAX) : 0;
    // op(A)(i, l): contiguous along i unless transposed; op(B)(l, j): along j only if transposed
    const bool ca = (pr.trans & 1) == 0, cb = (pr.trans & 2) != 0;
    const int64_t extent = rhs ? pr.n : pr.m;
    p.set(static_cast<const T*>(rhs ? pr.b : pr.a), rhs ? pr.ldb : pr.lda, rhs ? cb : ca,
          r == 32 ? int(rhs ? it.tile_n : it.tile_m) * 32 : 0, q * r, ls, r, ok ? extent : 0);
    how = uint32_t(r) | (ca ? 64u : 0u) | (cb ? 128u : 0u) | (r == 32 && p.step <= INT_MAX ? 256u : 0u);
  }
  template <class Src>
  __device__ __forceinline__ void open(const Src& src, const GroupedItem& it, int lane, PanelCopy<T>& pa,
                                       PanelCopy<T>& pb) {
    open(src, it, lane, true, pb);
    const uint32_t wide_b = how;
    open(src, it, lane, false, pa);
    how &= wide_b;
  }
  template <bool DEEP, bool SMALL>
  __device__ __forceinline__ void issue(PanelCopy<T>& p, const T* panel, bool rhs, const void* dummy) const {
    p.template issue<DEEP, SMALL>(smem_u32(panel), dummy, (how & (rhs ? 128u : 64u)) != 0u, left, int(how & 63u), (how & 256u) != 0u);
  }
};

__device__ __forceinline__ int item_stages(const GroupedItem& it) {
  return it.k > 0 ? (int(it.k) + kKc - 1) / kKc : 1;
}

// ---------------------------------------------------------------- FP64 compute
// NJ 8-column fragments of one 16-row block: sA, sB at the lane's K offset tig, row g / column g of
// the first fragment.  The m16n8k8 fragments are two m16n8k4 steps' taken in K order (same bits).
template <int NJ>
__device__ __forceinline__ void stage_f64(double (&acc)[4][4], const double* sA, const double* sB) {
  constexpr int kUp = 4 * kLineStride + kRowGap<double>;  // K offset 4
  const double a0 = sA[0], a1 = sA[8], a2 = sA[kUp], a3 = sA[kUp + 8];
#pragma unroll
  for (int j = 0; j < NJ; ++j)
    dmma_16x8x8_g(acc[j], a0, a1, a2, a3, sB[j * 8], sB[kUp + j * 8]);
}

// ---------------------------------------------------------------- FP32 compute
// Accumulator fragments: class 32: (row block i, column block j) -> i*4 + j; class 16:
// (problem p, column block j) -> p*2 + j; class 8: problem p -> p (rows 8-15 unused).
//
// FP32: the m16n8k8 A fragment of the 16 lines at l0 (rows 8-15 zero when `half`) and the B
// fragment of the 8 lines at l0, each as its three bf16 pieces.
__device__ __forceinline__ void frag_a(const float* sA, int l0, bool half, int g, int tig, uint32_t (&p)[3][2]) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    p[0][r] = p[1][r] = p[2][r] = 0u;
    const float* x = sA + (2 * tig) * kLineStride + l0 + g + 8 * r;
    if (!(half && r == 1)) split_pair(x[0], x[kLineStride], p[0][r], p[1][r], p[2][r]);
  }
}
__device__ __forceinline__ void frag_b(const float* sB, int l0, int g, int tig, uint32_t (&p)[3]) {
  const float* x = sB + (2 * tig) * kLineStride + l0 + g;
  split_pair(x[0], x[kLineStride], p[0], p[1], p[2]);
}
// C fragments' six piece products of one 8-deep chunk, smallest first, each into a fresh fragment that
// is then added to its result (round to nearest): fragment c is acc[slot(c)] += A piece ia(c) times B
// piece ib(c).  The chains of six go a step of each in turn, so that a warp with few others beside it
// does not wait for each MMA (100 products of 32 x 32 x 2048, A transposed: 215 -> 191 us with the
// unrolled copies).
template <int C, int NA, int NB, class Slot, class Ia, class Ib>
__device__ __forceinline__ void chunk_products(float (&acc)[8][4], const uint32_t (&pa)[NA][3][2],
                                               const uint32_t (&pb)[NB][3], Slot slot, Ia ia, Ib ib) {
  constexpr int kPieceA[6] = {0, 2, 1, 0, 1, 0}, kPieceB[6] = {2, 0, 1, 1, 0, 0};  // hl lh mm hm mh hh
  float d[C][4];
#pragma unroll
  for (int q = 0; q < 6; ++q)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (q == 0)
        mma_bf16_1688_fresh(d[c], pa[ia(c)][kPieceA[q]], pb[ib(c)][kPieceB[q]]);
      else
        mma_bf16_1688(d[c], pa[ia(c)][kPieceA[q]], pb[ib(c)][kPieceB[q]]);
    }
#pragma unroll
  for (int c = 0; c < C; ++c)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[slot(c)][e] = __fadd_rn(acc[slot(c)][e], d[c][e]);
}
// MI row blocks (of 16) by NJ column blocks (of 8) of a class-32 stage.
template <int MI, int NJ>
__device__ __forceinline__ void stage32(float (&acc)[8][4], const float* st, int g, int tig) {
  uint32_t pa[MI][3][2];
#pragma unroll
  for (int i = 0; i < MI; ++i) frag_a(st, i * 16, false, g, tig, pa[i]);
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    uint32_t pb[1][3];
    frag_b(st + kPanelElems, j * 8, g, tig, pb[0]);
    chunk_products<MI>(
        acc, pa, pb, [j](int i) { return i * 4 + j; }, [](int i) { return i; }, [](int) { return 0; });
  }
}

// A stage of two products of at most 16 x 16, or of four of at most 8 x 8.
__device__ __forceinline__ void stage_small(float (&acc)[8][4], const float* st, bool mid, int g, int tig) {
  const float* sA = st;
  const float* sB = st + kPanelElems;
  if (mid) {
    uint32_t pa[2][3][2], pb[4][3];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      frag_a(sA, p * 16, false, g, tig, pa[p]);
#pragma unroll
      for (int j = 0; j < 2; ++j) frag_b(sB, p * 16 + j * 8, g, tig, pb[p * 2 + j]);
    }
    chunk_products<4>(
        acc, pa, pb, [](int c) { return c; }, [](int c) { return c / 2; }, [](int c) { return c; });
  } else {
    uint32_t pa[4][3][2], pb[4][3];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      frag_a(sA, p * 8, true, g, tig, pa[p]);
      frag_b(sB, p * 8, g, tig, pb[p]);
    }
    chunk_products<4>(
        acc, pa, pb, [](int c) { return c; }, [](int c) { return c; }, [](int c) { return c; });
  }
}

// One stage of an item: the fragments it has (grouped_frags), nothing for padding.
template <bool SMALL>
__device__ __forceinline__ void compute_stage(float (&acc)[8][4], const float* st, const GroupedItem& it, int g,
                                              int tig) {
  if (SMALL || it.cls != 32) return stage_small(acc, st, it.cls == 16, g, tig);
  switch (it.frags >> 1) {
    case 0: return stage32<1, 2>(acc, st, g, tig);
    case 1: return stage32<1, 4>(acc, st, g, tig);
    case 2: return stage32<2, 2>(acc, st, g, tig);
    default: return stage32<2, 4>(acc, st, g, tig);
  }
}

// ---------------------------------------------------------------- epilogue
// C = alpha * acc + beta * C for the fragment elements of one product: element (h, c) of the
// fragment at rows r0.., columns c0.. is row r0 + g + 8h, column c0 + 2 tig + c.  The
// descriptor's fields are copied to registers first (C stores could otherwise alias them).
template <typename T>
struct ProductStore {
  T* c;
  int64_t ldc, m, n;
  T alpha, beta;
  __device__ __forceinline__ void load(const GroupedProblem& pr) {
    c = static_cast<T*>(pr.c);
    ldc = pr.ldc;
    m = pr.m;
    n = pr.n;
    alpha = T(pr.alpha);
    beta = T(pr.beta);
  }
  __device__ __forceinline__ void put(int64_t row, int64_t col, T v) const {
    if (row < m && col < n) put_at(c + row + col * ldc, v);
  }
  __device__ __forceinline__ void put_at(T* dst, T v) const {
    const T a = sizeof(T) == 8 ? T(__dmul_rn(double(alpha), double(v))) : T(__fmul_rn(float(alpha), float(v)));
    if (beta == T(0))
      *dst = a;
    else if constexpr (sizeof(T) == 8)
      *dst = __fma_rn(double(beta), double(*dst), double(a));
    else
      *dst = __fmaf_rn(float(beta), float(*dst), float(a));
  }
};

// C of NJ column fragments of ROWS rows: element e of fragment j of row block h is row 16h + 8 (e / 2),
// column 8j + e % 2 from (r0, c0), the lane's first place.
template <int H, int NJ, typename T, int F>
__device__ __forceinline__ void store_tile(const ProductStore<T>& ps, int64_t r0, int64_t c0, int nj,
                                           const T (&acc)[F][4]) {
  const int64_t rest_r = ps.m - r0, rest_c = ps.n - c0;
  const int rows = int(rest_r < 32 ? rest_r : 32), cols = int(rest_c < 32 ? rest_c : 32);
  T* cp = ps.c + r0 + c0 * ps.ldc;
  const int64_t next = 7 * ps.ldc;
#pragma unroll
  for (int j = 0; j < NJ; ++j, cp += next) {
    if (j >= nj) break;  // not computed
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (8 * j + c < cols) {
#pragma unroll
        for (int h = 0; h < 2 * H; ++h)
          if (8 * h < rows) ps.put_at(cp + 8 * h, acc[(h >> 1) * NJ + j][(h & 1) * 2 + c]);
      }
      if (c == 0) cp += ps.ldc;
    }
  }
}

template <bool SMALL, class Src>
__device__ __forceinline__ void epilogue_f32(const Src& src, const GroupedItem& it, float (&acc)[8][4], int g, int tig) {
  ProductStore<float> ps;
  if (!SMALL && it.cls == 32) {
    ps.load(src.problem(it.problem[0]));
    store_tile<2, 4>(ps, int64_t(it.tile_m) * 32 + g, int64_t(it.tile_n) * 32 + 2 * tig, (it.frags & 3) + 1, acc);
  } else if (it.cls == 16) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      const uint32_t pid = p == 0 ? it.problem[0] : it.problem[1];
      if (pid == kNoProblem) continue;
      ps.load(src.problem(pid));
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) ps.put(g + (e >> 1) * 8, j * 8 + tig * 2 + (e & 1), acc[p * 2 + j][e]);
    }
  } else {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const uint32_t pid = slot_problem(it, p);
      if (pid == kNoProblem) continue;
      ps.load(src.problem(pid));
#pragma unroll
      for (int e = 0; e < 2; ++e) ps.put(g, tig * 2 + e, acc[p][e]);
    }
  }
}

// ---------------------------------------------------------------- FP32: a warp's pipeline
// Items w0, w0 + W, w0 + 2W, ... in stage order; copies run S - 1 stages ahead of the
// compute, across item boundaries.
template <int S, bool DEEP, bool SMALL, class Src>
__device__ __forceinline__ void run_items_f32(const Src& src, int64_t w0, int64_t W, float* ring) {
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, tig = lane & 3;

  // producer position
  int64_t p_idx = w0;
  int p_left = 0;  // stages of the producer's item still to copy
  uint32_t p_next = 0;  // first problem of its next item
  ItemCopy<float> cp;
  PanelCopy<float> pa, pb;
  auto open_item = [&]() {
    const GroupedItem it = src.item(p_idx);
    cp.open(src, it, lane, pa, pb);
    p_left = item_stages(it);
    // the next item's record comes to L1 with this read, its problem one stage later
    p_next = src.first_problem(p_idx + W);
  };
  if (p_idx < src.count) open_item();
  const void* const dummy = src.dummy();
  auto produce = [&](int slot) {
    if (p_idx < src.count) {
      const float* stage = ring + slot * kStageElems;
      cp.template issue<DEEP, SMALL>(pa, stage, false, dummy);
      cp.template issue<DEEP, SMALL>(pb, stage + kPanelElems, true, dummy);
      cp.left -= kKc;
      if (--p_left == 0) {
        p_idx += W;
        if (p_idx < src.count) open_item();
      } else if (p_left == 1) {
        src.prefetch(p_next);
      }
    }
    cp_async_commit();  // an empty group past the end keeps the group count uniform
  };
#pragma unroll
  for (int s = 0; s < S - 1; ++s) produce(s);

  // consumer position
  int64_t c_idx = w0;
  int c_stages = 0;
  GroupedItem cur{};
  if (c_idx < src.count) {
    cur = src.item(c_idx);
    c_stages = item_stages(cur);
  }
  float acc[8][4];
#pragma unroll
  for (int f = 0; f < 8; ++f)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[f][e] = 0.f;
  int slot = 0;
  while (c_idx < src.count) {
    cp_async_wait<S - 2>();
    __syncwarp();  // every lane's copies of this stage have landed; the slot refilled below is free
    produce(slot == 0 ? S - 1 : slot - 1);
    compute_stage<SMALL>(acc, ring + slot * kStageElems, cur, g, tig);
    slot = slot == S - 1 ? 0 : slot + 1;
    if (--c_stages == 0) {
      epilogue_f32<SMALL>(src, cur, acc, g, tig);
#pragma unroll
      for (int f = 0; f < 8; ++f)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[f][e] = 0.f;
      c_idx += W;
      if (c_idx < src.count) {
        cur = src.item(c_idx);
        c_stages = item_stages(cur);
      }
    }
  }
  cp_async_wait<0>();  // no copy may outlive the warp (the trailing groups are empty)
}

// ---------------------------------------------------------------- FP64: a block's pipeline
// The same order for a block of two warps: warp 0 copies the items' rows of op(A), warp 1 their
// columns of op(B); each computes half of the fragments: a 16-row block of a 32 x 32 tile (or half
// of its columns when it has one row block), one of two products, two of four.  Half the FP64 sums
// per lane leaves registers for 24 warps per SM instead of 16, with half the copies each.
template <int S, bool DEEP, class Src>
__device__ __forceinline__ void run_items_f64(const Src& src, int64_t w0, int64_t W, double* ring) {
  const int warp = int(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int g = lane >> 2, tig = lane & 3;

  int64_t p_idx = w0;
  int p_left = 0;
  uint32_t p_next = 0;
  ItemCopy<double> cp;
  PanelCopy<double> pc;  // the warp's operand
  auto open_item = [&]() {
    const GroupedItem it = src.item(p_idx);
    cp.open(src, it, lane, warp != 0, pc);
    p_left = item_stages(it);
    p_next = src.first_problem(p_idx + W);
  };
  if (p_idx < src.count) open_item();
  const void* const dummy = src.dummy();
  auto produce = [&](int slot) {
    if (p_idx < src.count) {
      cp.template issue<DEEP, false>(pc, ring + slot * kStageElems + warp * kPanelElems, warp != 0, dummy);
      cp.left -= kKc;
      if (--p_left == 0) {
        p_idx += W;
        if (p_idx < src.count) open_item();
      } else if (p_left == 1) {
        src.prefetch(p_next);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < S - 1; ++s) produce(s);

  int64_t c_idx = w0;
  int c_stages = 0;
  GroupedItem cur{};
  // the warp's part of the item: fragments of row block rb from column block j0, nj of them (class 8:
  // one column block of products 2 warp and 2 warp + 1)
  int rb = 0, j0 = 0, nj = 0;
  auto take = [&]() {
    cur = src.item(c_idx);
    c_stages = item_stages(cur);
    const int n = (cur.frags & 3) + 1;
    if (cur.cls == 16) {
      rb = warp;
      j0 = 2 * warp;
      nj = 2;
    } else if (cur.cls == 8 || (cur.frags & 4)) {
      rb = warp;
      j0 = 0;
      nj = cur.cls == 8 ? 0 : n;
    } else {
      rb = 0;
      j0 = warp ? (n + 1) / 2 : 0;
      nj = warp ? n / 2 : (n + 1) / 2;
    }
  };
  if (c_idx < src.count) take();
  double acc[4][4];
#pragma unroll
  for (int f = 0; f < 4; ++f)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[f][e] = 0.0;
  int slot = 0;
  while (c_idx < src.count) {
    cp_async_wait<S - 2>();
    __syncthreads();  // both warps' copies of this stage have landed; the slot refilled below is free
    produce(slot == 0 ? S - 1 : slot - 1);
    const double* st = ring + slot * kStageElems + tig * kLineStride + g;
    if (cur.cls == 8) {
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const double* x = st + (2 * warp + p) * 8;
        constexpr int kUp = 4 * kLineStride + kRowGap<double>;
        dmma_16x8x8_g(acc[p], x[0], 0.0, x[kUp], 0.0, x[kPanelElems], x[kPanelElems + kUp]);
      }
    } else {
      const double *sA = st + 16 * rb, *sB = st + kPanelElems + 8 * j0;
      switch (nj) {
        case 1: stage_f64<1>(acc, sA, sB); break;
        case 2: stage_f64<2>(acc, sA, sB); break;
        case 3: stage_f64<3>(acc, sA, sB); break;
        case 4: stage_f64<4>(acc, sA, sB); break;
        default: break;
      }
    }
    slot = slot == S - 1 ? 0 : slot + 1;
    if (--c_stages == 0) {
      ProductStore<double> ps;
      if (cur.cls == 32) {
        ps.load(src.problem(cur.problem[0]));
        store_tile<1, 4>(ps, int64_t(cur.tile_m) * 32 + 16 * rb + g, int64_t(cur.tile_n) * 32 + 8 * j0 + 2 * tig, nj, acc);
      } else if (cur.cls == 16) {
        const uint32_t pid = warp == 0 ? cur.problem[0] : cur.problem[1];
        if (pid != kNoProblem) {
          ps.load(src.problem(pid));
          store_tile<1, 4>(ps, g, 2 * tig, 2, acc);
        }
      } else {
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const uint32_t pid = slot_problem(cur, 2 * warp + p);
          if (pid == kNoProblem) continue;
          ps.load(src.problem(pid));
#pragma unroll
          for (int e = 0; e < 2; ++e) ps.put(g, tig * 2 + e, acc[p][e]);
        }
      }
#pragma unroll
      for (int f = 0; f < 4; ++f)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[f][e] = 0.0;
      c_idx += W;
      if (c_idx < src.count) take();
    }
  }
  cp_async_wait<0>();
}

// Dynamic shared memory of a block: a ring per item at a time.
template <typename T>
constexpr size_t ring_bytes(int stages) {
  return size_t(stages) * kStageElems * sizeof(T) * (sizeof(T) == 8 ? 1 : kWarpsPerBlock);
}

template <bool DEEP>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, DEEP ? kDeepBlocks64 : kBlocks64)
    grouped_f64_kernel(const GroupedProblem* __restrict__ problems, const GroupedItem* __restrict__ items,
                       int64_t num_items) {
  extern __shared__ __align__(16) unsigned char grouped_smem[];
  run_items_f64<DEEP ? kDeepStages64 : kStages64, DEEP>(PlanItems{problems, items, num_items}, int64_t(blockIdx.x),
                                                        int64_t(gridDim.x), reinterpret_cast<double*>(grouped_smem));
}
template <bool DEEP, bool SMALL>
__global__ void __launch_bounds__(32 * kWarpsPerBlock, DEEP ? kDeepBlocks32 : kBlocks32)
    grouped_f32_kernel(const GroupedProblem* __restrict__ problems, const GroupedItem* __restrict__ items,
                       int64_t num_items) {
  extern __shared__ __align__(16) unsigned char grouped_smem[];
  const int warp = threadIdx.x >> 5;
  run_items_f32<kStages32, DEEP, SMALL>(
      PlanItems{problems, items, num_items}, int64_t(blockIdx.x) * kWarpsPerBlock + warp,
      int64_t(gridDim.x) * kWarpsPerBlock, reinterpret_cast<float*>(grouped_smem) + size_t(warp) * kStages32 * kStageElems);
}

// One FP32 product, one warp per 32 x 32 tile: the per-product launches of the same arithmetic.  A
// warp alone on its scheduler, so it takes the registers it can use (without a block count the
// compiler keeps to 104 of them: 10 products of 128 x 100 x 2000 2.53 / 1.80 ms).
__global__ void __launch_bounds__(32, 1) grouped_one_kernel(const GroupedProblem pr, int tiles_m, int64_t tiles) {
  extern __shared__ __align__(16) unsigned char grouped_smem[];
  run_items_f32<kStages32, false, false>(OneProduct{pr, tiles_m, tiles}, int64_t(blockIdx.x), int64_t(gridDim.x),
                                  reinterpret_cast<float*>(grouped_smem));
}

cudaError_t set_smem(const void* kern, size_t bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
}

struct GroupedKernel {
  void (*kern)(const GroupedProblem*, const GroupedItem*, int64_t);
  size_t smem;
};
GroupedKernel grouped_kernel(bool f64, GroupedVariant v) {
  if (f64)
    return v == GroupedVariant::kMany ? GroupedKernel{grouped_f64_kernel<false>, ring_bytes<double>(kStages64)}
                                      : GroupedKernel{grouped_f64_kernel<true>, ring_bytes<double>(kDeepStages64)};
  return GroupedKernel{v == GroupedVariant::kMany       ? grouped_f32_kernel<false, false>
                       : v == GroupedVariant::kFewSmall ? grouped_f32_kernel<true, true>
                                                        : grouped_f32_kernel<true, false>,
                       ring_bytes<float>(kStages32)};
}

}  // namespace

cudaError_t grouped_grid(bool f64, int64_t num_items, int64_t longest, bool small, int num_sms, GroupedGrid* grid) {
  const int64_t per_block = f64 ? 1 : kWarpsPerBlock;  // items at a time
  int64_t b = (num_items + per_block - 1) / per_block;
  const bool few = b <= int64_t(num_sms) * (f64 ? kDeepBlocks64 : kDeepBlocks32) && longest >= kDeepK;
  *grid = GroupedGrid{0, !few ? GroupedVariant::kMany : (small ? GroupedVariant::kFewSmall : GroupedVariant::kFew)};
  const GroupedKernel k = grouped_kernel(f64, grid->variant);
  cudaError_t e = set_smem(reinterpret_cast<const void*>(k.kern), k.smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, reinterpret_cast<const void*>(k.kern), 32 * kWarpsPerBlock,
                                                    k.smem);
  if (e != cudaSuccess) return e;
  const int64_t cap = int64_t(num_sms) * (per_sm > 0 ? per_sm : 1);
  if (b > cap) b = cap;
  grid->blocks = unsigned(b > 0 ? b : 0);
  return cudaSuccess;
}

cudaError_t launch_grouped_gemm(bool f64, const GroupedProblem* problems, const GroupedItem* items,
                                int64_t num_items, GroupedGrid grid, cudaStream_t stream) {
  if (num_items <= 0 || grid.blocks == 0) return cudaSuccess;
  const GroupedKernel k = grouped_kernel(f64, grid.variant);
  k.kern<<<grid.blocks, 32 * kWarpsPerBlock, k.smem, stream>>>(problems, items, num_items);
  return cudaGetLastError();
}

cudaError_t launch_grouped_one(const GroupedProblem& pr, cudaStream_t stream) {
  if (pr.m <= 0 || pr.n <= 0) return cudaSuccess;
  const int64_t tm = (pr.m + 31) / 32, tn = (pr.n + 31) / 32;
  if (tm > 65535 || tn > 65535) return cudaErrorInvalidValue;
  constexpr size_t kSmem = ring_bytes<float>(kStages32) / kWarpsPerBlock;
  const cudaError_t e = set_smem(reinterpret_cast<const void*>(grouped_one_kernel), kSmem);
  if (e != cudaSuccess) return e;
  const int64_t tiles = tm * tn;
  const unsigned grid = unsigned(tiles < 65535 ? tiles : 65535);
  grouped_one_kernel<<<grid, 32, kSmem, stream>>>(pr, int(tm), tiles);
  return cudaGetLastError();
}

}  // namespace eb2
