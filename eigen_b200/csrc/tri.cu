// tri.cu -- the element-wise kernels the symmetric and triangular level-3 routines need
// around the GEMM: expanding a stored symmetric or triangular matrix into a full one, merging a
// product into one triangle of C, scaling a triangle or a matrix, and applying a triangular
// diagonal block to a panel in place (a multiply, or a solve by blocked substitution).
//
// Eigen's routines (blas/level3_impl.h:98-760) feed the GEBP kernel through triangular and
// self-adjoint packing (GeneralMatrixMatrixTriangular.h, SelfadjointMatrixMatrix.h,
// TriangularMatrixMatrix.h, TriangularSolverMatrix.h).  Here every product of any size goes
// through the device GEMM, and these kernels handle the triangles: they are memory-bound
// (expand, merge, scale: one read and one write per element) or, for the diagonal blocks,
// work on vectors staged in shared memory.
#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.h"

namespace eb2 {
namespace {

constexpr int kTile = 32;  // 32 x 32 element tiles, 32 x 8 threads
constexpr int kRowsPerThread = kTile / 8;

__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }

__device__ __forceinline__ bool in_triangle(int64_t i, int64_t j, bool upper) { return upper ? i <= j : i >= j; }

// out (n x n, ld ldo) = the symmetric matrix whose triangle `upper` is stored in A (ld lda):
// out(i,j) = A(i,j) inside the triangle and A(j,i) outside.  The mirrored reads go through
// a shared-memory tile so that both the reads and the writes are coalesced; elements of A
// outside the stored triangle are never read.
template <typename T>
__global__ void expand_symmetric_kernel(const T* __restrict__ A, int64_t lda, int64_t n, bool upper,
                                        T* __restrict__ out, int64_t ldo) {
  __shared__ T mirror[kTile][kTile + 1];
  const int64_t bi = int64_t(blockIdx.x) * kTile, bj = int64_t(blockIdx.y) * kTile;
  const int tx = threadIdx.x, ty = threadIdx.y;
  // tile (bj, bi) of A, needed where tile (bi, bj) is (partly) outside the triangle
  const bool any_outside = upper ? (bi + kTile - 1 > bj) : (bi < bj + kTile - 1);
  if (any_outside) {
    for (int q = 0; q < kRowsPerThread; ++q) {
      const int jj = ty + 8 * q;  // column of the mirrored tile = row of the output tile
      const int64_t r = bj + tx, c = bi + jj;  // element A(r, c) = out(c, r)
      if (r < n && c < n && in_triangle(r, c, upper)) mirror[jj][tx] = A[r + c * lda];
    }
  }
  __syncthreads();
  for (int q = 0; q < kRowsPerThread; ++q) {
    const int jj = ty + 8 * q;
    const int64_t i = bi + tx, j = bj + jj;
    if (i >= n || j >= n) continue;
    out[i + j * ldo] = in_triangle(i, j, upper) ? A[i + j * lda] : mirror[tx][jj];
  }
}

// out (n x n, ld ldo) = the triangular matrix stored in the triangle `upper` of A: A(i,j)
// inside the triangle, 0 outside, 1 on the diagonal when `unit` (then the stored diagonal is
// not read).
template <typename T>
__global__ void expand_triangular_kernel(const T* __restrict__ A, int64_t lda, int64_t n, bool upper, bool unit,
                                         T* __restrict__ out, int64_t ldo) {
  const int64_t bi = int64_t(blockIdx.x) * kTile, bj = int64_t(blockIdx.y) * kTile;
  for (int q = 0; q < kRowsPerThread; ++q) {
    const int64_t i = bi + threadIdx.x, j = bj + threadIdx.y + 8 * q;
    if (i >= n || j >= n) continue;
    T v = T(0);
    if (i == j)
      v = unit ? T(1) : A[i + j * lda];
    else if (in_triangle(i, j, upper))
      v = A[i + j * lda];
    out[i + j * ldo] = v;
  }
}

// C(i,j) = P(i,j) + beta C(i,j) on the triangle `upper` of the n x n C; beta == 0 writes P
// and never reads C; P == null stands for a zero product (C := beta C, beta == 0 writing
// exact zeros).  The other triangle is not touched.  With `only_if_flag` the kernel does
// nothing unless *only_if_flag != 0.
template <typename T>
__global__ void merge_triangle_kernel(const T* __restrict__ P, int64_t ldp, int64_t n, bool upper, T beta,
                                      T* __restrict__ C, int64_t ldc, const int* only_if_flag) {
  if (only_if_flag && *only_if_flag == 0) return;
  const int64_t bi = int64_t(blockIdx.x) * kTile, bj = int64_t(blockIdx.y) * kTile;
  for (int q = 0; q < kRowsPerThread; ++q) {
    const int64_t i = bi + threadIdx.x, j = bj + threadIdx.y + 8 * q;
    if (i >= n || j >= n || !in_triangle(i, j, upper)) continue;
    const T p = P ? P[i + j * ldp] : T(0);
    T* c = C + i + j * ldc;
    *c = beta == T(0) ? p : fma_rn(beta, *c, p);
  }
}

// X := alpha X elementwise (m x n, ld ldx): a plain multiply, so non-finite entries stay
// non-finite even for alpha == 0.
template <typename T>
__global__ void multiply_kernel(int64_t m, int64_t n, T alpha, T* __restrict__ X, int64_t ldx) {
  const int64_t bi = int64_t(blockIdx.x) * kTile, bj = int64_t(blockIdx.y) * kTile;
  for (int q = 0; q < kRowsPerThread; ++q) {
    const int64_t i = bi + threadIdx.x, j = bj + threadIdx.y + 8 * q;
    if (i < m && j < n) X[i + j * ldx] *= alpha;
  }
}

// x := E x in place for `count` vectors x (element r of vector t at X[r*vs + t*ts]), E the
// triangular block (nb x nb, nb <= kTriBlock, element (r, c) at E[r*er + c*ec]; the triangle
// `lower` or upper is used, the diagonal is taken as 1 when `unit`).  One thread per vector;
// E and a tile of kTriVecs vectors are staged in shared memory with coalesced loads and stores
// (the vector index runs fastest when ts == 1, the element index otherwise).
template <typename T>
__global__ void __launch_bounds__(kTriVecs) tri_block_multiply_kernel(const T* __restrict__ E, int64_t er, int64_t ec,
                                                                      int nb, bool lower, bool unit,
                                                                      T* __restrict__ X, int64_t vs, int64_t ts,
                                                                      int64_t count) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Es = reinterpret_cast<T*>(smem_raw);  // [nb][nb]
  T* Xs = Es + nb * nb;                    // [nb][kTriVecs + 1], Xs[r * (kTriVecs+1) + t]
  constexpr int kXld = kTriVecs + 1;
  const int tid = threadIdx.x;
  for (int idx = tid; idx < nb * nb; idx += kTriVecs) {
    const int r = idx / nb, c = idx % nb;
    T v = T(0);
    if (r == c)
      v = unit ? T(1) : E[r * er + c * ec];
    else if (lower ? r > c : r < c)
      v = E[r * er + c * ec];
    Es[idx] = v;
  }
  const int64_t t0 = int64_t(blockIdx.x) * kTriVecs;
  const int nv = int(count - t0 < kTriVecs ? count - t0 : kTriVecs);
  const bool vec_fast = (ts == 1);
  for (int idx = tid; idx < nb * kTriVecs; idx += kTriVecs) {
    const int t = vec_fast ? idx % kTriVecs : idx / nb;
    const int r = vec_fast ? idx / kTriVecs : idx % nb;
    if (t < nv) Xs[r * kXld + t] = X[r * vs + (t0 + t) * ts];
  }
  __syncthreads();
  if (tid < nv) {
    T* x = Xs + tid;
    // each new x[r] uses only entries that are still old: descending rows for a lower
    // triangle, ascending for an upper one
    if (lower) {
      for (int r = nb - 1; r >= 0; --r) {
        T s = Es[r * nb + r] * x[r * kXld];
        for (int c = 0; c < r; ++c) s = fma_rn(Es[r * nb + c], x[c * kXld], s);
        x[r * kXld] = s;
      }
    } else {
      for (int r = 0; r < nb; ++r) {
        T s = Es[r * nb + r] * x[r * kXld];
        for (int c = r + 1; c < nb; ++c) s = fma_rn(Es[r * nb + c], x[c * kXld], s);
        x[r * kXld] = s;
      }
    }
  }
  __syncthreads();
  for (int idx = tid; idx < nb * kTriVecs; idx += kTriVecs) {
    const int t = vec_fast ? idx % kTriVecs : idx / nb;
    const int r = vec_fast ? idx / kTriVecs : idx % nb;
    if (t < nv) X[r * vs + (t0 + t) * ts] = Xs[r * kXld + t];
  }
}

// x := E^-1 x for a diagonal block E of up to kPanelMax rows and `count` vectors (laid out
// as above), V of them per CTA, resident in shared memory for the whole block.  Blocked
// substitution over 16-row sub-blocks:
//   * one lane per vector solves a sub-block against its 16 x 16 triangle in registers, column
//     by column with the reciprocal of each diagonal entry, in the order of Eigen's column-major
//     triangular solve kernel (Eigen/src/Core/products/TriangularSolverMatrix.h:61-82);
//   * its contribution is subtracted from the rows below as 16 x 8 tile products (DMMA for
//     double), the next sub-block's rows first, so that the next solve runs in one or two warps
//     while the others update the rest;
//   * the coefficients of a sub-block's columns (negated) alternate between two shared-memory
//     panels; the loads of the panel after next are in flight in registers meanwhile.
// An upper triangle is solved as the lower one of the index-reversed system (row r <->
// nb-1-r), so both run forward.  Rows and columns past nb behave as an identity.
//
// Bound by the serial chain of 16 sub-blocks (a solve, a small product and two barriers each),
// so V shrinks until the vectors fill the SMs.  A 4096 solve with 2048 vectors (16 blocks of 256)
// went from 3047 to 1820 us against 64 vectors per CTA, 32-row sub-blocks without look-ahead and
// FMA updates (129 us a block on 32 CTAs), and from 1704 to 1439 us (48 to 31 us a block) with one
// address step per staged coefficient and the diagonal's reciprocals formed once at the start.
constexpr int kPanelSub = 16;

template <typename T, int V>
struct PanelCfg {
  static constexpr int kThreads = V == 64 ? 512 : 256;
  static constexpr int kXld = V + 4;  // row stride of the vectors: fragment reads hit distinct banks
  static constexpr int kSolvers = V == 64 ? 2 : 1;  // solving warps
  static constexpr int kPer = kPanelMax * kPanelSub / kThreads;  // coefficients a thread stages per panel
  static size_t smem(int nb) {
    const size_t nbp = size_t(nb + kPanelSub - 1) / kPanelSub * kPanelSub;
    return (nbp * kXld + 2 * kPanelSub * (nbp + 4) + nbp) * sizeof(T);
  }
};

// rows r0 .. r0+15, columns c0 .. c0+7 of the resident vectors += (panel rows) x (the solved
// 16 rows at xs): the 16 x 8 accumulator in the m16n8 fragment layout.  The product is summed from
// zero and added once: a vector entry is rounded at its own size once per sub-block, not once per
// row of it.  Normwise error of a 256-row block against extended precision: 2.0e-16 (FP32 1.07e-7),
// 5.2e-16 when the products ran into the vectors directly, at the same time (1366 us for 4096 x 2048).
__device__ __forceinline__ void panel_tile(const double* pr, int ldp, const double* xs, double* xd, int xld, int g,
                                           int tig) {
  double u[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < kPanelSub; k += 4) {
    const double a0 = pr[(k + tig) * ldp + g], a1 = pr[(k + tig) * ldp + g + 8], b0 = xs[(k + tig) * xld + g];
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+d"(u[0]), "+d"(u[1]), "+d"(u[2]), "+d"(u[3])
        : "d"(a0), "d"(a1), "d"(b0));
  }
  double2* const x0 = reinterpret_cast<double2*>(xd + g * xld + 2 * tig);
  double2* const x1 = reinterpret_cast<double2*>(xd + (g + 8) * xld + 2 * tig);
  const double2 v0 = *x0, v1 = *x1;
  *x0 = make_double2(v0.x + u[0], v0.y + u[1]);
  *x1 = make_double2(v1.x + u[2], v1.y + u[3]);
}
__device__ __forceinline__ void panel_tile(const float* pr, int ldp, const float* xs, float* xd, int xld, int g,
                                           int tig) {
  float u[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int k = 0; k < kPanelSub; ++k) {
    const float a0 = pr[k * ldp + g], a1 = pr[k * ldp + g + 8];
    const float2 b = *reinterpret_cast<const float2*>(xs + k * xld + 2 * tig);
    u[0] = fma_rn(a0, b.x, u[0]);
    u[1] = fma_rn(a0, b.y, u[1]);
    u[2] = fma_rn(a1, b.x, u[2]);
    u[3] = fma_rn(a1, b.y, u[3]);
  }
  float2* const x0 = reinterpret_cast<float2*>(xd + g * xld + 2 * tig);
  float2* const x1 = reinterpret_cast<float2*>(xd + (g + 8) * xld + 2 * tig);
  const float2 v0 = *x0, v1 = *x1;
  *x0 = make_float2(v0.x + u[0], v0.y + u[1]);
  *x1 = make_float2(v1.x + u[2], v1.y + u[3]);
}

template <typename T, int V>
__global__ void __launch_bounds__(PanelCfg<T, V>::kThreads)
    tri_panel_solve_kernel(const T* __restrict__ E, int64_t er, int64_t ec, int nb, bool lower, bool unit,
                           T* __restrict__ X, int64_t vs, int64_t ts, int64_t count) {
  using C = PanelCfg<T, V>;
  constexpr int kThreads = C::kThreads, kXld = C::kXld, kWarps = kThreads / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nsub = (nb + kPanelSub - 1) / kPanelSub, nbp = nsub * kPanelSub, ldp = nbp + 4;
  T* Xs = reinterpret_cast<T*>(smem_raw);  // [nbp][kXld]: Xs[r * kXld + t], forward row order
  T* panel0 = Xs + nbp * kXld;             // [kPanelSub][ldp] each: -E'(jb + r, jb + c) at c * ldp + r
  T* panel1 = panel0 + kPanelSub * ldp;
  T* Dinv = panel1 + kPanelSub * ldp;      // [nbp]: reciprocals of the diagonal
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, tig = lane & 3;
  const int64_t t0 = int64_t(blockIdx.x) * V;
  const int nv = int(count - t0 < V ? count - t0 : V);
  // forward row r is row ro(r) of the stored system
  auto ro = [&](int r) -> int64_t { return lower ? r : nb - 1 - r; };
  // The coefficients are contiguous along the rows, or along the columns when transposed.  A
  // thread's elements of a panel are a row and kPer columns (or a column and kPer rows) at fixed
  // offsets from the panel's corner, so their addresses move by one step per element and panel.
  const bool row_fast = er == 1;
  const int rb = row_fast ? tid % kPanelMax : tid / kPanelSub, cb = row_fast ? tid / kPanelMax : tid % kPanelSub;
  const int rq = row_fast ? 0 : kThreads / kPanelSub, cq = row_fast ? kThreads / kPanelMax : 0;
  const int64_t sgn = lower ? 1 : -1;
  const int64_t qstep = sgn * (row_fast ? cq * ec : rq * er), sub_step = sgn * kPanelSub * (er + ec);
  const T* corner = E + ro(rb) * er + ro(cb) * ec;  // element q = 0 of the next panel
  int left = nb;                                    // rows from the next panel's corner to the end
  T cv[C::kPer];
  auto fetch = [&]() {  // the next panel into registers
    const T* p = corner;
#pragma unroll
    for (int q = 0; q < C::kPer; ++q, p += qstep) {
      const int r = rb + q * rq, c = cb + q * cq;
      cv[q] = r == c ? T(1) : T(0);
      if (r < left && (r > c || (r == c && !unit))) cv[q] = *p;
    }
    corner += sub_step;
    left -= kPanelSub;
  };
  auto stash = [&](int sub, T* panel) {
    const int rows = nbp - sub * kPanelSub;
    T* p = panel + cb * ldp + rb;
    const int pstep = cq * ldp + rq;
#pragma unroll
    for (int q = 0; q < C::kPer; ++q, p += pstep)
      if (rb + q * rq < rows) *p = -cv[q];
  };
  auto solve = [&](int sub, const T* panel) {  // the solving warps
    const T* const dinv = Dinv + sub * kPanelSub;
    const int t = warp * 32 + lane;
    if (t < V) {
      T* x = Xs + sub * kPanelSub * kXld + t;
      T sv[kPanelSub];
#pragma unroll
      for (int r = 0; r < kPanelSub; ++r) sv[r] = x[r * kXld];
#pragma unroll
      for (int c = 0; c < kPanelSub; ++c) {
        // x_c = s_c / d_c, then s_r -= d_rc x_c for every later row r: independent updates, so
        // the dependent chain is two operations per row
        const T xc = sv[c] * dinv[c];
        sv[c] = xc;
#pragma unroll
        for (int r = c + 1; r < kPanelSub; ++r) sv[r] = fma_rn(panel[c * ldp + r], xc, sv[r]);
      }
#pragma unroll
      for (int r = 0; r < kPanelSub; ++r) x[r * kXld] = sv[r];
    }
  };

  fetch();
  for (int r = tid; r < nbp; r += kThreads) Dinv[r] = r < nb && !unit ? T(1) / E[ro(r) * (er + ec)] : T(1);
  if (ts == 1) {
    for (int idx = tid; idx < nbp * V; idx += kThreads) {
      const int t = idx % V, r = idx / V;
      Xs[r * kXld + t] = (t < nv && r < nb) ? X[ro(r) * vs + t0 + t] : T(0);
    }
  } else {
    for (int t = warp; t < V; t += kWarps)
      for (int r = lane; r < nbp; r += 32)
        Xs[r * kXld + t] = (t < nv && r < nb) ? X[ro(r) * vs + (t0 + t) * ts] : T(0);
  }
  stash(0, panel0);
  if (nsub > 1) {
    fetch();
    stash(1, panel1);
  }
  __syncthreads();
  if (warp < C::kSolvers) solve(0, panel0);
  __syncthreads();
  for (int j = 0; j + 1 < nsub; ++j) {
    T* const panel = (j & 1) ? panel1 : panel0;       // sub-block j's columns
    const T* const next = (j & 1) ? panel0 : panel1;  // sub-block j+1's
    if (j + 2 < nsub) fetch();
    const T* xs = Xs + j * kPanelSub * kXld;
    // the next sub-block's rows
    if (warp < V / 8)
      panel_tile(panel + kPanelSub, ldp, xs + 8 * warp, Xs + (j + 1) * kPanelSub * kXld + 8 * warp, kXld, g, tig);
    __syncthreads();
    if (warp < C::kSolvers) {
      solve(j + 1, next);
    } else {
      // the rows below them
      const int tiles = (nsub - j - 2) * (V / 8);
      for (int w = warp - C::kSolvers; w < tiles; w += kWarps - C::kSolvers) {
        const int rt = w / (V / 8) + 2, ct = w % (V / 8);
        panel_tile(panel + rt * kPanelSub, ldp, xs + 8 * ct, Xs + (j + rt) * kPanelSub * kXld + 8 * ct, kXld, g, tig);
      }
    }
    __syncthreads();
    if (j + 2 < nsub) stash(j + 2, panel);  // read after the next iteration's first barrier
  }
  if (ts == 1) {
    for (int idx = tid; idx < nb * V; idx += kThreads) {
      const int t = idx % V, r = idx / V;
      if (t < nv) X[ro(r) * vs + t0 + t] = Xs[r * kXld + t];
    }
  } else {
    for (int t = warp; t < nv; t += kWarps)
      for (int r = lane; r < nb; r += 32) X[ro(r) * vs + (t0 + t) * ts] = Xs[r * kXld + t];
  }
}

dim3 tile_grid(int64_t m, int64_t n) {
  return dim3(unsigned((m + kTile - 1) / kTile), unsigned((n + kTile - 1) / kTile));
}

bool grid_fits(int64_t m, int64_t n) {
  return (m + kTile - 1) / kTile <= 0x7fffffff && (n + kTile - 1) / kTile <= 65535;
}

}  // namespace

template <typename T>
cudaError_t launch_expand_symmetric(const T* A, int64_t lda, int64_t n, bool upper, T* out, int64_t ldo,
                                    cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (!grid_fits(n, n)) return cudaErrorInvalidConfiguration;
  expand_symmetric_kernel<T><<<tile_grid(n, n), dim3(kTile, 8), 0, st>>>(A, lda, n, upper, out, ldo);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_expand_triangular(const T* A, int64_t lda, int64_t n, bool upper, bool unit, T* out, int64_t ldo,
                                     cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  if (!grid_fits(n, n)) return cudaErrorInvalidConfiguration;
  expand_triangular_kernel<T><<<tile_grid(n, n), dim3(kTile, 8), 0, st>>>(A, lda, n, upper, unit, out, ldo);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_merge_triangle(const T* P, int64_t ldp, int64_t n, bool upper, T beta, T* C, int64_t ldc,
                                  cudaStream_t st, const int* only_if_flag) {
  if (n == 0) return cudaSuccess;
  if (!grid_fits(n, n)) return cudaErrorInvalidConfiguration;
  merge_triangle_kernel<T><<<tile_grid(n, n), dim3(kTile, 8), 0, st>>>(P, ldp, n, upper, beta, C, ldc, only_if_flag);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_multiply(int64_t m, int64_t n, T alpha, T* X, int64_t ldx, cudaStream_t st) {
  if (m == 0 || n == 0) return cudaSuccess;
  if (!grid_fits(m, n)) return cudaErrorInvalidConfiguration;
  multiply_kernel<T><<<tile_grid(m, n), dim3(kTile, 8), 0, st>>>(m, n, alpha, X, ldx);
  return cudaGetLastError();
}

size_t tri_block_smem(int nb, size_t elem) { return (size_t(nb) * nb + size_t(nb) * (kTriVecs + 1)) * elem; }

template <typename T>
cudaError_t launch_tri_block_multiply(const T* E, int64_t er, int64_t ec, int nb, bool lower, bool unit, T* X,
                                      int64_t vs, int64_t ts, int64_t count, cudaStream_t st) {
  if (count == 0 || nb == 0) return cudaSuccess;
  if (nb < 0 || nb > kTriBlock || count < 0) return cudaErrorInvalidValue;
  const size_t smem = tri_block_smem(nb, sizeof(T));
  const int64_t blocks = (count + kTriVecs - 1) / kTriVecs;
  if (blocks > 0x7fffffff) return cudaErrorInvalidConfiguration;
  auto kern = tri_block_multiply_kernel<T>;
  // one attribute call per instantiation: the largest block's footprint
  static_assert(sizeof(T) <= 8, "element size");
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(tri_block_smem(kTriBlock, 8)));
  if (e != cudaSuccess) return e;
  kern<<<unsigned(blocks), kTriVecs, smem, st>>>(E, er, ec, nb, lower, unit, X, vs, ts, count);
  return cudaGetLastError();
}

namespace {

template <typename T, int V>
cudaError_t launch_panel(const T* E, int64_t er, int64_t ec, int nb, bool lower, bool unit, T* X, int64_t vs,
                         int64_t ts, int64_t count, cudaStream_t st) {
  using C = PanelCfg<T, V>;
  const int64_t blocks = (count + V - 1) / V;
  if (blocks > 0x7fffffff) return cudaErrorInvalidConfiguration;
  auto kern = tri_panel_solve_kernel<T, V>;
  const cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(C::smem(kPanelMax)));
  if (e != cudaSuccess) return e;
  kern<<<unsigned(blocks), C::kThreads, C::smem(nb), st>>>(E, er, ec, nb, lower, unit, X, vs, ts, count);
  return cudaGetLastError();
}

}  // namespace

template <typename T>
cudaError_t launch_tri_panel_solve(const T* E, int64_t er, int64_t ec, int nb, bool lower, bool unit, T* X, int64_t vs,
                                   int64_t ts, int64_t count, cudaStream_t st) {
  if (count == 0 || nb == 0) return cudaSuccess;
  if (nb < 0 || nb > kPanelMax || count < 0) return cudaErrorInvalidValue;
  // the fewest vectors per CTA that still leave one CTA per SM
  constexpr int64_t kSms = 148;
  if (count <= 16 * kSms) return launch_panel<T, 16>(E, er, ec, nb, lower, unit, X, vs, ts, count, st);
  if (count <= 32 * kSms) return launch_panel<T, 32>(E, er, ec, nb, lower, unit, X, vs, ts, count, st);
  return launch_panel<T, 64>(E, er, ec, nb, lower, unit, X, vs, ts, count, st);
}

#define EB2_TRI_INSTANTIATE(T)                                                                                     \
  template cudaError_t launch_expand_symmetric<T>(const T*, int64_t, int64_t, bool, T*, int64_t, cudaStream_t);     \
  template cudaError_t launch_expand_triangular<T>(const T*, int64_t, int64_t, bool, bool, T*, int64_t,             \
                                                   cudaStream_t);                                                  \
  template cudaError_t launch_merge_triangle<T>(const T*, int64_t, int64_t, bool, T, T*, int64_t, cudaStream_t,    \
                                                const int*);                                                       \
  template cudaError_t launch_multiply<T>(int64_t, int64_t, T, T*, int64_t, cudaStream_t);                          \
  template cudaError_t launch_tri_block_multiply<T>(const T*, int64_t, int64_t, int, bool, bool, T*, int64_t,       \
                                                    int64_t, int64_t, cudaStream_t);                               \
  template cudaError_t launch_tri_panel_solve<T>(const T*, int64_t, int64_t, int, bool, bool, T*, int64_t, int64_t, \
                                                 int64_t, cudaStream_t);
EB2_TRI_INSTANTIATE(double)
EB2_TRI_INSTANTIATE(float)
#undef EB2_TRI_INSTANTIATE

}  // namespace eb2
