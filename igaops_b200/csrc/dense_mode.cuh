// Dense mode products on the FP64 tensor cores (m8n8k4).
//
// One CTA computes MB rows x BN columns of Y = A X, A (rows x cols) a dense 1D
// factor (fast-diagonalisation eigenvectors, dense Kronecker factors), X the
// tensor with the contracted mode as rows and every other mode flattened into N
// columns. A column n = (n / lo) hi-stride + (n % lo) lo-stride: with the strides
// of the full control-point tensor the first and last product of a
// preconditioner apply gather and scatter the free box themselves.
//
// A and the X tile are staged whole (K = cols) in shared memory: the extents of
// one direction are a few hundred at most. Row strides are 4 mod 8 doubles, which
// makes both fragment loads (rows by k, and k by rows for the transposed second
// stage) conflict-free. FP32 tensors are converted on the way in and out: the
// products and sums are FP64.
//
// TWO stages compute A^T (s . (A X)) in one launch for the slowest mode of the
// fast diagonalisation (forward product, 1 / Lambda, backward product): the
// columns stay in shared memory between the two.
#pragma once

#include "common.cuh"

namespace iga {

template <typename T>
struct DenseMode {
  const T* A;           // A[r * ldr + c * ldc]
  int64_t ldr, ldc;
  int32_t rows, cols;
  const T* x;           // x[(n / xlo) * xhi + (n % xlo) * xls + c * xc]
  int64_t xhi, xls, xc;
  T* y;                 // y[(n / ylo) * yhi + (n % ylo) * yls + r * yr]
  int64_t yhi, yls, yr;
  int32_t xlo, ylo;
  int64_t N;
  const T* scale;       // s[(r * N + n) / scale_div]; null: none
  int32_t scale_div;
  int32_t accumulate;
  int32_t mb;           // rows per CTA
};

// 16 warps: the staging of the operands, instruction-bound, takes as long as the
// products with 8 (96^3 p3 apply 86 us, with 16 warps 72)
constexpr int kDenseThreads = 512;
constexpr int kDenseMax = 384;  // largest contracted extent

__host__ __device__ inline int dense_ld(int n) {  // smallest stride >= n, 4 mod 8
  return (n + 3) / 8 * 8 + 4;
}

// shared memory (bytes): A (mb x cols), the X tile, and the second stage's tile
inline size_t dense_smem(int mb, int cols, int bn, bool two) {
  const size_t kp = (cols + 3) / 4 * 4;
  const size_t a = (size_t)(two ? (kp + 7) / 8 * 8 : (mb + 7) / 8 * 8) * dense_ld(cols);
  const size_t xr = two ? (kp + 7) / 8 * 8 : kp;
  return (a + (two ? 2 : 1) * xr * (bn + 4)) * 8;
}

// ------------------------------------------------- device pieces
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}
__device__ __forceinline__ void cp8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// CONST: of a 1D factor, constant over the apply; else of a tensor, which the product
// before may still write when this kernel starts
template <bool CONST, typename T>
__device__ __forceinline__ void stage_elem(double* dst, const T* src) {
  if constexpr (sizeof(T) == 8) cp8(dst, src);
  else *dst = (double)(CONST ? __ldg(src) : ld_dependent(src));
}

// acc[i] += A(row block i) X(column block) over K: R row blocks at once. A[r][c]
// at a[r * sr + c * sc], X[c][n] at b[c * ldx + n] (lane offsets included).
// (ZERO: from zero.)
template <int R, bool ZERO>
__device__ __forceinline__ void block_rows(double (&acc)[R][2], const double* a, int sr8, int sc,
                                           const double* b, int ldx, int kp) {
  if (ZERO) {
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i][0] = acc[i][1] = 0.0;
  }
#pragma unroll 2
  for (int k = 0; k < kp; k += 4) {
    const double bv = b[k * ldx];
    double av[R];
#pragma unroll
    for (int i = 0; i < R; ++i) av[i] = a[i * sr8 + k * sc];
#pragma unroll
    for (int i = 0; i < R; ++i) dmma(acc[i], av[i], bv);
  }
}

template <typename T>
iga_status launch_dense_mode(const DenseMode<T>& p, bool two, bool dependent, cudaStream_t st);

// Whether a product of these extents runs on launch_dense_mode, and in two
// stages: the operands of the smallest tile fit shared memory.
inline bool dense_fits(int rows, int cols, int64_t N) {
  return rows >= 1 && cols >= 1 && cols <= kDenseMax && rows <= 1 << 16 && N < (1ll << 31);
}
inline bool dense_two_fits(int m) { return dense_smem(m, m, 32, true) <= 227 * 1024; }

// A mode product of a compact tensor (outer, cols, inner) -> (outer, rows, inner).
template <typename T>
inline DenseMode<T> dense_compact(const T* A, int64_t ldr, int64_t ldc, int rows, int cols,
                                  int64_t outer, int64_t inner, const T* x, T* y) {
  DenseMode<T> p;
  p.A = A;
  p.ldr = ldr;
  p.ldc = ldc;
  p.rows = rows;
  p.cols = cols;
  p.x = x;
  p.xlo = (int32_t)inner;
  p.xhi = cols * inner;
  p.xls = 1;
  p.xc = inner;
  p.y = y;
  p.ylo = (int32_t)inner;
  p.yhi = rows * inner;
  p.yls = 1;
  p.yr = inner;
  p.N = outer * inner;
  p.scale = nullptr;
  p.scale_div = 1;
  p.accumulate = 0;
  p.mb = rows;
  return p;
}

}  // namespace iga
