// Fast-diagonalisation (FD) preconditioner apply.
//
// P^{-1} v = (U_d (x) ... (x) U_1) Lambda^{-1} (U_d (x) ... (x) U_1)^T v on
// the free nodes, zero on the Dirichlet nodes (SpaceFD.apply,
// src/igaops/fastdiag/utils/space_precond.py:273-320).  The free nodes of a
// direction are a contiguous index range [lo_d, lo_d + m_d) (Dirichlet only
// removes the first and/or last control point, space_precond.py:159-168), so
// the free set is a box of the control-point tensor: gather and scatter are
// index arithmetic, fused with the first and last mode products' inputs.
//
// This file holds the FP64-arithmetic path (FP64 / FP32 tensors) on the dense
// mode products of dense_mode.cu; the BF16 tensor-core (tcgen05) mode products
// live in fd_tc.cu.
#include "common.cuh"
#include "dense_mode.cuh"

namespace iga {

struct Box {
  int32_t ndim;
  int32_t n[4];   // full extents, direction 1 first
  int32_t lo[4];  // first free index per direction
  int32_t m[4];   // free extents
};

// dst[f*ncols + k] = src[g(f)*ncols + k] (gather) or the reverse (scatter):
// f enumerates the box (direction 1 fastest), g(f) its position in the full
// tensor.
template <typename T, bool SCATTER>
__global__ void __launch_bounds__(256) box_copy_kernel(Box b, int64_t ncols, const T* __restrict__ src,
                                                       T* __restrict__ dst) {
  int64_t mfree = 1;
  for (int d = 0; d < b.ndim; ++d) mfree *= b.m[d];
  const int64_t total = mfree * ncols;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = idx % ncols;
    int64_t f = idx / ncols;
    int64_t g = 0, stride = 1;
    for (int d = 0; d < b.ndim; ++d) {
      const int64_t i = f % b.m[d];
      f /= b.m[d];
      g += (i + b.lo[d]) * stride;
      stride *= b.n[d];
    }
    if (SCATTER)
      dst[g * ncols + k] = src[idx];
    else
      dst[idx] = src[g * ncols + k];
  }
}

}  // namespace iga

using namespace iga;

extern "C" {

iga_status iga_mode_product(int dtype, const iga_factor* M, int64_t outer, int64_t inner,
                            const void* x, void* y, int accumulate, iga_stream stream);
iga_status iga_pointwise_scale(int dtype, int64_t nq, int64_t ncols, const void* coef,
                               int64_t coef_stride, const void* u, void* out, int accumulate,
                               iga_stream stream);

iga_status iga_box_copy(int dtype, int ndim, const int32_t* n, const int32_t* lo,
                        const int32_t* m, int64_t ncols, const void* src, void* dst, int scatter,
                        iga_stream stream) {
  clear_error();
  IGA_CHECK_ARG(ndim >= 1 && ndim <= 4, "ndim %d out of range", ndim);
  IGA_CHECK_ARG(n && lo && m && src && dst && ncols >= 1, "bad argument");
  IGA_CHECK_ARG(dtype == IGA_F64 || dtype == IGA_F32, "dtype %d not supported", dtype);
  Box b;
  b.ndim = ndim;
  int64_t M = 1;
  for (int d = 0; d < 4; ++d) {
    b.n[d] = d < ndim ? n[d] : 1;
    b.lo[d] = d < ndim ? lo[d] : 0;
    b.m[d] = d < ndim ? m[d] : 1;
    IGA_CHECK_ARG(b.lo[d] >= 0 && b.m[d] >= 0 && b.lo[d] + b.m[d] <= b.n[d],
                  "box of direction %d out of range", d);
    M *= b.m[d];
  }
  if (M == 0) return IGA_OK;
  int64_t blocks = ceil_div(M * ncols, 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  cudaStream_t st = as_stream(stream);
  if (dtype == IGA_F64) {
    if (scatter)
      box_copy_kernel<double, true><<<(unsigned)blocks, 256, 0, st>>>(b, ncols, (const double*)src,
                                                                      (double*)dst);
    else
      box_copy_kernel<double, false><<<(unsigned)blocks, 256, 0, st>>>(b, ncols, (const double*)src,
                                                                       (double*)dst);
  } else {
    if (scatter)
      box_copy_kernel<float, true><<<(unsigned)blocks, 256, 0, st>>>(b, ncols, (const float*)src,
                                                                     (float*)dst);
    else
      box_copy_kernel<float, false><<<(unsigned)blocks, 256, 0, st>>>(b, ncols, (const float*)src,
                                                                      (float*)dst);
  }
  IGA_LAUNCH_CHECK();
  return IGA_OK;
}

}  // extern "C"

namespace iga {

// The apply on y (already zero): forward products from direction 1 up to the
// slowest, the slowest direction's forward product, 1 / Lambda and backward
// product in one launch where its tile fits, backward products down to
// direction 1. Tensors of up to three directions gather in the first product and
// scatter in the last; the others copy the box. 2 d - 1 launches instead of
// 2 d + 3, each but the first set up while its predecessor runs. 96^3 p3 (m = 97,
// 1.06 GFLOP), us: 308 -> 72 (FP32 tensors 82); 256 threads per CTA 86.
template <typename T>
static iga_status fd_apply_t(const Box& b, const void* const* U, const T* inv, int64_t ncols,
                             const T* x, T* y, T* work0, T* work1, iga_stream stream) {
  cudaStream_t st = as_stream(stream);
  const int nd = b.ndim, last = nd - 1;
  const int dtype = sizeof(T) == 8 ? IGA_F64 : IGA_F32;
  int64_t M = 1;
  bool dense = true;
  for (int d = 0; d < nd; ++d) M *= b.m[d];
  for (int d = 0; d < nd; ++d) dense = dense && dense_fits(b.m[d], b.m[d], M * ncols / b.m[d]);
  const bool direct = dense && nd <= 3 && ncols == 1;  // gather and scatter in the products
  T* buf[2] = {work0, work1};
  const T* cur = x;
  int next = 0;
  bool dependent = false;
  if (!direct) {
    iga_status rc = iga_box_copy(dtype, nd, b.n, b.lo, b.m, ncols, x, work0, 0, stream);
    if (rc) return rc;
    cur = work0;
    next = 1;
  }
  // product of direction d: U^T (forward) or U; gather / scatter: full tensor
  auto mode = [&](int d, bool forward, bool two, bool scaled) -> iga_status {
    int64_t outer = 1, inner = ncols;
    for (int e = last; e > d; --e) outer *= b.m[e];
    for (int e = d - 1; e >= 0; --e) inner *= b.m[e];
    const int m = b.m[d];
    const bool gather = direct && cur == x, scatter = direct && !forward && d == 0;
    const bool to_y = scatter || (direct && two && nd == 1);
    T* dst = to_y ? y : buf[next];
    if (!dense) {
      iga_factor F;
      F.kind = 1;
      F.rows = F.cols = m;
      F.ld_row = forward ? 1 : m;
      F.ld_col = forward ? m : 1;
      F.dense = U[d];
      iga_status rc = iga_mode_product(dtype, &F, outer, inner, cur, dst, 0, stream);
      if (rc) return rc;
    } else {
      DenseMode<T> p = dense_compact<T>((const T*)U[d], forward ? 1 : m, forward ? m : 1, m, m,
                                        outer, inner, cur, dst);
      if (two || scaled) {
        p.scale = inv;
        p.scale_div = (int32_t)ncols;
      }
      // the box in the full tensor, columns of direction 1's products:
      // (i3, i2) -> (i3 n2 + i2) n1
      const int64_t n1 = b.n[0], n12 = n1 * b.n[1];
      const int64_t off = b.lo[0] + b.lo[1] * n1 + b.lo[2] * n12;
      if (gather) {
        p.x = x + off;
        p.xlo = b.m[1];
        p.xhi = n12;
        p.xls = n1;
        p.xc = 1;
      }
      if (to_y) {
        p.y = y + off;
        p.ylo = b.m[1];
        p.yhi = n12;
        p.yls = n1;
        p.yr = 1;
      }
      iga_status rc = launch_dense_mode<T>(p, two, dependent, st);
      if (rc) return rc;
      dependent = true;
    }
    cur = dst;
    next ^= 1;
    return IGA_OK;
  };
  const bool two = dense && dense_two_fits(b.m[last]);
  for (int d = 0; d < last; ++d) {
    iga_status rc = mode(d, true, false, false);
    if (rc) return rc;
  }
  if (two) {
    iga_status rc = mode(last, true, true, false);
    if (rc) return rc;
  } else {
    iga_status rc = mode(last, true, false, dense);
    if (rc) return rc;
    if (!dense) {
      T* dst = buf[next];
      rc = iga_pointwise_scale(dtype, M, ncols, inv, 1, cur, dst, 0, stream);
      if (rc) return rc;
      cur = dst;
      next ^= 1;
    }
    rc = mode(last, false, false, false);
    if (rc) return rc;
  }
  for (int d = last - 1; d >= 0; --d) {
    iga_status rc = mode(d, false, false, false);
    if (rc) return rc;
  }
  if (direct) return IGA_OK;
  return iga_box_copy(dtype, nd, b.n, b.lo, b.m, ncols, cur, y, 1, stream);
}

}  // namespace iga

extern "C" {

iga_status iga_fd_apply(int dtype, int ndim, const int32_t* n, const int32_t* lo, const int32_t* m,
                        const void* const* U, const void* inv_lambda, int64_t ncols, const void* x,
                        void* y, void* work0, void* work1, iga_stream stream) {
  clear_error();
  IGA_CHECK_ARG(ndim >= 1 && ndim <= 4, "ndim %d out of range", ndim);
  IGA_CHECK_ARG(n && lo && m && U && inv_lambda && x && y && work0 && work1, "null argument");
  IGA_CHECK_ARG(ncols >= 1, "ncols must be >= 1");
  IGA_CHECK_ARG(dtype == IGA_F64 || dtype == IGA_F32, "dtype %d not supported", dtype);
  Box b;
  b.ndim = ndim;
  int64_t N = 1, M = 1;
  for (int d = 0; d < 4; ++d) {
    b.n[d] = d < ndim ? n[d] : 1;
    b.lo[d] = d < ndim ? lo[d] : 0;
    b.m[d] = d < ndim ? m[d] : 1;
    IGA_CHECK_ARG(b.lo[d] >= 0 && b.m[d] >= 0 && b.lo[d] + b.m[d] <= b.n[d],
                  "free box of direction %d out of range", d);
    N *= b.n[d];
    M *= b.m[d];
  }
  cudaStream_t st = as_stream(stream);
  const size_t esz = dtype == IGA_F64 ? 8 : 4;
  IGA_CUDA_TRY(cudaMemsetAsync(y, 0, (size_t)N * ncols * esz, st));
  if (M == 0) return IGA_OK;
  return dtype == IGA_F64
             ? fd_apply_t<double>(b, U, (const double*)inv_lambda, ncols, (const double*)x,
                                  (double*)y, (double*)work0, (double*)work1, stream)
             : fd_apply_t<float>(b, U, (const float*)inv_lambda, ncols, (const float*)x, (float*)y,
                                 (float*)work0, (float*)work1, stream);
}

}  // extern "C"
