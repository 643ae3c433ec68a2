// Space-time fast-diagonalisation preconditioner (arrowhead form).
//
// SpTimeFD.apply / apply_transpose (src/igaops/fastdiag/utils/time_arrow.py:
// 112-192): on the free nodes (time indices 1..nt-1 times the spatial free
// box; time is the slowest direction)
//   x -> (U_s^T per space direction) -> (conj(Ut)^T in time)
//     -> arrowhead solve with H_ij = adv*Dt_i + Lambda_j
//     -> (Ut in time) -> (U_s per space direction) -> real part,
// where Ut (complex) diagonalises the time pencil except for one border row
// and column (the arrowhead g).  The transpose swaps Ut / conj(Ut) and uses
// -conj(g).  The arrowhead solve (operations.py:5-93) is one thread per
// spatial eigen-index j walking the time index i: block elimination of the
// border with the Schur complement computed on the fly, complex arithmetic
// in FP64, storage in the element type of the call.
#include "common.cuh"
#include "dense_mode.cuh"

extern "C" iga_status iga_box_copy(int dtype, int ndim, const int32_t* n, const int32_t* lo,
                                   const int32_t* m, int64_t ncols, const void* src, void* dst,
                                   int scatter, iga_stream stream);

namespace iga {

template <typename T>
__global__ void __launch_bounds__(256)
    arrowhead_kernel(int mt, int64_t ms, const double* __restrict__ dt,
                     const double* __restrict__ b, const double* __restrict__ lam,
                     T* __restrict__ re, T* __restrict__ im) {
  const int k = mt - 1;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < ms;
       j += (int64_t)gridDim.x * blockDim.x) {
    const double l = lam[j];
    double sr = dt[2 * k] + l, si = dt[2 * k + 1];  // H_last, then the Schur complement
    double ar = 0.0, ai = 0.0;                       // sum_i conj(b_i) y_i
    for (int i = 0; i < k; ++i) {
      const double hr = dt[2 * i] + l, hi = dt[2 * i + 1];
      const double den = hr * hr + hi * hi;
      const double br = b[2 * i], bi = b[2 * i + 1];
      const double bb = br * br + bi * bi;
      sr += bb * hr / den;
      si -= bb * hi / den;
      const int64_t o = (int64_t)i * ms + j;
      const double rr = (double)re[o], ri = (double)im[o];
      const double yr = (rr * hr + ri * hi) / den, yi = (ri * hr - rr * hi) / den;
      re[o] = (T)yr;
      im[o] = (T)yi;
      ar += br * yr + bi * yi;
      ai += br * yi - bi * yr;
    }
    const int64_t ol = (int64_t)k * ms + j;
    const double lr = (double)re[ol] + ar, li = (double)im[ol] + ai;
    const double sd = sr * sr + si * si;
    const double xr = (lr * sr + li * si) / sd, xi = (li * sr - lr * si) / sd;
    re[ol] = (T)xr;
    im[ol] = (T)xi;
    for (int i = 0; i < k; ++i) {
      const double hr = dt[2 * i] + l, hi = dt[2 * i + 1];
      const double den = hr * hr + hi * hi;
      const double br = b[2 * i], bi = b[2 * i + 1];
      const double mr = (br * hr + bi * hi) / den, mi = (bi * hr - br * hi) / den;
      const int64_t o = (int64_t)i * ms + j;
      re[o] = (T)((double)re[o] - (mr * xr - mi * xi));
      im[o] = (T)((double)im[o] - (mr * xi + mi * xr));
    }
  }
}

// The time part of the apply in one launch: forward rotation, arrowhead solves
// and backward rotation of BN spatial eigen-indices per CTA, the time vectors in
// shared memory throughout. The rotations are FP64 tensor-core products
// (dense_mode.cuh); a warp solves one column, lanes over the time index, the
// border's two sums by shuffles (the thread-per-column form above is a chain of
// mt complex divisions: 26 us at mt = 26, half of the whole apply).
//   re = Ur^T a, im = s Ui^T a;  arrowhead;  w = Ur re + s Ui im
// with s = -1 for the apply, +1 for its transpose.
constexpr int kTimeCols = 16;

template <typename T>
struct TimeArgs {
  const T* ur;
  const T* ui;
  const double* dt;
  const double* b;
  const double* lam;
  const T* x;  // (mt, ms)
  T* y;        // (mt, ms)
  int32_t mt;
  int32_t ms;
  double sign;
};

static size_t time_smem(int mt) {
  const size_t ar = (mt + 7) / 8 * 8;
  return (2 * ar * dense_ld(mt) + 3 * ar * (kTimeCols + 4)) * 8;
}

template <typename T>
__global__ void __launch_bounds__(kDenseThreads) sptime_time_kernel(const __grid_constant__ TimeArgs<T> p) {
  extern __shared__ __align__(16) double sm[];
  constexpr int BN = kTimeCols, LDX = BN + 4, CB = BN / 8, NW = kDenseThreads / 32, RG = NW / CB;
  static_assert(NW == BN, "one warp per column");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
  const int mt = p.mt, kp = (mt + 3) / 4 * 4, ar = (mt + 7) / 8 * 8, lda = dense_ld(mt);
  double* Ar = sm;
  double* Ai = Ar + ar * lda;
  double* Xs = Ai + ar * lda;
  double* Tr = Xs + ar * LDX;
  double* Ti = Tr + ar * LDX;
  const int j0 = blockIdx.x * BN, bn = min(BN, p.ms - j0);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  for (int r = warp; r < ar; r += NW)
    for (int c = lane; c < lda; c += 32) {
      if (r < mt && c < mt) {
        stage_elem<true>(Ar + r * lda + c, p.ur + (int64_t)r * mt + c);
        stage_elem<true>(Ai + r * lda + c, p.ui + (int64_t)r * mt + c);
      } else {
        Ar[r * lda + c] = Ai[r * lda + c] = 0.0;
      }
    }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int e = tid; e < ar * BN; e += kDenseThreads) {
    const int i = e / BN, j = e % BN;
    if (i < mt && j < bn) stage_elem<false>(Xs + i * LDX + j, p.x + (int64_t)i * p.ms + j0 + j);
    else Xs[i * LDX + j] = 0.0;
  }
  if constexpr (sizeof(T) == 8) asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int cb = warp % CB, rg = warp / CB, nc = cb * 8 + 2 * tq;
  // forward: rows k of U^T, A[k][i] = U[i][k]
  for (int rb = rg; rb < ar / 8; rb += RG) {
    double re[1][2], im[1][2];
    const double* bl = Xs + tq * LDX + cb * 8 + gq;
    block_rows<1, true>(re, Ar + rb * 8 + gq + tq * lda, 0, lda, bl, LDX, kp);
    block_rows<1, true>(im, Ai + rb * 8 + gq + tq * lda, 0, lda, bl, LDX, kp);
    double* dr = Tr + (rb * 8 + gq) * LDX + nc;
    double* di = Ti + (rb * 8 + gq) * LDX + nc;
    dr[0] = re[0][0];
    dr[1] = re[0][1];
    di[0] = p.sign * im[0][0];
    di[1] = p.sign * im[0][1];
  }
  __syncthreads();
  // arrowhead solve of column `warp`: H_i = dt_i + lambda, border b
  if (warp < bn) {
    const int k = mt - 1;
    const double l = __ldg(p.lam + j0 + warp);
    double* cr = Tr + warp;
    double* ci = Ti + warp;
    double sr = 0.0, si = 0.0, tr = 0.0, ti = 0.0;
    for (int i = lane; i < k; i += 32) {
      const double hr = __ldg(p.dt + 2 * i) + l, hi = __ldg(p.dt + 2 * i + 1);
      const double den = hr * hr + hi * hi;
      const double br = __ldg(p.b + 2 * i), bi = __ldg(p.b + 2 * i + 1);
      const double bb = br * br + bi * bi;
      sr += bb * hr / den;
      si -= bb * hi / den;
      const double rr = cr[i * LDX], ri = ci[i * LDX];
      const double yr = (rr * hr + ri * hi) / den, yi = (ri * hr - rr * hi) / den;
      cr[i * LDX] = yr;
      ci[i * LDX] = yi;
      tr += br * yr + bi * yi;
      ti += br * yi - bi * yr;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, o);
      si += __shfl_xor_sync(0xffffffffu, si, o);
      tr += __shfl_xor_sync(0xffffffffu, tr, o);
      ti += __shfl_xor_sync(0xffffffffu, ti, o);
    }
    sr += __ldg(p.dt + 2 * k) + l;  // the Schur complement of the border
    si += __ldg(p.dt + 2 * k + 1);
    const double lr = cr[k * LDX] + tr, li = ci[k * LDX] + ti;
    const double sd = sr * sr + si * si;
    const double xr = (lr * sr + li * si) / sd, xi = (li * sr - lr * si) / sd;
    __syncwarp();
    for (int i = lane; i < k; i += 32) {
      const double hr = __ldg(p.dt + 2 * i) + l, hi = __ldg(p.dt + 2 * i + 1);
      const double den = hr * hr + hi * hi;
      const double br = __ldg(p.b + 2 * i), bi = __ldg(p.b + 2 * i + 1);
      const double mr = (br * hr + bi * hi) / den, mi = (bi * hr - br * hi) / den;
      cr[i * LDX] -= mr * xr - mi * xi;
      ci[i * LDX] -= mr * xi + mi * xr;
    }
    if (lane == 0) {
      cr[k * LDX] = xr;
      ci[k * LDX] = xi;
    }
  }
  __syncthreads();
  // fold the sign of the imaginary part's backward rotation into the result
  for (int rb = rg; rb < ar / 8; rb += RG) {
    double re[1][2], im[1][2];
    const int o = tq * LDX + cb * 8 + gq;
    block_rows<1, true>(re, Ar + (rb * 8 + gq) * lda + tq, 0, 1, Tr + o, LDX, kp);
    block_rows<1, true>(im, Ai + (rb * 8 + gq) * lda + tq, 0, 1, Ti + o, LDX, kp);
    const int r = rb * 8 + gq;
    if (r < mt) {
      T* dst = p.y + (int64_t)r * p.ms + j0 + nc;
      if (nc < bn) dst[0] = (T)(re[0][0] + p.sign * im[0][0]);
      if (nc + 1 < bn) dst[1] = (T)(re[0][1] + p.sign * im[0][1]);
    }
  }
}

template <typename T>
static iga_status launch_time(const TimeArgs<T>& a, cudaStream_t st) {
  auto kern = sptime_time_kernel<T>;
  const size_t smem = time_smem(a.mt);
  static SmemOptIn optin;
  IGA_CUDA_TRY(optin.allow((const void*)kern, smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ceil_div(a.ms, kTimeCols));
  cfg.blockDim = dim3(kDenseThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  IGA_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, a));
  return IGA_OK;
}

// The apply on y (already zero) where the time vectors fit shared memory: space
// products, the time kernel, space products back; up to two space directions the
// first product gathers the box and the last scatters it. sdim = 2: 5 launches
// instead of 13 (2D p3 24^2 x 24: 134 -> 27 us a call).
template <typename T>
static iga_status sptime_fused(int sdim, const int32_t* n, const int32_t* lo, const int32_t* m,
                               const void* const* U, TimeArgs<T> ta, const T* x, T* y, T* work0,
                               T* work1, iga_stream stream) {
  cudaStream_t st = as_stream(stream);
  const int nd = sdim + 1;
  const bool direct = sdim <= 2;
  T* buf[2] = {work0, work1};
  const T* cur = x;
  int next = 0;
  bool dependent = false;
  if (!direct) {
    iga_status rc = iga_box_copy(sizeof(T) == 8 ? IGA_F64 : IGA_F32, nd, n, lo, m, 1, x, work0, 0, stream);
    if (rc) return rc;
    cur = work0;
    next = 1;
  }
  // columns of direction 1's products in the full tensor: (t, i2) or (t)
  const int64_t n0 = n[0], n01 = n0 * (sdim > 1 ? n[1] : 1);
  const int64_t off = lo[0] + (sdim > 1 ? lo[1] * n0 : 0) + lo[sdim] * n01;
  auto mode = [&](int d, bool forward) -> iga_status {
    int64_t outer = m[sdim], inner = 1;
    for (int e = sdim - 1; e > d; --e) outer *= m[e];
    for (int e = d - 1; e >= 0; --e) inner *= m[e];
    const bool gather = direct && cur == x, scatter = direct && !forward && d == 0;
    T* dst = scatter ? y : buf[next];
    DenseMode<T> p = dense_compact<T>((const T*)U[d], forward ? 1 : m[d], forward ? m[d] : 1, m[d],
                                      m[d], outer, inner, cur, dst);
    if (gather) {
      p.x = x + off;
      p.xlo = sdim > 1 ? m[1] : 1;
      p.xhi = n01;
      p.xls = n0;
      p.xc = 1;
    }
    if (scatter) {
      p.y = y + off;
      p.ylo = sdim > 1 ? m[1] : 1;
      p.yhi = n01;
      p.yls = n0;
      p.yr = 1;
    }
    iga_status rc = launch_dense_mode<T>(p, false, dependent, st);
    if (rc) return rc;
    dependent = true;
    cur = dst;
    next ^= 1;
    return IGA_OK;
  };
  iga_status rc;
  for (int d = 0; d < sdim; ++d)
    if ((rc = mode(d, true))) return rc;
  ta.x = cur;
  ta.y = buf[next];
  if ((rc = launch_time<T>(ta, st))) return rc;
  cur = buf[next];
  next ^= 1;
  for (int d = sdim - 1; d >= 0; --d)
    if ((rc = mode(d, false))) return rc;
  if (direct) return IGA_OK;
  return iga_box_copy(sizeof(T) == 8 ? IGA_F64 : IGA_F32, nd, n, lo, m, 1, cur, y, 1, stream);
}

// Triangular solves of the QZ (legacy) space-time FD (src/igaops/fastdiag/
// utils/time_legacy.py:61-170): for every spatial eigen-index j, the time
// vector (re, im)[i * ms + j], i < mt, is replaced by the solution of
//   (adv S + lam_j T) y = rhs        (upper triangular; apply)
//   (adv S + lam_j T)^T y = rhs      (lower triangular; transpose)
// with S, T the complex generalized Schur forms (row-major (re, im) pairs).
// One thread per j, complex arithmetic in FP64.
template <typename T>
__global__ void __launch_bounds__(256)
    qz_tri_kernel(int mt, int64_t ms, const double* __restrict__ S, const double* __restrict__ Tm,
                  double adv, const double* __restrict__ lam, int transpose, T* __restrict__ re,
                  T* __restrict__ im) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < ms;
       j += (int64_t)gridDim.x * blockDim.x) {
    const double l = lam[j];
    for (int s = 0; s < mt; ++s) {
      const int i = transpose ? s : mt - 1 - s;
      double ar = (double)re[(int64_t)i * ms + j], ai = (double)im[(int64_t)i * ms + j];
      const int k0 = transpose ? 0 : i + 1, k1 = transpose ? i : mt;
      for (int k = k0; k < k1; ++k) {
        // M_ik (apply) or M_ki (transpose), M = adv S + lam T
        const int64_t e = transpose ? ((int64_t)k * mt + i) : ((int64_t)i * mt + k);
        const double mr = adv * S[2 * e] + l * Tm[2 * e];
        const double mi = adv * S[2 * e + 1] + l * Tm[2 * e + 1];
        const double yr = (double)re[(int64_t)k * ms + j], yi = (double)im[(int64_t)k * ms + j];
        ar -= mr * yr - mi * yi;
        ai -= mr * yi + mi * yr;
      }
      const int64_t d = (int64_t)i * mt + i;
      const double dr = adv * S[2 * d] + l * Tm[2 * d], di = adv * S[2 * d + 1] + l * Tm[2 * d + 1];
      const double den = dr * dr + di * di;
      re[(int64_t)i * ms + j] = (T)((ar * dr + ai * di) / den);
      im[(int64_t)i * ms + j] = (T)((ai * dr - ar * di) / den);
    }
  }
}

}  // namespace iga

using namespace iga;

extern "C" {

iga_status iga_mode_product(int dtype, const iga_factor* M, int64_t outer, int64_t inner,
                            const void* x, void* y, int accumulate, iga_stream stream);
iga_status iga_axpby(int dtype, int64_t n, double alpha, const void* x, double beta, void* y,
                     iga_stream stream);
iga_status iga_box_copy(int dtype, int ndim, const int32_t* n, const int32_t* lo,
                        const int32_t* m, int64_t ncols, const void* src, void* dst, int scatter,
                        iga_stream stream);

iga_status iga_arrowhead_solve(int dtype, int mt, int64_t ms, const double* dt, const double* b,
                               const double* lam, void* re, void* im, iga_stream stream) {
  clear_error();
  IGA_CHECK_ARG(mt >= 1 && ms >= 0 && dt && lam && re && im && (mt == 1 || b), "bad argument");
  if (ms == 0) return IGA_OK;
  int64_t blocks = ceil_div(ms, 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  cudaStream_t st = as_stream(stream);
  if (dtype == IGA_F64)
    arrowhead_kernel<double><<<(unsigned)blocks, 256, 0, st>>>(mt, ms, dt, b, lam, (double*)re,
                                                               (double*)im);
  else if (dtype == IGA_F32)
    arrowhead_kernel<float><<<(unsigned)blocks, 256, 0, st>>>(mt, ms, dt, b, lam, (float*)re,
                                                              (float*)im);
  else {
    set_error("dtype %d not supported", dtype);
    return IGA_ERR_UNSUPPORTED;
  }
  IGA_LAUNCH_CHECK();
  return IGA_OK;
}

iga_status iga_fd_sptime_apply(int dtype, int sdim, const int32_t* n, const int32_t* lo,
                               const int32_t* m, const void* const* U, const void* ut_re,
                               const void* ut_im, const double* dt, const double* bfac,
                               const double* lam, int transpose, const void* x, void* y,
                               void* work0, void* work1, void* work2, iga_stream stream) {
  clear_error();
  IGA_CHECK_ARG(sdim >= 1 && sdim <= 3, "space dimension %d out of range", sdim);
  IGA_CHECK_ARG(n && lo && m && U && ut_re && ut_im && dt && lam && x && y && work0 && work1 &&
                    work2,
                "null argument");
  IGA_CHECK_ARG(dtype == IGA_F64 || dtype == IGA_F32, "dtype %d not supported", dtype);
  const int nd = sdim + 1;
  int64_t N = 1, M = 1, ms = 1;
  for (int d = 0; d < nd; ++d) {
    IGA_CHECK_ARG(m[d] >= 1 && lo[d] >= 0 && lo[d] + m[d] <= n[d], "box of direction %d", d);
    N *= n[d];
    M *= m[d];
    if (d < sdim) ms *= m[d];
  }
  const int mt = m[sdim];
  IGA_CHECK_ARG(mt == 1 || bfac, "null arrowhead border");
  cudaStream_t st = as_stream(stream);
  const size_t esz = dtype == IGA_F64 ? 8 : 4;
  IGA_CUDA_TRY(cudaMemsetAsync(y, 0, (size_t)N * esz, st));
  bool fused = ms < (1ll << 31) && time_smem(mt) <= 227 * 1024;
  for (int d = 0; d < sdim; ++d) fused = fused && dense_fits(m[d], m[d], M / m[d]);
  if (fused) {
    auto run = [&](auto tag) -> iga_status {
      using T = decltype(tag);
      TimeArgs<T> ta{(const T*)ut_re, (const T*)ut_im, dt, bfac, lam, nullptr, nullptr,
                     mt, (int32_t)ms, transpose ? 1.0 : -1.0};
      return sptime_fused<T>(sdim, n, lo, m, U, ta, (const T*)x, (T*)y, (T*)work0, (T*)work1, stream);
    };
    return dtype == IGA_F64 ? run(double{}) : run(float{});
  }
  iga_status rc = iga_box_copy(dtype, nd, n, lo, m, 1, x, work0, 0, stream);
  if (rc) return rc;
  void* buf[2] = {work0, work1};
  int cur = 0;
  auto dense = [&](const void* A, int rows, bool tr) {
    iga_factor F;
    memset(&F, 0, sizeof(F));
    F.kind = 1;
    F.rows = F.cols = rows;
    F.ld_row = tr ? 1 : rows;
    F.ld_col = tr ? rows : 1;
    F.dense = A;
    return F;
  };
  auto space_pass = [&](bool forward) -> iga_status {
    // tensor (mt, m_sdim-1, ..., m_0): direction d has outer = mt * prod_{d'>d} m,
    // inner = prod_{d'<d} m
    for (int d = sdim - 1; d >= 0; --d) {
      iga_factor F = dense(U[d], m[d], forward);
      int64_t outer = mt, inner = 1;
      for (int e = sdim - 1; e > d; --e) outer *= m[e];
      for (int e = d - 1; e >= 0; --e) inner *= m[e];
      iga_status r = iga_mode_product(dtype, &F, outer, inner, buf[cur], buf[cur ^ 1], 0, stream);
      if (r) return r;
      cur ^= 1;
    }
    return IGA_OK;
  };
  if ((rc = space_pass(true))) return rc;
  // time forward: re = Ut_re^T a, im = -+ Ut_im^T a (conj(Ut)^T for apply, Ut^T for transpose)
  void* a = buf[cur];
  void* re = buf[cur ^ 1];
  void* im = work2;
  {
    iga_factor Fr = dense(ut_re, mt, true), Fi = dense(ut_im, mt, true);
    if ((rc = iga_mode_product(dtype, &Fr, 1, ms, a, re, 0, stream))) return rc;
    if ((rc = iga_mode_product(dtype, &Fi, 1, ms, a, im, 0, stream))) return rc;
    if (!transpose && (rc = iga_axpby(dtype, M, -1.0, im, 0.0, im, stream))) return rc;
  }
  if ((rc = iga_arrowhead_solve(dtype, mt, ms, dt, bfac, lam, re, im, stream))) return rc;
  // time backward: w = Re(Ut z) = Ut_re z_re - Ut_im z_im (apply) or
  // Re(conj(Ut) z) = Ut_re z_re + Ut_im z_im (transpose)
  {
    if (!transpose && (rc = iga_axpby(dtype, M, -1.0, im, 0.0, im, stream))) return rc;
    iga_factor Fr = dense(ut_re, mt, false), Fi = dense(ut_im, mt, false);
    if ((rc = iga_mode_product(dtype, &Fr, 1, ms, re, a, 0, stream))) return rc;
    if ((rc = iga_mode_product(dtype, &Fi, 1, ms, im, a, 1, stream))) return rc;
  }
  if ((rc = space_pass(false))) return rc;
  return iga_box_copy(dtype, nd, n, lo, m, 1, buf[cur], y, 1, stream);
}


iga_status iga_fd_sptime_qz_apply(int dtype, int sdim, const int32_t* n, const int32_t* lo,
                                  const int32_t* m, const void* const* U, const void* q_re,
                                  const void* q_im, const void* z_re, const void* z_im,
                                  const double* S, const double* Tm, double adv,
                                  const double* lam, int transpose, const void* x, void* y,
                                  void* work0, void* work1, void* work2, iga_stream stream) {
  clear_error();
  IGA_CHECK_ARG(sdim >= 1 && sdim <= 3, "space dimension %d out of range", sdim);
  IGA_CHECK_ARG(n && lo && m && U && q_re && q_im && z_re && z_im && S && Tm && lam && x && y &&
                    work0 && work1 && work2,
                "null argument");
  IGA_CHECK_ARG(dtype == IGA_F64 || dtype == IGA_F32, "dtype %d not supported", dtype);
  const int nd = sdim + 1;
  int64_t N = 1, M = 1, ms = 1;
  for (int d = 0; d < nd; ++d) {
    IGA_CHECK_ARG(m[d] >= 1 && lo[d] >= 0 && lo[d] + m[d] <= n[d], "box of direction %d", d);
    N *= n[d];
    M *= m[d];
    if (d < sdim) ms *= m[d];
  }
  const int mt = m[sdim];
  cudaStream_t st = as_stream(stream);
  const size_t esz = dtype == IGA_F64 ? 8 : 4;
  IGA_CUDA_TRY(cudaMemsetAsync(y, 0, (size_t)N * esz, st));
  iga_status rc = iga_box_copy(dtype, nd, n, lo, m, 1, x, work0, 0, stream);
  if (rc) return rc;
  void* buf[2] = {work0, work1};
  int cur = 0;
  auto dense = [&](const void* A, int rows, bool tr) {
    iga_factor F;
    memset(&F, 0, sizeof(F));
    F.kind = 1;
    F.rows = F.cols = rows;
    F.ld_row = tr ? 1 : rows;
    F.ld_col = tr ? rows : 1;
    F.dense = A;
    return F;
  };
  auto space_pass = [&](bool forward) -> iga_status {
    for (int d = sdim - 1; d >= 0; --d) {
      iga_factor F = dense(U[d], m[d], forward);
      int64_t outer = mt, inner = 1;
      for (int e = sdim - 1; e > d; --e) outer *= m[e];
      for (int e = d - 1; e >= 0; --e) inner *= m[e];
      iga_status r = iga_mode_product(dtype, &F, outer, inner, buf[cur], buf[cur ^ 1], 0, stream);
      if (r) return r;
      cur ^= 1;
    }
    return IGA_OK;
  };
  if ((rc = space_pass(true))) return rc;
  // time forward: Q^H a (apply: re = Q_re^T a, im = -Q_im^T a) or Z^T a
  // (transpose: re = Z_re^T a, im = Z_im^T a)
  void* a = buf[cur];
  void* re = buf[cur ^ 1];
  void* im = work2;
  {
    iga_factor Fr = dense(transpose ? z_re : q_re, mt, true);
    iga_factor Fi = dense(transpose ? z_im : q_im, mt, true);
    if ((rc = iga_mode_product(dtype, &Fr, 1, ms, a, re, 0, stream))) return rc;
    if ((rc = iga_mode_product(dtype, &Fi, 1, ms, a, im, 0, stream))) return rc;
    if (!transpose && (rc = iga_axpby(dtype, M, -1.0, im, 0.0, im, stream))) return rc;
  }
  {
    int64_t blocks = ceil_div(ms, 256);
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (dtype == IGA_F64)
      qz_tri_kernel<double><<<(unsigned)blocks, 256, 0, st>>>(mt, ms, S, Tm, adv, lam, transpose,
                                                              (double*)re, (double*)im);
    else
      qz_tri_kernel<float><<<(unsigned)blocks, 256, 0, st>>>(mt, ms, S, Tm, adv, lam, transpose,
                                                             (float*)re, (float*)im);
    IGA_LAUNCH_CHECK();
  }
  // time backward: Re(Z y) = Z_re y_re - Z_im y_im (apply) or
  // Re(conj(Q) y) = Q_re y_re + Q_im y_im (transpose)
  {
    if (!transpose && (rc = iga_axpby(dtype, M, -1.0, im, 0.0, im, stream))) return rc;
    iga_factor Fr = dense(transpose ? q_re : z_re, mt, false);
    iga_factor Fi = dense(transpose ? q_im : z_im, mt, false);
    if ((rc = iga_mode_product(dtype, &Fr, 1, ms, re, a, 0, stream))) return rc;
    if ((rc = iga_mode_product(dtype, &Fi, 1, ms, im, a, 1, stream))) return rc;
  }
  if ((rc = space_pass(false))) return rc;
  return iga_box_copy(dtype, nd, n, lo, m, 1, buf[cur], y, 1, stream);
}

}  // extern "C"
