// Pointwise geometry at quadrature points: metric, determinant, pseudo-
// inverse of the Jacobian and the stiffness coefficient tensor.
//
// Follows Operations.inverse_rectangular_matrix and
// eval_inverse_and_determinant (src/igaops/geometry/mixin/operations.py:
// 73-159): G = J^T J, det J = sqrt(det G), J^+ = G^{-1} J^T, with the
// closed-form 1x1 / 2x2 / 3x3 inverse of G; the coefficient of the stiffness
// operator is C = det J * J^+ J^{+T} (how the reference's tests and examples
// build it from EvaluatedSpline, tests/test_assemble.py:116-123).
#include <algorithm>

#include "common.cuh"

namespace iga {

template <int D>
__device__ __forceinline__ void inv_det(const double (&G)[3][3], double (&inv)[3][3],
                                        double& det) {
  if (D == 1) {
    det = G[0][0];
    inv[0][0] = 1.0;
  } else if (D == 2) {
    det = G[0][0] * G[1][1] - G[0][1] * G[1][0];
    inv[0][0] = G[1][1];
    inv[1][1] = G[0][0];
    inv[0][1] = -G[0][1];
    inv[1][0] = -G[1][0];
  } else {
    det = G[0][1] * G[1][2] * G[2][0] - G[0][2] * G[1][1] * G[2][0] + G[0][2] * G[1][0] * G[2][1] -
          G[0][0] * G[1][2] * G[2][1] + G[0][0] * G[1][1] * G[2][2] - G[0][1] * G[1][0] * G[2][2];
    inv[0][0] = G[1][1] * G[2][2] - G[1][2] * G[2][1];
    inv[0][1] = G[0][2] * G[2][1] - G[0][1] * G[2][2];
    inv[0][2] = G[0][1] * G[1][2] - G[0][2] * G[1][1];
    inv[1][0] = G[1][2] * G[2][0] - G[1][0] * G[2][2];
    inv[1][1] = G[0][0] * G[2][2] - G[0][2] * G[2][0];
    inv[1][2] = G[0][2] * G[1][0] - G[0][0] * G[1][2];
    inv[2][0] = G[1][0] * G[2][1] - G[1][1] * G[2][0];
    inv[2][1] = G[0][1] * G[2][0] - G[0][0] * G[2][1];
    inv[2][2] = G[0][0] * G[1][1] - G[0][1] * G[1][0];
  }
#pragma unroll
  for (int i = 0; i < D; ++i)
#pragma unroll
    for (int j = 0; j < D; ++j) inv[i][j] = inv[i][j] / det;
}

// jac: (M, D, Nq) physical coordinate m, parametric direction j.
// Outputs (each optional): det (Nq), invjac (D, M, Nq), coef (D, D, Nq).
template <int D>
__global__ void __launch_bounds__(256) geometry_kernel(int64_t nq, int M,
                                                       const double* __restrict__ jac,
                                                       double* __restrict__ det_out,
                                                       double* __restrict__ invjac_out,
                                                       double* __restrict__ coef_out,
                                                       int32_t* __restrict__ status) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nq;
       q += (int64_t)gridDim.x * blockDim.x) {
    double J[3][3];
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int j = 0; j < D; ++j) J[m][j] = jac[((int64_t)m * D + j) * nq + q];
    double G[3][3];
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = 0; j < D; ++j) {
        double s = 0.0;
        for (int l = 0; l < M; ++l) s += J[l][i] * J[l][j];
        G[i][j] = s;
      }
    double inv[3][3], detG;
    inv_det<D>(G, inv, detG);
    // status bits: 1 = |det G| < 1e-14 (singular metric), 2 = det J <= 0 or NaN
    if (!(fabs(detG) >= 1e-14)) atomicOr(status, 1);
    const double dj = sqrt(detG);
    if (!(dj > 0.0)) atomicOr(status, 2);
    double P[3][3];  // J^+ = G^{-1} J^T : (D x M)
#pragma unroll
    for (int i = 0; i < D; ++i)
      for (int m = 0; m < M; ++m) {
        double s = 0.0;
#pragma unroll
        for (int l = 0; l < D; ++l) s += inv[i][l] * J[m][l];
        P[i][m] = s;
      }
    if (det_out) det_out[q] = dj;
    if (invjac_out)
#pragma unroll
      for (int i = 0; i < D; ++i)
        for (int m = 0; m < M; ++m) invjac_out[((int64_t)i * M + m) * nq + q] = P[i][m];
    if (coef_out)
#pragma unroll
      for (int i = 0; i < D; ++i)
#pragma unroll
        for (int j = 0; j < D; ++j) {
          double s = 0.0;
          for (int l = 0; l < M; ++l) s += P[i][l] * P[j][l];
          coef_out[((int64_t)i * D + j) * nq + q] = s * dj;
        }
  }
}

// ------------------------------------------------- coefficients in one pass
// det J and C = det J * J^+ J^{+T} of a 3D patch straight from its control
// points. J is square, so with its cofactors K (J^{-1} = K^T / det J)
// C_ij = K_i . K_j / |det J|: no product J^T J, whose condition number is squared.
// Rounding: directions are summed in the order 2, 1, 3 (the products: 3, 2, 1). Against
// extended precision both are off by 6.5e-15 (p3 64^3, 64 000 points, relative 2-norm of
// C); two FP64 results of different order differ by 8.9e-15.
//
// A warp owns 32 consecutive points of direction 1 at one point of direction 2
// and marches along a segment of direction 3: lane = point, with the trial
// planes (d1, d2 and value components) of W control planes of every coordinate
// in registers. A new plane is contracted over direction 2 (lanes = control
// points of the 32 points' range) and then direction 1 through a small
// warp-private buffer. Every store of a warp is 256 contiguous bytes.
//
// Bound by the 80 bytes written per point. Before, nine Kronecker products of
// three passes each and a pointwise pass moved about 1.3 KB per point: 3D p3 64^3
// (7.4 M points) 1537 us a call, now 206 (this kernel 169, written bytes alone 94:
// a warp's planes come one after the other, latency keeps it from the store rate).
template <int W>
struct Geo3Args {
  int32_t n[3], nq[3];
  const int32_t* start[3];
  const double* v0[3];
  const double* v1[3];
  const double* x;  // (3, N), direction 1 fastest
  double* det;
  double* coef;
  int32_t* status;
  int32_t nseg;
};

constexpr int kGeoWarps = 4;

template <int W>
__global__ void __launch_bounds__(32 * kGeoWarps)
    geometry3_kernel(const __grid_constant__ Geo3Args<W> a) {
  constexpr int CM = 31 + W + 1;  // control range of 32 points (unit steps), even
  __shared__ double s_t[kGeoWarps][2][3][2][CM];  // plane contracted over direction 2
  __shared__ double s_b1[kGeoWarps][2 * W][32];
  __shared__ __align__(16) double s_b3[kGeoWarps][2][2 * W];  // band values of this and the next point
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n1 = a.n[0], n2 = a.n[1], n3 = a.n[2];
  const int nq1 = a.nq[0], nq2 = a.nq[1], nq3 = a.nq[2];
  const int tiles1 = (nq1 + 31) / 32;
  const int64_t unit = (int64_t)blockIdx.x * kGeoWarps + warp;
  if (unit >= (int64_t)tiles1 * nq2 * a.nseg) return;
  const int t1 = (int)(unit % tiles1);
  const int64_t rest = unit / tiles1;
  const int q2 = (int)(rest % nq2), seg = (int)(rest / nq2);
  const int q1 = t1 * 32 + lane, q1c = min(q1, nq1 - 1);
  const int qa = (int)((int64_t)nq3 * seg / a.nseg);
  const int qb = (int)((int64_t)nq3 * (seg + 1) / a.nseg);
  const int c1lo = __ldg(a.start[0] + t1 * 32), s1 = __ldg(a.start[0] + q1c) - c1lo;
  const int C1r = __ldg(a.start[0] + min(t1 * 32 + 31, nq1 - 1)) - c1lo + W;
  const int c2lo = __ldg(a.start[1] + q2);
  double(*b1)[32] = s_b1[warp];
#pragma unroll
  for (int k = 0; k < W; ++k) {
    b1[k][lane] = __ldg(a.v0[0] + (int64_t)q1c * W + k);
    b1[W + k][lane] = __ldg(a.v1[0] + (int64_t)q1c * W + k);
  }
  const int64_t plane = (int64_t)n1 * n2, N = plane * n3, Nq = (int64_t)nq1 * nq2 * nq3;
  double F[3][3][W];  // [coordinate][d1, d2, value][plane]
  int buf = 0;
  // lane l touches a line of the next plane's 3 W rows (two lines cover the usual
  // 14 control points of 32 points), so that its reads hit L1
  const int prow = min(lane >> 1, 3 * W - 1);
  const double* pre = a.x + (prow / W) * N + (int64_t)min(c2lo + prow % W, n2 - 1) * n1 +
                      min(c1lo + (lane & 1) * (C1r - 1), n1 - 1);
  auto produce = [&](int c3) {
    buf ^= 1;
    const double* xp = a.x + min(c3, n3 - 1) * plane;
    asm volatile("prefetch.global.L1 [%0];" ::"l"(pre + min(c3 + 1, n3 - 1) * plane));
    for (int e = lane; e < 2 * C1r; e += 32) {
      const int b = e >= C1r, c = e - b * C1r;
      const double* bv = (b ? a.v1[1] : a.v0[1]) + (int64_t)q2 * W;
      const int g1 = min(c1lo + c, n1 - 1);
      double v[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int k = 0; k < W; ++k) {
        const double w = __ldg(bv + k);
        const double* xr = xp + (int64_t)min(c2lo + k, n2 - 1) * n1 + g1;
#pragma unroll
        for (int m = 0; m < 3; ++m) v[m] += w * __ldg(xr + m * N);
      }
#pragma unroll
      for (int m = 0; m < 3; ++m) s_t[warp][buf][m][b][c] = v[m];
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < W - 1; ++k) F[m][j][k] = F[m][j][k + 1];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      double d1 = 0.0, d2 = 0.0, v = 0.0;
#pragma unroll
      for (int k = 0; k < W; ++k) {
        const double t0 = s_t[warp][buf][m][0][s1 + k], tv = s_t[warp][buf][m][1][s1 + k];
        d1 += b1[W + k][lane] * t0;
        v += b1[k][lane] * t0;
        d2 += b1[k][lane] * tv;
      }
      F[m][0][W - 1] = d1;
      F[m][1][W - 1] = d2;
      F[m][2][W - 1] = v;
    }
  };
  int base = __ldg(a.start[2] + qa) - W;  // plane below the window
#pragma unroll 1
  for (int k = 0; k < W; ++k) produce(++base + W - 1);
  int flags = 0;
  double* out = a.coef + ((int64_t)qa * nq2 + q2) * nq1 + q1;
  double* dout = a.det + ((int64_t)qa * nq2 + q2) * nq1 + q1;
  // the next point's band values travel through a register of lanes 0 .. 2 W - 1
  auto band3 = [&](int q) {
    const int k = lane % W;
    return __ldg((lane < W ? a.v0[2] : a.v1[2]) + (int64_t)min(q, nq3 - 1) * W + k);
  };
  double nb = band3(qa);
  int s3n = __ldg(a.start[2] + qa);
#pragma unroll 1
  for (int q = qa; q < qb; ++q) {
    double* b3 = s_b3[warp][q & 1];
    if (lane < 2 * W) b3[lane] = nb;
    const int s3 = s3n;
    nb = band3(q + 1);
    s3n = __ldg(a.start[2] + min(q + 1, nq3 - 1));
    while (base < s3) produce(++base + W - 1);
    __syncwarp();
    double J[3][3];
#pragma unroll
    for (int m = 0; m < 3; ++m) J[m][0] = J[m][1] = J[m][2] = 0.0;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const double w0 = b3[k], w1 = b3[W + k];
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        J[m][0] += w0 * F[m][0][k];
        J[m][1] += w0 * F[m][1][k];
        J[m][2] += w1 * F[m][2][k];
      }
    }
    double K[3][3];  // K_i = J_j x J_k (columns): the cofactors of J
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int j = (i + 1) % 3, k = (i + 2) % 3;
      K[0][i] = J[1][j] * J[2][k] - J[2][j] * J[1][k];
      K[1][i] = J[2][j] * J[0][k] - J[0][j] * J[2][k];
      K[2][i] = J[0][j] * J[1][k] - J[1][j] * J[0][k];
    }
    const double dj = fabs(J[0][0] * K[0][0] + J[1][0] * K[1][0] + J[2][0] * K[2][0]);
    // status bits: 1 = |det G| < 1e-14 (singular metric), 2 = det J <= 0 or NaN
    if (!(dj * dj >= 1e-14)) flags |= 1;
    if (!(dj > 0.0)) flags |= 2;
    if (q1 < nq1) {
      if (a.det) *dout = dj;
      if (a.coef) {
        const double r = 1.0 / dj;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = i; j < 3; ++j) {
            const double c = (K[0][i] * K[0][j] + K[1][i] * K[1][j] + K[2][i] * K[2][j]) * r;
            out[(3 * i + j) * Nq] = c;
            if (j > i) out[(3 * j + i) * Nq] = c;
          }
      }
    }
    out += (int64_t)nq1 * nq2;
    dout += (int64_t)nq1 * nq2;
  }
  if (flags && q1 < nq1) atomicOr(a.status, flags);
}

template <int W>
static iga_status launch_geometry3(const iga_mf_plan* p, const double* x, double* det,
                                   double* coef, int32_t* status, cudaStream_t st) {
  Geo3Args<W> a;
  for (int d = 0; d < 3; ++d) {
    a.n[d] = p->n[d];
    a.nq[d] = p->nq[d];
    a.start[d] = p->trial[d].start;
    a.v0[d] = (const double*)p->trial[d].vals;
    a.v1[d] = (const double*)p->trial_d1[d];
  }
  a.x = x;
  a.det = det;
  a.coef = coef;
  a.status = status;
  // segments of at least 4 W points (a segment's first window costs W planes),
  // as many as keep about 32 warps per SM busy
  const int64_t rows = ceil_div(p->nq[0], 32) * p->nq[1];
  a.nseg = (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(148 * 32, rows), p->nq[2] / (4 * W)));
  const int64_t blocks = ceil_div(rows * a.nseg, kGeoWarps);
  IGA_CHECK_ARG(blocks < (1ll << 31), "too many points (%lld blocks)", (long long)blocks);
  geometry3_kernel<W><<<(unsigned)blocks, 32 * kGeoWarps, 0, st>>>(a);
  IGA_LAUNCH_CHECK();
  return IGA_OK;
}

}  // namespace iga

using namespace iga;

extern "C" {

iga_status iga_geometry_coefficients(const iga_mf_plan* plan, const double* ctrlpts, double* det_out,
                                     double* coef_out, int32_t* status, iga_stream stream) {
  clear_error();
  IGA_CHECK_ARG(plan && ctrlpts && status, "null argument");
  IGA_CHECK_ARG(plan->ndim == 3, "one-pass coefficients cover 3D patches, got ndim %d", plan->ndim);
  for (int d = 0; d < 3; ++d) {
    IGA_CHECK_ARG(plan->n[d] >= 1 && plan->nq[d] >= 1, "empty direction %d", d);
    IGA_CHECK_ARG(plan->trial[d].rows == plan->nq[d] && plan->trial[d].cols == plan->n[d] &&
                      plan->trial[d].width == plan->width,
                  "trial band of direction %d does not match the plan", d);
    IGA_CHECK_ARG(plan->trial[d].start && plan->trial[d].vals && plan->trial_d1[d],
                  "trial band of direction %d has null arrays", d);
  }
  cudaStream_t st = as_stream(stream);
  switch (plan->width) {
    case 2: return launch_geometry3<2>(plan, ctrlpts, det_out, coef_out, status, st);
    case 3: return launch_geometry3<3>(plan, ctrlpts, det_out, coef_out, status, st);
    case 4: return launch_geometry3<4>(plan, ctrlpts, det_out, coef_out, status, st);
    case 5: return launch_geometry3<5>(plan, ctrlpts, det_out, coef_out, status, st);
    case 6: return launch_geometry3<6>(plan, ctrlpts, det_out, coef_out, status, st);
    default: break;
  }
  set_error("one-pass coefficients cover band widths 2..6, got %d", plan->width);
  return IGA_ERR_UNSUPPORTED;
}

iga_status iga_geometry_pointwise(int ndim, int ncoord, int64_t nq, const double* jac,
                                  double* det_out, double* invjac_out, double* coef_out,
                                  int32_t* status, iga_stream stream) {
  clear_error();
  IGA_CHECK_ARG(ndim >= 1 && ndim <= 3, "ndim %d out of range", ndim);
  IGA_CHECK_ARG(ncoord >= ndim && ncoord <= 3, "ncoord %d out of range", ncoord);
  IGA_CHECK_ARG(jac && status && nq >= 0, "null argument");
  if (nq == 0) return IGA_OK;
  int64_t blocks = ceil_div(nq, 256);
  if (blocks > 148 * 32) blocks = 148 * 32;
  cudaStream_t st = as_stream(stream);
  switch (ndim) {
    case 1:
      geometry_kernel<1><<<(unsigned)blocks, 256, 0, st>>>(nq, ncoord, jac, det_out, invjac_out,
                                                           coef_out, status);
      break;
    case 2:
      geometry_kernel<2><<<(unsigned)blocks, 256, 0, st>>>(nq, ncoord, jac, det_out, invjac_out,
                                                           coef_out, status);
      break;
    default:
      geometry_kernel<3><<<(unsigned)blocks, 256, 0, st>>>(nq, ncoord, jac, det_out, invjac_out,
                                                           coef_out, status);
  }
  IGA_LAUNCH_CHECK();
  return IGA_OK;
}

}  // extern "C"
