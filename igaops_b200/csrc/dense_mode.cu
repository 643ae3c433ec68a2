// Kernel and launch rule of the dense mode products (see dense_mode.cuh).
#include <algorithm>
#include <type_traits>

#include "dense_mode.cuh"

namespace iga {

template <typename T, int BN, bool TWO>
__global__ void __launch_bounds__(kDenseThreads) dense_mode_kernel(const __grid_constant__ DenseMode<T> p) {
  extern __shared__ __align__(16) double sm[];
  constexpr int LDX = BN + 4;
  constexpr int CB = BN / 8;                       // column blocks
  constexpr int RG = (kDenseThreads / 32) / CB;    // warps per column block
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gq = lane >> 2, tq = lane & 3;
  const int K = p.cols, kp = (K + 3) / 4 * 4, lda = dense_ld(K);
  const int r_lo = blockIdx.y * p.mb, mr = min(p.mb, p.rows - r_lo);
  // rows of A in shared memory: the CTA's rows, in two stages also the k padding
  const int ar = TWO ? (kp + 7) / 8 * 8 : (mr + 7) / 8 * 8;
  const int xr = TWO ? ar : kp;
  double* As = sm;
  double* Xs = As + ar * lda;
  double* Ts = Xs + xr * LDX;  // TWO only
  const int64_t n_lo = (int64_t)blockIdx.x * BN;
  const int bn = (int)min((int64_t)BN, p.N - n_lo);

  // the next product may set itself up; it waits before it reads this output
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  constexpr int NW = kDenseThreads / 32;
  // A: lanes along the unit stride of the factor (U: rows; U^T: 8 rows x 4
  // columns per warp, 64-byte reads and conflict-free stores), zero padding
  if (p.ldc == 1) {
    for (int r = warp; r < mr; r += NW) {
      const T* src = p.A + (int64_t)(r_lo + r) * p.ldr;
      double* dst = As + r * lda;
#pragma unroll 4
      for (int c = lane; c < K; c += 32) stage_elem<true>(dst + c, src + c);
    }
  } else {
    for (int c = warp * 4 + tq; c < K; c += 4 * NW) {
      const T* src = p.A + (int64_t)r_lo * p.ldr + (int64_t)c * p.ldc;
      double* dst = As + c;
#pragma unroll 4
      for (int r = gq; r < mr; r += 8) stage_elem<true>(dst + r * lda, src + (int64_t)r * p.ldr);
    }
  }
  for (int r = tid; r < ar; r += kDenseThreads)
    for (int c = r < mr ? K : 0; c < kp; ++c) As[r * lda + c] = 0.0;
  // X tile [c][n]; padding rows and columns zero
  for (int e = tid; e < (xr - K) * BN; e += kDenseThreads) Xs[(K + e / BN) * LDX + e % BN] = 0.0;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (p.xc == 1) {  // the contracted mode is contiguous: 8 (c) x 4 (n) per warp
    for (int n = warp * 4 + (lane >> 3); n < BN; n += 4 * NW) {
      const uint32_t g = (uint32_t)n_lo + n;
      const T* src = p.x + (int64_t)(g / (uint32_t)p.xlo) * p.xhi + (int64_t)(g % (uint32_t)p.xlo) * p.xls;
      double* dst = Xs + n;
      if (n < bn) {
#pragma unroll 4
        for (int c = lane & 7; c < K; c += 8) stage_elem<false>(dst + c * LDX, src + c);
      } else {
        for (int c = lane & 7; c < K; c += 8) dst[c * LDX] = 0.0;
      }
    }
  } else {
    const int n = tid % BN;
    const uint32_t g = (uint32_t)n_lo + n;
    const T* src = p.x + (int64_t)(g / (uint32_t)p.xlo) * p.xhi + (int64_t)(g % (uint32_t)p.xlo) * p.xls;
    double* dst = Xs + n;
    if (n < bn) {
#pragma unroll 4
      for (int c = tid / BN; c < K; c += kDenseThreads / BN) stage_elem<false>(dst + c * LDX, src + c * p.xc);
    } else {
      for (int c = tid / BN; c < K; c += kDenseThreads / BN) dst[c * LDX] = 0.0;
    }
  }
  if constexpr (sizeof(T) == 8) asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  // warp: column block cb, row blocks rb = rg, rg + RG, ...
  const int cb = warp % CB, rg = warp / CB;
  // this lane's two output columns
  const int nc = cb * 8 + 2 * tq;
  int64_t yoff[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint32_t g = (uint32_t)n_lo + nc + j;
    yoff[j] = (int64_t)(g / (uint32_t)p.ylo) * p.yhi + (int64_t)(g % (uint32_t)p.ylo) * p.yls;
  }
  auto store = [&](int rb, const double (&acc)[2]) {
    const int r = rb * 8 + gq;
    if (r >= mr) return;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if (nc + j >= bn) continue;
      double v = acc[j];
      if (!TWO && p.scale) v *= (double)__ldg(p.scale + ((int64_t)(r_lo + r) * p.N + n_lo + nc + j) / p.scale_div);
      T* dst = p.y + yoff[j] + (int64_t)(r_lo + r) * p.yr;
      *dst = p.accumulate ? (T)((double)*dst + v) : (T)v;
    }
  };
  auto mid = [&](int rb, const double (&acc)[2]) {  // first stage's result, scaled
    const int r = rb * 8 + gq;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      double v = 0.0;
      if (r < mr && nc + j < bn)
        v = acc[j] * (double)__ldg(p.scale + ((int64_t)r * p.N + n_lo + nc + j) / p.scale_div);
      Ts[r * LDX + nc + j] = v;
    }
  };
  auto rows = [&](const double* a, int sr, int sc, const double* x, auto&& out) {
    const int nb = (ar + 7) / 8, mine = nb > rg ? (nb - rg + RG - 1) / RG : 0;
    const double* al = a + gq * sr + tq * sc;
    const double* bl = x + tq * LDX + cb * 8 + gq;
    for (int i = 0; i < mine;) {
      const int left = mine - i, passes = (left + 3) / 4, now = (left + passes - 1) / passes;
      const int rb = rg + i * RG;
      auto run = [&](auto tag) {
        constexpr int R = decltype(tag)::value;
        double acc[R][2];
        block_rows<R, true>(acc, al + rb * 8 * sr, RG * 8 * sr, sc, bl, LDX, kp);
#pragma unroll
        for (int k = 0; k < R; ++k) out(rb + k * RG, acc[k]);
      };
      switch (now) {
        case 4: run(std::integral_constant<int, 4>{}); break;
        case 3: run(std::integral_constant<int, 3>{}); break;
        case 2: run(std::integral_constant<int, 2>{}); break;
        default: run(std::integral_constant<int, 1>{}); break;
      }
      i += now;
    }
  };
  if constexpr (TWO) {
    rows(As, lda, 1, Xs, mid);
    __syncthreads();
    rows(As, 1, lda, Ts, store);
  } else {
    rows(As, lda, 1, Xs, store);
  }
}

// Tile choice: the (rows, columns) per CTA that the cost model ranks first. A CTA
// pays a fixed part (launch, first loads, epilogue; about 2500 cycles), the
// staging of its operands (8 elements a cycle) and its products (64 a cycle,
// shared by the CTAs of an SM); CTAs run in waves.
struct DenseTile {
  int mb, bn;
};
static DenseTile dense_tile(int rows, int cols, int64_t N, bool two) {
  DenseTile best{rows, 64};
  double cost = 1e300;
  const int full = (rows + 7) / 8 * 8;
  for (int bn = 16; bn <= 64; bn *= 2) {
    // the rows in 1 .. 16 equal parts, or in parts of 64 .. 8
    for (int split = 1; split <= 20; ++split) {
      const int mb = split <= 16 ? ((full + split - 1) / split + 7) / 8 * 8 : 64 >> (split - 17);
      if (split > 1 && (two || mb > full)) continue;
      const size_t sm = dense_smem(mb, cols, bn, two);
      if (sm > 227 * 1024) continue;
      const int occ = std::max(1, std::min(4, (int)(227 * 1024 / (sm + 1024))));
      const double ctas = (double)ceil_div(N, bn) * ceil_div(rows, mb);
      const double per_sm = std::min((double)occ, std::max(1.0, ctas / 148.0));
      const double work = ((double)mb * cols + (double)cols * bn) / 8.0 +
                          (two ? 2.0 : 1.0) * mb * bn * cols / 64.0;
      const double c = (2500.0 + per_sm * work) * std::max(1.0, (double)ceil_div((int64_t)ctas, 148 * occ));
      if (c < cost) {
        cost = c;
        best = {mb, bn};
      }
    }
  }
  return best;
}

template <typename T, int BN, bool TWO>
static iga_status launch_tile(const DenseMode<T>& p, size_t smem, bool dependent, cudaStream_t st) {
  auto kern = dense_mode_kernel<T, BN, TWO>;
  static SmemOptIn optin;
  IGA_CUDA_TRY(optin.allow((const void*)kern, smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ceil_div(p.N, BN), (unsigned)ceil_div(p.rows, p.mb));
  cfg.blockDim = dim3(kDenseThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = dependent ? 1 : 0;
  IGA_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p));
  return IGA_OK;
}

template <typename T>
iga_status launch_dense_mode(const DenseMode<T>& q, bool two, bool dependent, cudaStream_t st) {
  DenseMode<T> p = q;
  const DenseTile t = dense_tile(p.rows, p.cols, p.N, two);
  p.mb = t.mb;
  const size_t smem = dense_smem(t.mb, p.cols, t.bn, two);
#define IGA_BN(B)                                                                   \
  return two ? launch_tile<T, B, true>(p, smem, dependent, st)                      \
             : launch_tile<T, B, false>(p, smem, dependent, st)
  switch (t.bn) {
    case 16: IGA_BN(16);
    case 32: IGA_BN(32);
    default: IGA_BN(64);
  }
#undef IGA_BN
}

template iga_status launch_dense_mode<double>(const DenseMode<double>&, bool, bool, cudaStream_t);
template iga_status launch_dense_mode<float>(const DenseMode<float>&, bool, bool, cudaStream_t);

}  // namespace iga
