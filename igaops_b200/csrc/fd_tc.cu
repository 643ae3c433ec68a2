// Fast-diagonalisation apply on the 5th-generation tensor cores (tcgen05).
//
// P^{-1} v = (U_3 x U_2 x U_1) Lambda^{-1} (U_3 x U_2 x U_1)^T v on the free
// box (SpaceFD.apply, src/igaops/fastdiag/utils/space_precond.py:273-320) is
// 2*d mode products with dense m x m eigenvector matrices.  Each mode product
// here is one GEMM
//     D[row][a] = sum_k T[row][k] * B[k][a]
// whose data operand T is K-major: every GEMM stores its output with the
// tensor dims rotated (the contracted dim becomes the slowest, the next
// contraction dim the fastest), so after d products the order is natural
// again.  Operands are BF16 in shared memory (no-swizzle canonical UMMA
// layout), the accumulator is FP32 in tensor memory (TMEM); one CTA of 4
// warps owns 128 rows and the whole N (= m <= 256):
//   * warps stage the A tile (128 rows x Kp) with 16-byte vector loads, or
//     gather it from the FP32/FP64 input vector (first product);
//   * thread 0 brings the pre-tiled B image with one TMA bulk copy, issues
//     Kp/16 tcgen05.mma (M=128, N=Np, K=16) and tcgen05.commit;
//   * each warp reads its 32 TMEM lanes (tcgen05.ld 32x32b) and stores the
//     rotated output as BF16 (optionally times 1/Lambda), or scatters the
//     final product into the output vector.
// Boxes of extents up to 128 take the products over directions 1 and 2 in one
// kernel, four kernels in all (further down); larger ones run the six products.
#include <vector>

#include "common.cuh"

#include <cuda_bf16.h>

namespace iga {

namespace tc {

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  // SWIZZLE_NONE canonical layout; version 1 (sm_100) at bit 46
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

// kind::f16 instruction descriptor: BF16 x BF16 -> F32, both K-major
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

__device__ __forceinline__ void mma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc,
                                         uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Programmatic dependent launch: products 2..6 of an apply are launched
// while the previous product still runs.  A CTA signals that the next
// product may be scheduled once it holds its tensor memory (so a CTA that
// can still block in tcgen05.alloc always belongs to the newest grid, and
// the older grids never wait on it), and waits for the previous product's
// completion before it reads any data that product writes.
__device__ __forceinline__ void launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_prerequisites() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace tc

// Threads of a product CTA: 8 warps; warps w and w + 4 share TMEM lanes
// 32 (w mod 4) .. +31 and split the output columns in 16-column chunks.
constexpr int kTcThreads = 256;

// Output columns of a product are split over two CTAs per 128-row tile
// (the halves' widths multiples of 16, as tcgen05.mma with M = 128 needs),
// so that the MMA chain and the epilogue on a product's critical path are
// half as long and the products run on twice the CTAs.
__host__ __device__ __forceinline__ int tc_nsplit(int Np) { return Np >= 32 ? 2 : 1; }
__host__ __device__ __forceinline__ int tc_first_half(int Np) { return (Np / 16 + 1) / 2 * 16; }

// Gathers the CTA's 128 x Kp A tile (rows (i3, i2) of the free box, k = i1)
// from the input vector into the canonical K-major BF16 layout, in which
// the 8 elements (row r, k = 8 kc .. 8 kc + 7) are the 16 bytes at
// kc * 2048 + r * 16.  rowbase[r] is the vector index of (row r, k = 0).
// Thread t owns row t mod 128 and one half of its chunks, so a warp's
// 16-byte stores cover 512 contiguous bytes (no bank conflicts).  A row's
// elements are read as the aligned 16-byte blocks that hold them (VW
// elements each; every block read holds an element of the row, so it lies
// in memory the row's own elements occupy), VW chunks per round from a
// register window of 9 blocks shifted by the row's misalignment.  Padding
// columns k >= m0 and rows r >= nvalid are written as zeros.
template <typename TX>
__device__ __forceinline__ void gather_tile(const TX* __restrict__ xp, const int64_t* rowbase,
                                            int nvalid, int Kp, int m0, __nv_bfloat16* As,
                                            int tid) {
  constexpr int VW = 16 / (int)sizeof(TX);  // elements per 16-byte block: 4 or 2
  constexpr int G = VW;                     // chunks per round: G * 8 / VW = 8 blocks
  constexpr int NW = 9;                     // blocks in the window (+1 for misalignment)
  const int r = tid & 127;
  const int nkc = Kp / 8, halfc = (nkc + 1) / 2;
  const int kc0 = (tid >> 7) ? halfc : 0, kc1 = (tid >> 7) ? nkc : halfc;
  unsigned char* rowp = reinterpret_cast<unsigned char*>(As) + (size_t)r * 16;
  const int64_t b = r < nvalid ? rowbase[r] : -1;
  uintptr_t a16 = 0;
  int lead = 0, qlast = -1;
  if (b >= 0) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(xp + b);
    a16 = a & ~(uintptr_t)15;
    lead = (int)((a & 15) / sizeof(TX));
    qlast = (lead + m0 - 1) / VW;  // last block holding an element of the row
  }
  for (int kg = kc0; kg < kc1; kg += G) {
    // window: blocks q0 .. q0 + NW - 1, element k = 8 kg at position p0
    const int e0 = lead + 8 * kg;
    const int q0 = e0 / VW, p0 = e0 - q0 * VW;
    TX w[NW * VW];
#pragma unroll
    for (int t = 0; t < NW; ++t) {
      uint4 v = make_uint4(0, 0, 0, 0);
      if (b >= 0 && q0 + t <= qlast)
        v = __ldg(reinterpret_cast<const uint4*>(a16 + (uintptr_t)(q0 + t) * 16));
      const TX* pv = reinterpret_cast<const TX*>(&v);
#pragma unroll
      for (int i = 0; i < VW; ++i) w[t * VW + i] = pv[i];
    }
    // w[i] <- w[i + p0] (p0 < VW), one select per bit of p0
#pragma unroll
    for (int sh = VW / 2; sh >= 1; sh /= 2) {
      const bool on = (p0 & sh) != 0;
#pragma unroll
      for (int i = 0; i + sh < NW * VW; ++i) w[i] = on ? w[i + sh] : w[i];
    }
#pragma unroll
    for (int c = 0; c < G; ++c) {
      const int kc = kg + c;
      if (kc >= kc1) break;
      uint32_t pk[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = 8 * kc + 2 * j;
        const float lo = (b >= 0 && k < m0) ? (float)w[8 * c + 2 * j] : 0.f;
        const float hi = (b >= 0 && k + 1 < m0) ? (float)w[8 * c + 2 * j + 1] : 0.f;
        const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        pk[j] = *reinterpret_cast<const uint32_t*>(&h);
      }
      *reinterpret_cast<uint4*>(rowp + (size_t)kc * 2048) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
    }
  }
}


// one mode product
struct TcGemm {
  // rows and their split into (r_slow, r_fast): row = r_slow * rfast + r_fast
  int32_t R, rfast;
  int32_t Kp, K;   // padded contraction length (multiple of 16), true length
  int32_t N, Np;   // outputs per row (m of this direction) and its padding
  int32_t kpn;     // padded fastest length of the output tensor
  // A source
  const __nv_bfloat16* A;  // [R][Kp] (mode 0)
  // gather (first product): A[row][k] = x[box(row, k)]
  const void* x;
  int32_t x_f64;
  // output
  __nv_bfloat16* out;      // [N][R/rfast][kpn] (modes 0/1)
  const float* inv_lambda; // scaling (mode 1), index a*R + row
  void* y;                 // scatter target (mode 2)
  int32_t y_f64;
  // box of the free nodes (gather / scatter), direction 1 first
  int32_t n[3], lo[3], m[3];
  const __nv_bfloat16* Bimg;  // pre-tiled B (Np x Kp, canonical K-major)
  int32_t* status;
};

// a_mode: 0 = BF16 tensor, 1 = gather from x (rows (i3,i2), k = i1)
// o_mode: 0 = rotated BF16 store, 1 = same times 1/Lambda, 2 = scatter to y
template <int A_MODE, int O_MODE>
__device__ __forceinline__ void fd_tc_body(const TcGemm& g, const int bx) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ uint64_t bars[2];
  __shared__ uint32_t tmem_base;
  __shared__ int s_fail;
  __shared__ int64_t rowbase[128];
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int Kp = g.Kp, Np = g.Np;
  __nv_bfloat16* As = reinterpret_cast<__nv_bfloat16*>(smem_raw);            // 128 x Kp
  __nv_bfloat16* Bs = reinterpret_cast<__nv_bfloat16*>(smem_raw + 128 * Kp * 2);  // Np x Kp
  // CTA bx: rows of tile bx / nsplit, output columns [n_off, n_off + n_cnt)
  const int nsplit = tc_nsplit(Np);
  const int tile = bx / nsplit, half = bx - tile * nsplit;
  const int n1 = tc_first_half(Np);
  const int n_off = half ? n1 : 0, n_cnt = nsplit == 1 ? Np : (half ? Np - n1 : n1);
  const int row0 = tile * 128;
  uint32_t ncols = 32;
  while ((int)ncols < n_cnt) ncols <<= 1;

  if (tid == 0) {
    mbar_init(smem_u32(&bars[0]), 1);
    mbar_init(smem_u32(&bars[1]), 1);
    s_fail = 0;
    fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(smem_u32(&tmem_base), ncols);
  __syncthreads();
  // this CTA holds its tensor memory: the next product may be scheduled
  tc::launch_dependents();
  if (tid == 0) {
    // the B image is constant (eigenvectors), independent of the previous product
    const uint32_t bytes = (uint32_t)(Np * Kp * 2);
    mbar_arrive_expect_tx(smem_u32(&bars[0]), bytes);
    bulk_g2s(smem_u32(Bs), g.Bimg, bytes, smem_u32(&bars[0]));
  }
  // everything below reads the previous product's output (or the input
  // vector, written before the first product, which is launched in order)
  tc::wait_prerequisites();
  // ---- A tile in canonical K-major layout: core (grp, kc) at (kc*16 + grp)*128 B
  // Loads are issued in groups (all of a group before any of its shared
  // stores), so a thread keeps a group of global reads in flight instead of
  // one.
  // Descriptor fields used inside the loops are copied to registers first:
  // the descriptor may sit in shared memory (batch kernel), and every store
  // below could alias it for the compiler, forcing a re-read per element.
  const int kchunks = Kp / 8, Kt = g.K;
  const int R = g.R;
  if (A_MODE == 0) {
    // thread t owns row t mod 128 and half of its 16-byte chunks: a warp's
    // stores for one chunk index cover 512 contiguous bytes of the
    // canonical layout (chunk (kc, r) at kc * 2048 + r * 16), no conflicts
    constexpr int U = 8;
    const int r = tid & 127;
    const int halfc = (kchunks + 1) / 2;
    const int kc0 = (tid >> 7) ? halfc : 0, kc1 = (tid >> 7) ? kchunks : halfc;
    const bool live = row0 + r < R;
    const uint4* Arow =
        reinterpret_cast<const uint4*>(g.A + (size_t)(live ? row0 + r : 0) * Kp);
    unsigned char* dst = smem_raw + (size_t)r * 16;
    // Padding is not read: it holds other products' values (the work arrays change
    // layout from product to product), finite only while all inputs were. The chunk
    // with the last column is masked.
    const int tailc = Kt & 7 ? Kt >> 3 : -1;
    uint4 tail = make_uint4(0, 0, 0, 0);
    if (live && tailc >= kc0 && tailc < kc1) {
      tail = ld_dependent(Arow + tailc);
      uint32_t* w = reinterpret_cast<uint32_t*>(&tail);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        w[j] &= ((Kt & 7) > 2 * j ? 0xffffu : 0u) | ((Kt & 7) > 2 * j + 1 ? 0xffff0000u : 0u);
    }
    for (int k0 = kc0; k0 < kc1; k0 += U) {
      uint4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        v[u] = make_uint4(0, 0, 0, 0);
        if (live && k0 + u < min(kc1, Kt >> 3)) v[u] = ld_dependent(Arow + k0 + u);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k0 + u < kc1) *reinterpret_cast<uint4*>(dst + (size_t)(k0 + u) * 2048) = v[u];
    }
    if (tailc >= kc0 && tailc < kc1)
      *reinterpret_cast<uint4*>(dst + (size_t)tailc * 2048) = tail;
  } else {
    // rows (i3, i2) of the free box, k = i1: the vector index of each row's
    // first element once per CTA, then one add per element
    if (tid < 128) {
      const int row = row0 + tid;
      int64_t b = -1;
      if (row < R) {
        const int i3 = row / g.m[1], i2 = row - i3 * g.m[1];
        b = ((int64_t)(g.lo[2] + i3) * g.n[1] + g.lo[1] + i2) * g.n[0] + g.lo[0];
      }
      rowbase[tid] = b;
    }
    __syncthreads();
    const int nvalid = R - row0 < 128 ? R - row0 : 128;
    if (g.x_f64)
      gather_tile(reinterpret_cast<const double*>(g.x), rowbase, nvalid, Kp, g.m[0], As, tid);
    else
      gather_tile(reinterpret_cast<const float*>(g.x), rowbase, nvalid, Kp, g.m[0], As, tid);
  }
  tc::fence_proxy_async_smem();
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tbase = tmem_base;
  if (tid == 0) {
    if (!mbar_wait_bounded(smem_u32(&bars[0]), 0)) {
      s_fail = 1;
      if (g.status) atomicExch(g.status, IGA_ERR_TIMEOUT);
    } else {
      const uint32_t idesc = tc::idesc_bf16(128, n_cnt);
      // this CTA's output columns are B rows n_off .. n_off + n_cnt - 1: the
      // core matrices from group n_off / 8 on, same K stride as the full image
      const uint32_t a0 = smem_u32(As), b0 = smem_u32(Bs) + (uint32_t)(n_off / 8) * 128;
      const uint32_t lbo_a = 16 * 128, lbo_b = (uint32_t)(Np / 8) * 128;
      for (int kk = 0; kk < Kp / 16; ++kk) {
        const uint64_t ad = tc::smem_desc(a0 + 2 * kk * lbo_a, lbo_a, 128);
        const uint64_t bd = tc::smem_desc(b0 + 2 * kk * lbo_b, lbo_b, 128);
        tc::mma_bf16(tbase, ad, bd, idesc, kk > 0 ? 1u : 0u);
      }
      tc::mma_commit(smem_u32(&bars[1]));
    }
  }
  __syncthreads();
  // epilogue rows: warp w reads TMEM lanes 32 (w mod 4) .. +31 (= tile rows),
  // column chunks 16 (w div 4), +32, ...
  const int wq = warp & 3;
  const int r = wq * 32 + lane;
  const int row = row0 + r;
  const bool rv = row < R;
  const int Nout = g.N;
  const float* __restrict__ inv_lambda = g.inv_lambda;
  // 1/Lambda factors of a column chunk (scaling product only); the first
  // chunk's are read while the MMA chain runs, the next one's while the
  // current chunk is stored
  float lam[16], lamn[16];
  auto load_lam = [&](int c, float (&d)[16]) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      d[i] = (rv && c + i < Nout) ? __ldg(inv_lambda + (int64_t)(c + i) * R + row) : 0.f;
  };
  if (O_MODE == 1) load_lam(n_off + 16 * (warp >> 2), lam);
  bool ok = (s_fail == 0);
  if (ok) ok = mbar_wait_bounded(smem_u32(&bars[1]), 0);
  if (!__syncthreads_and(ok)) {
    if (tid == 0 && g.status) atomicExch(g.status, IGA_ERR_TIMEOUT);
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tbase, ncols);
    return;
  }
  tc::tc_fence_after();
  // ---- epilogue
  const int rs = rv ? row / g.rfast : 0, rf = rv ? row - rs * g.rfast : 0;
  const int nslow = R / g.rfast;
  // rotated store (modes 0/1): out[a][rs][rf]; scatter (mode 2): row =
  // (i2, i1) of the box, a = i3
  __nv_bfloat16* const out = g.out;
  const int64_t ostride = (int64_t)nslow * g.kpn, obase = (int64_t)rs * g.kpn + rf;
  const int64_t yplane = (int64_t)g.n[1] * g.n[0];
  int64_t ybase = 0;
  if (O_MODE == 2 && rv) {
    const int i1 = row % g.m[0], i2 = row / g.m[0];
    ybase = ((int64_t)g.lo[2] * g.n[1] + g.lo[1] + i2) * g.n[0] + g.lo[0] + i1;
  }
  const bool yf64 = g.y_f64 != 0;
  void* const yp = g.y;
  for (int c0 = 16 * (warp >> 2); c0 < n_cnt; c0 += 32) {
    if (O_MODE == 1 && c0 + 32 < n_cnt) load_lam(n_off + c0 + 32, lamn);
    float v[16];
    tc::tmem_ld16(tbase + ((uint32_t)(wq * 32) << 16) + (uint32_t)c0, v);
    if (rv) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int a = n_off + c0 + i;
        if (a >= Nout) break;
        if (O_MODE == 2) {
          const int64_t idx = ybase + (int64_t)a * yplane;
          if (yf64)
            reinterpret_cast<double*>(yp)[idx] = (double)v[i];
          else
            reinterpret_cast<float*>(yp)[idx] = v[i];
        } else {
          float val = v[i];
          if (O_MODE == 1) val *= lam[i];
          out[obase + (int64_t)a * ostride] = __float2bfloat16(val);
        }
      }
    }
    if (O_MODE == 1) {
#pragma unroll
      for (int i = 0; i < 16; ++i) lam[i] = lamn[i];
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tbase, ncols);
}

template <int A_MODE, int O_MODE>
__global__ void __launch_bounds__(kTcThreads) fd_tc_kernel(const __grid_constant__ TcGemm g) {
  fd_tc_body<A_MODE, O_MODE>(g, blockIdx.x);
}

// Many patches in one launch: patch p owns CTAs [cta0[p], cta0[p+1]); its
// product descriptor gs[p] goes to shared memory, with the gather source /
// scatter target moved to element offset offs[p] of the flat x / y.
template <int A_MODE, int O_MODE>
__global__ void __launch_bounds__(kTcThreads)
    fd_tc_batch_kernel(const TcGemm* __restrict__ gs, const int32_t* __restrict__ cta0, int np,
                       const int64_t* __restrict__ offs, const void* xb, void* yb,
                       const int32_t* __restrict__ skip) {
  __shared__ TcGemm sg;
  __shared__ int sp;
  if (threadIdx.x == 0) {
    int lo = 0, hi = np;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(cta0 + mid) <= (int)blockIdx.x) lo = mid;
      else hi = mid;
    }
    sp = lo;
  }
  __syncthreads();
  const int p = sp;
  // one round of independent reads: the skip flag, one word of the product
  // descriptor per thread, the patch's vector offset and its first CTA
  constexpr int kWords = (int)(sizeof(TcGemm) / sizeof(int));
  static_assert(kWords <= kTcThreads, "descriptor copy: one word per thread");
  const int sk = skip ? __ldg(skip + p) : -1;
  const int word = threadIdx.x < kWords
                       ? __ldg(reinterpret_cast<const int*>(gs + p) + threadIdx.x) : 0;
  const int64_t off = (A_MODE == 1 || O_MODE == 2) ? __ldg(offs + p) : 0;
  const int first = __ldg(cta0 + p);
  if (sk >= 0) return;  // patch done: its output stays zero (same p for the whole CTA)
  if (threadIdx.x < kWords) reinterpret_cast<int*>(&sg)[threadIdx.x] = word;
  __syncthreads();
  if (threadIdx.x == 0) {
    if (A_MODE == 1) sg.x = (const char*)xb + off * (sg.x_f64 ? 8 : 4);
    if (O_MODE == 2) sg.y = (char*)yb + off * (sg.y_f64 ? 8 : 4);
  }
  __syncthreads();
  fd_tc_body<A_MODE, O_MODE>(sg, (int)blockIdx.x - first);
}

// ---------------------------------------------------------------------------
// The apply in four kernels (every free extent up to kTcFusedMax):
//   plane: W0[i3][a2][a1] = products over i1, then i2 of plane i3 of the box
//   line:  W1[a3][a2][a1] = product over i3, times 1/Lambda
//   plane: W0[a3][i2][i1] = products over a1, then a2 of plane a3
//   line:  y[i3][i2][i1]  = product over a3
// (index 1 padded to Kp1 in W0 and W1). A CTA of the six separate products spends
// its time waiting: for its operands, one short chain of MMAs, its epilogue, the end
// of the grid before it. A plane's two products share one such chain, and what the
// first one passes on stays on the SM: its accumulator, rounded to BF16 as it was
// for memory, becomes an operand of the second. For that its rows have to be the
// rows of the second product and its columns the contracted index, so the first
// product takes the eigenvector image as A and the plane's rows as B (accumulator
// row a1, column i2). A thread then holds 16 neighbouring columns of one row and
// writes the two 16-byte chunks they are in the canonical layout. A line's CTA reads
// 128 rows x 8 planes as pairs of rows and transposes them in registers. The
// products, their order and their roundings are those of the separate products and
// so are the results, bit for bit. (Direction 3 in one kernel with 1/Lambda between
// its two products makes three kernels and 2 us less, but reorders the backward
// products, hence the roundings.)
// Measured (FP64 vectors, us, separate -> here): 9^3 22.6 -> 18, 31^3 25.7 -> 20.9,
// 64^3 33.3 -> 25.0, 97^3 45.2 -> 33.4, 123^3 79 -> 41. Launches and waits bound the
// small ones; at 97^3 97 planes leave 51 SMs idle, and the gather of x (8.1 MB) and
// the clearing of y make the first kernel the longest (12 us of 33).
// Beyond 128 the first product's rows need two tiles that stage the same plane, one
// CTA a SM: the planes in pairs took 72 us against 62 separate at 133^3, 109 against
// 106 at 150^3, so those keep the separate products.
// ---------------------------------------------------------------------------
struct TcFused {
  int32_t n[3], lo[3], m[3], kp[3];  // vector, free box, extents padded to 16
  int32_t io_f64;
  const __nv_bfloat16* F[3];         // images of U_d^T
  const __nv_bfloat16* B[3];         // images of U_d
  const float* inv_lambda;
  const void* x;
  void* y;
  __nv_bfloat16 *w0, *w1;
  int32_t* status;
};

constexpr int kTcFusedMax = 128;
// what an A operand of fewer than 128 rows reads behind its last K chunk (the
// accumulator rows that come of it are never used)
constexpr int kTcOverread = 2048;
// Threads of a CTA (NT): 512, warps w, w + 4, w + 8, w + 12 sharing 32 rows of the
// accumulator and taking its columns 16 at a time in turn; 256 while a CTA's
// operands take up to this much (extents up to 48: 9^3 15.0 us against 17.0, 31^3 17.0
// against 18.8, 45^3 the same; beyond, 97^3 35.5 against 28.5; three-kernel form)
constexpr size_t kTcSmallSmem = 24 * 1024;

static size_t tc_plane_smem(const int* kp) {
  return ((size_t)kp[0] * kp[0] + (size_t)kp[0] * kp[1] + (size_t)kp[1] * kp[1]) * 2 + kTcOverread;
}
static size_t tc_line_smem(const int* kp) { return ((size_t)128 + kp[2]) * kp[2] * 2; }

// A CTA's shared state beside its operands
struct TcShared {
  uint64_t bars[2];  // images landed; MMA chain done
  uint32_t tmem;
  int fail;
};

__device__ __forceinline__ uint32_t tc_begin(TcShared& s, int ncols_min, uint32_t& ncols) {
  ncols = 32;
  while ((int)ncols < ncols_min) ncols <<= 1;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&s.bars[0]), 1);
    mbar_init(smem_u32(&s.bars[1]), 1);
    s.fail = 0;
    fence_mbar_init();
  }
  if (threadIdx.x < 32) tc::tmem_alloc(smem_u32(&s.tmem), ncols);
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  // this CTA holds its tensor memory: the next kernel may be scheduled
  tc::launch_dependents();
  return s.tmem;
}

__device__ __forceinline__ void tc_end(uint32_t tmem, uint32_t ncols) {
  tc::tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) tc::tmem_dealloc(tmem, ncols);
}

// D = A B over K (shared memory written by all threads before the call, or by
// bulk copies on bars[0]); false in every thread when a wait ran out.
__device__ __forceinline__ bool tc_product(TcShared& s, uint32_t tmem, uint32_t a, uint32_t lbo_a,
                                           uint32_t b, uint32_t lbo_b, int N, int K,
                                           uint32_t parity, int32_t* status) {
  tc::fence_proxy_async_smem();
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  if (threadIdx.x == 0) {  // the others sleep at the barrier below
    bool ok = mbar_wait_bounded(smem_u32(&s.bars[0]), 0);
    if (ok) {
      const uint32_t idesc = tc::idesc_bf16(128, N);
      for (int kk = 0; kk < K / 16; ++kk)
        tc::mma_bf16(tmem, tc::smem_desc(a + 2 * kk * lbo_a, lbo_a, 128),
                     tc::smem_desc(b + 2 * kk * lbo_b, lbo_b, 128), idesc, kk > 0 ? 1u : 0u);
      tc::mma_commit(smem_u32(&s.bars[1]));
      ok = mbar_wait_bounded(smem_u32(&s.bars[1]), parity);
    }
    if (!ok) {
      s.fail = 1;
      if (status) atomicExch(status, IGA_ERR_TIMEOUT);
    }
  }
  __syncthreads();
  tc::tc_fence_after();
  return s.fail == 0;
}

__device__ __forceinline__ uint4 tc_pack8(const float* v) {
  uint4 q;
  uint32_t* p = reinterpret_cast<uint32_t*>(&q);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
    p[j] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return q;
}

// Plane i3 of the box as K-major rows: row i2, k = i1; zero beyond the box.  A
// warp takes 4 rows x 8 columns per load, eight loads under way.
template <int NT, typename TX>
__device__ __forceinline__ void tc_stage_box(const TcFused& g, const TX* __restrict__ x, int i3,
                                             unsigned char* xs) {
  const int m1 = g.m[0], m2 = g.m[1], nkc = g.kp[0] / 8, rows = g.kp[1];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, lr = lane >> 3, lk = lane & 7;
  const int64_t ld = g.n[0];
  const TX* const src = x + (((int64_t)g.lo[2] + i3) * g.n[1] + g.lo[1]) * ld + g.lo[0];
  int r = 4 * (warp / nkc), kc = warp % nkc;  // task: rows r .. r + 3, chunk kc
  constexpr int U = 13, NW = NT / 32;
  while (r < rows) {
    float v[U];
    int at[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int rr = r + lr, k = 8 * kc + lk;
      at[u] = r < rows ? kc * rows * 16 + rr * 16 + 2 * lk : -1;
      v[u] = rr < m2 && k < m1 ? (float)__ldg(src + rr * ld + k) : 0.f;
      kc += NW;
      while (kc >= nkc) kc -= nkc, r += 4;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at[u] >= 0) *reinterpret_cast<__nv_bfloat16*>(xs + at[u]) = __float2bfloat16(v[u]);
  }
}

// Plane i3 of W1 as K-major rows: row a2, k = a1.  A warp takes 8 rows x 4 chunks
// per load, all of a plane's loads under way up to 128 x 128; a row's padding is not
// trusted to be finite.
template <int NT>
__device__ __forceinline__ void tc_stage_w1(const TcFused& g, int i3, unsigned char* xs) {
  const int m1 = g.m[0], m2 = g.m[1], kp1 = g.kp[0], nkc = kp1 / 8, rows = g.kp[1];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, lr = lane & 7, lc = lane >> 3;
  const __nv_bfloat16* const src = g.w1 + (size_t)i3 * m2 * kp1;
  const int ngc = (nkc + 3) / 4;
  int r = 8 * (warp / ngc), gc = warp % ngc;
  constexpr int U = 4, NW = NT / 32;
  while (r < rows) {
    uint4 v[U];
    int at[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int rr = r + lr, kc = 4 * gc + lc;
      at[u] = r < rows && kc < nkc ? kc * rows * 16 + rr * 16 : -1;
      v[u] = make_uint4(0, 0, 0, 0);
      if (rr < m2 && kc < nkc)
        v[u] = ld_dependent(reinterpret_cast<const uint4*>(src + (size_t)rr * kp1 + 8 * kc));
      uint32_t* w = reinterpret_cast<uint32_t*>(&v[u]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = 8 * kc + 2 * j;
        w[j] &= (k < m1 ? 0xffffu : 0u) | (k + 1 < m1 ? 0xffff0000u : 0u);
      }
      gc += NW;
      while (gc >= ngc) gc -= ngc, r += 8;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at[u] >= 0) *reinterpret_cast<uint4*>(xs + at[u]) = v[u];
  }
}

// The grid's share of a zero fill (y is zero outside the box; the last kernel
// writes the box two launches later).
template <int NT>
__device__ __forceinline__ void tc_zero(void* y, int64_t bytes) {
  const int64_t id = (int64_t)blockIdx.x * NT + threadIdx.x;
  const int64_t all = (int64_t)gridDim.x * NT;
  const int64_t head = min(bytes, (int64_t)((0 - (uintptr_t)y) & 15)), n16 = (bytes - head) / 16;
  char* const p = (char*)y + head;
  for (int64_t i = id; i < n16; i += all) reinterpret_cast<uint4*>(p)[i] = make_uint4(0, 0, 0, 0);
  const int64_t nw = (bytes - 16 * n16) / 4;  // head and tail, 4-byte words
  if (id < nw)
    *reinterpret_cast<uint32_t*>(4 * id < head ? (char*)y + 4 * id : p + 16 * n16 + 4 * id - head) = 0u;
}

// FWD: box of x -> W0; else W1 -> W0.  CTA i3: plane i3.
template <int NT, bool FWD>
__device__ __forceinline__ void fd_tc_plane(const TcFused& g, const int i3, void* yall,
                                            int64_t zero_bytes) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ TcShared sh;
  const int Kp1 = g.kp[0], Np2 = g.kp[1], m1 = g.m[0], m2 = g.m[1];
  const int tid = threadIdx.x;
  unsigned char* const us = smem_raw;                    // first image
  unsigned char* const xs = us + (size_t)Kp1 * Kp1 * 2;  // plane, then first result
  unsigned char* const vs = xs + (size_t)Kp1 * Np2 * 2;  // second image
  uint32_t ncols;
  const uint32_t tmem = tc_begin(sh, Np2, ncols);
  if (tid == 0) {
    // the images are constant, independent of the previous kernel
    const uint32_t bar = smem_u32(&sh.bars[0]);
    mbar_arrive_expect_tx(bar, (uint32_t)(Kp1 * Kp1 + Np2 * Np2) * 2);
    bulk_g2s(smem_u32(us), FWD ? g.F[0] : g.B[0], (uint32_t)(Kp1 * Kp1 * 2), bar);
    bulk_g2s(smem_u32(vs), FWD ? g.F[1] : g.B[1], (uint32_t)(Np2 * Np2 * 2), bar);
  }
  tc::wait_prerequisites();
  if (FWD) {
    if (g.io_f64) tc_stage_box<NT>(g, reinterpret_cast<const double*>(g.x), i3, xs);
    else tc_stage_box<NT>(g, reinterpret_cast<const float*>(g.x), i3, xs);
    if (zero_bytes) tc_zero<NT>(yall, zero_bytes);
  } else {
    tc_stage_w1<NT>(g, i3, xs);
  }
  bool ok = tc_product(sh, tmem, smem_u32(us), Kp1 * 16, smem_u32(xs), Np2 * 16, Np2, Kp1, 0,
                       g.status);
  const int warp = tid / 32, wq = warp & 3, r = wq * 32 + tid % 32;
  const uint32_t tq = tmem + ((uint32_t)(wq * 32) << 16);
  if (ok) {
    // accumulator row a1, columns i2 -> row a1 of the second product, k = i2
    for (int c = 16 * (warp >> 2); c < Np2; c += NT / 8) {
      float v[16];
      tc::tmem_ld16(tq + c, v);
      if (r < Kp1) {
        *reinterpret_cast<uint4*>(xs + ((size_t)(c / 8) * Kp1 + r) * 16) = tc_pack8(v);
        *reinterpret_cast<uint4*>(xs + ((size_t)(c / 8 + 1) * Kp1 + r) * 16) = tc_pack8(v + 8);
      }
    }
    ok = tc_product(sh, tmem, smem_u32(xs), Kp1 * 16, smem_u32(vs), Np2 * 16, Np2, Np2, 1,
                    g.status);
    if (ok) {
      const bool live = r < m1;
      __nv_bfloat16* const w = g.w0 + (size_t)i3 * m2 * Kp1 + r;
      for (int c = 16 * (warp >> 2); c < Np2; c += NT / 8) {
        float v[16];
        tc::tmem_ld16(tq + c, v);
        if (!live) continue;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int a2 = c + i;
          if (a2 >= m2) break;
          w[(size_t)a2 * Kp1] = __float2bfloat16(v[i]);
        }
      }
    }
  }
  tc_end(tmem, ncols);
}

// Rows (a2, a1 padded) of W0, contraction over direction 3.  FWD: times 1/Lambda
// into W1; else into the box of y.  CTA bx: 128 rows, half of the columns.
template <int NT, bool FWD>
__device__ __forceinline__ void fd_tc_line(const TcFused& g, const int bx) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ TcShared sh;
  const int Kp1 = g.kp[0], Kp3 = g.kp[2], m1 = g.m[0], m3 = g.m[2], tid = threadIdx.x;
  const int ns = tc_nsplit(Kp3), half = bx % ns, row0 = bx / ns * 128;
  const int n1 = ns == 1 ? Kp3 : tc_first_half(Kp3);
  const int n_off = half ? n1 : 0, n_cnt = half ? Kp3 - n1 : n1;
  const int R = g.m[1] * Kp1;
  unsigned char* const as = smem_raw;                    // data
  unsigned char* const bs = as + (size_t)128 * Kp3 * 2;  // image
  uint32_t ncols;
  const uint32_t tmem = tc_begin(sh, n_cnt, ncols);
  if (tid == 0) {
    const uint32_t bytes = (uint32_t)(Kp3 * Kp3 * 2), bar = smem_u32(&sh.bars[0]);
    mbar_arrive_expect_tx(bar, bytes);
    bulk_g2s(smem_u32(bs), FWD ? g.F[2] : g.B[2], bytes, bar);
  }
  const int warp = tid / 32, lane = tid % 32, wq = warp & 3, r = wq * 32 + lane;
  const int row = row0 + r, a2 = row / Kp1, a1 = row - a2 * Kp1;
  const bool live = row < R && a1 < m1;
  // 1/Lambda of a chunk of columns; the first one's is under way before the wait
  const float* const lam = g.inv_lambda + (live ? (size_t)a2 * m1 + a1 : 0);
  const size_t lstride = (size_t)g.m[1] * m1;
  auto load_lam = [&](int c, float (&d)[16]) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      d[i] = live && c + i < m3 ? __ldg(lam + (c + i) * lstride) : 0.f;
  };
  float l0[16], l1[16];
  if (FWD) load_lam(n_off + 16 * (warp >> 2), l0);
  tc::wait_prerequisites();
  {
    // a warp takes 64 rows (a pair per lane) x 8 planes per task
    const int nkc = Kp3 / 8;
    constexpr int U = 2, NW = NT / 32;
    for (int t = warp; t < 2 * nkc; t += U * NW) {
      uint32_t v[U][8];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int s = t + u * NW, rr = row0 + (s & 1) * 64 + 2 * lane, k0 = (s >> 1) * 8;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          v[u][j] = rr < R && k0 + j < m3
                        ? ld_dependent(reinterpret_cast<const uint32_t*>(g.w0 + (size_t)(k0 + j) * R + rr)) : 0u;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int s = t + u * NW;
        if (s >= 2 * nkc) break;
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          lo[j] = __byte_perm(v[u][2 * j], v[u][2 * j + 1], 0x5410);
          hi[j] = __byte_perm(v[u][2 * j], v[u][2 * j + 1], 0x7632);
        }
        uint4* d = reinterpret_cast<uint4*>(as + ((size_t)(s >> 1) * 128 + (s & 1) * 64 + 2 * lane) * 16);
        d[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        d[1] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      }
    }
  }
  const bool ok = tc_product(sh, tmem, smem_u32(as), 2048, smem_u32(bs) + n_off * 16, Kp3 * 16,
                             n_cnt, Kp3, 0, g.status);
  const uint32_t tq = tmem + ((uint32_t)(wq * 32) << 16);
  if (ok) {
    const int64_t yplane = (int64_t)g.n[1] * g.n[0];
    const int64_t yb = (int64_t)g.lo[2] * yplane + ((int64_t)g.lo[1] + a2) * g.n[0] + g.lo[0] + a1;
    const bool f64 = g.io_f64 != 0;
    void* const y = g.y;
    for (int c = 16 * (warp >> 2); c < n_cnt; c += NT / 8) {
      if (FWD) load_lam(n_off + c + NT / 8, l1);
      float v[16];
      tc::tmem_ld16(tq + c, v);
      if (FWD) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] *= l0[i], l0[i] = l1[i];
        // lanes 2 l, 2 l + 1 swap columns: each writes two neighbouring rows of one
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
          const float mine = lane & 1 ? v[i + 1] : v[i];
          const float other = __shfl_xor_sync(0xffffffffu, lane & 1 ? v[i] : v[i + 1], 1);
          const int a3 = n_off + c + i + (lane & 1);
          if (row < R && a3 < m3)
            *reinterpret_cast<__nv_bfloat162*>(g.w1 + (size_t)a3 * R + (row & ~1)) =
                __floats2bfloat162_rn(lane & 1 ? other : mine, lane & 1 ? mine : other);
        }
      } else if (live) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int i3 = n_off + c + i;
          if (i3 >= m3) break;
          if (f64) reinterpret_cast<double*>(y)[yb + i3 * yplane] = (double)v[i];
          else reinterpret_cast<float*>(y)[yb + i3 * yplane] = v[i];
        }
      }
    }
  }
  tc_end(tmem, ncols);
}

// STAGE 0 .. 3: the four kernels; zero_bytes > 0: the first one clears y
template <int NT, int STAGE>
__device__ __forceinline__ void fd_tc_stage(const TcFused& g, int bx, void* yall, int64_t zero_bytes) {
  if (STAGE & 1) fd_tc_line<NT, STAGE == 1>(g, bx);
  else fd_tc_plane<NT, STAGE == 0>(g, bx, yall, zero_bytes);
}

template <int NT, int STAGE>
__global__ void __launch_bounds__(NT)
    fd_tc_fused_kernel(const __grid_constant__ TcFused g, int64_t zero_bytes) {
  fd_tc_stage<NT, STAGE>(g, blockIdx.x, g.y, zero_bytes);
}

template <int NT, int STAGE>
__global__ void __launch_bounds__(NT)
    fd_tc_fused_batch_kernel(const TcFused* __restrict__ gs, const int32_t* __restrict__ cta0,
                             int np, const int64_t* __restrict__ offs, const void* xb, void* yb,
                             const int32_t* __restrict__ skip, int64_t zero_bytes) {
  __shared__ TcFused sg;
  __shared__ int sp;
  if (threadIdx.x == 0) {
    int lo = 0, hi = np;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(cta0 + mid) <= (int)blockIdx.x) lo = mid;
      else hi = mid;
    }
    sp = lo;
  }
  __syncthreads();
  const int p = sp;
  constexpr int kWords = (int)(sizeof(TcFused) / sizeof(int));
  static_assert(kWords <= NT, "descriptor copy: one word per thread");
  const int sk = skip ? __ldg(skip + p) : -1;
  const int word = threadIdx.x < kWords
                       ? __ldg(reinterpret_cast<const int*>(gs + p) + threadIdx.x) : 0;
  const int64_t off = __ldg(offs + p);
  const int first = __ldg(cta0 + p);
  if (sk >= 0) {  // patch done: its output stays zero (same p for the whole CTA)
    // a grid never ends before the one it follows: the zero fill is the first one's
    if (STAGE == 0 && zero_bytes) tc_zero<NT>(yb, zero_bytes);
    tc::wait_prerequisites();
    return;
  }
  if (threadIdx.x < kWords) reinterpret_cast<int*>(&sg)[threadIdx.x] = word;
  __syncthreads();
  if (threadIdx.x == 0) {
    sg.x = (const char*)xb + off * (sg.io_f64 ? 8 : 4);
    sg.y = (char*)yb + off * (sg.io_f64 ? 8 : 4);
  }
  __syncthreads();
  fd_tc_stage<NT, STAGE>(sg, (int)blockIdx.x - first, yb, zero_bytes);
}

// Launch configuration of one product: products after the first of an
// apply overlap their launch and prologue with the previous product
// (programmatic stream serialization; the kernels wait for it in-kernel).
struct TcLaunch {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  TcLaunch(unsigned grid, size_t smem, cudaStream_t st, bool overlap,
           unsigned threads = kTcThreads) {
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
  }
};

template <int A_MODE, int O_MODE>
static iga_status launch_tc_batch(const TcGemm* gs, const int32_t* cta0, int np,
                                  const int64_t* offs, int grid, size_t smem, const void* x,
                                  void* y, const int32_t* skip, cudaStream_t st, bool overlap) {
  static SmemOptIn optin;
  IGA_CUDA_TRY(optin.allow((const void*)fd_tc_batch_kernel<A_MODE, O_MODE>, smem));
  TcLaunch L((unsigned)grid, smem, st, overlap);
  IGA_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, fd_tc_batch_kernel<A_MODE, O_MODE>, gs, cta0, np, offs,
                                  x, y, skip));
  IGA_LAUNCH_CHECK();
  return IGA_OK;
}

static bool tc_fits_fused(const int32_t* m) {
  return m[0] <= kTcFusedMax && m[1] <= kTcFusedMax && m[2] <= kTcFusedMax;
}

// The six rotated products of one patch (see iga_fd_apply_tc).
static void tc_stages(TcGemm g[6], const int32_t* n, const int32_t* lo, const int32_t* m,
                      const void* const* Bfwd, const void* const* Bbwd, const float* inv_lambda,
                      const void* x, void* y, int io_f64, void* work0, void* work1,
                      int32_t* status) {
  int kp[3];
  for (int d = 0; d < 3; ++d) kp[d] = (int)ceil_div(m[d], 16) * 16;
  const int m1 = m[0], m2 = m[1], m3 = m[2];
  __nv_bfloat16* w0 = (__nv_bfloat16*)work0;
  __nv_bfloat16* w1 = (__nv_bfloat16*)work1;
  TcGemm b;
  memset(&b, 0, sizeof(b));
  for (int d = 0; d < 3; ++d) {
    b.n[d] = n[d];
    b.lo[d] = lo[d];
    b.m[d] = m[d];
  }
  b.status = status;
  b.x = x;
  b.x_f64 = io_f64;
  b.y = y;
  b.y_f64 = io_f64;
  b.inv_lambda = inv_lambda;
  const __nv_bfloat16* F[3] = {(const __nv_bfloat16*)Bfwd[0], (const __nv_bfloat16*)Bfwd[1],
                               (const __nv_bfloat16*)Bfwd[2]};
  const __nv_bfloat16* Bk[3] = {(const __nv_bfloat16*)Bbwd[0], (const __nv_bfloat16*)Bbwd[1],
                                (const __nv_bfloat16*)Bbwd[2]};
  // (R, rfast, K dir, out fastest dir, A, B, out)
  auto set = [&](TcGemm& g, int R, int rfast, int kd, int od, const __nv_bfloat16* A,
                 const __nv_bfloat16* B, __nv_bfloat16* out) {
    g = b;
    g.R = R;
    g.rfast = rfast;
    g.Kp = kp[kd];
    g.K = m[kd];
    g.N = m[kd];
    g.Np = kp[kd];
    g.kpn = kp[od];
    g.A = A;
    g.Bimg = B;
    g.out = out;
  };
  set(g[0], m3 * m2, m2, 0, 1, nullptr, F[0], w0);  // gather -> [a1][i3][Kp2]
  set(g[1], m1 * m3, m3, 1, 2, w0, F[1], w1);       // -> [a2][a1][Kp3]
  set(g[2], m2 * m1, m1, 2, 0, w1, F[2], w0);       // -> [a3][a2][Kp1] / Lambda
  set(g[3], m3 * m2, m2, 0, 1, w0, Bk[0], w1);      // -> [i1][a3][Kp2]
  set(g[4], m1 * m3, m3, 1, 2, w1, Bk[1], w0);      // -> [i2][i1][Kp3]
  set(g[5], m2 * m1, m1, 2, 0, w0, Bk[2], nullptr); // -> scatter y
}

template <int A_MODE, int O_MODE>
static iga_status launch_tc(const TcGemm& g, cudaStream_t st, bool overlap) {
  const size_t smem = (size_t)(128 + g.Np) * g.Kp * 2;
  auto kern = fd_tc_kernel<A_MODE, O_MODE>;
  static SmemOptIn optin;
  IGA_CUDA_TRY(optin.allow((const void*)kern, smem));
  TcLaunch L((unsigned)(ceil_div(g.R, 128) * tc_nsplit(g.Np)), smem, st, overlap);
  IGA_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, kern, g));
  IGA_LAUNCH_CHECK();
  return IGA_OK;
}

static void tc_fused_desc(TcFused& g, const int32_t* n, const int32_t* lo, const int32_t* m,
                          const void* const* Bfwd, const void* const* Bbwd,
                          const float* inv_lambda, const void* x, void* y, int io_f64, void* work0,
                          void* work1, int32_t* status) {
  memset(&g, 0, sizeof(g));
  for (int d = 0; d < 3; ++d) {
    g.n[d] = n[d];
    g.lo[d] = lo[d];
    g.m[d] = m[d];
    g.kp[d] = (int)ceil_div(m[d], 16) * 16;
    g.F[d] = (const __nv_bfloat16*)Bfwd[d];
    g.B[d] = (const __nv_bfloat16*)Bbwd[d];
  }
  g.io_f64 = io_f64;
  g.inv_lambda = inv_lambda;
  g.x = x;
  g.y = y;
  g.w0 = (__nv_bfloat16*)work0;
  g.w1 = (__nv_bfloat16*)work1;
  g.status = status;
}

// CTAs and shared memory of the four kernels
static int64_t tc_fused_ctas(const TcFused& g, int stage) {
  if (stage & 1)
    return ceil_div((int64_t)g.m[1] * g.kp[0], 128) * tc_nsplit(g.kp[2]);
  return g.m[2];
}
static size_t tc_fused_smem(const TcFused& g, int stage) {
  return stage & 1 ? tc_line_smem(g.kp) : tc_plane_smem(g.kp);
}

static size_t tc_fused_smem_max(const TcFused& g) {
  return std::max(tc_fused_smem(g, 0), tc_fused_smem(g, 1));
}

// The first kernel clears y itself while a CTA's share stays below this; a small
// box in a large vector is left to a memset (HBM speed, no CTA waits for it).
constexpr int64_t kTcZeroPerCta = 256 * 1024;

template <typename K, typename... A>
static iga_status launch_tc_fused(K kern, SmemOptIn& optin, int threads, int64_t grid, size_t smem,
                                  cudaStream_t st, bool overlap, A... args) {
  IGA_CUDA_TRY(optin.allow((const void*)kern, smem));
  TcLaunch L((unsigned)grid, smem, st, overlap, (unsigned)threads);
  IGA_CUDA_TRY(cudaLaunchKernelEx(&L.cfg, kern, args...));
  IGA_LAUNCH_CHECK();
  return IGA_OK;
}
template <int NT, int STAGE>
static iga_status launch_tc_stage(const TcFused& g, int64_t zero_bytes, cudaStream_t st) {
  static SmemOptIn optin;
  return launch_tc_fused(fd_tc_fused_kernel<NT, STAGE>, optin, NT, tc_fused_ctas(g, STAGE),
                         tc_fused_smem(g, STAGE), st, STAGE > 0, g, zero_bytes);
}
template <int NT>
static iga_status launch_tc_apply(const TcFused& g, int64_t zero_bytes, cudaStream_t st) {
  iga_status rc;
  if ((rc = launch_tc_stage<NT, 0>(g, zero_bytes, st))) return rc;
  if ((rc = launch_tc_stage<NT, 1>(g, 0, st))) return rc;
  if ((rc = launch_tc_stage<NT, 2>(g, 0, st))) return rc;
  return launch_tc_stage<NT, 3>(g, 0, st);
}

struct TcBatchArgs {
  const TcFused* gs;
  const int32_t* cta0[4];
  const int64_t* offs;
  const int32_t *grid, *skip;
  const void* x;
  void* y;
  size_t smem;
  int np;
};
template <int NT, int STAGE>
static iga_status launch_tc_batch_stage(const TcBatchArgs& b, int64_t zero_bytes, cudaStream_t st) {
  static SmemOptIn optin;
  return launch_tc_fused(fd_tc_fused_batch_kernel<NT, STAGE>, optin, NT, b.grid[STAGE], b.smem,
                         st, STAGE > 0, b.gs, b.cta0[STAGE], b.np, b.offs, b.x, b.y, b.skip,
                         zero_bytes);
}
template <int NT>
static iga_status launch_tc_batch_apply(const TcBatchArgs& b, int64_t zero_bytes, cudaStream_t st) {
  iga_status rc;
  if ((rc = launch_tc_batch_stage<NT, 0>(b, zero_bytes, st))) return rc;
  if ((rc = launch_tc_batch_stage<NT, 1>(b, 0, st))) return rc;
  if ((rc = launch_tc_batch_stage<NT, 2>(b, 0, st))) return rc;
  return launch_tc_batch_stage<NT, 3>(b, 0, st);
}

}  // namespace iga

using namespace iga;

extern "C" {

iga_status iga_fd_tc_workspace(const int32_t* m, int64_t* elems) {
  clear_error();
  IGA_CHECK_ARG(m && elems, "null argument");
  int64_t kp[3];
  for (int d = 0; d < 3; ++d) kp[d] = ceil_div(m[d], 16) * 16;
  // rotated intermediates: [a1][m3][Kp2], [a2][m1][Kp3], [a3][m2][Kp1] and
  // the backward ones; the largest bounds all
  int64_t big = 0;
  big = std::max<int64_t>(big, (int64_t)m[0] * m[2] * kp[1]);
  big = std::max<int64_t>(big, (int64_t)m[1] * m[0] * kp[2]);
  big = std::max<int64_t>(big, (int64_t)m[2] * m[1] * kp[0]);
  *elems = big;
  return IGA_OK;
}

// 3D FD apply with BF16 tensor-core mode products.  Bfwd[d] / Bbwd[d]: the
// pre-tiled images of U_d^T / U_d (Np_d x Kp_d BF16, canonical K-major, see
// igaops_b200/fastdiag.py); inv_lambda: FP32, prod(m) entries (direction 1
// fastest); x, y: FP32 or FP64 (io_dtype), full control-point vectors; y is
// zeroed outside the box.  work0 / work1: BF16, iga_fd_tc_workspace elements
// each, of any content (their padding does not reach a result).
iga_status iga_fd_apply_tc(int io_dtype, const int32_t* n, const int32_t* lo, const int32_t* m,
                           const void* const* Bfwd, const void* const* Bbwd,
                           const float* inv_lambda, const void* x, void* y, void* work0,
                           void* work1, int32_t* status, iga_stream stream) {
  clear_error();
  IGA_CHECK_ARG(n && lo && m && Bfwd && Bbwd && inv_lambda && x && y && work0 && work1,
                "null argument");
  IGA_CHECK_ARG(io_dtype == IGA_F64 || io_dtype == IGA_F32, "io dtype %d", io_dtype);
  for (int d = 0; d < 3; ++d) {
    IGA_CHECK_ARG(m[d] >= 1 && m[d] <= 256, "free extent %d of direction %d not in 1..256", m[d],
                  d);
    IGA_CHECK_ARG(lo[d] >= 0 && lo[d] + m[d] <= n[d], "free box out of range in direction %d", d);
    IGA_CHECK_ARG(Bfwd[d] && Bbwd[d] && ((uintptr_t)Bfwd[d] & 15) == 0 &&
                      ((uintptr_t)Bbwd[d] & 15) == 0,
                  "B images must be 16-byte aligned");
  }
  IGA_CHECK_ARG(((uintptr_t)work0 & 15) == 0 && ((uintptr_t)work1 & 15) == 0,
                "work buffers must be 16-byte aligned");
  cudaStream_t st = as_stream(stream);
  int64_t N = (int64_t)n[0] * n[1] * n[2];
  const int64_t ybytes = N * (io_dtype == IGA_F64 ? 8 : 4);
  if (tc_fits_fused(m)) {
    TcFused f;
    tc_fused_desc(f, n, lo, m, Bfwd, Bbwd, inv_lambda, x, y, io_dtype == IGA_F64, work0, work1,
                  status);
    const bool own = ybytes <= kTcZeroPerCta * tc_fused_ctas(f, 0);
    if (!own) IGA_CUDA_TRY(cudaMemsetAsync(y, 0, (size_t)ybytes, st));
    return tc_fused_smem_max(f) <= kTcSmallSmem ? launch_tc_apply<256>(f, own ? ybytes : 0, st)
                                                : launch_tc_apply<512>(f, own ? ybytes : 0, st);
  }
  IGA_CUDA_TRY(cudaMemsetAsync(y, 0, (size_t)ybytes, st));
  TcGemm g[6];
  tc_stages(g, n, lo, m, Bfwd, Bbwd, inv_lambda, x, y, io_dtype == IGA_F64, work0, work1, status);
  iga_status rc;
  if ((rc = launch_tc<1, 0>(g[0], st, false))) return rc;
  if ((rc = launch_tc<0, 0>(g[1], st, true))) return rc;
  if ((rc = launch_tc<0, 1>(g[2], st, true))) return rc;
  if ((rc = launch_tc<0, 0>(g[3], st, true))) return rc;
  if ((rc = launch_tc<0, 0>(g[4], st, true))) return rc;
  if ((rc = launch_tc<0, 2>(g[5], st, true))) return rc;
  return IGA_OK;
}


static inline int64_t tc_align(int64_t b) { return (b + 255) / 256 * 256; }

iga_status iga_fd_tc_batch_table_bytes(int npatch, int64_t* bytes) {
  clear_error();
  IGA_CHECK_ARG(npatch >= 1 && bytes, "bad argument");
  *bytes = 6 * tc_align((int64_t)npatch * sizeof(TcGemm)) + 6 * tc_align((int64_t)(npatch + 1) * 4) +
           (int64_t)npatch * 8;
  return IGA_OK;
}

// Multi-patch FD apply: per patch p the arrays hold n/lo/m at [3p..3p+2],
// Bfwd/Bbwd images at [3p..3p+2], inv_lambda[p], work0[p], work1[p] and the
// element offset of its vectors in the flat x / y.  Fills the device table
// (synchronous copies) and returns the grid of each of the six products and
// the dynamic shared memory of the largest patch.
iga_status iga_fd_tc_batch_prepare(int npatch, const int32_t* n, const int32_t* lo,
                                   const int32_t* m, const void* const* Bfwd,
                                   const void* const* Bbwd, const float* const* inv_lambda,
                                   void* const* work0, void* const* work1,
                                   const int64_t* offsets, int io_dtype, int32_t* status,
                                   void* table, int32_t* grid, int64_t* smem) {
  clear_error();
  IGA_CHECK_ARG(npatch >= 1 && n && lo && m && Bfwd && Bbwd && inv_lambda && work0 && work1 &&
                    offsets && table && grid && smem,
                "null argument");
  IGA_CHECK_ARG(io_dtype == IGA_F64 || io_dtype == IGA_F32, "io dtype %d", io_dtype);
  IGA_CHECK_ARG(((uintptr_t)table & 255) == 0, "table must be 256-byte aligned");
  static_assert(sizeof(TcFused) <= sizeof(TcGemm) * 3, "the table is sized for TcGemm");
  std::vector<TcFused> fused((size_t)npatch);
  // One path for the whole batch: a launch's kernels overlap all patches. Five patches of
  // 43^3 and one of 133 x 43 x 43 points: 41 us through the six products; in a set of
  // their own the five take 24 us in four kernels, the one 32 us.
  bool all_fused = true;
  std::vector<TcGemm> st((size_t)6 * npatch);
  std::vector<int32_t> cta((size_t)6 * (npatch + 1));
  std::vector<int64_t> offs((size_t)npatch);
  int64_t tot[6] = {0, 0, 0, 0, 0, 0};
  size_t sm = 0;
  for (int p = 0; p < npatch; ++p) {
    for (int d = 0; d < 3; ++d) {
      const int mm = m[3 * p + d];
      IGA_CHECK_ARG(mm >= 1 && mm <= 256, "patch %d: free extent %d not in 1..256", p, mm);
      IGA_CHECK_ARG(lo[3 * p + d] >= 0 && lo[3 * p + d] + mm <= n[3 * p + d],
                    "patch %d: free box out of range", p);
      IGA_CHECK_ARG(Bfwd[3 * p + d] && Bbwd[3 * p + d] && ((uintptr_t)Bfwd[3 * p + d] & 15) == 0 &&
                        ((uintptr_t)Bbwd[3 * p + d] & 15) == 0,
                    "patch %d: B images must be 16-byte aligned", p);
      const size_t kp = (size_t)ceil_div(mm, 16) * 16;
      sm = std::max(sm, (128 + kp) * kp * 2);
    }
    IGA_CHECK_ARG(inv_lambda[p] && work0[p] && work1[p] && ((uintptr_t)work0[p] & 15) == 0 &&
                      ((uintptr_t)work1[p] & 15) == 0 && offsets[p] >= 0,
                  "patch %d: bad Lambda / work / offset", p);
    all_fused = all_fused && tc_fits_fused(m + 3 * p);
    tc_fused_desc(fused[p], n + 3 * p, lo + 3 * p, m + 3 * p, Bfwd + 3 * p, Bbwd + 3 * p,
                  inv_lambda[p], nullptr, nullptr, io_dtype == IGA_F64, work0[p], work1[p], status);
    TcGemm g[6];
    tc_stages(g, n + 3 * p, lo + 3 * p, m + 3 * p, Bfwd + 3 * p, Bbwd + 3 * p, inv_lambda[p],
              nullptr, nullptr, io_dtype == IGA_F64, work0[p], work1[p], status);
    for (int s = 0; s < 6; ++s) {
      st[(size_t)s * npatch + p] = g[s];
      cta[(size_t)s * (npatch + 1) + p] = (int32_t)tot[s];
      tot[s] += ceil_div(g[s].R, 128) * tc_nsplit(g[s].Np);
    }
    offs[p] = offsets[p];
  }
  if (all_fused) {
    // four kernels: the descriptors in the first slot, no CTAs in the last two
    sm = 0;
    for (int s = 0; s < 6; ++s) {
      tot[s] = 0;
      for (int p = 0; p < npatch && s < 4; ++p) {
        cta[(size_t)s * (npatch + 1) + p] = (int32_t)tot[s];
        tot[s] += tc_fused_ctas(fused[p], s);
        sm = std::max(sm, tc_fused_smem(fused[p], s));
      }
    }
  }
  for (int s = 0; s < 6; ++s) {
    IGA_CHECK_ARG(tot[s] < (1ll << 31), "too many CTAs");
    cta[(size_t)s * (npatch + 1) + npatch] = (int32_t)tot[s];
    grid[s] = (int32_t)tot[s];
  }
  char* t = (char*)table;
  const int64_t gb = tc_align((int64_t)npatch * sizeof(TcGemm));
  const int64_t cb = tc_align((int64_t)(npatch + 1) * 4);
  for (int s = 0; s < 6; ++s) {
    if (!all_fused)
      IGA_CUDA_TRY(cudaMemcpy(t + s * gb, st.data() + (size_t)s * npatch, npatch * sizeof(TcGemm),
                              cudaMemcpyHostToDevice));
    IGA_CUDA_TRY(cudaMemcpy(t + 6 * gb + s * cb, cta.data() + (size_t)s * (npatch + 1),
                            (npatch + 1) * 4, cudaMemcpyHostToDevice));
  }
  if (all_fused)
    IGA_CUDA_TRY(cudaMemcpy(t, fused.data(), npatch * sizeof(TcFused), cudaMemcpyHostToDevice));
  IGA_CUDA_TRY(cudaMemcpy(t + 6 * gb + 6 * cb, offs.data(), npatch * 8, cudaMemcpyHostToDevice));
  *smem = (int64_t)sm;
  return IGA_OK;
}

iga_status iga_fd_tc_batch_apply(int io_dtype, int npatch, const void* table, const int32_t* grid,
                                 int64_t smem, const void* x, void* y, int64_t ntot,
                                 const int32_t* skip, iga_stream stream) {
  clear_error();
  IGA_CHECK_ARG(npatch >= 1 && table && grid && x && y && ntot >= 0 && smem > 0 &&
                    smem <= 227 * 1024,
                "bad argument");
  IGA_CHECK_ARG(io_dtype == IGA_F64 || io_dtype == IGA_F32, "io dtype %d", io_dtype);
  cudaStream_t st = as_stream(stream);
  const int64_t ybytes = ntot * (io_dtype == IGA_F64 ? 8 : 4);
  const bool fused = grid[4] == 0;
  const bool own = fused && ybytes <= kTcZeroPerCta * grid[0];
  if (!own) IGA_CUDA_TRY(cudaMemsetAsync(y, 0, (size_t)ybytes, st));
  const char* t = (const char*)table;
  const int64_t gb = tc_align((int64_t)npatch * sizeof(TcGemm));
  const int64_t cb = tc_align((int64_t)(npatch + 1) * 4);
  const int64_t* offs = (const int64_t*)(t + 6 * gb + 6 * cb);
  auto G = [&](int s) { return (const TcGemm*)(t + s * gb); };
  auto C = [&](int s) { return (const int32_t*)(t + 6 * gb + s * cb); };
  iga_status rc;
  if (fused) {
    const TcBatchArgs b = {(const TcFused*)t, {C(0), C(1), C(2), C(3)}, offs, grid, skip, x, y,
                           (size_t)smem, npatch};
    return (size_t)smem <= kTcSmallSmem ? launch_tc_batch_apply<256>(b, own ? ybytes : 0, st)
                                        : launch_tc_batch_apply<512>(b, own ? ybytes : 0, st);
  }
  if ((rc = launch_tc_batch<1, 0>(G(0), C(0), npatch, offs, grid[0], smem, x, y, skip, st,
                                     false)))
    return rc;
  if ((rc = launch_tc_batch<0, 0>(G(1), C(1), npatch, offs, grid[1], smem, x, y, skip, st,
                                     true)))
    return rc;
  if ((rc = launch_tc_batch<0, 1>(G(2), C(2), npatch, offs, grid[2], smem, x, y, skip, st,
                                     true)))
    return rc;
  if ((rc = launch_tc_batch<0, 0>(G(3), C(3), npatch, offs, grid[3], smem, x, y, skip, st,
                                     true)))
    return rc;
  if ((rc = launch_tc_batch<0, 0>(G(4), C(4), npatch, offs, grid[4], smem, x, y, skip, st,
                                     true)))
    return rc;
  if ((rc = launch_tc_batch<0, 2>(G(5), C(5), npatch, offs, grid[5], smem, x, y, skip, st,
                                     true)))
    return rc;
  return IGA_OK;
}

}  // extern "C"
