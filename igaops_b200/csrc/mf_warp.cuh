// Warp-per-tile form of the fused 3D matrix-free operator (see mf_fused.cuh for
// the operator and its patterns).
//
// A CTA is one warp. It owns a tile of 8 x 8 quadrature pencils (directions 1, 2) and
// a segment of direction 3, two pencils per lane. Nothing is shared between warps, so
// the march has no CTA barrier, a point's band values are loaded once for the whole
// tile, and everything that belongs to the tile (pointers, counters, branches) is
// uniform over the CTA and lives on the uniform datapath.
//
// The points of direction 3 are taken in groups: runs of at most kGroupPts
// points between window moves (an element, usually). Before a group
//   * the test window moves: the oldest accumulator plane is final and two chains
//     of FP64 tensor-core products (m8n8k4) contract it over q2 and q1;
//   * the trial window moves: the next control plane's slab (copied one plane
//     ahead) is contracted over directions 1 and 2, on the tensor cores too.
// A lane owns the pencils (q1 = lane / 4, q2 = 2 (lane mod 4) + i), i = 0, 1: with
// the k-steps of a product taking the even and the odd members of the contracted
// index, the accumulators of one product are the operand of the next and the
// window entries come out at their owners, so only the slab and the weight
// fragments pass through shared memory.
// At a point the coefficients mix the W-long trial dot products and the result
// is spread over the W test accumulators. A group's coefficients are one bulk
// copy (packed [group][tile][point][stream][pencil], padding pencils zero) with
// the group's step rows beside them, in an NB-deep ring. The warps of a wave
// march through the groups at about the same pace, so with the group outermost
// they read one moving window of the stream instead of a page each.
//
// What bounds it: HBM for the stiffness (FP64 p3 128^3 2861 MB in 468 us, 6.1 TB/s,
// until the power cap lowers the SM clock to 1.7 GHz), latency and issue of the
// per-group chain for the mass, whose points carry eight bytes each. Against the
// CTA-per-tile kernel (16 x 8 tiles, shared chunks, CTA barriers; B200, us a launch
// with the clearing of y, back to back, best segment count): FP64 stiffness 3D p3 128^3 919 -> 468, p4 96^3
// 576 -> 216, p5 96^3 663 -> 420; FP64 mass p3 128^3 438 -> 155, p2 96^3 177 -> 62;
// FP32 stiffness p3 128^3 606 -> 268, p4 61 x 57 x 63 94 -> 46; FP64 gradu_v p2 40^3
// 34 -> 18. On the way: plane work through shared memory (a barrier per stage, the
// shared-memory pipe at 78 %) 525 and 214 us for the first two and four; four warps
// per CTA with batches of fixed length 25 % slower (per-warp values in vector
// registers); prefetching a third group into L2 and broadcasting tile constants by
// shuffles changed nothing.
#pragma once

#include "mf_fused.cuh"

namespace iga {

constexpr int kWarpFace = 8;                      // pencils per direction of a tile
constexpr int kWarpTile = kWarpFace * kWarpFace;  // pencils of a tile

// Step rows: the needed derivative orders of the trial group, then of the test
// group (step_group<T>(W) values each).
template <class P>
__host__ __device__ constexpr int trial_slot(int b) {
  return (b == 1 && P::last_trial_needed(0)) ? 1 : 0;
}
template <class P>
__host__ __device__ constexpr int ntrial_last() {
  return (P::last_trial_needed(0) ? 1 : 0) + (P::last_trial_needed(1) ? 1 : 0);
}
template <class P>
__host__ __device__ constexpr int test_slot(int a) {
  return ntrial_last<P>() + ((a == 1 && P::last_test_needed(0)) ? 1 : 0);
}
template <class P>
__host__ __device__ constexpr int ntest_last() {
  return (P::last_test_needed(0) ? 1 : 0) + (P::last_test_needed(1) ? 1 : 0);
}
template <typename T, class P>
__host__ __device__ constexpr int warp_row_len(int W) {
  return (ntrial_last<P>() + ntest_last<P>()) * step_group<T>(W);
}

// derivative orders of the test factors of direction 2
template <class P>
__host__ __device__ constexpr bool a2_needed(int b) {
  return P::tpair_needed(2 * b) || P::tpair_needed(2 * b + 1);
}
template <class P>
__host__ __device__ constexpr int na2() {
  return (a2_needed<P>(0) ? 1 : 0) + (a2_needed<P>(1) ? 1 : 0);
}
template <class P>
__host__ __device__ constexpr int a2_slot(int b) {
  return (b == 1 && a2_needed<P>(0)) ? 1 : 0;
}

// derivative orders of the trial factors of direction 2
template <class P>
__host__ __device__ constexpr bool b2_needed(int b) {
  return P::combo_needed(2 * b) || P::combo_needed(2 * b + 1);
}
template <class P>
__host__ __device__ constexpr int nb2() {
  return (b2_needed<P>(0) ? 1 : 0) + (b2_needed<P>(1) ? 1 : 0);
}
template <class P>
__host__ __device__ constexpr int b2_slot(int b) {
  return (b == 1 && b2_needed<P>(0)) ? 1 : 0;
}

// Points per group: the elements of a type-2 rule have three. (Groups of three are
// unrolled; the groups of two that Gauss rules of degrees 3 and 4 have take a loop, whose
// cost was not timed apart.)
constexpr int kGroupPts = 3;

// Groups in the coefficient ring.
constexpr int kWarpRing = 2;

// Resident CTAs (warps) per SM that the register budget is set for. Measured at
// 96^3 / 128^3 (us, best segment count): FP64 stiffness p3 8: 478, 12: 523, p4 8:
// 216, 12: 405 (spills); FP64 gradu_v p3 8: 170, 12: 124, p5 8: 262, 12: 317; FP64
// mass p2 16: 68, 20: 62, 24: 69, p5 16: 140, 20: 148; FP32 stiffness p4 12: 148,
// 16: 150, p5 12: 245, 16: 291; FP32 mass 20 (80 registers). FP64 stiffness of widths 3
// and 6 takes width 4's and 5's (not timed by themselves).
__host__ __device__ constexpr int warp_resident(bool f64, int S, int W) {
  return f64 ? (S > 3 ? 8 : S > 1 ? (W <= 4 ? 12 : 8) : (W <= 4 ? 20 : 16)) : (S > 1 ? 12 : 20);
}

// Shared memory of a CTA (byte offsets; every region 16-byte aligned). Band
// starts advance by at most one control plane per point, so a tile's control
// ranges are at most W + 7 wide. WIDE: some tile's range exceeds eight (degree 5,
// or elements of fewer than three points) and takes a second 8-block.
template <typename T, class P, int W, bool WIDE>
struct WarpSmem {
  static constexpr int E = (int)sizeof(T);
  static constexpr int range = W + kWarpFace - 1;           // widest control range
  static constexpr int NBK = WIDE ? 2 : 1;                  // 8-blocks of a range
  static constexpr int KC = WIDE ? (range + 3) / 4 : 2;     // k-steps over a slab row
  static constexpr int rows = 8 * NBK;                      // slab rows
  static constexpr int xrow = KC <= 3 ? 12 : 20;            // slab row stride, 4 mod 8
  static constexpr int row = warp_row_len<T, P>(W);
  static constexpr int chunk = P::S * kWarpTile;            // elements per point
  static constexpr int slot = kGroupPts * (chunk + row);    // elements per group
  static constexpr int ring = 64;  // after the mbarriers
  static constexpr int xs = ring + kWarpRing * slot * E;
  static constexpr int xhalf = rows * xrow * E;
  // weight fragments, 32 doubles each
  static constexpr int a1 = xs + 2 * xhalf;                 // [b1][kt]: trial bands of q1
  static constexpr int b2 = a1 + nb1<P>() * KC * 256;       // [b2][block][i]: of q2
  static constexpr int w2 = b2 + nb2<P>() * NBK * 2 * 256;  // [a2][block][i]: test weights of q2
  static constexpr int w1 = w2 + na2<P>() * NBK * 2 * 256;  // [a1][block][j]: of q1
  static constexpr int total = w1 + ng<P>() * NBK * 2 * 256;
};

// Asynchronous copy of one element to shared memory, where `in` holds.
template <int BYTES>
__device__ __forceinline__ void cp_async_elem(uint32_t dst, const void* src, bool in) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t"
      "@p cp.async.ca.shared.global [%0], [%1], %2;\n\t}" ::"r"(dst),
      "l"(src), "n"(BYTES), "r"((uint32_t)in)
      : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Group list behind the step rows: [0] number of groups, [1 + g] = first point
// of group g << 2 | moves before it (1 trial, 2 test), [1 + ngroups] = nq << 2.
template <typename T>
__host__ __device__ inline int64_t group_list_offset(int nq, int row) {  // bytes
  return ((int64_t)nq * row * (int)sizeof(T) + 15) / 16 * 16;
}

template <typename T, int W, class P, bool WIDE>
__device__ __forceinline__ void mfw_body(const FusedArgs<T>& a, const int unit, const int col) {
  using L = WarpSmem<T, P, W, WIDE>;
  constexpr int S = P::S, I = P::I, J = P::J;
  constexpr int NCOMBO = ncombo3<P>();
  constexpr int NB = kWarpRing;
  constexpr int G = step_group<T>(W);
  constexpr int F = kWarpFace, XR = L::xrow, E = L::E, NBK = L::NBK;
  static_assert(NB * 8 <= L::ring, "barrier area");
  extern __shared__ __align__(128) unsigned char smem[];

  const int lane = threadIdx.x;
  const int n1 = a.n[0], n2 = a.n[1], n3 = a.n[2];
  const int nq1 = a.nq[0], nq2 = a.nq[1], nq3 = a.nq[2];
  const int seg = unit % a.nseg, tile = unit / a.nseg;
  const int t1 = tile % a.tiles1, t2 = tile / a.tiles1;
  const int q1lo = t1 * F, w1 = min(F, nq1 - q1lo);
  const int q2lo = t2 * F, w2 = min(F, nq2 - q2lo);

  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
  T* ring = reinterpret_cast<T*>(smem + L::ring);
  T* xs = reinterpret_cast<T*>(smem + L::xs);

  // ----------------------------------------------------- groups of the segment
  const int* glist = reinterpret_cast<const int*>(reinterpret_cast<const char*>(a.step_table) +
                                                  group_list_offset<T>(nq3, L::row));
  // what depends on the tile alone is loaded before any of it is used; wide bands
  // have no registers to hold it over the ring's prologue and load it at its use
  int early[10];
  if constexpr (!WIDE) {
    early[0] = __ldg(a.tstart[0] + q1lo), early[1] = __ldg(a.tstart[0] + q1lo + w1 - 1);
    early[2] = __ldg(a.tstart[1] + q2lo), early[3] = __ldg(a.tstart[1] + q2lo + w2 - 1);
    early[4] = __ldg(a.wtstart[0] + q1lo), early[5] = __ldg(a.wtstart[0] + q1lo + w1 - 1);
    early[6] = __ldg(a.wtstart[1] + q2lo), early[7] = __ldg(a.wtstart[1] + q2lo + w2 - 1);
    early[8] = __ldg(a.tstart[0] + q1lo + min(lane >> 2, w1 - 1));
    early[9] = __ldg(a.tstart[1] + q2lo + min(lane >> 2, w2 - 1));
  }
  auto tile_int = [&](int slot, const int* at) { return WIDE ? __ldg(at) : early[slot]; };
  auto entry = [&](int g) { return __shfl_sync(0xffffffffu, __ldg(glist + 1 + g), 0); };
  const int ngrp = __shfl_sync(0xffffffffu, __ldg(glist), 0);
  const int ga = (int)((int64_t)ngrp * seg / a.nseg), gb = (int)((int64_t)ngrp * (seg + 1) / a.nseg);
  if (ga >= gb) return;
  // entries of the groups g .. g + NB + 1
  int en[NB + 2];
#pragma unroll
  for (int k = 0; k < NB + 2; ++k) en[k] = entry(min(ga + k, ngrp));
  const int qa = en[0] >> 2;

  // ------------------------------------------------------- coefficient ring
  // (running source pointers; csrc: the next group's chunks of the first tile)
  const int ntiles = a.tiles1 * a.tiles2;
  const T* csrc = a.packed + (int64_t)qa * ntiles * L::chunk;
  const T* rsrc = a.step_table + (int64_t)qa * L::row;
  auto issue = [&](int slot, int np) {
    const uint32_t bar = smem_u32(bars) + slot * 8;
    const uint32_t dst = smem_u32(ring) + slot * (L::slot * E);
    if (lane == 0) {
      mbar_arrive_expect_tx(bar, (uint32_t)(np * ((L::chunk + L::row) * E)));
      bulk_g2s(dst, csrc + (int64_t)(tile * np) * L::chunk, (uint32_t)(np * (L::chunk * E)), bar);
      bulk_g2s(dst + kGroupPts * L::chunk * E, rsrc, (uint32_t)(np * (L::row * E)), bar);
    }
  };
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < NB; ++s) mbar_init(smem_u32(&bars[s]), 1);
    fence_mbar_init();
  }
#pragma unroll
  for (int s = 0; s < NB; ++s) {
    const int np = (en[s + 1] >> 2) - (en[s] >> 2);
    // the wait test hook withholds the first group: its wait runs out
    if (ga + s < gb && !(a.wait_test && s == 0)) issue(s, np);
    csrc += (int64_t)(np * ntiles) * L::chunk;
    rsrc += np * L::row;
  }

  // ------------------------------------------------------------ tile tables
  const int c1lo = tile_int(0, a.tstart[0] + q1lo);
  const int C1r = tile_int(1, a.tstart[0] + q1lo + w1 - 1) - c1lo + W;
  const int c2lo = tile_int(2, a.tstart[1] + q2lo);
  const int C2r = tile_int(3, a.tstart[1] + q2lo + w2 - 1) - c2lo + W;
  const int d1lo = tile_int(4, a.wtstart[0] + q1lo);
  const int D1r = min(tile_int(5, a.wtstart[0] + q1lo + w1 - 1) + W - 1, n1 - 1) - d1lo + 1;
  const int d2lo = tile_int(6, a.wtstart[1] + q2lo);
  const int D2r = min(tile_int(7, a.wtstart[1] + q2lo + w2 - 1) + W - 1, n2 - 1) - d2lo + 1;
  // Weight fragments (lane = 4 gq + tq holds A[gq][tq] or B[tq][gq]), zero outside
  // the bands and the tile. A lane's pencils are (q1 = gq, q2 = 2 tq + i), so with
  // the k index of a product standing for point 2 tq + i (i = k-step) or control
  // row 2 tq + i, the accumulators of one product are operands of the next.
  const int gq = lane >> 2, tq = lane & 3;
  double* fa1 = reinterpret_cast<double*>(smem + L::a1) + lane;
  double* fb2 = reinterpret_cast<double*>(smem + L::b2) + lane;
  double* fw2 = reinterpret_cast<double*>(smem + L::w2) + lane;
  double* fw1 = reinterpret_cast<double*>(smem + L::w1) + lane;
  {
    const int q1 = q1lo + min(gq, w1 - 1), q2 = q2lo + min(gq, w2 - 1);
    const int s1 = tile_int(8, a.tstart[0] + q1) - c1lo, s2 = tile_int(9, a.tstart[1] + q2) - c2lo;
    auto band = [&](const T* v, int q, int k) {
      return k >= 0 && k < W ? (double)__ldg(v + (int64_t)q * W + k) : 0.0;
    };
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      if (P::b1_needed(b)) {
#pragma unroll
        for (int kt = 0; kt < L::KC; ++kt)
          fa1[(b1_slot<P>(b) * L::KC + kt) * 32] = band(b ? a.tB1[0] : a.tB0[0], q1, 4 * kt + tq - s1);
      }
      if (b2_needed<P>(b)) {
#pragma unroll
        for (int m = 0; m < 2 * NBK; ++m)
          fb2[(b2_slot<P>(b) * 2 * NBK + m) * 32] =
              band(b ? a.tB1[1] : a.tB0[1], q2, 8 * (m >> 1) + 2 * tq + (m & 1) - s2);
      }
    }
#pragma unroll 1
    for (int m = 0; m < 2 * NBK; ++m) {
      const int r = 8 * (m >> 1) + gq, l = 2 * tq + (m & 1);
      double v2[2] = {0.0, 0.0}, v1[2] = {0.0, 0.0};
      if (r < D2r && l < w2) {
        const int k = q2lo + l - __ldg(a.rstart[1] + d2lo + r);
        if (k >= 0 && k < a.RW) {
          const int64_t at = (int64_t)(d2lo + r) * a.RW + k;
          if (a2_needed<P>(0)) v2[0] = (double)__ldg(a.wR0[1] + at);
          if (a2_needed<P>(1)) v2[1] = (double)__ldg(a.wR1[1] + at);
        }
      }
      if (r < D1r && l < w1) {
        const int k = q1lo + l - __ldg(a.rstart[0] + d1lo + r);
        if (k >= 0 && k < a.RW) {
          const int64_t at = (int64_t)(d1lo + r) * a.RW + k;
          if (P::a1_needed(0)) v1[0] = (double)__ldg(a.wR0[0] + at);
          if (P::a1_needed(1)) v1[1] = (double)__ldg(a.wR1[0] + at);
        }
      }
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        if (a2_needed<P>(b)) fw2[(a2_slot<P>(b) * 2 * NBK + m) * 32] = v2[b];
        if (P::a1_needed(b)) fw1[(g_slot<P>(b) * 2 * NBK + m) * 32] = v1[b];
      }
    }
  }

  const int64_t pstride = (int64_t)n1 * n2;  // control points per plane
  // x slab of one control plane, copied one plane ahead into the other half of
  // xs, 4 rows x 8 columns per pass (rows paired so that a half-warp's two rows
  // fall on different banks). Entries past the control range or the patch stay
  // zero; they meet zero weights. (So do entries that an output does not reach: an
  // infinity or NaN of x or of a coefficient makes every output of the tiles whose
  // control ranges or points hold it NaN, as it did in the 16 x 8 tiles.)
  for (int e = lane; e < 2 * L::xhalf / E; e += 32) xs[e] = T(0);
  const int xr0 = ((lane >> 3) & 1) * 2 + (lane >> 4), xc0 = lane & 7;
  const int xrows = min(C2r, n2 - c2lo), xcols = min(C1r, n1 - c1lo);
  const bool xin0 = xr0 < xrows && xc0 < xcols, xin1 = xr0 + 4 < xrows && xc0 < xcols;
  const T* xsrc = a.x + (int64_t)col * a.N + (int64_t)c2lo * n1 + c1lo;
  int xplane = __ldg(a.tstart[2] + qa);
  xsrc += min(xplane, n3 - 1) * pstride;
  const int xg0 = xr0 * n1 + xc0, xg1 = xg0 + 4 * n1;
  const uint32_t xdst = smem_u32(xs) + (xr0 * XR + xc0) * E;
  int xflip = 0;  // half (bytes) that the next copy fills
  auto fetch = [&]() {
    cp_async_elem<E>(xdst + xflip, xsrc + xg0, xin0);
    cp_async_elem<E>(xdst + xflip + 4 * XR * E, xsrc + xg1, xin1);
    if constexpr (WIDE) {
      for (int r = 8; r < xrows; r += 4)
        cp_async_elem<E>(xdst + xflip + r * XR * E, xsrc + xg0 + r * n1,
                         xr0 + r < xrows && xc0 < xcols);
      for (int c = 8; c < xcols; c += 4)  // 8 rows x 4 columns per pass
        for (int r = lane >> 2; r < xrows; r += 8)
          cp_async_elem<E>(smem_u32(xs) + xflip + (r * XR + c + (lane & 3)) * E,
                           xsrc + r * n1 + c + (lane & 3), c + (lane & 3) < xcols);
    }
    cp_async_commit();
    if (++xplane < n3) xsrc += pstride;
  };

  T win[NCOMBO][W][2];  // trial planes at the lane's pencils
  const T* xl = xs + gq * XR + tq;
  // a slab (entry (row 8 nb + gq, column 4 kt + tq) from get) contracted over q1,
  // then q2, both on the tensor cores, the first product's accumulators being the
  // second's A operand; the result enters the window
  auto contract = [&](auto&& get, auto&& then) {
    double d2[NCOMBO][2];
#pragma unroll
    for (int c = 0; c < NCOMBO; ++c) d2[c][0] = d2[c][1] = 0.0;
#pragma unroll
    for (int nb = 0; nb < NBK; ++nb) {
      if (nb == 1 && C2r <= 8) break;
      double d1[2][2];
      d1[0][0] = d1[0][1] = d1[1][0] = d1[1][1] = 0.0;
#pragma unroll
      for (int kt = 0; kt < L::KC; ++kt) {
        if (kt >= 2 && C1r <= 4 * kt) break;
        const double xv = (double)get(nb, kt);
        if (P::b1_needed(0)) dmma_8x8x4(d1[0][0], d1[0][1], fa1[kt * 32], xv);
        if (P::b1_needed(1)) dmma_8x8x4(d1[1][0], d1[1][1], fa1[(b1_slot<P>(1) * L::KC + kt) * 32], xv);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (P::combo_needed(c))
            dmma_8x8x4(d2[combo_slot<P>(c)][0], d2[combo_slot<P>(c)][1], d1[c & 1][i],
                       fb2[(b2_slot<P>(c >> 1) * 2 * NBK + 2 * nb + i) * 32]);
    }
    then();
#pragma unroll
    for (int c = 0; c < NCOMBO; ++c)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int m = 0; m < W - 1; ++m) win[c][m][i] = win[c][m + 1][i];
        win[c][W - 1][i] = (T)d2[c][i];
      }
  };
  // the next plane: its slab has landed, the one after it gets under way
  auto produce = [&]() {
    cp_async_wait_all();
    __syncwarp();
    const T* xb = xl + xflip / E;
    xflip = L::xhalf - xflip;
    contract([&](int nb, int kt) { return xb[8 * nb * XR + 4 * kt]; }, fetch);
  };

  T acc[I][W][2];  // test planes
#pragma unroll
  for (int i = 0; i < I; ++i)
#pragma unroll
    for (int k = 0; k < W; ++k) acc[i][k][0] = acc[i][k][1] = T(0);
  int yleft = n3 - __ldg(a.wtstart[2] + qa);  // planes of y from the oldest one on
  T* ydst = a.y + (int64_t)col * a.N + (int64_t)d2lo * n1 + d1lo + (n3 - yleft) * pstride;
  const int ylane = gq * n1 + 2 * tq;
  // the oldest test plane is final: contracted over q2 (the accumulators are the B
  // operand), then q1, and added into y
  auto retire = [&]() {
    if (yleft > 0) {
      double v[4][2];
#pragma unroll
      for (int pr = 0; pr < 4; ++pr) {
        if (!P::tpair_needed(pr)) continue;
        T v0 = T(0), v1 = T(0);
#pragma unroll
        for (int i = 0; i < I; ++i)
          if (P::tpair(i) == pr) {
            v0 += acc[i][0][0];
            v1 += acc[i][0][1];
          }
        v[pr][0] = (double)v0;
        v[pr][1] = (double)v1;
      }
#pragma unroll
      for (int mt = 0; mt < NBK; ++mt) {
        if (mt == 1 && D2r <= 8) break;
        double e[2][2];
        e[0][0] = e[0][1] = e[1][0] = e[1][1] = 0.0;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int pr = 0; pr < 4; ++pr)
            if (P::tpair_needed(pr))
              dmma_8x8x4(e[pr & 1][0], e[pr & 1][1],
                         fw2[(a2_slot<P>(pr >> 1) * 2 * NBK + 2 * mt + i) * 32], v[pr][i]);
#pragma unroll
        for (int nt = 0; nt < NBK; ++nt) {
          if (nt == 1 && D1r <= 8) break;
          double c0 = 0.0, c1 = 0.0;
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            if (!P::a1_needed(g)) continue;
#pragma unroll
            for (int j = 0; j < 2; ++j)
              dmma_8x8x4(c0, c1, e[g][j], fw1[(g_slot<P>(g) * 2 * NBK + 2 * nt + j) * 32]);
          }
          T* yr = ydst + ylane + mt * 8 * n1 + nt * 8;
          const bool in = mt * 8 + gq < D2r;
          if (in && nt * 8 + 2 * tq < D1r) atomicAdd(yr, (T)c0);
          if (in && nt * 8 + 2 * tq + 1 < D1r) atomicAdd(yr + 1, (T)c1);
        }
      }
    }
    --yleft;
    ydst += pstride;
#pragma unroll
    for (int i = 0; i < I; ++i)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int k = 0; k < W - 1; ++k) acc[i][k][c] = acc[i][k + 1][c];
        acc[i][W - 1][c] = T(0);
      }
  };

  auto point = [&](const T* cs, const T* row) {
    T u[J][2];
#pragma unroll
    for (int j = 0; j < J; ++j) {
      T bq[G];
      load_group<T, G>(row + trial_slot<P>(P::beta(j, 2)) * G, bq);
      const int c = combo_slot<P>(P::combo(j));
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        T v0 = bq[0] * win[c][0][i], v1 = bq[1] * win[c][1][i];
#pragma unroll
        for (int k = 2; k < W; ++k) {
          if (k & 1) v1 += bq[k] * win[c][k][i];
          else v0 += bq[k] * win[c][k][i];
        }
        u[j][i] = v0 + v1;
      }
    }
    T cv[S][2];
#pragma unroll
    for (int s = 0; s < S; ++s) ld2(cs + s * kWarpTile + lane * 2, cv[s][0], cv[s][1]);
#pragma unroll
    for (int i = 0; i < I; ++i) {
      T g[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        g[c] = cv[P::cidx(i, 0)][c] * u[0][c];
#pragma unroll
        for (int j = 1; j < J; ++j) g[c] += cv[P::cidx(i, j)][c] * u[j][c];
      }
      T wq[G];
      load_group<T, G>(row + test_slot<P>(P::alpha(i, 2)) * G, wq);
#pragma unroll
      for (int k = 0; k < W; ++k) {
        acc[i][k][0] += wq[k] * g[0];
        acc[i][k][1] += wq[k] * g[1];
      }
    }
  };

  // -------------------------------------------------------------- the march
  __syncwarp();
  if constexpr (WIDE) {
    fetch();
#pragma unroll 1
    for (int k = 0; k < W; ++k) produce();
  } else {
    // The first window's planes straight from global memory, all loads at once: a
    // segment's start was a chain of W slab copies. Mass, degree 3, 8^3 and 16^3:
    // 10.4 -> 8.5 us; stiffness, degree 3, 48^3: 39.0 -> 37.2 us, 128^3: 476 -> 468 us
    // (burst). Wide bands keep the copies: W x 2 more registers would spill.
    T xi[W][2];
#pragma unroll
    for (int k = 0; k < W; ++k) {
#pragma unroll
      for (int kt = 0; kt < 2; ++kt)
        xi[k][kt] = gq < xrows && 4 * kt + tq < xcols ? __ldg(xsrc + gq * n1 + 4 * kt + tq) : T(0);
      if (++xplane < n3) xsrc += pstride;
    }
    fetch();
#pragma unroll
    for (int k = 0; k < W; ++k)
      contract([&](int, int kt) { return xi[k][kt]; }, [] {});
  }
  int slot = 0;
  uint32_t parity = 0;
#pragma unroll 1
  for (int g = ga; g < gb; ++g) {
    const int enew = __ldg(glist + 1 + min(g + NB + 2, ngrp));
    if (g > ga) {  // the segment's first windows are in place
      if (en[0] & 2) retire();
      if (en[0] & 1) produce();
    }
    const int np = (en[1] >> 2) - (en[0] >> 2);
    const bool ok = mbar_wait_bounded_ns(smem_u32(bars) + slot * 8, parity,
                                         a.wait_test ? kWaitTestLimitNs : kWaitLimitNs);
    if (!__all_sync(0xffffffffu, ok)) {
      if (lane == 0) {
        // the copies still in flight land before the CTA leaves
        for (int o = 1; o < NB && g + o < gb; ++o)
          (void)mbar_wait_bounded(smem_u32(&bars[(slot + o) % NB]),
                                  slot + o >= NB ? parity ^ 1u : parity);
        report_status(a.status, IGA_ERR_TIMEOUT);
      }
      cp_async_wait_all();
      return;
    }
    const T* cs = ring + slot * L::slot;
    const T* row = cs + kGroupPts * L::chunk;
    if (np == kGroupPts) {
#pragma unroll
      for (int t = 0; t < kGroupPts; ++t) point(cs + t * L::chunk, row + t * L::row);
    } else {
#pragma unroll 1
      for (int t = 0; t < np; ++t) point(cs + t * L::chunk, row + t * L::row);
    }
    __syncwarp();  // every lane is done with the group: its slot is refilled
    if (g + NB < gb) {
      const int nn = (en[NB + 1] >> 2) - (en[NB] >> 2);
      issue(slot, nn);
      csrc += (int64_t)(nn * ntiles) * L::chunk;
      rsrc += nn * L::row;
    }
    if (++slot == NB) {
      slot = 0;
      parity ^= 1u;
    }
#pragma unroll
    for (int k = 0; k < NB + 1; ++k) en[k] = en[k + 1];
    en[NB + 1] = __shfl_sync(0xffffffffu, enew, 0);
  }
#pragma unroll(WIDE ? 1 : W)
  for (int k = 0; k < W; ++k) retire();
  cp_async_wait_all();
}

template <typename T, int W, class P, bool WIDE>
__global__ void __launch_bounds__(32, warp_resident(sizeof(T) == 8, P::S, W))
    mfw_kernel(const __grid_constant__ FusedArgs<T> a) {
  mfw_body<T, W, P, WIDE>(a, blockIdx.x, blockIdx.y);
}

// Arguments of the CTA's patch in a multi-patch launch (patch p owns CTAs
// [cta0[p], cta0[p+1]), its vectors start at offs[p]): the patch, or -1 when it is
// done (its output stays zero).
template <typename T>
__device__ __forceinline__ int mfw_batch_args(const FusedArgs<T>* __restrict__ args,
                                              const int32_t* __restrict__ cta0, int npatch,
                                              const int64_t* __restrict__ offs, const T* xb, T* yb,
                                              const int32_t* __restrict__ skip, FusedArgs<T>& sa) {
  int lo = 0, hi = npatch;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(cta0 + mid) <= (int)blockIdx.x) lo = mid;
    else hi = mid;
  }
  const int p = lo;
  if (skip && __ldg(skip + p) >= 0) return -1;
  const int* src = reinterpret_cast<const int*>(args + p);
  int* dst = reinterpret_cast<int*>(&sa);
  for (int i = threadIdx.x; i < (int)(sizeof(FusedArgs<T>) / sizeof(int)); i += 32) dst[i] = src[i];
  __syncwarp();
  if (threadIdx.x == 0) {
    sa.x = xb + offs[p];
    sa.y = yb + offs[p];
  }
  __syncwarp();
  return p;
}

// Many patches of one pattern and band width in one launch.
template <typename T, int W, class P, bool WIDE>
__global__ void __launch_bounds__(32, warp_resident(sizeof(T) == 8, P::S, W))
    mfw_batch_kernel(const FusedArgs<T>* __restrict__ args, const int32_t* __restrict__ cta0,
                     int npatch, const int64_t* __restrict__ offs, const T* xb, T* yb,
                     const int32_t* __restrict__ skip) {
  __shared__ FusedArgs<T> sa;
  const int p = mfw_batch_args<T>(args, cta0, npatch, offs, xb, yb, skip, sa);
  if (p < 0) return;
  mfw_body<T, W, P, WIDE>(sa, (int)blockIdx.x - __ldg(cta0 + p), 0);
}

}  // namespace iga
