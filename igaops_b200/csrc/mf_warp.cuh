// Warp-per-tile form of the fused 3D matrix-free operator (see mf_fused.cuh for
// the operator and its patterns).
//
// A CTA is one warp. It owns a tile of 8 x 8 quadrature pencils (directions
// 1, 2) and a segment of direction 3; lane (ly, lx2) owns the neighbouring
// pencils 2 lx2, 2 lx2 + 1 of row ly. Nothing is shared between warps, so the march has no CTA
// barrier, a point's band values are loaded once for the whole tile, and
// everything that belongs to the tile (pointers, counters, branches) is uniform
// over the CTA and lives on the uniform datapath.
//
// The points of direction 3 are taken in groups: runs of at most kGroupPts
// points between window moves (an element, usually). Before a group
//   * the test window moves: the oldest accumulator plane is final; it goes to
//     shared memory and two chains of FP64 tensor-core products (m8n8k4)
//     contract it over q2 and q1. The first chain's result fragment is the
//     second chain's A operand when the second contraction takes the even
//     points of q1 in its first k-step and the odd ones in its second, so the
//     intermediate stays in registers;
//   * the trial window moves: the next control plane's slab (copied one plane
//     ahead) is contracted over directions 1 and 2.
// At a point the coefficients mix the W-long trial dot products and the result
// is spread over the W test accumulators. A group's coefficients are one bulk
// copy (packed [group][tile][point][stream][pencil], padding pencils zero) with
// the group's step rows beside them, in an NB-deep ring. The warps of a wave
// march through the groups at about the same pace, so with the group outermost
// they read one moving window of the stream instead of a page each.
//
// What bounds it: instruction issue and the latency of the per-group chain
// (production, points, flush) at the residency that registers allow; FP64
// stiffness at 2 KB of registers per lane pair of pencils runs eight warps per
// SM and comes within 15-20 % of the measured copy bandwidth. Measured against
// the CTA-per-tile kernel (16 x 8 tiles, shared chunks, CTA barriers; B200, CUDA
// events, best segment count, us): FP64 stiffness 3D p3 128^3 919 -> 520
// (2861 MB, 5.5 TB/s; 600 once the power cap lowers the SM clock to 1.7 GHz),
// p4 96^3 576 -> 275, p5 96^3 663 -> 491; FP64 mass p3 128^3 438 -> 210, p2 96^3
// 177 -> 85; FP32 stiffness p3 128^3 606 -> 310, p4 61 x 57 x 63 94 -> 53; FP64
// gradu_v p2 40^3 34 -> 22; 9.5 -> 4.1 (stiffness) and 5.4 -> 1.9 (mass) warp
// instructions per point. Four warps per CTA with a batch of fixed length cost
// 25 % more (per-warp values in vector registers), two blocks of pencils per
// lane gained 5 % for FP64 mass and lost 20 % for FP32 stiffness.
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

// Points per group: the elements of a type-2 rule have three.
constexpr int kGroupPts = 3;

// Groups in the coefficient ring.
constexpr int kWarpRing = 2;

// Resident CTAs (warps) per SM that the register budget is set for. Measured at
// 96^3 / 128^3 (us, best segment count): FP64 stiffness p3 8: 520, 12: 627
// (spills), p4 8: 282, 12: 471; FP64 gradu_v p3 8: 170, 12: 149, p5 8: 262, 12:
// 335; FP64 mass p2 16: 94, 20: 85, 24: 91, p5 16: 155, 20: 189; FP32 stiffness
// p4 8: 205, 12: 172, 16: 177; FP32 mass p4 16: 85, 20: 76, 24: 80.
__host__ __device__ constexpr int warp_resident(bool f64, int S, int W) {
  return f64 ? (S > 3 ? 8 : S > 1 ? (W <= 4 ? 12 : 8) : (W <= 4 ? 20 : 16)) : (S > 1 ? 12 : 20);
}

// Shared memory of a CTA (byte offsets; every region 16-byte aligned). Band
// starts advance by at most one control plane per point, so a block's control
// ranges are at most W + 7 wide and every offset is a compile-time constant.
template <typename T, class P, int W>
struct WarpSmem {
  static constexpr int E = (int)sizeof(T);
  static constexpr int range = W + kWarpFace - 1;
  static constexpr int rows = (range + 3) / 4 * 4;          // rows of the slab (whole passes)
  static constexpr int xrow = range;                        // slab row stride
  static constexpr int nblk = (range + 7) / 8;              // 8-blocks of a control range
  static constexpr int row = warp_row_len<T, P>(W);
  static constexpr int chunk = P::S * kWarpTile;            // elements per point
  static constexpr int slot = kGroupPts * (chunk + row);    // elements per group
  static constexpr int bw = W % 2 ? 2 * W : 2 * W + 2;      // band row stride (conflict-free)
  __host__ __device__ static constexpr int up(int b) { return (b + 15) / 16 * 16; }
  static constexpr int ring = 64;  // after the mbarriers
  static constexpr int done = ring + kWarpRing * slot * E;
  static constexpr int a1s = done + npair3<P>() * kWarpTile * 8;
  static constexpr int xs = a1s + up(nb1<P>() * rows * kWarpFace * E);
  static constexpr int xhalf = up(rows * xrow * E);
  static constexpr int b1 = xs + 2 * xhalf;
  static constexpr int b2 = b1 + up(kWarpFace * bw * E);
  static constexpr int f2 = b2 + up(kWarpFace * bw * E);    // [mt][b][kt][lane]
  static constexpr int f1 = f2 + nblk * na2<P>() * 2 * 32 * 8;  // [nt][g][kt][lane]
  static constexpr int total = f1 + nblk * ng<P>() * 2 * 32 * 8;
};

// Asynchronous copy of one element to shared memory.
template <int BYTES>
__device__ __forceinline__ void cp_async_elem(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Group list behind the step rows: [0] number of groups, [1 + g] = first point
// of group g << 2 | moves before it (1 trial, 2 test), [1 + ngroups] = nq << 2.
template <typename T>
__host__ __device__ inline int64_t group_list_offset(int nq, int row) {  // bytes
  return ((int64_t)nq * row * (int)sizeof(T) + 15) / 16 * 16;
}

template <typename T, int W, class P>
__device__ __forceinline__ void mfw_body(const FusedArgs<T>& a, const int unit, const int col) {
  using L = WarpSmem<T, P, W>;
  constexpr int S = P::S, I = P::I, J = P::J;
  constexpr int NCOMBO = ncombo3<P>();
  constexpr int NB = kWarpRing;
  constexpr int G = step_group<T>(W);
  constexpr int F = kWarpFace, XR = L::xrow, ROWS = L::rows, E = L::E;
  static_assert(NB * 8 <= L::ring, "barrier area");
  static_assert(L::nblk == 2, "two 8-blocks cover a control range");
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
  double* done = reinterpret_cast<double*>(smem + L::done);
  T* a1s = reinterpret_cast<T*>(smem + L::a1s);
  T* xs = reinterpret_cast<T*>(smem + L::xs);
  T* b1t = reinterpret_cast<T*>(smem + L::b1);
  T* b2t = reinterpret_cast<T*>(smem + L::b2);
  double* f2 = reinterpret_cast<double*>(smem + L::f2);
  double* f1 = reinterpret_cast<double*>(smem + L::f1);

  // ----------------------------------------------------- groups of the segment
  const int* glist = reinterpret_cast<const int*>(reinterpret_cast<const char*>(a.step_table) +
                                                  group_list_offset<T>(nq3, L::row));
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
  const int c1lo = __ldg(a.tstart[0] + q1lo);
  const int C1r = __ldg(a.tstart[0] + q1lo + w1 - 1) - c1lo + W;
  const int c2lo = __ldg(a.tstart[1] + q2lo);
  const int C2r = __ldg(a.tstart[1] + q2lo + w2 - 1) - c2lo + W;
  const int d1lo = __ldg(a.wtstart[0] + q1lo);
  const int D1r = min(__ldg(a.wtstart[0] + q1lo + w1 - 1) + W - 1, n1 - 1) - d1lo + 1;
  const int d2lo = __ldg(a.wtstart[1] + q2lo);
  const int D2r = min(__ldg(a.wtstart[1] + q2lo + w2 - 1) + W - 1, n2 - 1) - d2lo + 1;
  for (int e = lane; e < F * 2 * W; e += 32) {
    const int l = e / (2 * W), r = e - l * 2 * W, b = r / W, k = r - b * W;
    b1t[l * L::bw + r] =
        __ldg((b ? a.tB1[0] : a.tB0[0]) + (int64_t)(q1lo + min(l, w1 - 1)) * W + k);
    b2t[l * L::bw + r] =
        __ldg((b ? a.tB1[1] : a.tB0[1]) + (int64_t)(q2lo + min(l, w2 - 1)) * W + k);
  }
  const int gq = lane >> 2, tq = lane & 3;  // fragment coordinates
  // fragments of the test weights, zero outside the band and the tile.
  // q2: A operand, rows r2, columns l2 = 4 kt + tq; q1: B operand, rows
  // l1 = 2 tq + kt, columns r1
#pragma unroll 1
  for (int m = 0; m < L::nblk * 4; ++m) {
    const int r = (m >> 2) * 8 + gq, b = (m >> 1) & 1, kt = m & 1;
    double v2 = 0.0, v1 = 0.0;
    if (r < D2r && 4 * kt + tq < w2) {
      const int k = q2lo + 4 * kt + tq - __ldg(a.rstart[1] + d2lo + r);
      if (k >= 0 && k < a.RW)
        v2 = (double)__ldg((b ? a.wR1[1] : a.wR0[1]) + (int64_t)(d2lo + r) * a.RW + k);
    }
    if (r < D1r && 2 * tq + kt < w1) {
      const int k = q1lo + 2 * tq + kt - __ldg(a.rstart[0] + d1lo + r);
      if (k >= 0 && k < a.RW)
        v1 = (double)__ldg((b ? a.wR1[0] : a.wR0[0]) + (int64_t)(d1lo + r) * a.RW + k);
    }
    const int mt = m >> 2;
    if (b ? a2_needed<P>(1) : a2_needed<P>(0))
      f2[((mt * na2<P>() + (b ? a2_slot<P>(1) : 0)) * 2 + kt) * 32 + lane] = v2;
    if (b ? P::a1_needed(1) : P::a1_needed(0))
      f1[((mt * ng<P>() + (b ? g_slot<P>(1) : 0)) * 2 + kt) * 32 + lane] = v1;
  }

  const int64_t pstride = (int64_t)n1 * n2;  // control points per plane
  // lane roles: production over q1 (column lx, rows r0 + 4 i), production over
  // q2 and the points (row ly, pencils px, px + 1)
  const int ly = lane >> 2, px = 2 * (lane & 3);
  const int lx = lane & 7, r0 = lane >> 3;
  const int s1 = __ldg(a.tstart[0] + q1lo + min(lx, w1 - 1)) - c1lo;
  const int s2 = __ldg(a.tstart[1] + q2lo + min(ly, w2 - 1)) - c2lo;
  const T* b1l = b1t + lx * L::bw;
  const T* b2l = b2t + ly * L::bw;
  const T* xr0 = xs + r0 * XR + s1;
  T* a1w = a1s + r0 * F + lx;
  const T* a1r = a1s + s2 * F + px;
  double* dnw = done + ly * F + (px ^ ((ly & 2) << 1));
  const double* dnr = done + tq * F + (gq ^ ((tq & 2) << 1));

  // x slab of one control plane, copied one plane ahead into the other half of
  // xs: 4 rows x 8 columns per pass, columns beyond the eighth in a remainder
  // loop. Control points beyond the patch only meet zero band values: their
  // copies read the nearest point of the patch instead.
  auto xoff = [&](int r, int c) { return min(r, n2 - 1 - c2lo) * n1 + min(c, n1 - 1 - c1lo); };
  const int xg0 = xoff(r0, min(lx, C1r - 1)), xg1 = xoff(min(r0 + 4, C2r - 1), min(lx, C1r - 1));
  const T* xsrc = a.x + (int64_t)col * a.N + (int64_t)c2lo * n1 + c1lo;
  int xplane = __ldg(a.tstart[2] + qa);
  xsrc += min(xplane, n3 - 1) * pstride;
  const uint32_t xdst = smem_u32(xs) + (r0 * XR + lx) * E;
  const bool wide = C1r > 8 || C2r > 8;
  int xflip = 0;  // half (bytes) that the next copy fills
  auto fetch = [&]() {
    cp_async_elem<E>(xdst + xflip, xsrc + xg0);
    cp_async_elem<E>(xdst + xflip + 4 * XR * E, xsrc + xg1);
    if (wide) {
      if (C2r > 8)
        cp_async_elem<E>(xdst + xflip + 8 * XR * E,
                         xsrc + xoff(min(r0 + 8, C2r - 1), min(lx, C1r - 1)));
#pragma unroll 1
      for (int e = lane; e < (C1r - 8) * ROWS; e += 32) {
        const int c = 8 + e / ROWS, r = e % ROWS;
        cp_async_elem<E>(smem_u32(xs) + xflip + (r * XR + c) * E, xsrc + xoff(min(r, C2r - 1), c));
      }
    }
    cp_async_commit();
    if (++xplane < n3) xsrc += pstride;
  };

  T win[NCOMBO][W][2];  // trial planes at the lane's pencils
  // q1 contraction of the landed slab, the next one on its way
  auto produce_q1 = [&]() {
    const T* xr = xr0 + xflip / E;
    xflip = L::xhalf - xflip;
    fetch();
    T bv[2][W];
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int k = 0; k < W; ++k)
        if (P::b1_needed(b)) bv[b][k] = b1l[b * W + k];
    // rows past the control range hold stale slab entries; nothing reads them
#pragma unroll
    for (int rb = 0; rb < ROWS; rb += 4) {
      if (rb >= 8 && rb >= C2r) break;
      T v0 = T(0), v1 = T(0);
#pragma unroll
      for (int k = 0; k < W; ++k) {
        const T xv = xr[rb * XR + k];
        if (P::b1_needed(0)) v0 += bv[0][k] * xv;
        if (P::b1_needed(1)) v1 += bv[1][k] * xv;
      }
      if (P::b1_needed(0)) a1w[(b1_slot<P>(0) * ROWS + rb) * F] = v0;
      if (P::b1_needed(1)) a1w[(b1_slot<P>(1) * ROWS + rb) * F] = v1;
    }
  };
  // q2 contraction into the new plane of the window
  auto produce_q2 = [&](T (&nw)[NCOMBO][2]) {
#pragma unroll
    for (int b1 = 0; b1 < 2; ++b1) {
      if (!P::b1_needed(b1)) continue;
      T xw[W][2];
#pragma unroll
      for (int k = 0; k < W; ++k) ld2(a1r + (b1_slot<P>(b1) * ROWS + k) * F, xw[k][0], xw[k][1]);
#pragma unroll
      for (int b2 = 0; b2 < 2; ++b2) {
        const int c = b1 | (b2 << 1);
        if (!P::combo_needed(c)) continue;
        T v0 = T(0), v1 = T(0);
#pragma unroll
        for (int k = 0; k < W; ++k) {
          const T bb = b2l[b2 * W + k];
          v0 += bb * xw[k][0];
          v1 += bb * xw[k][1];
        }
        nw[combo_slot<P>(c)][0] = v0;
        nw[combo_slot<P>(c)][1] = v1;
      }
    }
  };
  auto shift_win = [&](const T (&nw)[NCOMBO][2]) {
#pragma unroll
    for (int c = 0; c < NCOMBO; ++c)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int m = 0; m < W - 1; ++m) win[c][m][i] = win[c][m + 1][i];
        win[c][W - 1][i] = nw[c][i];
      }
  };

  auto produce = [&]() {
    cp_async_wait_all();
    __syncwarp();
    produce_q1();
    __syncwarp();
    T nw[NCOMBO][2];
    produce_q2(nw);
    asm volatile("" ::: "memory");
    shift_win(nw);
  };

  T acc[I][W][2];  // test planes
#pragma unroll
  for (int i = 0; i < I; ++i)
#pragma unroll
    for (int k = 0; k < W; ++k) acc[i][k][0] = acc[i][k][1] = T(0);
  int yleft = n3 - __ldg(a.wtstart[2] + qa);  // planes of y from the oldest one on
  T* ydst = a.y + (int64_t)col * a.N + (int64_t)d2lo * n1 + d1lo + (n3 - yleft) * pstride;
  const int ylane = gq * n1 + 2 * tq;
  // one 8-row block of the q2 contraction
  auto flush_q2 = [&](int mt, double (&ks)[2][2]) {
    ks[0][0] = ks[0][1] = ks[1][0] = ks[1][1] = 0.0;
#pragma unroll
    for (int pr = 0; pr < 4; ++pr) {
      if (!P::tpair_needed(pr)) continue;
#pragma unroll
      for (int kt = 0; kt < 2; ++kt)
        dmma_8x8x4(ks[pr & 1][0], ks[pr & 1][1], f2[((mt * na2<P>() + a2_slot<P>(pr >> 1)) * 2 + kt) * 32 + lane],
                   dnr[pair_slot<P>(pr) * kWarpTile + kt * 4 * F]);
    }
  };
  // one 8-column block of the q1 contraction of a q2 block
  auto flush_q1 = [&](int mt, int nt, const double (&ks)[2][2]) {
    double c0 = 0.0, c1 = 0.0;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      if (!P::a1_needed(g)) continue;
#pragma unroll
      for (int kt = 0; kt < 2; ++kt)
        dmma_8x8x4(c0, c1, ks[g][kt], f1[((nt * ng<P>() + g_slot<P>(g)) * 2 + kt) * 32 + lane]);
    }
    T* yr = ydst + ylane + mt * 8 * n1 + nt * 8;
    const bool in = mt * 8 + gq < D2r;
    if (in && nt * 8 + 2 * tq < D1r) atomicAdd(yr, (T)c0);
    if (in && nt * 8 + 2 * tq + 1 < D1r) atomicAdd(yr + 1, (T)c1);
  };
  // the oldest test plane is final: its entries to shared memory ...
  auto retire_store = [&]() {
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
      *reinterpret_cast<double2*>(dnw + pair_slot<P>(pr) * kWarpTile) =
          make_double2((double)v0, (double)v1);
    }
  };
  // ... contracted over q2, then q1, added into y: the first block, and the
  // others where a control range exceeds eight
  auto flush_first = [&]() {
    double ks[2][2];
    flush_q2(0, ks);
    flush_q1(0, 0, ks);
    if (D1r > 8) flush_q1(0, 1, ks);
  };
  auto flush_second = [&]() {
    if (D2r > 8) {
      double ks[2][2];
      flush_q2(1, ks);
      flush_q1(1, 0, ks);
      if (D1r > 8) flush_q1(1, 1, ks);
    }
  };
  auto shift_acc = [&]() {
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
  auto retire = [&]() {
    __syncwarp();  // the previous plane's fragments are read
    retire_store();
    if (yleft > 0) {
      __syncwarp();
      flush_first();
      flush_second();
    }
    asm volatile("" ::: "memory");
    shift_acc();
  };
  // both windows move (the usual case): the two chains share their barriers and
  // fill each other's latencies
  auto move = [&]() {
    cp_async_wait_all();
    __syncwarp();
    retire_store();
    produce_q1();
    __syncwarp();
    T nw[NCOMBO][2];
    produce_q2(nw);
    if (yleft > 0) {
      flush_first();
      flush_second();
    }
    asm volatile("" ::: "memory");
    shift_win(nw);
    shift_acc();
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
  fetch();
#pragma unroll 1
  for (int k = 0; k < W; ++k) produce();
  int slot = 0;
  uint32_t parity = 0;
#pragma unroll 1
  for (int g = ga; g < gb; ++g) {
    const int enew = __ldg(glist + 1 + min(g + NB + 2, ngrp));
    if (g > ga) {  // the segment's first windows are in place
      const int mv = en[0] & 3;
      if (mv == 3) {
        move();
      } else {
        if (mv & 2) retire();
        if (mv & 1) produce();
      }
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
#pragma unroll 1
  for (int k = 0; k < W; ++k) retire();
  cp_async_wait_all();
}

template <typename T, int W, class P>
__global__ void __launch_bounds__(32, warp_resident(sizeof(T) == 8, P::S, W))
    mfw_kernel(const __grid_constant__ FusedArgs<T> a) {
  mfw_body<T, W, P>(a, blockIdx.x, blockIdx.y);
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
template <typename T, int W, class P>
__global__ void __launch_bounds__(32, warp_resident(sizeof(T) == 8, P::S, W))
    mfw_batch_kernel(const FusedArgs<T>* __restrict__ args, const int32_t* __restrict__ cta0,
                     int npatch, const int64_t* __restrict__ offs, const T* xb, T* yb,
                     const int32_t* __restrict__ skip) {
  __shared__ FusedArgs<T> sa;
  const int p = mfw_batch_args<T>(args, cta0, npatch, offs, xb, yb, skip, sa);
  if (p < 0) return;
  mfw_body<T, W, P>(sa, (int)blockIdx.x - __ldg(cta0 + p), 0);
}

}  // namespace iga
