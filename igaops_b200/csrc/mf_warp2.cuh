// Warp-per-tile form of the fused 2D matrix-free operator: a CTA is one warp, it
// owns 32 quadrature pencils of direction 1 (one per lane) and a segment of
// direction 2, and marches through the same point groups, ring and step rows as
// the 3D kernel (mf_warp.cuh). A trial row is W products per lane with x values
// loaded one row ahead; a final test row goes to shared memory and lane o adds
// its output's weights (tabulated per tile) times the row.
//
// Small problems are what 2D is used for: the time is a chain of latencies, so
// the segments are short (the wave model decides) and nothing waits for another
// warp. Against the CTA-per-tile kernel (128 pencils, two CTA barriers and a band
// lookup per point, segments of 48 points), B200, us a whole call: FP64 stiffness
// p3 64^2 58 -> 13 (launch-bound), p5 301 x 283 67 -> 28, p3 1000^2 176 -> 90,
// FP32 p3 128^2 48 -> 15, FP64 mass p4 320^2 54 -> 19.
#pragma once

#include "mf_warp.cuh"

namespace iga {

constexpr int kWarpFace2 = 32;   // pencils per tile
constexpr int kWarpRing2 = 4;    // groups in the ring
constexpr int kWarpResident2 = 16;

// Shared memory of a CTA (byte offsets); the weight table's depth kw is the
// number of points an output of the tile can read (run time).
template <typename T, class P, int W>
struct WarpSmem2 {
  static constexpr int E = (int)sizeof(T);
  static constexpr int row = warp_row_len<T, P>(W);
  static constexpr int chunk = P::S * kWarpFace2;
  static constexpr int slot = kGroupPts * (chunk + row);
  static constexpr int nout = kWarpFace2 + W - 1;  // outputs of a tile (unit steps)
  static constexpr int ng = (P::a1_needed(0) ? 1 : 0) + (P::a1_needed(1) ? 1 : 0);
  static constexpr int ring = 64;
  // finished rows, with kWarpFace2 zeros before, between and after them
  static constexpr int done = ring + kWarpRing2 * slot * E;
  static constexpr int nrow = 2 * kWarpFace2;
  static constexpr int wtab = done + (kWarpFace2 + ng * nrow) * E;
  __host__ __device__ static int total(int kw) { return wtab + (ng * kw * nout * E + 15) / 16 * 16; }
};

template <typename T, int W, class P>
__global__ void __launch_bounds__(32, kWarpResident2)
    mfw2_kernel(const __grid_constant__ FusedArgs<T> a) {
  using L = WarpSmem2<T, P, W>;
  constexpr int S = P::S, I = P::I, J = P::J, NB = kWarpRing2, E = L::E;
  constexpr int G = step_group<T>(W);
  constexpr int FB = nb1<P>();
  extern __shared__ __align__(128) unsigned char smem[];

  const int lane = threadIdx.x;
  const int n1 = a.n[0], n2 = a.n[1], nq1 = a.nq[0], nq2 = a.nq[1];
  const int unit = blockIdx.x, seg = unit % a.nseg, tile = unit / a.nseg;
  const int q1lo = tile * kWarpFace2, w1 = min(kWarpFace2, nq1 - q1lo);
  const int q1 = q1lo + min(lane, w1 - 1);
  const int kw = min(a.RW, kWarpFace2);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);
  T* ring = reinterpret_cast<T*>(smem + L::ring);
  T* done = reinterpret_cast<T*>(smem + L::done) + kWarpFace2;
  T* wtab = reinterpret_cast<T*>(smem + L::wtab);

  const int* glist = reinterpret_cast<const int*>(reinterpret_cast<const char*>(a.step_table) +
                                                  group_list_offset<T>(nq2, L::row));
  auto entry = [&](int g) { return __shfl_sync(0xffffffffu, __ldg(glist + 1 + g), 0); };
  const int ngrp = __shfl_sync(0xffffffffu, __ldg(glist), 0);
  const int ga = (int)((int64_t)ngrp * seg / a.nseg), gb = (int)((int64_t)ngrp * (seg + 1) / a.nseg);
  if (ga >= gb) return;
  int en[NB + 2];  // entries of the groups g .. g + NB + 1
#pragma unroll
  for (int k = 0; k < NB + 2; ++k) en[k] = entry(min(ga + k, ngrp));
  const int qa = en[0] >> 2;

  const int ntiles = a.tiles1;
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
    csrc += (int64_t)(np * ntiles) * L::chunk;
    rsrc += np * L::row;
  };
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < NB; ++s) mbar_init(smem_u32(&bars[s]), 1);
    fence_mbar_init();
  }
#pragma unroll
  for (int s = 0; s < NB; ++s)
    if (ga + s < gb) issue(s, (en[s + 1] >> 2) - (en[s] >> 2));

  // trial bands of the lane's point; its x values of a control row
  T b1[FB][W];
  const int c1 = __ldg(a.tstart[0] + q1);
  int xo[W];
#pragma unroll
  for (int k = 0; k < W; ++k) {
    if (P::b1_needed(0)) b1[b1_slot<P>(0)][k] = __ldg(a.tB0[0] + (int64_t)q1 * W + k);
    if (P::b1_needed(1)) b1[b1_slot<P>(1)][k] = __ldg(a.tB1[0] + (int64_t)q1 * W + k);
    xo[k] = min(c1 + k, n1 - 1);  // columns beyond the patch only meet zero band values
  }
  int xrow = __ldg(a.tstart[1] + qa);
  const T* x = a.x + (int64_t)blockIdx.y * a.N;
  T xn[W];  // the next row's values
  auto fetch = [&]() {
    const T* xr = x + (int64_t)min(xrow, n2 - 1) * n1;
#pragma unroll
    for (int k = 0; k < W; ++k) xn[k] = __ldg(xr + xo[k]);
    ++xrow;
  };
  T win[FB][W];
  auto produce = [&]() {
    T v[FB];
#pragma unroll
    for (int b = 0; b < FB; ++b) {
      v[b] = T(0);
#pragma unroll
      for (int k = 0; k < W; ++k) v[b] += b1[b][k] * xn[k];
    }
    fetch();
#pragma unroll
    for (int b = 0; b < FB; ++b) {
#pragma unroll
      for (int k = 0; k < W - 1; ++k) win[b][k] = win[b][k + 1];
      win[b][W - 1] = v[b];
    }
  };
  fetch();

  // outputs of the tile: lane o (and o + 32) reads the kw points from l0 on with
  // the tabulated weights: its band, and zeros of `done` where that leaves the tile
  // (not other points with zero weights: an infinity or NaN of theirs is not its own)
  const int d1lo = __ldg(a.wtstart[0] + q1lo);
  const int D1r = min(__ldg(a.wtstart[0] + q1lo + w1 - 1) + W - 1, n1 - 1) - d1lo + 1;
  int l0[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int o = lane + 32 * h;
    l0[h] = 0;
    if (o < D1r) {
      const int rs = __ldg(a.rstart[0] + d1lo + o) - q1lo;
      l0[h] = rs < 0 ? max(min(rs + a.RW - kw, 0), -kWarpFace2) : min(rs, kWarpFace2);
#pragma unroll 1
      for (int k = 0; k < kw; ++k) {
        const int l = l0[h] + k, kk = l - rs;
        const bool in = l >= 0 && l < w1 && kk >= 0 && kk < a.RW;
        const int64_t at = (int64_t)(d1lo + o) * a.RW + kk;
        if (P::a1_needed(0)) wtab[(g_slot<P>(0) * kw + k) * L::nout + o] = in ? __ldg(a.wR0[0] + at) : T(0);
        if (P::a1_needed(1)) wtab[(g_slot<P>(1) * kw + k) * L::nout + o] = in ? __ldg(a.wR1[0] + at) : T(0);
      }
    }
  }
  done[lane - kWarpFace2] = T(0);
#pragma unroll
  for (int g = 0; g < L::ng; ++g) done[g * L::nrow + kWarpFace2 + lane] = T(0);

  T acc[I][W];
#pragma unroll
  for (int i = 0; i < I; ++i)
#pragma unroll
    for (int k = 0; k < W; ++k) acc[i][k] = T(0);
  int yrow = __ldg(a.wtstart[1] + qa);
  T* y = a.y + (int64_t)blockIdx.y * a.N + d1lo;
  auto retire = [&]() {
    __syncwarp();  // the previous row is read
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      if (!P::a1_needed(g)) continue;
      T v = T(0);
#pragma unroll
      for (int i = 0; i < I; ++i)
        if (P::alpha(i, 0) == g) v += acc[i][0];
      done[g_slot<P>(g) * L::nrow + lane] = v;  // padding pencils: zero coefficients
    }
    __syncwarp();
    if (yrow < n2) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int o = lane + 32 * h;
        if (o < D1r) {
          T v[2] = {T(0), T(0)};
          const T* dn = done + l0[h];
          const T* wt = wtab + o;
#pragma unroll 4
          for (int k = 0; k < kw; ++k)
#pragma unroll
            for (int g = 0; g < L::ng; ++g) v[g] += wt[(g * kw + k) * L::nout] * dn[g * L::nrow + k];
          atomicAdd(y + (int64_t)yrow * n1 + o, v[0] + v[1]);
        }
      }
    }
    ++yrow;
#pragma unroll
    for (int i = 0; i < I; ++i) {
#pragma unroll
      for (int k = 0; k < W - 1; ++k) acc[i][k] = acc[i][k + 1];
      acc[i][W - 1] = T(0);
    }
  };
  auto point = [&](const T* cs, const T* row) {
    T u[J];
#pragma unroll
    for (int j = 0; j < J; ++j) {
      T bq[G];
      load_group<T, G>(row + trial_slot<P>(P::beta(j, 1)) * G, bq);
      const T* f = win[b1_slot<P>(P::beta(j, 0))];
      T v0 = bq[0] * f[0], v1 = bq[1] * f[1];
#pragma unroll
      for (int k = 2; k < W; ++k) {
        if (k & 1) v1 += bq[k] * f[k];
        else v0 += bq[k] * f[k];
      }
      u[j] = v0 + v1;
    }
    T cv[S];
#pragma unroll
    for (int s = 0; s < S; ++s) cv[s] = cs[s * kWarpFace2 + lane];
#pragma unroll
    for (int i = 0; i < I; ++i) {
      T g = cv[P::cidx(i, 0)] * u[0];
#pragma unroll
      for (int j = 1; j < J; ++j) g += cv[P::cidx(i, j)] * u[j];
      T wq[G];
      load_group<T, G>(row + test_slot<P>(P::alpha(i, 1)) * G, wq);
#pragma unroll
      for (int k = 0; k < W; ++k) acc[i][k] += wq[k] * g;
    }
  };

  __syncwarp();
#pragma unroll 1
  for (int k = 0; k < W; ++k) produce();
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
    const bool ok = mbar_wait_bounded(smem_u32(bars) + slot * 8, parity);
    if (!__all_sync(0xffffffffu, ok)) {
      if (lane == 0) {
        // the copies still in flight land before the CTA leaves
        for (int o = 1; o < NB && g + o < gb; ++o)
          (void)mbar_wait_bounded(smem_u32(&bars[(slot + o) % NB]),
                                  slot + o >= NB ? parity ^ 1u : parity);
        report_status(a.status, IGA_ERR_TIMEOUT);
      }
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
    if (g + NB < gb) issue(slot, (en[NB + 1] >> 2) - (en[NB] >> 2));
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
}

}  // namespace iga
