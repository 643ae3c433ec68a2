// Host entry points of the fused matrix-free operator: layout, packing of the
// reference-layout coefficients, and the matvec launch.
#include <vector>

#include "mf_fused.cuh"
#include "mf_warp.cuh"
#include "mf_warp2.cuh"

namespace iga {

static int pattern_nstream(int ndim, int op, int st, int sym) {
  const int sp = st ? ndim - 1 : ndim;
  switch (op) {
    case IGA_OP_MASS: return 1;
    case IGA_OP_STIFF: return sym ? sp * (sp + 1) / 2 : sp * sp;
    case IGA_OP_GRADU_V:
    case IGA_OP_U_GRADV: return sp;
    default: return -1;
  }
}

static iga_status check_plan(const iga_mf_plan* p) {
  IGA_CHECK_ARG(p, "null plan");
  IGA_CHECK_ARG(p->ndim == 2 || p->ndim == 3, "fused matvec supports ndim 2 or 3, got %d", p->ndim);
  IGA_CHECK_ARG(p->op >= IGA_OP_MASS && p->op <= IGA_OP_U_GRADV, "bad op %d", p->op);
  IGA_CHECK_ARG(p->spacetime == 0 || p->spacetime == 1, "bad spacetime flag");
  IGA_CHECK_ARG(p->time_test == 0 || p->time_test == 1, "time_test must be 0 or 1");
  IGA_CHECK_ARG(p->time_trial == 0 || p->time_trial == 1, "time_trial must be 0 or 1");
  const int S = pattern_nstream(p->ndim, p->op, p->spacetime, p->sym);
  IGA_CHECK_ARG(S == p->nstream && S >= 1 && S <= 9, "nstream %d does not match op (%d)",
                p->nstream, S);
  IGA_CHECK_ARG(p->nseg >= 1, "nseg must be >= 1");
  for (int d = 0; d < p->ndim; ++d) {
    IGA_CHECK_ARG(p->n[d] >= 1 && p->nq[d] >= 1, "empty direction %d", d);
    IGA_CHECK_ARG(p->trial[d].rows == p->nq[d] && p->trial[d].cols == p->n[d],
                  "trial band %d has shape %dx%d, expected %dx%d", d, p->trial[d].rows,
                  p->trial[d].cols, p->nq[d], p->n[d]);
    IGA_CHECK_ARG(p->testT[d].rows == p->nq[d] && p->testT[d].cols == p->n[d],
                  "testT band %d shape mismatch", d);
    IGA_CHECK_ARG(p->testR[d].rows == p->n[d] && p->testR[d].cols == p->nq[d],
                  "testR band %d shape mismatch", d);
    IGA_CHECK_ARG(p->trial[d].width == p->width && p->testT[d].width == p->width,
                  "band widths of direction %d differ from plan width %d", d, p->width);
    IGA_CHECK_ARG(p->testR[d].width == p->rwidth, "testR width mismatch in direction %d", d);
  }
  const int last = p->ndim - 1;
  IGA_CHECK_ARG(p->nseg <= p->nq[last], "nseg %d exceeds nq of the streamed direction", p->nseg);
  IGA_CHECK_ARG(p->face[0] >= 1 && (p->ndim == 2 || p->face[1] >= 1), "bad face");
  return IGA_OK;
}

// The face selects the kernel: 8 x 8 (3D) and 32 (2D) are the warp-per-tile
// kernels, whose chunks hold the whole tile (padding pencils zero).
static bool warp_face(const iga_mf_plan* p) {
  return p->ndim == 3 ? p->face[0] == kWarpFace && p->face[1] == kWarpFace
                      : p->face[0] == kWarpFace2;
}

static int64_t layout_elems(const iga_mf_plan* p, int dtype, int64_t* tile_off) {
  if (warp_face(p)) {
    const bool d3 = p->ndim == 3;
    const int64_t tiles = ceil_div(p->nq[0], p->face[0]) * (d3 ? ceil_div(p->nq[1], kWarpFace) : 1);
    // [group][tile][point][stream][pencil]: a tile has no offset of its own
    if (tile_off)
      for (int64_t t = 0; t < tiles; ++t) tile_off[t] = 0;
    return tiles * p->nq[p->ndim - 1] * p->nstream * (d3 ? kWarpTile : kWarpFace2);
  }
  const int FX = p->face[0];
  const int FY = p->ndim == 3 ? p->face[1] : 1;
  const int tiles1 = (int)ceil_div(p->nq[0], FX);
  const int tiles2 = p->ndim == 3 ? (int)ceil_div(p->nq[1], FY) : 1;
  const int nlast = p->nq[p->ndim - 1];
  int64_t off = 0;
  for (int t2 = 0; t2 < tiles2; ++t2) {
    const int w2 = p->ndim == 3 ? std::min(FY, p->nq[1] - t2 * FY) : 1;
    for (int t1 = 0; t1 < tiles1; ++t1) {
      const int w1 = std::min(FX, p->nq[0] - t1 * FX);
      if (tile_off) tile_off[(int64_t)t2 * tiles1 + t1] = off;
      const int64_t cs = dtype == IGA_F64 ? chunk_stride_elems<double>(p->nstream, w1, w2)
                                          : chunk_stride_elems<float>(p->nstream, w1, w2);
      off += cs * nlast;
    }
  }
  return off;
}

// pack: thread per (stream, q) in reference order
template <typename Tin, typename Tout>
__global__ void __launch_bounds__(256) mf_pack_kernel(int ndim, int nq1, int nq2, int nq3, int FX,
                                                      int FY, int S, int tiles1,
                                                      const int64_t* __restrict__ tile_off,
                                                      SrcRows rows, const Tin* __restrict__ coefs,
                                                      int64_t ld, Tout* __restrict__ packed) {
  const int64_t Nq = (int64_t)nq1 * nq2 * (ndim == 3 ? nq3 : 1);
  const int64_t total = Nq * S;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int s = (int)(idx / Nq);
    const int64_t q = idx - (int64_t)s * Nq;
    const int q1 = (int)(q % nq1);
    const int64_t r = q / nq1;
    const Tout v = (Tout)coefs[(int64_t)rows.r[s] * ld + q];
    const int t1 = q1 / FX, l1 = q1 - t1 * FX;
    const int w1 = min(FX, nq1 - t1 * FX);
    int64_t off;
    if (ndim == 3) {
      const int q2 = (int)(r % nq2);
      const int q3 = (int)(r / nq2);
      const int t2 = q2 / FY, l2 = q2 - t2 * FY;
      const int w2 = min(FY, nq2 - t2 * FY);
      off = tile_off[(int64_t)t2 * tiles1 + t1] + (int64_t)q3 * chunk_stride_elems<Tout>(S, w1, w2) +
            (point_major3(S) ? ((int64_t)l2 * w1 + l1) * S + s
                             : (int64_t)s * w1 * w2 + (int64_t)l2 * w1 + l1);
    } else {
      const int q2 = (int)r;
      off = tile_off[t1] + (int64_t)q2 * chunk_stride_elems<Tout>(S, w1, 1) + (int64_t)s * w1 + l1;
    }
    packed[off] = v;
  }
}

// pack of point-major 3D chunks: one CTA per (face tile, q3) chunk, one
// thread per face point; each thread reads its point's streams (coalesced
// along q1 per stream) and writes them contiguously (the chunk is one
// contiguous run of the packed buffer)
template <typename Tin, typename Tout>
__global__ void __launch_bounds__(256) mf_pack3_pm_kernel(int nq1, int nq2, int FX, int FY, int S,
                                                          int tiles1,
                                                          const int64_t* __restrict__ tile_off,
                                                          SrcRows rows, const Tin* __restrict__ coefs,
                                                          int64_t ld, Tout* __restrict__ packed) {
  const int tile = blockIdx.x, q3 = blockIdx.y;
  const int t1 = tile % tiles1, t2 = tile / tiles1;
  const int w1 = min(FX, nq1 - t1 * FX), w2 = min(FY, nq2 - t2 * FY);
  const int l = threadIdx.x, l1 = l % FX, l2 = l / FX;
  if (l1 >= w1 || l2 >= w2) return;
  const int64_t q = ((int64_t)q3 * nq2 + t2 * FY + l2) * nq1 + t1 * FX + l1;
  Tout* dst = packed + tile_off[tile] + (int64_t)q3 * chunk_stride_elems<Tout>(S, w1, w2) +
              ((int64_t)l2 * w1 + l1) * S;
  for (int s = 0; s < S; ++s) dst[s] = (Tout)coefs[(int64_t)rows.r[s] * ld + q];
}

// pack for the warp-per-tile kernels, [group][tile][point][stream][pencil], tiles
// of F1 x F2 pencils (F2 = 1 in 2D, where nq2 = 1 and q3 counts direction 2): one
// CTA per (row of tiles, q3), both on the x axis of the grid (the others end at 65535);
// a warp walks one row of points (coalesced reads) and writes its pieces into the row's
// tiles (pencil l1 F2 + l2), zeros beyond the grid.
template <typename Tin, typename Tout, int F1, int F2>
__global__ void __launch_bounds__(256)
    mf_pack_warp_kernel(int nq1, int nq2, int nq3, int S, int tiles1, int tiles2,
                        const int32_t* __restrict__ groups, SrcRows rows,
                        const Tin* __restrict__ coefs, int64_t ld, Tout* __restrict__ packed) {
  constexpr int FT = F1 * F2;
  const int q3 = blockIdx.x / tiles2, t2 = blockIdx.x - q3 * tiles2;
  int lo = 0, hi = __ldg(groups);  // the group of q3
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if ((__ldg(groups + 1 + mid) >> 2) <= q3) lo = mid;
    else hi = mid;
  }
  const int qg = __ldg(groups + 1 + lo) >> 2, np = (__ldg(groups + 2 + lo) >> 2) - qg;
  const int64_t chunk = (int64_t)S * FT, tstride = np * chunk;
  Tout* base = packed + ((int64_t)qg * tiles1 * tiles2 + (int64_t)t2 * tiles1 * np + (q3 - qg)) * chunk;
  for (int row = threadIdx.x >> 5; row < S * F2; row += 8) {
    const int s = row / F2, l2 = row % F2;
    const int q2 = t2 * F2 + l2;
    const Tin* src = coefs + (int64_t)rows.r[s] * ld + ((int64_t)q3 * nq2 + q2) * nq1;
    Tout* dst = base + s * FT + l2;
    for (int q1 = threadIdx.x & 31; q1 < tiles1 * F1; q1 += 32)
      dst[(q1 / F1) * tstride + q1 % F1 * F2] = (q1 < nq1 && q2 < nq2) ? (Tout)src[q1] : Tout(0);
  }
}

// step rows of the warp-per-tile kernel: the pattern's value groups (src)
template <typename T>
struct RowSrc {
  const T* p[4];
  int n;
};
template <typename T>
__global__ void mf_table_warp_kernel(int nq, int W, RowSrc<T> src, T* __restrict__ table) {
  const int G = step_group<T>(W), rlen = src.n * G;
  const int64_t total = (int64_t)nq * rlen;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int q = (int)(idx / rlen), j = (int)(idx - (int64_t)q * rlen);
    const int grp = j / G, k = j - grp * G;
    table[idx] = k < W ? src.p[grp][(int64_t)q * W + k] : T(0);
  }
}

// group list behind the step rows (see group_list_offset): runs of points
// between window moves, cut into pieces of at most kGroupPts points of nearly
// equal size; one CTA, thread q0 + t decides for point q whether a group starts
// there, a running prefix sum numbers them
__global__ void __launch_bounds__(256) mf_groups_kernel(int nq, const int32_t* __restrict__ ts,
                                                        const int32_t* __restrict__ ws,
                                                        int32_t* __restrict__ list) {
  __shared__ int s_cnt[256];
  auto moves = [&](int q) {
    return q <= 0 ? 0 : (ts[q] != ts[q - 1] ? 1 : 0) | (ws[q] != ws[q - 1] ? 2 : 0);
  };
  int base = 0;
  for (int q0 = 0; q0 < nq; q0 += 256) {
    const int q = q0 + threadIdx.x;
    bool start = false;
    if (q < nq) {
      int lo = q, hi = q + 1;  // the run [lo, hi) of q
      while (lo > 0 && !moves(lo)) --lo;
      while (hi < nq && !moves(hi)) ++hi;
      const int len = hi - lo, np = (len + kGroupPts - 1) / kGroupPts;
      for (int k = 0; k < np; ++k) start |= q == lo + (int)((int64_t)len * k / np);
    }
    s_cnt[threadIdx.x] = start;
    __syncthreads();
    int rank = 0, total = 0;
    for (int t = 0; t < 256; ++t) {
      rank += t < (int)threadIdx.x ? s_cnt[t] : 0;
      total += s_cnt[t];
    }
    if (start) list[1 + base + rank] = q << 2 | moves(q);
    base += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    list[0] = base;
    list[1 + base] = nq << 2;
  }
}

// derivative orders of the streamed direction that an operator reads: bit 0 /
// bit 1 = order 0 / 1 of the trial bands, bit 2 / 3 of the test bands
static int last_orders(const iga_mf_plan* p) {
  if (p->spacetime) return (1 << p->time_trial) | (4 << p->time_test);
  const bool tg = p->op == IGA_OP_STIFF || p->op == IGA_OP_U_GRADV;
  const bool wg = p->op == IGA_OP_STIFF || p->op == IGA_OP_GRADU_V;
  return (tg ? 3 : 1) | (wg ? 12 : 4);
}

// byte offset of the group list in the step table
static int64_t group_list_bytes(const iga_mf_plan* p, int dtype) {
  const int o = last_orders(p), n = (o & 1) + (o >> 1 & 1) + (o >> 2 & 1) + (o >> 3);
  const int nq = p->nq[p->ndim - 1];
  return dtype == IGA_F64 ? group_list_offset<double>(nq, n * step_group<double>(p->width))
                          : group_list_offset<float>(nq, n * step_group<float>(p->width));
}

template <typename T>
static iga_status table_warp(const iga_mf_plan* p, int64_t* elems, void* table, cudaStream_t st) {
  const int o = last_orders(p), last = p->ndim - 1;
  RowSrc<T> src;
  src.n = 0;
  if (o & 1) src.p[src.n++] = (const T*)p->trial[last].vals;
  if (o & 2) src.p[src.n++] = (const T*)p->trial_d1[last];
  if (o & 4) src.p[src.n++] = (const T*)p->testT[last].vals;
  if (o & 8) src.p[src.n++] = (const T*)p->testT_d1[last];
  const int rlen = src.n * step_group<T>(p->width), nq = p->nq[last];
  const int64_t off = group_list_offset<T>(nq, rlen);
  // at most one group per point, the count and the end mark
  *elems = (off + 4 * ((int64_t)nq + 2) + (int64_t)sizeof(T) - 1) / (int64_t)sizeof(T);
  if (!table) return IGA_OK;
  for (int i = 0; i < src.n; ++i) IGA_CHECK_ARG(src.p[i], "band values missing");
  IGA_CHECK_ARG(p->trial[last].start && p->testT[last].start, "band starts missing");
  const unsigned g = (unsigned)std::min<int64_t>(ceil_div((int64_t)nq * rlen, 256), 148 * 8);
  mf_table_warp_kernel<T><<<g, 256, 0, st>>>(nq, p->width, src, (T*)table);
  mf_groups_kernel<<<1, 256, 0, st>>>(nq, p->trial[last].start, p->testT[last].start,
                                      (int32_t*)((char*)table + off));
  IGA_LAUNCH_CHECK();
  return IGA_OK;
}

// step table rows of the last direction: B0, B1, W0T, W1T (W each), starts
template <typename T>
__global__ void mf_table_kernel(int nq, int W, int rlen, const int32_t* __restrict__ ts,
                                const T* __restrict__ b0, const T* __restrict__ b1,
                                const int32_t* __restrict__ ws, const T* __restrict__ w0,
                                const T* __restrict__ w1, T* __restrict__ table) {
  const int64_t total = (int64_t)nq * rlen;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int q = (int)(idx / rlen), j = (int)(idx - (int64_t)q * rlen);
    const int G = step_group<T>(W);
    const int grp = j / G, k = j - grp * G;
    T v = T(0);
    if (grp < 4) {
      if (k < W) {
        const T* src = grp == 0 ? b0 : grp == 1 ? b1 : grp == 2 ? w0 : w1;
        v = src[(int64_t)q * W + k];
      }
    } else if (j == 4 * G) {
      v = step_start_enc(ts[q], T(0));
    } else if (j == 4 * G + 1) {
      v = step_start_enc(ws[q], T(0));
    }
    table[idx] = v;
  }
}

template <typename T>
static void fill_args(FusedArgs<T>& a, const iga_mf_plan* p, const void* packed, const void* x,
                      void* y) {
  for (int d = 0; d < 3; ++d) {
    a.n[d] = d < p->ndim ? p->n[d] : 1;
    a.nq[d] = d < p->ndim ? p->nq[d] : 1;
    a.tstart[d] = d < p->ndim ? p->trial[d].start : nullptr;
    a.tB0[d] = d < p->ndim ? (const T*)p->trial[d].vals : nullptr;
    a.tB1[d] = d < p->ndim ? (const T*)p->trial_d1[d] : nullptr;
    a.wtstart[d] = d < p->ndim ? p->testT[d].start : nullptr;
    a.wT0[d] = d < p->ndim ? (const T*)p->testT[d].vals : nullptr;
    a.wT1[d] = d < p->ndim ? (const T*)p->testT_d1[d] : nullptr;
    a.rstart[d] = d < p->ndim ? p->testR[d].start : nullptr;
    a.wR0[d] = d < p->ndim ? (const T*)p->testR[d].vals : nullptr;
    a.wR1[d] = d < p->ndim ? (const T*)p->testR_d1[d] : nullptr;
  }
  a.W = p->width;
  a.RW = p->rwidth;
  a.tiles1 = (int)ceil_div(p->nq[0], p->face[0]);
  a.tiles2 = p->ndim == 3 ? (int)ceil_div(p->nq[1], p->face[1]) : 1;
  a.nseg = p->nseg;
  a.cmax1 = p->cmax[0];
  a.cmax2 = p->cmax[1];
  a.dmax1 = p->dmax[0];
  a.dmax2 = p->dmax[1];
  int64_t N = 1;
  for (int d = 0; d < p->ndim; ++d) N *= p->n[d];
  a.N = N;
  a.tile_off = p->tile_off;
  a.step_table = (const T*)p->step_table;
  a.rlen = step_row_len<T>(p->width);
  a.packed = (const T*)packed;
  a.x = (const T*)x;
  a.y = (T*)y;
  a.status = p->status;
  a.wait_test = p->wait_test;
}

template <typename T>
static iga_status launch_dispatch(const FusedArgs<T>& a, const LaunchInfo& li);

template <>
iga_status launch_dispatch<double>(const FusedArgs<double>& a, const LaunchInfo& li) {
#define IGA_W_CASES(D)                                  \
  switch (li.W) {                                       \
    case 3: return launch_mf##D##_f64_w3(a, li);        \
    case 4: return launch_mf##D##_f64_w4(a, li);        \
    case 5: return launch_mf##D##_f64_w5(a, li);        \
    case 6: return launch_mf##D##_f64_w6(a, li);        \
    default: break;                                     \
  }
  if (li.ndim == 3) { IGA_W_CASES(3) } else { IGA_W_CASES(2) }
#undef IGA_W_CASES
  set_error("no fused kernel for band width %d", li.W);
  return IGA_ERR_UNSUPPORTED;
}

template <>
iga_status launch_dispatch<float>(const FusedArgs<float>& a, const LaunchInfo& li) {
#define IGA_W_CASES(D)                                  \
  switch (li.W) {                                       \
    case 3: return launch_mf##D##_f32_w3(a, li);        \
    case 4: return launch_mf##D##_f32_w4(a, li);        \
    case 5: return launch_mf##D##_f32_w5(a, li);        \
    case 6: return launch_mf##D##_f32_w6(a, li);        \
    default: break;                                     \
  }
  if (li.ndim == 3) { IGA_W_CASES(3) } else { IGA_W_CASES(2) }
#undef IGA_W_CASES
  set_error("no fused kernel for band width %d", li.W);
  return IGA_ERR_UNSUPPORTED;
}

static LaunchInfo launch_info(const iga_mf_plan* p, int64_t ncols, cudaStream_t st) {
  LaunchInfo li;
  li.ndim = p->ndim;
  li.op = p->op;
  li.st = p->spacetime;
  li.tt = p->time_test;
  li.tr = p->time_trial;
  li.sym = p->sym;
  li.W = p->width;
  li.FX = p->face[0];
  li.FY = p->ndim == 3 ? p->face[1] : 1;
  li.NST = kStages;
  li.ncols = ncols;
  li.stream = st;
  li.resident = nullptr;
  return li;
}

// shared memory of the multi-patch kernel for one patch of a pattern
template <typename T>
static size_t batch_smem(const iga_mf_plan* p, int rlen) {
  const int W = p->width, RW = p->rwidth;
  auto f = [&](auto pat) -> size_t {
    using P = decltype(pat);
    if (warp_face(p)) {
      const bool wide = std::max({p->cmax[0], p->cmax[1], p->dmax[0], p->dmax[1]}) > kWarpFace;
      switch (W) {
        case 3: return wide ? WarpSmem<T, P, 3, true>::total : WarpSmem<T, P, 3, false>::total;
        case 4: return wide ? WarpSmem<T, P, 4, true>::total : WarpSmem<T, P, 4, false>::total;
        case 5: return wide ? WarpSmem<T, P, 5, true>::total : WarpSmem<T, P, 5, false>::total;
        default: return wide ? WarpSmem<T, P, 6, true>::total : WarpSmem<T, P, 6, false>::total;
      }
    }
    return mf3d_smem_bytes<T, P>(kFace3X, kFace3Y, W, RW, rlen, p->cmax[0], p->cmax[1],
                                 p->dmax[0], p->dmax[1]);
  };
  switch (p->op) {
    case IGA_OP_MASS: return f(Pat<3, IGA_OP_MASS, 0, 0, 0, 0>{});
    case IGA_OP_STIFF:
      return p->sym ? f(Pat<3, IGA_OP_STIFF, 0, 0, 0, 1>{}) : f(Pat<3, IGA_OP_STIFF, 0, 0, 0, 0>{});
    case IGA_OP_GRADU_V: return f(Pat<3, IGA_OP_GRADU_V, 0, 0, 0, 0>{});
    default: return f(Pat<3, IGA_OP_U_GRADV, 0, 0, 0, 0>{});
  }
}

static inline int64_t align256(int64_t b) { return (b + 255) / 256 * 256; }

template <typename T>
static int64_t batch_table_bytes(int npatch) {
  return align256((int64_t)npatch * sizeof(FusedArgs<T>)) + align256((int64_t)(npatch + 1) * 4) +
         (int64_t)npatch * 8;
}

template <typename T>
static iga_status batch_prepare(const iga_mf_plan* plans, int npatch, const void* const* packed,
                                const int64_t* offsets, void* table, int32_t* total_ctas,
                                int64_t* smem_bytes) {
  std::vector<FusedArgs<T>> args((size_t)npatch);
  std::vector<int32_t> cta0((size_t)npatch + 1);
  std::vector<int64_t> offs((size_t)npatch);
  int64_t total = 0;
  size_t smem = 0;
  const iga_mf_plan& p0 = plans[0];
  for (int i = 0; i < npatch; ++i) {
    const iga_mf_plan* p = plans + i;
    iga_status rc = check_plan(p);
    if (rc) return rc;
    IGA_CHECK_ARG(p->ndim == 3 && !p->spacetime, "patch %d: multi-patch matvec covers 3D space operators", i);
    IGA_CHECK_ARG(p->op == p0.op && p->sym == p0.sym &&
                      (p->width == p0.width || (warp_face(p) && p->op == IGA_OP_STIFF)) &&
                      p->face[0] == p0.face[0] && p->face[1] == p0.face[1] &&
                      (warp_face(p) || (p->face[0] == kFace3X && p->face[1] == kFace3Y)),
                  "patch %d: operator, symmetry, face and (but for stiffness with face (8, 8)) band "
                  "width must match patch 0",
                  i);
    const int range = p->width + kWarpFace - 1;
    IGA_CHECK_ARG(!warp_face(p) || std::max({p->cmax[0], p->cmax[1], p->dmax[0], p->dmax[1]}) <= range,
                  "patch %d: control ranges of a tile exceed %d", i, range);
    IGA_CHECK_ARG(packed[i] && ((uintptr_t)packed[i] & 15) == 0 && p->step_table,
                  "patch %d: packed coefficients (16-byte aligned) and step table required", i);
    fill_args<T>(args[i], p, packed[i], nullptr, nullptr);
    IGA_CHECK_ARG(offsets[i] >= 0, "patch %d: negative offset", i);
    offs[i] = offsets[i];
    cta0[i] = (int32_t)total;
    total += (int64_t)args[i].tiles1 * args[i].tiles2 * args[i].nseg;
    smem = std::max(smem, batch_smem<T>(p, args[i].rlen));
  }
  IGA_CHECK_ARG(total < (1ll << 31), "too many CTAs (%lld)", (long long)total);
  cta0[npatch] = (int32_t)total;
  char* t = (char*)table;
  const int64_t a_bytes = align256((int64_t)npatch * sizeof(FusedArgs<T>));
  const int64_t c_bytes = align256((int64_t)(npatch + 1) * 4);
  IGA_CUDA_TRY(cudaMemcpy(t, args.data(), npatch * sizeof(FusedArgs<T>), cudaMemcpyHostToDevice));
  IGA_CUDA_TRY(cudaMemcpy(t + a_bytes, cta0.data(), (npatch + 1) * 4, cudaMemcpyHostToDevice));
  IGA_CUDA_TRY(cudaMemcpy(t + a_bytes + c_bytes, offs.data(), npatch * 8, cudaMemcpyHostToDevice));
  *total_ctas = (int32_t)total;
  *smem_bytes = (int64_t)smem;
  return IGA_OK;
}

template <typename T>
static iga_status batch_dispatch(const BatchLaunch& b, const T* x, T* y);

template <>
iga_status batch_dispatch<double>(const BatchLaunch& b, const double* x, double* y) {
  if (b.W == 0) return launch_mf3_multi(b, x, y);
  switch (b.W) {
    case 3: return launch_mf3_batch_f64_w3(b, x, y);
    case 4: return launch_mf3_batch_f64_w4(b, x, y);
    case 5: return launch_mf3_batch_f64_w5(b, x, y);
    case 6: return launch_mf3_batch_f64_w6(b, x, y);
    default: break;
  }
  set_error("no multi-patch kernel for band width %d", b.W);
  return IGA_ERR_UNSUPPORTED;
}

template <>
iga_status batch_dispatch<float>(const BatchLaunch& b, const float* x, float* y) {
  if (b.W == 0) return launch_mf3_multi(b, x, y);
  switch (b.W) {
    case 3: return launch_mf3_batch_f32_w3(b, x, y);
    case 4: return launch_mf3_batch_f32_w4(b, x, y);
    case 5: return launch_mf3_batch_f32_w5(b, x, y);
    case 6: return launch_mf3_batch_f32_w6(b, x, y);
    default: break;
  }
  set_error("no multi-patch kernel for band width %d", b.W);
  return IGA_ERR_UNSUPPORTED;
}

}  // namespace iga

using namespace iga;

extern "C" {

iga_status iga_mf_batch_table_bytes(int dtype, int npatch, int64_t* bytes) {
  clear_error();
  IGA_CHECK_ARG(npatch >= 1 && bytes, "bad argument");
  if (dtype == IGA_F64) *bytes = batch_table_bytes<double>(npatch);
  else if (dtype == IGA_F32) *bytes = batch_table_bytes<float>(npatch);
  else {
    set_error("dtype %d not supported", dtype);
    return IGA_ERR_UNSUPPORTED;
  }
  return IGA_OK;
}

iga_status iga_mf_batch_prepare(const iga_mf_plan* plans, int npatch, int dtype,
                                const void* const* packed, const int64_t* offsets, void* table,
                                int32_t* total_ctas, int64_t* smem_bytes) {
  clear_error();
  IGA_CHECK_ARG(plans && npatch >= 1 && packed && offsets && table && total_ctas && smem_bytes,
                "null argument");
  IGA_CHECK_ARG(((uintptr_t)table & 255) == 0, "table must be 256-byte aligned");
  for (int i = 0; i < npatch; ++i)
    IGA_CHECK_ARG(plans[i].width >= 3 && plans[i].width <= 6, "band width %d", plans[i].width);
  if (dtype == IGA_F64)
    return batch_prepare<double>(plans, npatch, packed, offsets, table, total_ctas, smem_bytes);
  if (dtype == IGA_F32)
    return batch_prepare<float>(plans, npatch, packed, offsets, table, total_ctas, smem_bytes);
  set_error("dtype %d not supported", dtype);
  return IGA_ERR_UNSUPPORTED;
}

iga_status iga_mf_batch_matvec(const iga_mf_plan* plan0, int dtype, int npatch, const void* table,
                               int32_t total_ctas, int64_t smem_bytes, const void* x, void* y,
                               int64_t ntot, int zero_y, const int32_t* skip,
                               iga_stream stream) {
  clear_error();
  IGA_CHECK_ARG(plan0 && table && x && y && npatch >= 1 && total_ctas >= 1 && ntot >= 0,
                "bad argument");
  cudaStream_t st = as_stream(stream);
  const size_t esz = dtype == IGA_F64 ? 8 : 4;
  if (zero_y) IGA_CUDA_TRY(cudaMemsetAsync(y, 0, (size_t)ntot * esz, st));
  BatchLaunch b;
  b.op = plan0->op;
  b.sym = plan0->sym;
  b.W = plan0->width;
  b.warp = warp_face(plan0);
  IGA_CHECK_ARG(b.W != 0 || (b.warp && b.op == IGA_OP_STIFF && plan0->nstream > 3),
                "mixed band widths need the stiffness operator with face (8, 8)");
  b.npatch = npatch;
  b.total_ctas = total_ctas;
  b.smem = (size_t)smem_bytes;
  const char* t = (const char*)table;
  const int64_t a_bytes =
      align256((int64_t)npatch * (dtype == IGA_F64 ? sizeof(FusedArgs<double>) : sizeof(FusedArgs<float>)));
  const int64_t c_bytes = align256((int64_t)(npatch + 1) * 4);
  b.args = t;
  b.cta0 = (const int32_t*)(t + a_bytes);
  b.offs = (const int64_t*)(t + a_bytes + c_bytes);
  b.skip = skip;
  b.stream = st;
  if (dtype == IGA_F64) return batch_dispatch<double>(b, (const double*)x, (double*)y);
  if (dtype == IGA_F32) return batch_dispatch<float>(b, (const float*)x, (float*)y);
  set_error("dtype %d not supported", dtype);
  return IGA_ERR_UNSUPPORTED;
}

iga_status iga_mf_resident(const iga_mf_plan* plan, int dtype, int32_t* ctas) {
  clear_error();
  iga_status rc = check_plan(plan);
  if (rc) return rc;
  IGA_CHECK_ARG(dtype == IGA_F64 || dtype == IGA_F32, "dtype %d not supported", dtype);
  IGA_CHECK_ARG(ctas, "null ctas");
  *ctas = 0;
  if (!warp_face(plan)) return IGA_OK;
  LaunchInfo li = launch_info(plan, 1, nullptr);
  int n = 0;
  li.resident = &n;
  if (dtype == IGA_F64) {
    FusedArgs<double> a;
    fill_args<double>(a, plan, nullptr, nullptr, nullptr);
    rc = launch_dispatch<double>(a, li);
  } else {
    FusedArgs<float> a;
    fill_args<float>(a, plan, nullptr, nullptr, nullptr);
    rc = launch_dispatch<float>(a, li);
  }
  if (rc) return rc;
  *ctas = n;
  return IGA_OK;
}

iga_status iga_mf_layout(const iga_mf_plan* plan, int dtype, int64_t* elems,
                         int64_t* tile_off_host) {
  clear_error();
  iga_status rc = check_plan(plan);
  if (rc) return rc;
  IGA_CHECK_ARG(dtype == IGA_F64 || dtype == IGA_F32, "dtype %d not supported", dtype);
  IGA_CHECK_ARG(elems, "null elems");
  *elems = layout_elems(plan, dtype, tile_off_host);
  return IGA_OK;
}

iga_status iga_mf_table(const iga_mf_plan* plan, int dtype, int64_t* elems, void* table,
                        iga_stream stream) {
  clear_error();
  iga_status rc = check_plan(plan);
  if (rc) return rc;
  IGA_CHECK_ARG(elems, "null elems");
  IGA_CHECK_ARG(dtype == IGA_F64 || dtype == IGA_F32, "dtype %d not supported", dtype);
  if (warp_face(plan))
    return dtype == IGA_F64 ? table_warp<double>(plan, elems, table, as_stream(stream))
                            : table_warp<float>(plan, elems, table, as_stream(stream));
  const int last = plan->ndim - 1;
  const int W = plan->width;
  const int nq = plan->nq[last];
  const int rlen = dtype == IGA_F64 ? step_row_len<double>(W) : step_row_len<float>(W);
  *elems = (int64_t)nq * rlen;
  if (!table) return IGA_OK;
  const iga_band& tb = plan->trial[last];
  const iga_band& wb = plan->testT[last];
  IGA_CHECK_ARG(tb.start && tb.vals && plan->trial_d1[last] && wb.start && wb.vals &&
                    plan->testT_d1[last],
                "band arrays of the last direction missing");
  const unsigned g = (unsigned)std::min<int64_t>(ceil_div(*elems, 256), 148 * 8);
  cudaStream_t st = as_stream(stream);
  if (dtype == IGA_F64)
    mf_table_kernel<double><<<g, 256, 0, st>>>(
        nq, W, rlen, tb.start, (const double*)tb.vals, (const double*)plan->trial_d1[last],
        wb.start, (const double*)wb.vals, (const double*)plan->testT_d1[last], (double*)table);
  else
    mf_table_kernel<float><<<g, 256, 0, st>>>(
        nq, W, rlen, tb.start, (const float*)tb.vals, (const float*)plan->trial_d1[last],
        wb.start, (const float*)wb.vals, (const float*)plan->testT_d1[last], (float*)table);
  IGA_LAUNCH_CHECK();
  return IGA_OK;
}

iga_status iga_mf_pack(const iga_mf_plan* plan, int dtype_in, const void* coefs, int64_t ld,
                       int dtype_out, void* packed, iga_stream stream) {
  clear_error();
  iga_status rc = check_plan(plan);
  if (rc) return rc;
  IGA_CHECK_ARG(coefs && packed && plan->tile_off, "null pointer");
  IGA_CHECK_ARG(dtype_in == IGA_F64 || dtype_in == IGA_F32, "dtype_in %d", dtype_in);
  IGA_CHECK_ARG(dtype_out == IGA_F64 || dtype_out == IGA_F32, "dtype_out %d", dtype_out);
  const int S = plan->nstream;
  SrcRows rows;
  for (int s = 0; s < 9; ++s) {
    rows.r[s] = plan->src_row[s];
    if (s < S) IGA_CHECK_ARG(rows.r[s] >= 0, "src_row[%d] negative", s);
  }
  cudaStream_t st = as_stream(stream);
  const int64_t elems = layout_elems(plan, dtype_out, nullptr);
  const size_t esz = dtype_out == IGA_F64 ? 8 : 4;
  int64_t Nq = 1;
  for (int d = 0; d < plan->ndim; ++d) Nq *= plan->nq[d];
  IGA_CHECK_ARG(ld >= Nq, "ld %lld smaller than Nq %lld", (long long)ld, (long long)Nq);
  if (warp_face(plan)) {
    const bool d3 = plan->ndim == 3;
    const int nq2 = d3 ? plan->nq[1] : 1, nq3 = plan->nq[plan->ndim - 1];
    const int tiles1 = (int)ceil_div(plan->nq[0], plan->face[0]);
    const int tiles2 = d3 ? (int)ceil_div(nq2, kWarpFace) : 1;
    const int64_t ctas = (int64_t)tiles2 * nq3;
    IGA_CHECK_ARG(ctas < (1ll << 31), "%lld rows of tiles exceed the grid", (long long)ctas);
    IGA_CHECK_ARG(plan->step_table, "this face packs by the step table's groups (iga_mf_table)");
    const dim3 grid((unsigned)ctas);
    const int32_t* groups =
        (const int32_t*)((const char*)plan->step_table + group_list_bytes(plan, dtype_out));
#define IGA_PACK(TI, TO)                                                                         \
  do {                                                                                           \
    if (d3)                                                                                      \
      mf_pack_warp_kernel<TI, TO, kWarpFace, kWarpFace>                                          \
          <<<grid, 256, 0, st>>>(plan->nq[0], nq2, nq3, S, tiles1, tiles2, groups, rows,         \
                                 (const TI*)coefs, ld, (TO*)packed);                             \
    else                                                                                         \
      mf_pack_warp_kernel<TI, TO, kWarpFace2, 1>                                                 \
          <<<grid, 256, 0, st>>>(plan->nq[0], nq2, nq3, S, tiles1, tiles2, groups, rows,         \
                                 (const TI*)coefs, ld, (TO*)packed);                             \
  } while (0)
    if (dtype_in == IGA_F64 && dtype_out == IGA_F64) IGA_PACK(double, double);
    else if (dtype_in == IGA_F64 && dtype_out == IGA_F32) IGA_PACK(double, float);
    else if (dtype_in == IGA_F32 && dtype_out == IGA_F64) IGA_PACK(float, double);
    else IGA_PACK(float, float);
#undef IGA_PACK
    IGA_LAUNCH_CHECK();
    return IGA_OK;
  }
  IGA_CUDA_TRY(cudaMemsetAsync(packed, 0, (size_t)elems * esz, st));
  int64_t blocks = ceil_div(Nq * S, 256);
  if (blocks > 148 * 64) blocks = 148 * 64;
  const int nq3 = plan->ndim == 3 ? plan->nq[2] : 1;
  const int FY = plan->ndim == 3 ? plan->face[1] : 1;
  const int tiles1 = (int)ceil_div(plan->nq[0], plan->face[0]);
  const bool pm3 = plan->ndim == 3 && point_major3(S) && plan->face[0] * FY <= 256;
  const int tiles2 = plan->ndim == 3 ? (int)ceil_div(plan->nq[1], FY) : 1;
  IGA_CHECK_ARG(!pm3 || nq3 <= 65535, "streamed direction of %d points exceeds the grid", nq3);
#define IGA_PACK(TI, TO)                                                                      \
  do {                                                                                        \
    if (pm3)                                                                                  \
      mf_pack3_pm_kernel<TI, TO><<<dim3((unsigned)(tiles1 * tiles2), (unsigned)nq3),         \
                                   (unsigned)(plan->face[0] * FY), 0, st>>>(                  \
          plan->nq[0], plan->nq[1], plan->face[0], FY, S, tiles1, plan->tile_off, rows,       \
          (const TI*)coefs, ld, (TO*)packed);                                                 \
    else                                                                                      \
      mf_pack_kernel<TI, TO><<<(unsigned)blocks, 256, 0, st>>>(                               \
          plan->ndim, plan->nq[0], plan->nq[1], nq3, plan->face[0], FY, S, tiles1,            \
          plan->tile_off, rows, (const TI*)coefs, ld, (TO*)packed);                           \
  } while (0)
  if (dtype_in == IGA_F64 && dtype_out == IGA_F64) IGA_PACK(double, double);
  else if (dtype_in == IGA_F64 && dtype_out == IGA_F32) IGA_PACK(double, float);
  else if (dtype_in == IGA_F32 && dtype_out == IGA_F64) IGA_PACK(float, double);
  else IGA_PACK(float, float);
#undef IGA_PACK
  IGA_LAUNCH_CHECK();
  return IGA_OK;
}

iga_status iga_mf_matvec(const iga_mf_plan* plan, int dtype, const void* packed, int64_t ncols,
                         const void* x, void* y, iga_stream stream) {
  clear_error();
  iga_status rc = check_plan(plan);
  if (rc) return rc;
  IGA_CHECK_ARG(packed && x && y && plan->tile_off, "null pointer");
  IGA_CHECK_ARG(ncols >= 1 && ncols <= 65535, "ncols %lld out of range", (long long)ncols);
  IGA_CHECK_ARG(((uintptr_t)packed & 15) == 0, "packed coefficients must be 16-byte aligned");
  IGA_CHECK_ARG(plan->width >= 3 && plan->width <= 6,
                "fused matvec supports band width 3..6 (degree 2..5), got %d", plan->width);
  cudaStream_t st = as_stream(stream);
  int64_t N = 1;
  for (int d = 0; d < plan->ndim; ++d) N *= plan->n[d];
  const size_t esz = dtype == IGA_F64 ? 8 : 4;
  IGA_CUDA_TRY(cudaMemsetAsync(y, 0, (size_t)N * ncols * esz, st));
  const LaunchInfo li = launch_info(plan, ncols, st);
  if (dtype == IGA_F64) {
    FusedArgs<double> a;
    fill_args<double>(a, plan, packed, x, y);
    return launch_dispatch<double>(a, li);
  }
  if (dtype == IGA_F32) {
    FusedArgs<float> a;
    fill_args<float>(a, plan, packed, x, y);
    return launch_dispatch<float>(a, li);
  }
  set_error("dtype %d not supported by iga_mf_matvec", dtype);
  return IGA_ERR_UNSUPPORTED;
}

}  // extern "C"
