// Stiffness product of many 3D patches of any band widths in one launch: patch p
// owns CTAs [cta0[p], cta0[p+1]) and its width picks the body. One launch per
// width, one after the other, left the SMs idle at the end of each: six mixed
// patches (p 2 .. 4, 20 .. 50 elements) 156 us per product in three launches,
// 117 in this one; 111 with the segment starts of mf_warp.cuh since.
#include "mf_fused.cuh"
#include "mf_warp.cuh"

namespace iga {

template <typename T, class P>
__global__ void __launch_bounds__(32, warp_resident(sizeof(T) == 8, P::S, 6))
    mfw_multi_kernel(const FusedArgs<T>* __restrict__ args, const int32_t* __restrict__ cta0,
                     int npatch, const int64_t* __restrict__ offs, const T* xb, T* yb,
                     const int32_t* __restrict__ skip) {
  __shared__ FusedArgs<T> sa;
  const int p = mfw_batch_args<T>(args, cta0, npatch, offs, xb, yb, skip, sa);
  if (p < 0) return;
  const int unit = (int)blockIdx.x - __ldg(cta0 + p);
  const bool wide = max(max(sa.cmax1, sa.cmax2), max(sa.dmax1, sa.dmax2)) > kWarpFace;
  switch (2 * sa.W + wide) {
    case 6: mfw_body<T, 3, P, false>(sa, unit, 0); break;
    case 7: mfw_body<T, 3, P, true>(sa, unit, 0); break;
    case 8: mfw_body<T, 4, P, false>(sa, unit, 0); break;
    case 9: mfw_body<T, 4, P, true>(sa, unit, 0); break;
    case 10: mfw_body<T, 5, P, false>(sa, unit, 0); break;
    case 11: mfw_body<T, 5, P, true>(sa, unit, 0); break;
    case 12: mfw_body<T, 6, P, false>(sa, unit, 0); break;
    default: mfw_body<T, 6, P, true>(sa, unit, 0);
  }
}

template <typename T, int SYM>
static iga_status launch(const BatchLaunch& b, const T* x, T* y) {
  using P = Pat<3, IGA_OP_STIFF, 0, 0, 0, SYM>;
  mfw_multi_kernel<T, P><<<(unsigned)b.total_ctas, 32, b.smem, b.stream>>>(
      (const FusedArgs<T>*)b.args, b.cta0, b.npatch, b.offs, x, y, b.skip);
  IGA_LAUNCH_CHECK();
  return IGA_OK;
}

iga_status launch_mf3_multi(const BatchLaunch& b, const double* x, double* y) {
  return b.sym ? launch<double, 1>(b, x, y) : launch<double, 0>(b, x, y);
}
iga_status launch_mf3_multi(const BatchLaunch& b, const float* x, float* y) {
  return b.sym ? launch<float, 1>(b, x, y) : launch<float, 0>(b, x, y);
}

}  // namespace iga
