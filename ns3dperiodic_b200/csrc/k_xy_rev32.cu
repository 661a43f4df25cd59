// x and y pass instantiations with the reversed radix schedules, FP32 lines
// (FP64: k_xy_rev.cu).
#include "dispatch.h"
#include "k_xy_rev.cuh"

namespace ns3d {

cudaError_t run_inv_x_rev(const InvXArgs<3, float2>& a, const PassGeom& g, cudaStream_t st) {
  return launch_inv_x<3, float2, 1>(a, g, st);
}
cudaError_t run_inv_x_rev(const InvXArgs<6, float2>& a, const PassGeom& g, cudaStream_t st) {
  return launch_inv_x<6, float2, 1>(a, g, st);
}
cudaError_t run_inv_y_rev(const InvYArgs<3, float2>& a, const PassGeom& g, cudaStream_t st) {
  return launch_inv_y<3, float2, 1>(a, g, st);
}
cudaError_t run_inv_y_rev(const InvYArgs<6, float2>& a, const PassGeom& g, cudaStream_t st) {
  return launch_inv_y<6, float2, 1>(a, g, st);
}
cudaError_t run_fwd_y_rev(const FwdYArgs<float2>& a, const PassGeom& g, cudaStream_t st) {
  return launch_fwd_y<float2, 1>(a, g, st);
}

cudaError_t prepare_xy_rev_f32(const PassGeom& g, int tile) {
  return prepare_rev_prec<float2>(g, tile);
}

}  // namespace ns3d
