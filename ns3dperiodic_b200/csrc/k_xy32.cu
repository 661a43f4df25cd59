// x and y pass instantiations, FP32 lines of the precision mode (FP64: k_xy.cu).
#include "dispatch.h"
#include "k_xy.cuh"

namespace ns3d {

cudaError_t run_inv_x(const InvXArgs<3, float2>& a, const PassGeom& g, cudaStream_t st) {
  if (g.tile[kTileInvX] >= 3) return run_inv_x_rev(a, g, st);
  return launch_inv_x<3>(a, g, st);
}
cudaError_t run_inv_x(const InvXArgs<6, float2>& a, const PassGeom& g, cudaStream_t st) {
  if (g.tile[kTileInvX] >= 3) return run_inv_x_rev(a, g, st);
  return launch_inv_x<6>(a, g, st);
}
cudaError_t run_inv_y(const InvYArgs<3, float2>& a, const PassGeom& g, cudaStream_t st) {
  if (g.tile[kTileInvY] >= 3) return run_inv_y_rev(a, g, st);
  return launch_inv_y<3>(a, g, st);
}
cudaError_t run_inv_y(const InvYArgs<6, float2>& a, const PassGeom& g, cudaStream_t st) {
  if (g.tile[kTileInvY] >= 3) return run_inv_y_rev(a, g, st);
  return launch_inv_y<6>(a, g, st);
}
cudaError_t run_fwd_y(const FwdYArgs<float2>& a, const PassGeom& g, cudaStream_t st) {
  if (g.tile[kTileFwdY] >= 3) return run_fwd_y_rev(a, g, st);
  return launch_fwd_y(a, g, st);
}

cudaError_t prepare_xy_f32(const PassGeom& g) { return prepare_xy_tiles<float2>(g); }

}  // namespace ns3d
