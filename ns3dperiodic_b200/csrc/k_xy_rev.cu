// x and y pass instantiations with the reversed radix schedules (tiles 3 and
// 4 of the inv_x, inv_y and fwd_y families), compiled apart from k_xy.cu so
// the parts build in parallel (FP32 lines: k_xy_rev32.cu).
#include "dispatch.h"
#include "k_xy_rev.cuh"

namespace ns3d {

bool rev_tile_exists(int n, int tile) { return rev_tile_exists_inline(n, tile); }

cudaError_t run_inv_x_rev(const InvXArgs<3>& a, const PassGeom& g, cudaStream_t st) {
  return launch_inv_x<3, double2, 1>(a, g, st);
}
cudaError_t run_inv_x_rev(const InvXArgs<6>& a, const PassGeom& g, cudaStream_t st) {
  return launch_inv_x<6, double2, 1>(a, g, st);
}
cudaError_t run_inv_y_rev(const InvYArgs<3>& a, const PassGeom& g, cudaStream_t st) {
  return launch_inv_y<3, double2, 1>(a, g, st);
}
cudaError_t run_inv_y_rev(const InvYArgs<6>& a, const PassGeom& g, cudaStream_t st) {
  return launch_inv_y<6, double2, 1>(a, g, st);
}
cudaError_t run_fwd_y_rev(const FwdYArgs<>& a, const PassGeom& g, cudaStream_t st) {
  return launch_fwd_y<double2, 1>(a, g, st);
}

cudaError_t prepare_xy_rev(const PassGeom& g) {
  for (int tile = 3; tile <= 4; ++tile) {
    cudaError_t e = prepare_rev_prec<double2>(g, tile);
    if (e == cudaSuccess) e = prepare_xy_rev_f32(g, tile);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace ns3d
