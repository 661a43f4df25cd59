// Launch-attribute preparation of the reversed-schedule tiles, shared by the
// FP64 and FP32 translation units (k_xy_rev.cu, k_xy_rev32.cu).
#pragma once

#include "launch.cuh"

namespace ns3d {
namespace {
template <typename C>
cudaError_t prepare_rev_prec(const PassGeom& g, int tile) {
  PassGeom gt = g;
  cudaError_t e;
  gt.tile[kTileInvX] = tile;
  if (rev_tile_exists_inline(g.Nx, tile)) {
    if ((e = launch_inv_x<3, C, 1>(InvXArgs<3, C>{}, gt, nullptr, true)) != cudaSuccess) return e;
    if ((e = launch_inv_x<6, C, 1>(InvXArgs<6, C>{}, gt, nullptr, true)) != cudaSuccess) return e;
  }
  gt.tile[kTileInvY] = gt.tile[kTileFwdY] = tile;
  if (rev_tile_exists_inline(g.Ny, tile)) {
    if ((e = launch_inv_y<3, C, 1>(InvYArgs<3, C>{}, gt, nullptr, true)) != cudaSuccess) return e;
    if ((e = launch_inv_y<6, C, 1>(InvYArgs<6, C>{}, gt, nullptr, true)) != cudaSuccess) return e;
    if ((e = launch_fwd_y<C, 1>(FwdYArgs<C>{}, gt, nullptr, true)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}
}  // namespace

}  // namespace ns3d
