// Launch-attribute preparation of the x / y passes, shared by the FP64 and FP32
// translation units (k_xy.cu, k_xy32.cu).
#pragma once

#include "launch.cuh"

namespace ns3d {
namespace {
template <typename C>
cudaError_t prepare_xy_prec(const PassGeom& g) {
  cudaError_t e;
  if ((e = launch_inv_x<3>(InvXArgs<3, C>{}, g, nullptr, true)) != cudaSuccess) return e;
  if ((e = launch_inv_x<6>(InvXArgs<6, C>{}, g, nullptr, true)) != cudaSuccess) return e;
  if ((e = launch_inv_y<3>(InvYArgs<3, C>{}, g, nullptr, true)) != cudaSuccess) return e;
  if ((e = launch_inv_y<6>(InvYArgs<6, C>{}, g, nullptr, true)) != cudaSuccess) return e;
  return launch_fwd_y(FwdYArgs<C>{}, g, nullptr, true);
}
}  // namespace

namespace {
// both tiles of every pass family, then the inv_y family's bulk-copy tile
template <typename C>
cudaError_t prepare_xy_tiles(const PassGeom& g) {
  for (int tile = 0; tile < 3; ++tile) {
    PassGeom gt = g;
    for (int& f : gt.tile) f = tile < 2 ? tile : 0;
    if (tile == 2) gt.tile[kTileInvY] = 2;
    const cudaError_t e = prepare_xy_prec<C>(gt);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
}  // namespace

}  // namespace ns3d
