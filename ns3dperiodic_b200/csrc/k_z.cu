// z pass instantiations (paired C2R, products, R2C), FP64 lines (FP32: k_z32.cu).
#include "dispatch.h"
#include "launch.cuh"

namespace ns3d {

cudaError_t run_z(const ZArgs<3>& a, const PassGeom& g, cudaStream_t st) {
  return launch_z(a, g, st);
}
cudaError_t run_z(const ZArgs<6>& a, const PassGeom& g, cudaStream_t st) {
  return launch_z(a, g, st);
}

}  // namespace ns3d
