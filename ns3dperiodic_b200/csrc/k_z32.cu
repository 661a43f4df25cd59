// z pass instantiations, FP32 lines of the precision mode (FP64: k_z.cu).
#include "dispatch.h"
#include "launch.cuh"

namespace ns3d {

cudaError_t run_z(const ZArgs<3, float2>& a, const PassGeom& g, cudaStream_t st) {
  return launch_z(a, g, st);
}
cudaError_t run_z(const ZArgs<6, float2>& a, const PassGeom& g, cudaStream_t st) {
  return launch_z(a, g, st);
}

}  // namespace ns3d
