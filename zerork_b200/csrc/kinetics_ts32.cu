// kinetics_ts32.cu -- the rates + Jacobian kernels with 32 states per tile.
#include "kinetics_kernel.cuh"

namespace zrk {
template cudaError_t launch_ts<32>(const DevMech &, const RatesJacArgs &, const KinParams &, const LaunchCfg &,
                                  cudaStream_t);
}  // namespace zrk
