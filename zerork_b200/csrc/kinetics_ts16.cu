// kinetics_ts16.cu -- the rates + Jacobian kernels with 16 states per tile.
#include "kinetics_kernel.cuh"

namespace zrk {
template cudaError_t launch_ts<16>(const DevMech &, const RatesJacArgs &, const KinParams &, const LaunchCfg &,
                                  cudaStream_t);
}  // namespace zrk
