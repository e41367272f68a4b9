// kinetics_ts8.cu -- the rates + Jacobian kernels with 8 states per tile.
#include "kinetics_kernel.cuh"

namespace zrk {
template cudaError_t launch_ts<8>(const DevMech &, const RatesJacArgs &, const KinParams &, const LaunchCfg &,
                                  cudaStream_t);
}  // namespace zrk
