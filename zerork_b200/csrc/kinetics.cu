// kinetics.cu -- workspace sizes and dispatch of the fused rates + Jacobian
// kernels (kinetics_kernel.cuh; one translation unit per tile size).
#include "kinetics_kernel.cuh"

namespace zrk {

extern template cudaError_t launch_ts<8>(const DevMech &, const RatesJacArgs &, const KinParams &, const LaunchCfg &,
                                         cudaStream_t);
extern template cudaError_t launch_ts<16>(const DevMech &, const RatesJacArgs &, const KinParams &, const LaunchCfg &,
                                          cudaStream_t);
extern template cudaError_t launch_ts<32>(const DevMech &, const RatesJacArgs &, const KinParams &, const LaunchCfg &,
                                          cudaStream_t);

namespace {

size_t ws_bytes(const DevMech &m, const LaunchCfg &cfg, int part_rows) {
  return (size_t)make_layout(m.nsp, m.nstep, part_rows).rows * cfg.ts * sizeof(double);
}

}  // namespace

int rates_jac_part_rows(const DevMech &m, const LaunchCfg &cfg) {
  const int few = 2 * cfg.warps, groups = std::min(cfg.warps * 32 / (cfg.ts / cfg.v), m.nsp + 1);
  if (groups <= few) return few;
  // (a global slice has to fit in the no-alloc entry point's 8 MiB)
  const size_t bytes = ws_bytes(m, cfg, groups), limit = cfg.global_ws ? 8u << 20 : 227 * 1024;
  return bytes + (cfg.stage && !cfg.global_ws ? (size_t)m.hot_bytes : 0) <= limit ? groups : few;
}

size_t rates_jac_ws_bytes(const DevMech &m, const LaunchCfg &cfg) {
  return ws_bytes(m, cfg, rates_jac_part_rows(m, cfg));
}

bool rates_jac_species_fit(const DevMech &m, const LaunchCfg &cfg) {
  if (cfg.stage) return false;  // among the staged tables
  const size_t ws = cfg.global_ws ? 0 : rates_jac_ws_bytes(m, cfg);
  // (two resident CTAs share the SM's 228 KB, 1 KB of it the system's for each)
  return ws + m.spc_bytes <= (cfg.minb == 2 ? 113 * 1024 : 227 * 1024);
}

size_t rates_jac_smem_bytes(const DevMech &m, const LaunchCfg &cfg) {
  const size_t tables = cfg.stage ? m.hot_bytes : rates_jac_species_fit(m, cfg) ? m.spc_bytes : 0;
  return (cfg.global_ws ? 0 : rates_jac_ws_bytes(m, cfg)) + tables;
}

bool rates_jac_mapping_ok(const LaunchCfg &c) {
  if (c.warps < 1 || c.warps > 32) return false;
  if (c.minb != 1 && (c.minb != 2 || c.warps > 8 || c.ts > 16 || c.stage)) return false;
  if (c.warps > 16 && c.v != 1) return false;  // 64 registers per thread: one state each
  return (c.ts == 8 || c.ts == 16 || c.ts == 32) && (c.v == 1 || c.v == 2 || c.v == 4);
}

cudaError_t launch_rates_jac(const DevMech &m, const RatesJacArgs &a, const KinParams &kp,
                             const LaunchCfg &cfg, cudaStream_t stream) {
  switch (cfg.ts) {
    case 8: return launch_ts<8>(m, a, kp, cfg, stream);
    case 16: return launch_ts<16>(m, a, kp, cfg, stream);
    case 32: return launch_ts<32>(m, a, kp, cfg, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace zrk
