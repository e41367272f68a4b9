// integrator_group.h -- the plain FP64 GPU path (integrator_group.cu): one
// BDF integration per group of reactors with a shared step size, order and
// WRMS norm, driven from the host kernel by kernel, as the reference's GPU
// branch of the cfd_plugin integrates a batch with one CVODE instance.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "integrator.h"

namespace zrk {

struct GroupCounters {
  long groups = 0, group_steps = 0, group_newton = 0, launches = 0, syncs = 0;
  long first_fail = 0;  // status of the first group whose attempts all failed
};

// Dynamic shared memory of the group kernels, in doubles: 128 reduction slots,
// then the rates workspace of 3 nsp + nstep doubles and the net rates' partial
// sums (part doubles).  A factorization has its pivot rows (rows doubles) over
// the rates and, when it fits in `limit`, the matrix of `matrix` doubles behind
// the larger of the two, over the partial sums, which are dead by then.  A
// mechanism whose partial sums do not fit sums its net rates without them.
struct GroupSmem {
  size_t matrix_at, eval, fac;  // offset of the matrix; sizes without and with it
  bool chunks, fac_smem;        // partial sums used; matrix in shared memory
};
inline GroupSmem group_smem(size_t nsp, size_t nstep, size_t part, size_t rows, size_t matrix, size_t limit) {
  const size_t ws = 3 * nsp + nstep;
  GroupSmem g;
  g.matrix_at = 128 + (ws > rows ? ws : rows);
  g.chunks = part > 0 && 128 + ws + part <= limit;
  g.eval = 128 + ws + (g.chunks ? part : 0);
  if (g.eval < g.matrix_at) g.eval = g.matrix_at;
  g.fac = g.matrix_at + matrix;
  if (g.fac < g.eval) g.fac = g.eval;
  g.fac_smem = g.fac <= limit;
  if (!g.fac_smem) g.fac = g.eval;
  return g;
}

// Doubles of device workspace per reactor of a group (the reactor's BDF
// vectors, history, Jacobian and Newton-matrix inverse).
size_t group_slot_doubles(const DevMech &m);
// Group sizes for n reactors and at most group_max per group, the last two
// groups split evenly (zerork_reactor_manager.cpp:933-940).
int group_sizes(int n, int group_max, std::vector<int> &sizes);
// Integrate a.n_reactors reactors (order_dev: reactor indices in group
// order) group by group.  slots: group_max * group_slot_doubles doubles;
// part_dev / part_host (pinned): group_max * 6 doubles each.  Per-reactor
// statistics go to a.stats (every reactor of a group gets the group's
// counters and status).  a.state / a.lu / a.order / a.queue_head unused.
cudaError_t integrate_group(const DevMech &m, const IntegOpts &o, const IntegArgs &a, const int *order_dev,
                            int group_max, int threads, double *slots, double *part_dev,
                            double *part_host, cudaStream_t stream, GroupCounters *gc);

}  // namespace zrk
