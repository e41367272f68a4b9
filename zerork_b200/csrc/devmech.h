// devmech.h -- mechanism tables laid out for the sm_100a kinetics kernels.
//
// One reaction record per reaction drives the rate-constant phase: each
// record carries the forward Arrhenius triple, the reverse rule (explicit
// REV triple or equilibrium constant), the third-body / falloff index and the
// reactant / product species, so one work item computes both steps of a
// reaction (rate_const.cpp:539-582 ordering: Arrhenius, Keq, third body,
// falloff; then perf_net.cpp:190-274 limiter and concentration products).
// Species-production and Jacobian phases use gather lists (per species and
// per Jacobian nonzero) so every sum is deterministic and atomic-free.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "mech.h"

namespace zrk {

constexpr int kMaxSide = 6;  // max species per reaction side (CHEMKIN limit)

enum RxnFlags : int {
  kRevKeq = 1,       // reverse step from the equilibrium constant
  kRevArr = 2,       // reverse step from explicit REV parameters
  kThirdBody = 4,
  kFalloff = 8,
  kPlog = 16,        // forward rate from the PLOG table (aux: PLOG index)
  kNoRxn = 32,       // padding of rxn_slots: no reaction
};

struct alignas(16) RxnRec {
  double lnA, n, Ta;        // forward (converted units)
  double lnA_r, n_r, Ta_r;  // explicit reverse, or dn in lnA_r for Keq
  int fwd, rev;             // step indices (rev = -1: irreversible)
  short flags, ne;          // ne efficiencies, from eff[e0] on
  int aux, e0;              // aux: falloff or PLOG index
  short nr, np;
  short r[kMaxSide], p[kMaxSide];
};
static_assert(sizeof(RxnRec) % 16 == 0, "RxnRec alignment");

struct alignas(16) Eff {
  double alpha;  // efficiency minus one
  int spc, pad;
};

// Plain-pointer view of the device tables (all device addresses).
struct DevMech {
  int nsp, nrxn, nstep, nnz;
  const double *mw, *inv_mw, *ru_inv_mw, *thermo;  // thermo: [nsp*16]
  const double *thermo_t;  // the same, coefficient by coefficient: [16][nsp]
  const RxnRec *rxn;
  // third-body and falloff efficiencies, one 16-byte entry each
  const Eff *eff;
  const int *fo_type, *fo_spc;
  const double *fo_par;  // 8 a reaction: the loader's, with -1 / T for Troe's T*** and T*
  // PLOG reactions: distinct pressures per reaction (plog_pt_ptr), Arrhenius
  // lines per pressure (plog_ln_ptr); see MechTables
  const int *plog_pt_ptr, *plog_ln_ptr;
  const double *plog_p, *plog_lnp, *plog_lnA, *plog_sgn, *plog_n, *plog_Ta;
  // species production gather lists (step indices in ascending step order)
  const int *sd_ptr, *sd_step, *sc_ptr, *sc_step;
  // Both lists of all species as one list for one reactor per CTA, cut into
  // net_chunks equal chunks of net_quads * 4 entries whatever species they
  // belong to: step | 1 << 31 for a destruction term | 1 << 30 where a partial
  // sum ends (a species' or the chunk's last term).  Chunk c's partial sums go
  // to the slots from net_slot[c] on, and species k's net rate is the sum of
  // the slots [net_ptr[k], net_ptr[k + 1]).  Stored quad by quad in blocks of 32
  // chunks ([block][net_quads][32]).
  // For mechanisms of up to kFewBlocks blocks of reactions instead: {species,
  // first, end, 0} by decreasing length, and the terms (net_chunks = 0 then).
  const int4 *sn_rec;
  const int *sn_step;
  int net_chunks, net_quads;
  const int4 *net_ent;
  const int *net_slot, *net_ptr;
  // both lists of a species for the rates kernel, longest first: {species,
  // number of terms, first record, number of destruction terms} and records of
  // four 16-bit steps, destruction first (unused places repeat the last step)
  const int4 *sq_rec;
  const int2 *sq_step;
  // Jacobian pattern and per-nonzero gather lists
  const int *col_ptr, *row_idx;
  const int *nzd_ptr, *nzd_step, *nzc_ptr, *nzc_step;
  // Species-column Jacobian entries as one flat list in column-major order
  // without each column's temperature row (nj items; column j holds items
  // [jf_ptr[j], jf_ptr[j+1]), and item f is nonzero f + j of the compressed
  // columns).  jw / jt: per item {row, n_des | n_cre << 16} and its
  // destruction then creation step indices from jt[jt_ptr[f]].  jit: the same
  // as 16-byte records {row | n_des << 16, the first four steps as 16-bit
  // indices, the item's first record of further steps}, four further steps a
  // record of jext; unused places hold nstep, the workspace's row of zeros;
  // one sentinel item ends the list.  jcost: the cumulative work estimate (12
  // and 4 per record of four steps) that splits the list into equal shares for
  // the thread groups of the rates kernel.
  int nj;
  const int2 *jw, *jext;
  const int4 *jit;
  const unsigned short *jt;
  const int *jt_ptr, *jcost, *jf_ptr;
  const int *jf_col;  // column of each item
  // row-wise view of the Jacobian pattern: row i has entries jr_kk[p] (index
  // into the compressed-column values) in columns jr_col[p], p in
  // [jr_ptr[i], jr_ptr[i+1])
  const int *jr_ptr, *jr_kk, *jr_col;
  const int *nz_rc;  // per Jacobian nonzero: row | column << 16
  // work lists for snake-order assignment to thread groups: species by
  // decreasing length of their lists (production gathers), and the reaction
  // records by kind and decreasing estimated cost
  const int *spc_order;
  const RxnRec *rxn_by_cost;
  // The same records for one reactor per CTA, a reaction a lane: grouped by
  // kind (PLOG, falloff, third body, the rest) in blocks of 32 of one kind,
  // padded with kNoRxn records, so that a warp runs one kind's code and the
  // long falloff chains run beside the others instead of after them.  The six
  // 16-byte parts of a block's records are stored part by part ([block][6][32]),
  // so that a warp reads each in one piece.
  const int4 *rxn_slots;
  int nblocks;
  // The tables the rates kernel reads form the first hot_bytes bytes of the
  // allocation at base (16-byte aligned), so a CTA can stage them in shared
  // memory and address them at a fixed offset from their global copies.
  const unsigned char *base;
  int hot_bytes;
  // molecular weights, their reciprocals and the thermodynamic fits: bytes from mw on
  int spc_bytes;
};

constexpr int kFewBlocks = 4;

// Doubles of the partial sums of net_ent's chunks: at most 3 nsp + 2 chunks,
// and a species boundary each.
__host__ __device__ inline int net_slots(int nsp) { return 4 * nsp + 2; }

// Host-side builder; owns the device allocation.
class DeviceMechanism {
 public:
  DeviceMechanism(const MechTables &t, const JacPattern &p);
  ~DeviceMechanism();
  DeviceMechanism(const DeviceMechanism &) = delete;
  DeviceMechanism &operator=(const DeviceMechanism &) = delete;
  const DevMech &view() const { return view_; }
  size_t bytes() const { return bytes_; }
  // host copies of the gather lists (for tests / cost models)
  int n_terms() const { return n_terms_; }

 private:
  void *blob_ = nullptr;
  size_t bytes_ = 0;
  int n_terms_ = 0;
  DevMech view_{};
};

}  // namespace zrk
