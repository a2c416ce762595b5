// Density with the factored density matrix: interface between the factored kernel
// (density_factored.cu) and the density dispatch and batches (density_tc.cu).
#pragma once

#include <vector>

#include "density.cuh"

namespace qmt {

// What a factor's rank decides in the kernel.
struct FactShape {
  int refused;             // 1: the unfactored launch of the pair does the work
  int r16;                 // rank rounded up to 16
  int sets;                // TMEM buffers of [H.. | S]: two (2 r16 <= 256 columns each) or one
  int na;                  // H accumulators: up to three where two buffers hold them, else one
};

// Shared memory of a launch: the ring, then the factor where it stays.
struct FactPlan {
  uint32_t nslots;         // ring slots
  uint32_t slot_magic;     // ceil(2^32 / nslots): group / nslots = umulhi(group, magic) below 2^28
  uint32_t slot_bytes;     // A pieces, then (streamed factor) the factor's K-step block
  uint32_t resident;       // the whole factor behind the ring, loaded once (single molecule)
};

// What the device leaves for a launch whose rank the host does not know.
struct FactDecision {
  FactShape shape;
  FactPlan plan;
  int rank;                // 0: refused
};

// One molecule of a factored launch.  A launch covers the tiles of one or more molecules; global
// tile t belongs to the molecule with tile0 <= t < tile0 + ntiles.
struct FactMol {
  PointMap pm;
  int64_t tile0, ntiles;
  int nunits;              // K-steps (units of 16 columns)
  int r16, sets, na;       // FactShape of the rank, where the host knows it
  const uint8_t* B;        // factor blocks (fact_split_kernel)
  const int4* units;       // unit and class tables
  const float* coords;
  const float* hscale;     // 2^-h_k of the factor columns
  float* qube;
  double* partials;        // per tile of this molecule
  double outscale;
};

constexpr int kFactorMaxR16 = 256;   // [H0 | S] of the rank's columns fill the 512 of TMEM

// Unit tables of the molecule's basis (fs: column scales 2^s_j), once per basis.
qmt_status ensure_unit_tables(qmt_mol* m, const std::vector<float>& fs, cudaStream_t s);
// Largest rank that a call may take: half of N; with `any_rank` (fp16x3 and many sample points) any rank of up to
// 256 functions.  0 when the nuclear charge already bounds the rank above it.
int factor_limit(const qmt_mol* m, int fmt, bool any_rank);
// Enqueues P = L L^T and the split factor, where they are not there yet, without waiting unless it may.
qmt_status ensure_factor(qmt_mol* m, int prec, int fmt, int nsplit, int kpad, bool any_rank, bool wait,
                         cudaStream_t s);
// The factor's rank, 0 when there is none that passed its check; -1 while only the device knows (wait: never).
qmt_status factor_rank(qmt_mol* m, bool wait, int* rank, cudaStream_t s);
// Descriptor of the molecule in a launch, its tiles starting at global tile `tile0`, for a factor of rank `rank`.
void fact_mol_desc(const qmt_mol* m, int rank, const PointMap& pm, int64_t tile0, int64_t ntiles, float* qube,
                   double outscale, FactMol& d);
// One persistent launch over the tiles of one molecule (host descriptor), or of nmol > 1 (device
// array `dev`, host copies for the shared-memory plan).
qmt_status launch_factored(const FactMol* host, const FactMol* dev, int nmol, int64_t ntiles, int fmt, int nsplit,
                           int* err, cudaStream_t s);
// The launch of a molecule whose rank only the device knows, `d` described for the largest rank that the call takes:
// the device decides first, and what it decided is left in *decision.
qmt_status launch_factored_on_device(qmt_mol* m, const FactMol& d, int limit, int fmt, int nsplit, int* err,
                                     const FactDecision** decision, cudaStream_t s);

// Column scales and producer tables, once per molecule (density_tc.cu).
qmt_status ensure_basis_operands(qmt_mol* m, int K, cudaStream_t s);

}  // namespace qmt
