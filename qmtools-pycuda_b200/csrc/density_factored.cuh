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
// Enqueues P = L L^T and the split factor, where they are not there yet, without waiting.
qmt_status ensure_factor(qmt_mol* m, int prec, int fmt, int nsplit, int kpad, bool any_rank, cudaStream_t s);
// The factor's rank, 0 when there is none that passed its check; -1 while only the device knows (wait: never).
qmt_status factor_rank(qmt_mol* m, bool wait, int* rank, cudaStream_t s);
// Enqueues the device's own decision for a call that takes ranks up to `limit`; the shape it leaves on the device.
qmt_status decide_on_device(qmt_mol* m, int limit, const FactShape** shape, cudaStream_t s);
// Descriptor of the molecule in a launch, its tiles starting at global tile `tile0`, for a factor of rank `rank`.
void fact_mol_desc(const qmt_mol* m, int rank, const PointMap& pm, int64_t tile0, int64_t ntiles, float* qube,
                   double outscale, FactMol& d);
// One persistent launch over the tiles of one molecule (host descriptor), or of nmol > 1 (device
// array `dev`, host copies for the shared-memory plan).  With `shape` (one molecule) the device has the rank, and the
// host's descriptor the largest one that it may be.
qmt_status launch_factored(const FactMol* host, const FactMol* dev, int nmol, int64_t ntiles, int fmt, int nsplit,
                           int* err, const FactShape* shape, cudaStream_t s);

// Column scales and producer tables, once per molecule (density_tc.cu).
qmt_status ensure_basis_operands(qmt_mol* m, int K, cudaStream_t s);

}  // namespace qmt
