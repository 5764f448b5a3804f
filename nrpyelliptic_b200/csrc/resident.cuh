// On-chip relaxation (kernels_resident.cu): jobs of one cooperative launch
// and the host driver's interface.
#pragma once

#include <math.h>

#include <vector>

#include "driver.cuh"
#include "substep.cuh"

namespace nrpyell {

// One grid of a launch.
template <typename T>
struct ResJob {
  int cta0;                 // first block
  int n0t, n1t, nrad, hmax;  // interior tiles along i0 and i1, radiation blocks, rows of the tallest tile
  int Nxx0, Nxx1, Nxx2, half2, N0, N1;
  long long N01, Ntot;
  T* y;                          // y_n: loaded at the start of a launch, stored at its end
  const T* aux;
  const T* R0;                   // correction form, else nullptr
  const T* coef;
  const double* colgeo;
  const double* w;               // L2 weights
  // exchanged values tagged with the substep that wrote them (kernels_resident.cu):
  // uu on [i2][i1][xu_row >= Nxx0 + 5], vv on [i2][i1][12] (the last 7 planes along
  // i0 and the outer 5), each in eight rotating slots
  void* xu;
  long long xu_slot;             // entries of a slot: uu, then vv from xv0 on
  int xu_row, xu_plane, xv0, xv_plane;
  double2* part;                 // [2][interior blocks]: shares of the residual norm
  int* state;                    // [0] n, [1] 0 or the stop mark, [2] converged
  double* sums;                  // weighted sum of squares of every evaluated residual
  int* err;
  double volume, log10_tol;
  double sum_met, sum_not_met;   // sums at or below / above which the stop test needs no logarithm (NaN: none)
  int max_steps, check_every;
  T dt, eta;
  T cOB[2];
  double invdx0, invdx1;
  int n_start;                   // filled in by the kernel
};

// The stop mark of a job that ended at step n.  Blocks read it as they start, and
// block 0 may write it meanwhile (nothing orders its first stop test after the
// start of a radiation block), so a mark made by the launch itself must read
// as none: with the launch's first step, passed by the host, both values mean
// the same to every block.
__host__ __device__ inline int stop_mark(int n) { return n + 1; }
__host__ __device__ inline bool stopped_before(int mark, int first) { return mark != 0 && mark <= first; }

// Whether a weighted sum of squares meets the tolerance: finalize_l2's test,
// without its logarithm where the sum alone decides.
template <typename Job>
__host__ __device__ inline bool residual_met(const Job& J, double s) {
  if (s <= J.sum_met) return true;
  if (s >= J.sum_not_met) return false;
  const double l2 = log10(1e-16 + sqrt(s / J.volume));
  return J.check_every > 0 ? l2 < J.log10_tol : l2 <= J.log10_tol;
}

// One grid to relax on chip.
struct ResGrid {
  Dims d;
  RfmTables* rt;
  BcTables* bt;
  L2Tables* lt;
  StateBuffers b;
  RelaxParams rp;
  int* state;       // 8 ints on the device
  double* history;  // entry of step 0
};

// How a grid is laid out on the GPU's SMs; blocks == 0: it does not fit.
struct ResPlan {
  int tx, p, threads, n0t, n1t, nrad, hmax, blocks;
  size_t smem;
  double cost;  // estimated cycles of a substep
};
template <typename T>
ResPlan resident_plan(const Dims& d, int max_blocks);

// Whether a grid relaxes on chip (its plan fits and no tile shape is forced).
template <typename T>
bool resident_ok(const Dims& d);

// How many grids of these dimensions, of `available`, share the SMs best (0: they
// do not fit).
template <typename T>
int resident_team(const Dims& d, int available);
int sm_count();

// Which grids of a batch relax on chip: the size of the teams for each grid, 0
// for those that take the batched launches (batch.cu).
template <typename T>
std::vector<int> chip_route(const std::vector<Dims>& grids);

// Relaxes the grids, all of the same dimensions, together in launches of many
// RK4 steps; results[i] as relax_loop's.  Returns false on error.
template <typename T>
bool relax_resident(const std::vector<ResGrid>& grids, std::vector<RelaxResult>* results);

void release_resident();

}  // namespace nrpyell
