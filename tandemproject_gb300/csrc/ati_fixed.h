// ati_fixed.h — fixed-point line sweeps of the FP64 fast path: interface.
//
// GB300 issues an FP64 multiply-add once in 64 clocks per SM sub-partition, a 32 x 32 + 64 bit integer multiply-add
// once in 4 and an integer addition once in 2 (measured, 16 warps an SM).  A compact derivative or filter is a linear
// map whose coefficients are known when the handle is made, so its line solves can run in 64-bit fixed point: every
// multiplication by a coefficient is three integer multiply-adds, and a few rows at a time share one scale
// (ati_fixed_line.h).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "ati_kernels.h"

namespace ati {

struct FixArgs {
  const BlockDev *blk;
  const LTile *lt;
  const int *rows;          // row table (first row after the padding)
  const int64_t *ends;      // end tables, FX_ET per (block * 3 + direction - 1)
  SweepIO<double, double> io;
  double *drva;
  FixScale fs;
  bool rowtiles;
};

namespace fast {
// a sweep of direction nn on the fixed-point kernels; the caller has checked e.fx_ok[filt][nn]
void sweep_fixed(const Eng<double> &e, cudaStream_t st, int nn, bool filt, const SweepIO<double, double> &io);
cudaError_t fixed_init();
}  // namespace fast

}  // namespace ati
