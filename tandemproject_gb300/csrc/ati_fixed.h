// ati_fixed.h — fixed-point line sweeps of the FP64 fast path: interface and table layout.
//
// GB300 issues an FP64 multiply-add once in 64 clocks per SM sub-partition, a 32 x 32 + 64 bit integer multiply-add
// once in 2 and an integer addition once in 1 (measured, 16 warps an SM).  A compact derivative or filter is a linear
// map whose coefficients are known when the handle is made, so its line solves can run in 64-bit fixed point: each
// line is scaled so that its largest difference of neighbouring values fills the range the operator's amplification
// leaves free, and every multiplication by a coefficient is three integer multiply-adds.  Values on the line are kept
// modulo 2^64 (only differences enter the operator), so the scale follows the differences and not the values.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "ati_kernels.h"

namespace ati {

// Row table, FX_RT 32-bit words per LU-factor row.  A coefficient c, |c| < 4, is the pair (hi, lo) with
// c = hi 2^-29 + lo 2^-61, both signed.  The forward values are carried as u = c2 v, as in the FU_RT table:
//   u(i) = A d1 + B d2 + C d3 + m0 u(i-2) + m1 u(i-1),  b(i) = u(i) + n1 b(i+1) + n2 b(i+2)
//   [0] A, [2] B, [4] C, [6] m0 = -l0', [8] m1 = -l1', [12] n1 = -c3, [14] n2 = -c4,
//   [16] R, [18] T: the row's results from incoming u(s0-2) = 1, u(s0-1) = 1 (back substitution within the segment);
//   [20] G, [22] H: from b(s1) = 1, b(s1+1) = 1; [24] g, [26] h: forward values from the incoming ones ([10] unused)
//   ([16]..[23] of the filter, whose responses are larger: FX_CBITS_FILTER in the place of 29)
constexpr int FX_BITS = 29, FX_CBITS_FILTER = 26, FX_RT = 28;
constexpr int FX_PAD = 8;  // rows of zero padding on each side of the table (reads ahead of a segment)
// End table, FX_ET pairs of words per (block, direction); pairs with FX_END_BITS in the place of 29 but for [54..149]:
//   [0..17]  start rows 0-2: six weights each on (f(q) - f(r)), q = 0..6 without r
//   [18..35] end rows L-1-r: the same on (f(L-1-q) - f(L-1-r))
//   [36..41] m0, m1 of rows 0-2;  [42..47] m0, m1 of rows L-1, L-2, L-3;  [48..53] n1, n2 of rows 0-2
//   [54..101] lines periodic onto their own block: start rows 0, 1: 24 weights each (29 bits), 11 on
//             the differences f(q+1) - f(q) from the line's start, one on f(L-1) - f(0), 12 on f(L-2-q) - f(L-1-q);
//             [102..149] end rows L-1, L-2: the same with the line reversed
//   [150..152] A, B, C and [153..154] m0, m1 of row 3
constexpr int FX_ET = 156;
constexpr int FX_END_BITS = 24;
// Longest line the tile of 32 lines holds in shared memory; on the shortest ones the two ends' rows meet
constexpr int FX_LMIN = 13, FX_LMAX = 800;
inline bool fx_line(int L) { return L >= FX_LMIN && L <= FX_LMAX; }
// largest bits of a scaled difference, and the operator's extra scale 2^k (ati_api.cu: fix_tables)
struct FixArgs {
  const BlockDev *blk;
  const LTile *lt;
  const int *rows;          // row table (first row after the padding)
  const int64_t *ends;      // end tables, FX_ET per (block * 3 + direction - 1)
  SweepIO<double, double> io;
  double *drva;
  int gbits, kscale;
  bool rowtiles;
};

namespace fast {
// a sweep of direction nn on the fixed-point kernels; the caller has checked e.fx_ok[filt][nn]
void sweep_fixed(const Eng<double> &e, cudaStream_t st, int nn, bool filt, const SweepIO<double, double> &io);
cudaError_t fixed_init();
}  // namespace fast

}  // namespace ati
