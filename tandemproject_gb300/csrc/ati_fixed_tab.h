// ati_fixed_tab.h — tables of the fixed-point line sweeps (ati_fixed_line.h), made on the host when a handle is made.
#pragma once
#include <cstdint>
#include <vector>

#include "ati_seg.h"

namespace ati {

// Row table, FX_RT 32-bit words per LU-factor row.  A coefficient c, |c| < 4, is the pair (hi, lo) with
// c = hi 2^-29 + lo 2^-61, both signed.  The forward values are carried as u = c2 v, as in the FU_RT table:
//   u(i) = A d1 + B d2 + C d3 + m0 u(i-2) + m1 u(i-1),  b(i) = u(i) + n1 b(i+1) + n2 b(i+2)
//   [0] A, [2] B, [4] C, [6] m0 = -l0', [8] m1 = -l1', [12] n1 = -c3, [14] n2 = -c4,
//   [16] R, [18] T: the row's results from incoming u(s0-2) = 1, u(s0-1) = 1 (back substitution within the segment);
//   [20] G, [22] H: from b(s1) = 1, b(s1+1) = 1; [24] g, [26] h: forward values from the incoming ones.
// Responses die out along a segment, so they are stored times a power of two that brings the largest to [1/2, 1):
//   [10]: that of R, T (low half word, signed) and of G, H (high half word) of the row's group, [11]: of g, h of the
//   segment's last two rows
constexpr int FX_BITS = 29, FX_RT = 28;
constexpr int FX_PAD = 8;  // rows of zero padding on each side of the table (reads ahead of a segment)
// End table, FX_ET pairs of words per (block, direction); pairs with FX_END_BITS in the place of 29 but for [54..149]:
//   [0..17]  start rows 0-2: six weights each on (f(q) - f(r)), q = 0..6 without r
//   [18..35] end rows L-1-r: the same on (f(L-1-q) - f(L-1-r))
//   [36..41] m0, m1 of rows 0-2;  [42..47] m0, m1 of rows L-1, L-2, L-3;  [48..53] n1, n2 of rows 0-2
//   [54..101] lines periodic onto their own block: rows 0 and 1 from either end, 24 weights each (29 bits): 11 on the
//             differences f(q+1) - f(q) from that end, one on f(L-1) - f(0), 12 on f(L-2-q) - f(L-1-q) (for the end's rows
//             with the line reversed); [102..103] what the start's sums are multiplied by, [104..105] the end's
//   [150..152] A, B, C and [153..154] m0, m1 of row 3
constexpr int FX_ET = 156;
constexpr int FX_END_BITS = 24;
// A segment's rows fall into groups, whose values share one scale: of FX_GR rows, the last one too; what does not divide is
// a group of its own before the last one (five to seven rows) or goes with the one there (up to twelve); up to 15 rows are
// one group.  Values change by a factor of 0.73 a row at most where nothing drives them, 3.6 bits a group, which the
// integers' spare bits over FP64's cover.  The first and the last group hold the seven points that one-sided end rows read,
// the two groups at either end the thirteen of a periodic line's.
constexpr int FX_GR = 8;
ATI_HD int fx_groups(int n) {
  return n < 2 * FX_GR ? 1 : (n - FX_GR) / FX_GR + ((n - FX_GR) % FX_GR >= 5) + 1;
}
// rows before group g of ng in a segment of n rows (g = ng: n)
ATI_HD int fx_group_start(int g, int ng, int n) {
  return g < ng - 1 || g == 0 ? FX_GR * g : (g == ng ? n : n - FX_GR);
}
// values carried from segment to segment stay below 2^FX_CARRY
constexpr int FX_CARRY = 59;
// Longest line the tile of 32 lines holds in shared memory; on the shortest ones the two ends' rows meet
constexpr int FX_LMIN = 13, FX_LMAX = 800;
inline bool fx_line(int L) { return L >= FX_LMIN && L <= FX_LMAX; }

struct SchemeHost;

// One operator's scales (the filter's, or the derivative's), the same for every handle of one scheme, so that a case's
// results do not depend on the other cases of a batch: the bits that a scaled difference may take, the extra scale 2^k its
// coefficients carry, the bits that values carried from group to group may take, and, in an open line's last group, whose
// rows amplify most, the spare bits of the differences and the bits of the carried values.  gbits 0: an extreme filter, which
// the FP64 sweeps take.
struct FixScale {
  int gbits = 0, k = 0, carry = 0, spare = 0, carry_end = 0;
};
struct FixOp : FixScale {
  double vfwd = 0, vinner = 0, vback = 0;  // largest values of the solve, in units of 2^gbits
};
FixOp fix_operator(const SchemeHost &H, bool filt);
// The largest values that a group's rows can take on a line of L points (per: periodic): in units of the largest
// difference that the group reads, forward (inner: those that inner rows read) and back, and per unit of its carried
// values; [1]: the line's last group.
struct FixBounds {
  double forward[2] = {0, 0}, inner[2] = {0, 0}, forward_carry[2] = {0, 0}, backward[2] = {0, 0}, backward_carry[2] = {0, 0};
};
FixBounds fix_bounds(const SchemeHost &H, bool filt, int L, bool per);
// The rows (L FX_RT words) and ends (2 FX_ET words) of a line with LU factors fac; false where a coefficient or a sum of
// products could leave its range.
bool fix_line(const SchemeHost &H, const FixOp &op, bool filt, int L, bool per, const double *fac, int *rows, int *ends);

}  // namespace ati
