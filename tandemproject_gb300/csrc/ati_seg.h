// ati_seg.h — the cut of a line into segments, for device and host.
//
// The segmentation is a function of the line length alone, so a block's results do not depend on the other blocks or
// cases of a handle (the segmented sweeps: ati_kernels.h, ati_fixed.h).
#pragma once

#ifndef ATI_HD
#ifdef __CUDACC__
#define ATI_HD __host__ __device__ __forceinline__
#else
#define ATI_HD inline
#endif
#endif

namespace ati {

// segments of about SEG_CUT points, at most SEG_CUTS of them
constexpr int SEG_CUT = 48, SEG_CUTS = 16;
ATI_HD int seg_count(int L) {
  const int s = (L + SEG_CUT - 1) / SEG_CUT;
  return s < 1 ? 1 : (s > SEG_CUTS ? SEG_CUTS : s);
}
// first row of segment k of S on a line of L points (the first L % S segments hold one row more)
ATI_HD int seg_start(int k, int L, int S) {
  const int q = L / S, r = L % S;
  return k * q + (k < r ? k : r);
}

}  // namespace ati
