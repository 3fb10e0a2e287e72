// How the weight-streaming GEMMs (gemm_stream.cu) split a call's (slab, K group) units over the CTAs.
#pragma once

#ifdef __CUDACC__
#define B200MOE_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define B200MOE_HOST_DEVICE inline
#endif

namespace b200moe {

// Units (K groups) of a CTA's range.  Equal ranges cut slabs anywhere: a CTA then writes up to two sets of partial sums and
// a slab's last arrival adds several.  Ranges of whole slabs, or of a share that divides a slab's groups, cost a single set or
// none, and are taken when they are at most kCutCost units longer (a cut costs about as much).  Measured with 4 / 8 / 12 /
// 16 / 24 units, us a call: 3 active experts 51.2 / 47.3 / 43.4 / 43.2 / 43.0, 7 active 77.4 / 77.2 / 76.6 / 81.7 / 81.5, 14
// active 135.6 / 130.7 / 130.3 / 130.3 / 130.7, 30 active 249 / 241 / 241 / 262 / 261, the others within 1 %.
// A share that does not divide the groups is no gain: its cuts drift across the slabs as those of equal ranges do.  28 groups
// where equal ranges would be 5, 8 or 9 long (one active expert, intermediate size 1408, 2560, 2816), us at 1 / 12 tokens: equal
// 43.0 / 53.2, 47.1 / 61.4, 49.2 / 63.5; shares of 6, 10, 10: 39.0 / 51.2, 45.1 / 61.4, 49.2 / 61.5; of 7, 14, 14: 36.9 / 49.2,
// 41.0 / 57.3, 43.0 / 59.4.
constexpr int kCutCost = 12;
B200MOE_HOST_DEVICE int stream_range(int units, int groups, int ctas) {
  const int per = (units + ctas - 1) / ctas;
  if (per == 0) return 0;
  int share;
  if (per < groups) {
    int pieces = groups / per;   // the most pieces of a slab that are not shorter than `per`, and all as long
    while (groups % pieces != 0) --pieces;
    share = groups / pieces;
  } else {
    share = (per + groups - 1) / groups * groups;
  }
  return share - per <= kCutCost ? share : per;
}

}  // namespace b200moe
