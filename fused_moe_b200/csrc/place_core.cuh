// Pieces shared by the kernels that lay the packed rows out (permute.cu, front_small.cu).
#pragma once

#include "common.cuh"

namespace b200moe {

// Thread e < 256 of the block's first eight warps brings the padded and the real rows of expert e; on return
// `row0` is the sum of `padded` over the experts before it, the other two are the totals.  Contains one __syncthreads
// that every thread of the block must reach (threads past 256 pass zeros and ignore the results).
__device__ __forceinline__ void block_scan_256(int padded, int total, int lane, int warp, int* s_pad, int* s_rows,
                                               int& row0, int& padded_all, int& rows_all) {
  int incl = padded;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += v;
  }
  const int rows = __reduce_add_sync(0xffffffffu, total);
  if (warp < 8 && lane == 31) {
    s_pad[warp] = incl;
    s_rows[warp] = rows;
  }
  __syncthreads();
  row0 = incl - padded;
  padded_all = 0;
  rows_all = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (i < warp) row0 += s_pad[i];
    padded_all += s_pad[i];
    rows_all += s_rows[i];
  }
}

// Where the rows of a local expert lie, kept in shared memory between the scan and the writing of the tables.
struct ExpertRows {
  int row0, total, padded;
};

// M-tile entries and padding marks (fewer than 128 a tile column of one expert), an expert per warp in turn: independent
// stores by 32 lanes instead of a chain of 127 by one thread.
__device__ __forceinline__ void write_expert_tables(const Workspace& ws, const ExpertRows* rows, int e_local, int lane,
                                                    int warp, int n_warps) {
  int* tile_expert = ws.at<int>(ws.L.tile_expert);
  int* row_token = ws.at<int>(ws.L.row_token);
  for (int e = warp; e < e_local; e += n_warps) {
    const ExpertRows x = rows[e];
    for (int t = lane; t < x.padded / kTileM; t += 32) tile_expert[x.row0 / kTileM + t] = e;
    for (int r = x.total + lane; r < x.padded; r += 32) row_token[x.row0 + r] = -1;
  }
}

}  // namespace b200moe
