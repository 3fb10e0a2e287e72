// Routing, scan and placement of a decode-size call (at most 32 tokens) in ONE block.
//
// At these sizes the three kernels it stands for (route.cu, and scan + place of permute.cu,
// which replace the reference's `fused_route_topk_kernel`, `exclusive_scan_kernel` and
// `dispatch_place_kernel`, solution/python/moe_fused.cu:568-698, 888-1051) do a few
// microseconds of work between them and two launch boundaries; the reference folds scan and
// placement into `fused_dispatch_single_block_kernel` for the same reason.  Results are
// identical to the separate kernels: same routing arithmetic (route_core.cuh), segments padded
// to `pad_rows`, placement stable by token id.
#include "common.cuh"
#include "kernels.cuh"
#include "place_core.cuh"
#include "route_core.cuh"

namespace b200moe {

namespace {

constexpr int kFrontWarps = kFrontSmallMaxTokens;   // at most: one warp per token, never fewer than the scan's eight

// What it takes is latency (one block, a few microseconds of dependent steps).  A warp's first eight lanes keep its
// token's (expert, weight) pairs in registers from the routing to the placement; an expert's tokens are a bit mask
// in shared memory (count: population count, a pair's place: the lower bits), so neither the count nor the placement
// loops over tokens or experts, and the whole kernel has four barriers instead of twenty: 11.4 -> 8.2 us at one token
// (cold caches).
__global__ void __launch_bounds__(kFrontWarps * 32, 1)
route_place_small_kernel(Workspace ws, const void* __restrict__ logits, int logits_dtype,
                         const void* __restrict__ bias, int bias_dtype, int T, float rsf, int local_off, int e_local,
                         int pad_rows) {
  __shared__ uint32_t s_mask[kNumExperts];   // tokens of each local expert
  __shared__ ExpertRows s_experts[kNumExperts];
  __shared__ int s_pad[8], s_rows[8];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int e = threadIdx.x;
  chain_release();   // launched in plain stream order itself (the first kernel of a call)
  // The call's counters (status word, meta, split-K and slab arrival counts): cleared here instead of by a
  // memset of its own, one launch boundary less.  Nothing of them is read before the barriers below.
  {
    uint32_t* z = ws.at<uint32_t>(ws.L.status);
    const int n = (int)((ws.L.chunk_counts - ws.L.status) / 4);
    for (int i = threadIdx.x; i < n; i += blockDim.x) z[i] = 0u;
  }
  if (e < kNumExperts) s_mask[e] = 0u;

  // ---- route: warp t routes token t; lane k < 8 keeps its k-th expert
  int my_id = -1, le = -1;
  float my_w = 0.f;
  if (warp < T) {
    float b[kNumGroups];
    load8_as_float(bias, bias_dtype, lane, b);
    route_one_token(logits, logits_dtype, warp, b, rsf, lane, my_id, my_w);
    if (lane < kTopK && my_id >= local_off && my_id < local_off + e_local) le = my_id - local_off;
  }
  __syncthreads();   // masks and counters are zero
  if (le >= 0) atomicOr(&s_mask[le], 1u << warp);
  __syncthreads();

  // ---- scan: thread e counts the pairs of local expert e, pads, prefix-sums
  int total = 0, padded = 0;
  if (e < kNumExperts) {
    total = __popc(s_mask[e]);
    padded = (total + pad_rows - 1) / pad_rows * pad_rows;
  }
  int row0, padded_all, rows_all;
  block_scan_256(padded, total, lane, warp, s_pad, s_rows, row0, padded_all, rows_all);
  if (e < kNumExperts) s_experts[e] = {row0, total, padded};
  __syncthreads();

  // ---- place
  if (warp < T && lane < kTopK) {
    const size_t i = (size_t)warp * kTopK + lane;
    int r = -1;   // "not local"
    if (le >= 0) {
      r = s_experts[le].row0 + __popc(s_mask[le] & ((1u << warp) - 1u));   // stable by token id
      ws.at<int>(ws.L.row_token)[r] = warp;
      ws.at<float>(ws.L.row_weight)[r] = my_w;
      ws.at<unsigned>(ws.L.row_amax)[r] = 0u;   // GEMM1's epilogue takes the running maximum with atomicMax
    }
    ws.at<int>(ws.L.tok_rows)[i] = r;
    ws.at<int32_t>(ws.L.topk_ids)[i] = my_id;
    ws.at<float>(ws.L.topk_w)[i] = my_w;
  }
  if (e < kNumExperts) {
    int* expert_row0 = ws.at<int>(ws.L.expert_row0);
    if (e < e_local) {
      expert_row0[e] = row0;
      ws.at<int>(ws.L.expert_count)[e] = total;
    }
    if (e == 0) {
      expert_row0[e_local] = padded_all;
      int* meta = ws.at<int>(ws.L.meta);
      meta[0] = padded_all / kTileM;
      meta[1] = padded_all;
      meta[2] = rows_all;
      meta[3] = pad_rows;
    }
  }
  write_expert_tables(ws, s_experts, e_local, lane, warp, blockDim.x / 32);
}

}  // namespace

cudaError_t launch_route_place_small(const Workspace& ws, const void* logits, int logits_dtype, const void* bias,
                                     int bias_dtype, int T, float rsf, int local_off, int e_local, int pad_rows,
                                     cudaStream_t stream) {
  if (T <= 0 || T > kFrontSmallMaxTokens) return cudaErrorInvalidValue;
  const int warps = T < 8 ? 8 : T;
  route_place_small_kernel<<<1, warps * 32, 0, stream>>>(ws, logits, logits_dtype, bias, bias_dtype, T, rsf, local_off,
                                                         e_local, pad_rows);
  return cudaGetLastError();
}

}  // namespace b200moe
