// Permutation of (token, k) pairs into per-expert row segments padded to 128-row tiles.
//
// Replaces the reference's `exclusive_scan_kernel`, `dispatch_place_kernel`,
// `fused_dispatch_single_block_kernel` (solution/python/moe_fused.cu:888-1051) and
// `fused_gather_hidden_scales_kernel` (moe_fused.cu:736-768).  Unlike the reference's
// atomic cursor, placement is stable by token id, so the packed order (and every later
// intermediate) is identical from run to run.
//
//   scan   : per-expert totals from the per-chunk histogram, 128-padded segment starts,
//            the M-tile -> expert table, per-chunk bases, padding rows marked -1
//   place  : one block per 256-token chunk; a pair's place is its rank in a bit mask of the expert's tokens
//   place  also records, per (token, k), the packed row it went to (-1: expert not local)
//   gather : one warp per packed row copies the e4m3 row and its 1x128 scales
#include "common.cuh"
#include "kernels.cuh"
#include "place_core.cuh"

namespace b200moe {

namespace {

// One block; what it takes is latency, so the chain is kept short: the chunk counts in rounds of eight independent
// loads, the prefix sum as warp shuffles plus eight warp totals (two barriers instead of eighteen), and the tables of
// an expert (M tiles, up to 127 padding marks) written by a whole warp instead of by one thread: 4.4 -> 3.6 us at 56
// tokens, 5.2 -> 4.0 us at 901 (32 experts, cold caches).
constexpr int kScanThreads = 1024;

__global__ void __launch_bounds__(kScanThreads)
scan_kernel(Workspace ws, int e_local, int n_chunks, int pad_rows) {
  __shared__ int s_pad[8], s_rows[8];
  __shared__ ExpertRows s_experts[kNumExperts];
  const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
  chain_wait();
  chain_release();
  int* chunk_counts = ws.at<int>(ws.L.chunk_counts);
  int* chunk_base = ws.at<int>(ws.L.chunk_base);
  int total = 0;
  if (e < e_local) {
    // eight independent loads in flight per round instead of one load per chunk in a chain
    for (int c0 = 0; c0 < n_chunks; c0 += 8) {
      int cnt[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) cnt[j] = c0 + j < n_chunks ? chunk_counts[(c0 + j) * e_local + e] : 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (c0 + j < n_chunks) chunk_base[(c0 + j) * e_local + e] = total;
        total += cnt[j];
      }
    }
  }
  const int padded = (total + pad_rows - 1) / pad_rows * pad_rows;   // whole M tiles
  int row0, padded_all, rows_all;
  block_scan_256(padded, total, lane, warp, s_pad, s_rows, row0, padded_all, rows_all);
  int* expert_row0 = ws.at<int>(ws.L.expert_row0);
  if (e < e_local) {
    expert_row0[e] = row0;
    ws.at<int>(ws.L.expert_count)[e] = total;
    s_experts[e] = {row0, total, padded};
  }
  __syncthreads();
  write_expert_tables(ws, s_experts, e_local, lane, warp, kScanThreads / 32);
  if (e == 0) {
    expert_row0[e_local] = padded_all;
    int* meta = ws.at<int>(ws.L.meta);
    meta[0] = padded_all / kTileM;
    meta[1] = padded_all;
    meta[2] = rows_all;   // rows with a local expert (for reporting)
    meta[3] = pad_rows;
  }
}

// One block per chunk of 256 tokens, two (token, k) pairs per thread.  The tokens of an expert are a 256-bit mask in
// shared memory, a pair's place among them the number of lower bits: order by token id as before, without a warp per
// expert that walks the chunk in e_local / 32 rounds of dependent loads: 6.0 -> 4.1 us at 56 tokens, 9.2 -> 5.0 us at 901
// (32 experts, cold caches); a call of 64 tokens over 256 experts takes 15 us less.
__global__ void __launch_bounds__(1024)
place_kernel(Workspace ws, const int32_t* __restrict__ ids, long long ids_stride,
             const float* __restrict__ w, long long w_stride, int T, int local_off, int e_local,
             const int* __restrict__ n_rows_dev) {
  constexpr int kWords = kChunkTokens / 32;
  constexpr int kPairs = kChunkTokens * kTopK / 1024;   // pairs per thread
  __shared__ uint32_t s_mask[kNumExperts][kWords];
  for (int i = threadIdx.x; i < kNumExperts * kWords; i += blockDim.x) (&s_mask[0][0])[i] = 0u;
  chain_wait();
  chain_release();
  if (n_rows_dev) T = min(T, *n_rows_dev);   // T was the capacity; rows past the count hold nothing
  const int c = blockIdx.x;
  const int t0 = c * kChunkTokens;
  const int k = threadIdx.x % kTopK;
  const int* chunk_base = ws.at<int>(ws.L.chunk_base) + (size_t)c * e_local;
  const int* expert_row0 = ws.at<int>(ws.L.expert_row0);
  int le[kPairs], base[kPairs];
  float wt[kPairs];
#pragma unroll
  for (int j = 0; j < kPairs; ++j) {
    const int t = t0 + (threadIdx.x + j * 1024) / kTopK;
    const int id = t < T ? ids[(size_t)t * ids_stride + k] - local_off : -1;
    le[j] = id >= 0 && id < e_local ? id : -1;
    // a token that names an expert twice is placed once, with the weight of the last one
#pragma unroll
    for (int d = 1; d < kTopK; ++d) {
      const int other = __shfl_down_sync(0xffffffffu, id, d, kTopK);
      if (k + d < kTopK && other == id) le[j] = -1;
    }
    base[j] = 0;
    wt[j] = 0.f;
    if (le[j] >= 0) {
      base[j] = expert_row0[le[j]] + chunk_base[le[j]];
      wt[j] = w[(size_t)t * w_stride + k];
    }
  }
  __syncthreads();   // masks are zero
#pragma unroll
  for (int j = 0; j < kPairs; ++j) {
    const int tl = (threadIdx.x + j * 1024) / kTopK;
    if (le[j] >= 0) atomicOr(&s_mask[le[j]][tl / 32], 1u << (tl % 32));
  }
  __syncthreads();
  int* row_token = ws.at<int>(ws.L.row_token);
  float* row_weight = ws.at<float>(ws.L.row_weight);
  int* tok_rows = ws.at<int>(ws.L.tok_rows);
#pragma unroll
  for (int j = 0; j < kPairs; ++j) {
    const int tl = (threadIdx.x + j * 1024) / kTopK, t = t0 + tl;
    if (t >= T) continue;
    int r = -1;   // "not local"
    if (le[j] >= 0) {
      r = base[j] + __popc(s_mask[le[j]][tl / 32] & ((1u << (tl % 32)) - 1u));
      for (int v = 0; v < tl / 32; ++v) r += __popc(s_mask[le[j]][v]);
      row_token[r] = t;
      row_weight[r] = wt[j];
    }
    tok_rows[(size_t)t * kTopK + k] = r;
  }
}

__global__ void __launch_bounds__(256)
gather_kernel(Workspace ws, const uint8_t* __restrict__ hidden, long long hidden_row_stride,
              const float* __restrict__ hscale, long long sstride_t, long long sstride_kb, int hidden_dim,
              RowSegments segs, __nv_bfloat16* __restrict__ out, long long out_stride, int T,
              const RowSegments* __restrict__ segs_dev, const int* __restrict__ n_rows_dev) {
  const int lane = threadIdx.x & 31;
  const int warps_per_block = blockDim.x >> 5;
  chain_wait();
  chain_release();
  if (segs_dev) segs = *segs_dev;            // the table was built on the device (see launch_ep_segments_pull)
  if (n_rows_dev) T = min(T, *n_rows_dev);
  // The layer's output starts as zeros: GEMM2's epilogue adds every packed row into its token's row, and a
  // token that no local expert took stays exactly 0.  Zeroed here, by all blocks, instead of by a memset
  // of its own (one launch boundary less), unless the grouped GEMM1 does it.
  if (out) {
    const int vec_per_row = hidden_dim / 8;   // 8 bf16 = 16 bytes
    const long long total = (long long)T * vec_per_row;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
      const long long t = i / vec_per_row;
      reinterpret_cast<uint4*>(out + t * out_stride)[i - t * vec_per_row] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  const int rows = ws.at<int>(ws.L.meta)[1];
  const int* row_token = ws.at<int>(ws.L.row_token);
  uint8_t* a_packed = ws.at<uint8_t>(ws.L.a_packed);
  float* a_scale = ws.at<float>(ws.L.a_scale);
  unsigned* row_amax = ws.at<unsigned>(ws.L.row_amax);
  const int m_cap = ws.L.m_cap;
  const int vecs = hidden_dim / 16;
  const int kblocks = hidden_dim / kBlockK;
  for (int m = blockIdx.x * warps_per_block + (threadIdx.x >> 5); m < rows; m += gridDim.x * warps_per_block) {
    int t = row_token[m];
    if (t < 0) continue;
    if (lane == 0) row_amax[m] = 0u;   // GEMM1's epilogue takes the running maximum with atomicMax
    uint4* dst = reinterpret_cast<uint4*>(a_packed + (size_t)m * hidden_dim);
    if (segs.n > 0) {
      // the row is a send row of some rank of the group (payload, then its scales), read where it was packed:
      // plain loads from this GPU's or a peer's memory, so the dispatch and the gather are one pass
      const uint8_t* row = segs.row(t);
      const uint4* src = reinterpret_cast<const uint4*>(row);
      for (int v = lane; v < vecs; v += 32) dst[v] = src[v];
      const float* sc = reinterpret_cast<const float*>(row + hidden_dim);
      for (int kb = lane; kb < kblocks; kb += 32) a_scale[(size_t)kb * m_cap + m] = sc[kb];
      continue;
    }
    const uint4* src = reinterpret_cast<const uint4*>(hidden + (size_t)t * hidden_row_stride);
    for (int v = lane; v < vecs; v += 32) dst[v] = __ldg(src + v);
    for (int kb = lane; kb < kblocks; kb += 32)
      a_scale[(size_t)kb * m_cap + m] = hscale[(size_t)t * sstride_t + (size_t)kb * sstride_kb];
  }
}

}  // namespace

cudaError_t launch_permute(const Workspace& ws, const int32_t* ids, long long ids_stride, const float* w,
                           long long w_stride, const uint8_t* hidden, long long hidden_row_stride,
                           const float* hscale, long long sstride_t, long long sstride_kb, int T, int e_local,
                           int local_off, int hidden_dim, int pad_rows, int num_sms, cudaStream_t stream,
                           bool placed, const RowSegments* segs, void* out_bf16, long long out_row_stride, bool zero_out,
                           const RowSegments* segs_dev, const int* n_rows_dev) {
  const int n_chunks = (T + kChunkTokens - 1) / kChunkTokens;
  cudaError_t err = cudaSuccess;
  if (!placed) {
    err = launch_chained(scan_kernel, dim3(1), dim3(kScanThreads), 0, stream, ws, e_local, n_chunks, pad_rows);
    if (err != cudaSuccess) return err;
  }
  if (n_chunks > 0) {
    if (!placed) {
      err = launch_chained(place_kernel, dim3(n_chunks), dim3(1024), 0, stream, ws, ids, ids_stride, w, w_stride, T,
                           local_off, e_local, n_rows_dev);
      if (err != cudaSuccess) return err;
    }
    // padded rows of this call: at most 8 T pairs plus 127 rows of padding per expert that has any
    const long long pairs = (long long)T * kTopK;
    long long cap_rows = pairs + (long long)(kTileM - 1) * (pairs < e_local ? pairs : e_local);
    if (cap_rows > ws.L.m_cap) cap_rows = ws.L.m_cap;
    int blocks = (int)((cap_rows + 7) / 8);
    int cap = num_sms * 8;
    if (blocks > cap) blocks = cap;
    RowSegments none;
    none.n = 0;
    err = launch_chained(gather_kernel, dim3(blocks), dim3(256), 0, stream, ws, hidden, hidden_row_stride, hscale,
                         sstride_t, sstride_kb, hidden_dim, segs ? *segs : none,
                         reinterpret_cast<__nv_bfloat16*>(zero_out ? out_bf16 : nullptr), out_row_stride, T, segs_dev, n_rows_dev);
  }
  return err;
}

}  // namespace b200moe
