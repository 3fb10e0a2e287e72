// C ABI of the library (declared in include/b200moe.h): argument checks, workspace
// carve-up, TMA descriptors, and the launch sequence of one layer call.
//
// Launch sequence of b200moe_run (all on the caller's stream, nothing allocated):
//   memset counters | route (+histogram) | scan | place | gather | GEMM1(+SwiGLU,+row max)
//   | requant | GEMM2(+row scale * routing weight, each row added into its token's zeroed bf16 output row)
// It replaces the two Python pipelines of the reference
// (solution/python/kernel.py:381-429 and 432-572), which need a host synchronisation
// above 2048 tokens (kernel.py:196); here tile counts stay on the device.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "common.cuh"
#include "kernels.cuh"

using namespace b200moe;

namespace {

thread_local char g_cuda_error[256] = "";

int cuda_fail(cudaError_t e, const char* what) {
  snprintf(g_cuda_error, sizeof(g_cuda_error), "%s: %s", what, cudaGetErrorString(e));
  return B200MOE_ERR_CUDA;
}

#define CUDA_TRY(expr)                                  \
  do {                                                  \
    cudaError_t _e = (expr);                            \
    if (_e != cudaSuccess) return cuda_fail(_e, #expr); \
  } while (0)

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

struct DeviceInfo {
  bool ready = false;
  int num_sms = 0;
};

// Optional cudaEvent_t pair recorded around the GEMM1 launch of this thread's next
// b200moe_experts call (then forgotten); lets a benchmark time the dominant kernel in place.
thread_local cudaEvent_t g_prof_start = nullptr;
thread_local cudaEvent_t g_prof_stop = nullptr;

// Optional host-mapped int32[4] of this thread's calls: a kernel that gives up on a bounded wait copies the
// status word there, so a host can notice without a device-to-host copy per call.
thread_local int* g_status_mirror = nullptr;

std::mutex g_mutex;
EncodeTiledFn g_encode = nullptr;
DeviceInfo g_dev[64];

// Once per process: the driver entry point for tensor-map encoding; once per device: the
// SM count and the opt-in shared memory sizes of the GEMM kernels.
int ensure_device(int* num_sms) {
  int dev = 0;
  CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return B200MOE_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(g_mutex);
  if (!g_encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    CUDA_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
    if (qres != cudaDriverEntryPointSuccess || !fn) {
      snprintf(g_cuda_error, sizeof(g_cuda_error), "cuTensorMapEncodeTiled not available from this driver");
      return B200MOE_ERR_CUDA;
    }
    g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  if (!g_dev[dev].ready) {
    cudaDeviceProp prop;
    CUDA_TRY(cudaGetDeviceProperties(&prop, dev));
    if (prop.major != 10) {
      snprintf(g_cuda_error, sizeof(g_cuda_error), "device %d is sm_%d%d; this library is built for sm_100a only",
               dev, prop.major, prop.minor);
      return B200MOE_ERR_CUDA;
    }
    g_dev[dev].num_sms = prop.multiProcessorCount;
    CUDA_TRY(configure_grouped_gemm());
    CUDA_TRY(configure_stream_gemm());
    g_dev[dev].ready = true;
  }
  *num_sms = g_dev[dev].num_sms;
  return B200MOE_OK;
}

// Bytes in boxes with 128-byte swizzle.
int encode_tmap(CUtensorMap* map, const void* base, uint32_t rank, const cuuint64_t* dims, const cuuint64_t* strides,
                const cuuint32_t* box) {
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(g_cuda_error, sizeof(g_cuda_error), "cuTensorMapEncodeTiled (%uD) failed with CUresult %d", rank, (int)r);
    return B200MOE_ERR_CUDA;
  }
  return B200MOE_OK;
}

// rows x K e4m3 matrix, row pitch `pitch` bytes; box = box_rows x 128 bytes, 128-byte swizzle.
int make_tmap(CUtensorMap* map, const void* base, uint64_t rows, uint64_t k, uint64_t pitch, uint32_t box_rows) {
  cuuint64_t dims[2] = {k, rows};
  cuuint64_t strides[1] = {pitch};
  cuuint32_t box[2] = {(cuuint32_t)kBlockK, box_rows};
  return encode_tmap(map, base, 2, dims, strides, box);
}

// GEMM1 weights [e_local][2*inter][k] seen as planes: plane 2e holds expert e's gate rows, plane
// 2e+1 its up rows.  One box = the same `box_rows` rows of two consecutive planes (gate rows,
// then the matching up rows), 128 bytes of K wide, 128-byte swizzle: one TMA operation
// instead of two per K block (a box costs the issuing thread and the TMA unit a few hundred
// cycles whatever its size).
int make_tmap_gate_up(CUtensorMap* map, const void* base, uint64_t e_local, uint64_t inter, uint64_t k,
                      uint32_t box_rows) {
  cuuint64_t dims[3] = {k, inter, 2 * e_local};
  cuuint64_t strides[2] = {k, inter * k};
  cuuint32_t box[3] = {(cuuint32_t)kBlockK, box_rows, 2};
  return encode_tmap(map, base, 3, dims, strides, box);
}

// The same with the K blocks as a dimension of their own (128 bytes apart), so that one box brings `box_kb` K blocks, each
// as a swizzled tile behind the other: rows x K, and the gate and up planes of GEMM1.
int make_tmap_kblocks(CUtensorMap* map, const void* base, uint64_t rows, uint64_t k, uint32_t box_rows, uint32_t box_kb) {
  cuuint64_t dims[3] = {(cuuint64_t)kBlockK, rows, k / kBlockK};
  cuuint64_t strides[2] = {k, (cuuint64_t)kBlockK};
  cuuint32_t box[3] = {(cuuint32_t)kBlockK, box_rows, box_kb};
  return encode_tmap(map, base, 3, dims, strides, box);
}
int make_tmap_gate_up_kblocks(CUtensorMap* map, const void* base, uint64_t e_local, uint64_t inter, uint64_t k,
                              uint32_t box_rows, uint32_t box_kb) {
  cuuint64_t dims[4] = {(cuuint64_t)kBlockK, inter, 2 * e_local, k / kBlockK};
  cuuint64_t strides[3] = {k, inter * k, (cuuint64_t)kBlockK};
  cuuint32_t box[4] = {(cuuint32_t)kBlockK, box_rows, 2, box_kb};
  return encode_tmap(map, base, 4, dims, strides, box);
}

uint64_t align_up(uint64_t x, uint64_t a) { return (x + a - 1) / a * a; }

constexpr long long kZeroInGemmBytes = 126ll << 20;   // L2
constexpr int kZeroInGemmExperts = 4;
constexpr int kDirectRowsMaxTokens = 8;   // largest call whose decode GEMM1 reads the caller's rows in place

// Decode-size calls (up to 16 tokens) requantise inside GEMM1 (B200MOE_DECODE=0 turns that off, B200MOE_DECODE=64
// extends it to 64 tokens).  Above 16 tokens the pass of its own is the default: the CTA that stores an expert's last slab
// turns up to 64 rows into codes alone, which takes longer than the launch it saves once experts hold more than a few rows.  us a
// call, pass / inside GEMM1 (32 experts): 17 tokens, 5 active experts 81.9 / 79.9, 8 active 98.3 / 102.4; 56 tokens, 14 active
// 147.5 / 149.5, 17 active 163.9 / 170.0; a Zipf load 17 tokens 108.5 / 120.8, 32 tokens 112.6 / 137.2, 64 tokens 116.8 / 170.0.
// Returns the token tile of the streaming kernels for such a call, or 0.
int decode_tile(int T) {
  static const bool decode_on = [] {
    const char* v = getenv("B200MOE_DECODE");
    return !(v && v[0] == '0');
  }();
  static const int decode_max_t = [] {
    const char* v = getenv("B200MOE_DECODE");
    return (v && v[0] == '6') ? 64 : 16;
  }();
  return (decode_on && T <= decode_max_t) ? (T <= 16 ? 16 : 64) : 0;
}

// Calls above the decode sizes and up to this many tokens take the weight-streaming GEMMs if few enough experts are local.
// The 128 x 256 tiles of the grouped kernel come in whole waves of SMs: with some ten to twenty active experts (two waves
// of GEMM1 items) the second is mostly idle, with more than a hundred it does not matter and the grouped kernel's larger
// boxes win.  us a call, grouped / streaming: 32 experts, 17 tokens on 8 active 104.5 / 98.3, 20 on 10 137.2 / 116.8, 33 on 17
// 172.1 / 163.9, 56 on 14 153.7 / 147.5, 64 on 19 204.8 / 180.3; 64 experts, 33 tokens on 28 270.4 / 239.6, 64 on 34 288.8 /
// 278.6; 256 experts, 64 tokens 915 / 945.  A Zipf load, all rows on nine experts: 17 tokens 110.7 / 108.5, 32 tokens 114.8 /
// 112.6, 40 tokens 114.7 / 114.7, 48 to 60 tokens 114.8 / 116.7, 64 tokens 116.7 / 116.8.  (Between 64 and 256 experts nothing was
// measured; they keep the grouped kernels.)  B200MOE_STREAM=0: never.
constexpr int kStreamMaxTokens = 64;
constexpr int kStreamMaxExperts = 64;
// Returns the most token rows of a tile (an expert of a call of at most 64 tokens has no more), or 0 for the grouped kernels.
int stream_tile(int T, int e_local) {
  static const bool on = [] {
    const char* v = getenv("B200MOE_STREAM");
    return !(v && v[0] == '0');
  }();
  // (smaller calls have no scratch for 64 token rows: they stream with decode_tile or not at all)
  return on && T > 16 && T <= kStreamMaxTokens && e_local <= kStreamMaxExperts ? 64 : 0;
}

int shape_ok(int T, int e_local, int hidden, int inter) {
  if (T < 0 || e_local < 1) return B200MOE_ERR_INVALID_ARGUMENT;
  if (e_local > kNumExperts || hidden < 256 || hidden % 256 != 0 || inter < 128 || inter % 128 != 0)
    return B200MOE_ERR_UNSUPPORTED_SHAPE;
  if ((long long)T * kTopK > (1ll << 30)) return B200MOE_ERR_UNSUPPORTED_SHAPE;
  // the GEMMs keep one weight scale per K block of an item in shared-memory panels
  if (hidden / kBlockK > grouped_gemm_max_kblocks() || inter / kBlockK > grouped_gemm_max_kblocks())
    return B200MOE_ERR_UNSUPPORTED_SHAPE;
  return B200MOE_OK;
}

void compute_layout(int T, int e_local, int hidden, int inter, b200moe_ws_layout* L) {
  memset(L, 0, sizeof(*L));
  const int n_chunks = T > 0 ? (T + kChunkTokens - 1) / kChunkTokens : 1;
  const long long pairs = (long long)T * (e_local < kTopK ? e_local : kTopK);
  // every expert segment is padded to a whole 128-row M tile; m_cap stays a multiple of 256
  const long long m_cap = (long long)align_up((uint64_t)pairs, 2 * kTileM) + (long long)2 * kTileM * e_local;
  L->m_cap = (int32_t)m_cap;
  L->max_tiles = (int32_t)(m_cap / kTileM);
  L->n_chunks = n_chunks;
  L->chunk_tokens = kChunkTokens;
  uint64_t off = 0;
  auto take = [&](uint64_t bytes) { uint64_t o = off; off = align_up(off + bytes, 256); return o; };
  L->status = take(16 * 4);
  L->meta = take(8 * 4);
  L->splitk_count = take(2 * kStreamMaxCtas * 4);   // inside the range that clear_counters() zeroes
  L->tile_done = take((uint64_t)L->max_tiles * 4);   // likewise
  L->chunk_counts = take((uint64_t)n_chunks * e_local * 4);
  L->chunk_base = take((uint64_t)n_chunks * e_local * 4);
  L->expert_count = take((uint64_t)e_local * 4);
  L->expert_row0 = take((uint64_t)(e_local + 1) * 4);
  L->tile_expert = take((uint64_t)L->max_tiles * 4);
  L->row_token = take((uint64_t)m_cap * 4);
  L->row_weight = take((uint64_t)m_cap * 4);
  L->a_packed = take((uint64_t)m_cap * hidden);
  L->a_scale = take((uint64_t)(hidden / kBlockK) * m_cap * 4);
  L->act = take((uint64_t)m_cap * inter * 2);
  L->row_amax = take((uint64_t)m_cap * 4);
  L->act_q = take((uint64_t)m_cap * inter);
  L->row_scale = take((uint64_t)m_cap * 4);
  L->tok_rows = take((uint64_t)(T > 0 ? T : 1) * kTopK * 4);
  L->topk_ids = take((uint64_t)(T > 0 ? T : 1) * kTopK * 4);
  L->topk_w = take((uint64_t)(T > 0 ? T : 1) * kTopK * 4);
  L->trace = take(2 * 8 * 64 * 8);   // room for one-off probes: absolute cycle stamps of CTA 0's first 64 K blocks
  // two cut tiles per CTA of the streaming GEMMs: 2.5 MiB at decode sizes, 10 MiB (64 token rows) up to kStreamMaxTokens, above
  // which no call streams
  const int stream_rows = T <= 16 ? 16 : T <= kStreamMaxTokens ? 64 : 0;
  L->splitk_scratch = take((uint64_t)2 * kStreamMaxCtas * stream_rows * 128 * 4);
  L->ep_segments = take(256);   // RowSegments at +0, int32 row count at +192 (b200moe_ep_local_experts)
  L->total_bytes = off;
  if (T > kStreamMaxTokens) {   // a workspace for so many tokens holds every smaller call, the largest that streams among them
    b200moe_ws_layout at_limit;
    compute_layout(kStreamMaxTokens, e_local, hidden, inter, &at_limit);
    if (at_limit.total_bytes > off) L->total_bytes = at_limit.total_bytes;
  }
}

int bind_workspace(int T, int e_local, int hidden, int inter, void* workspace, size_t bytes, Workspace* ws) {
  int rc = shape_ok(T, e_local, hidden, inter);
  if (rc != B200MOE_OK) return rc;
  if (!workspace) return B200MOE_ERR_INVALID_ARGUMENT;
  if (reinterpret_cast<uintptr_t>(workspace) % 256 != 0) return B200MOE_ERR_MISALIGNED;
  compute_layout(T, e_local, hidden, inter, &ws->L);
  if (bytes < ws->L.total_bytes) return B200MOE_ERR_WORKSPACE_TOO_SMALL;
  ws->base = reinterpret_cast<uint8_t*>(workspace);
  return B200MOE_OK;
}

// K blocks of a box of the streaming kernels
uint32_t group_kblocks(int k) { return k / kBlockK < kStreamGroup ? k / kBlockK : kStreamGroup; }

// What the streaming kernels take beside a GEMM's ordinary arguments: the packed rows ([m_cap][k] at `rows_off`) in boxes
// of 16 rows and, where a tile may hold more (`nt` 64), 32 and 64.  Only what the kernel reads is encoded: a map costs the host a
// good part of a microsecond, and a call at new addresses pays for each.
int make_stream_params(StreamParams* sp, const GemmParams& g, const Workspace& ws, uint64_t rows_off, int k, int nt) {
  memset(sp, 0, sizeof(*sp));
  sp->g = g;
  sp->expert_row0 = ws.at<int>(ws.L.expert_row0);
  const int n_maps = g.direct_a ? 0 : nt <= 16 ? 1 : 3;
  for (int c = 0; c < n_maps; ++c) {
    const int rc = make_tmap_kblocks(&sp->tmap_tok[c], ws.base + rows_off, (uint64_t)ws.L.m_cap, (uint64_t)k, 16u << c,
                                     group_kblocks(k));
    if (rc != B200MOE_OK) return rc;
  }
  return B200MOE_OK;
}

// Clears the status word and the histogram (start of a layer call).
int clear_counters(const Workspace& ws, int e_local, cudaStream_t stream) {
  // status, meta, splitk_count, tile_done, chunk_counts are adjacent: one memset covers them
  size_t bytes = (size_t)(ws.L.chunk_counts - ws.L.status) + (size_t)ws.L.n_chunks * e_local * 4;
  CUDA_TRY(cudaMemsetAsync(ws.base + ws.L.status, 0, bytes, stream));
  return B200MOE_OK;
}

}  // namespace

extern "C" {

int b200moe_version(void) { return 1; }

const char* b200moe_status_string(int status) {
  switch (status) {
    case B200MOE_OK: return "ok";
    case B200MOE_ERR_INVALID_ARGUMENT: return "invalid argument";
    case B200MOE_ERR_UNSUPPORTED_SHAPE: return "unsupported shape";
    case B200MOE_ERR_WORKSPACE_TOO_SMALL: return "workspace too small";
    case B200MOE_ERR_CUDA: return "CUDA call failed";
    case B200MOE_ERR_DEVICE_TIMEOUT: return "a bounded device-side wait timed out";
    case B200MOE_ERR_MISALIGNED: return "misaligned pointer or stride";
    default: return "unknown status";
  }
}

const char* b200moe_last_cuda_error(void) { return g_cuda_error; }

int b200moe_workspace_layout(int T, int e_local, int hidden, int inter, b200moe_ws_layout* layout) {
  int rc = shape_ok(T, e_local, hidden, inter);
  if (rc != B200MOE_OK) return rc;
  b200moe_ws_layout L;
  compute_layout(T, e_local, hidden, inter, &L);
  if (layout) *layout = L;
  return B200MOE_OK;
}

int b200moe_set_status_mirror(void* host_mapped_int4) {
  g_status_mirror = reinterpret_cast<int*>(host_mapped_int4);
  return B200MOE_OK;
}

int b200moe_profile_next_gemm1(void* start_event, void* stop_event) {
  g_prof_start = reinterpret_cast<cudaEvent_t>(start_event);
  g_prof_stop = reinterpret_cast<cudaEvent_t>(stop_event);
  return B200MOE_OK;
}

int b200moe_launches_per_run(int T, int e_local) {
  (void)e_local;
  if (T <= 0) return 0;
  const char* front = getenv("B200MOE_FRONT");
  const bool fused_front = T <= kFrontSmallMaxTokens && !(front && front[0] == '0');
  // route, scan, place, gather, gemm1, requant, gemm2 (+ weighted unpermute / reduce into the output); calls of at
  // most 32 tokens fuse the first three, the decode GEMM1 (at most 16 tokens) also requantises
  static const bool decode_on = [] {
    const char* v = getenv("B200MOE_DECODE");
    return !(v && v[0] == '0');
  }();
  static const int decode_max_t = [] {
    const char* v = getenv("B200MOE_DECODE");
    return (v && v[0] == '6') ? 64 : 16;
  }();
  const int requant = (decode_on && T <= decode_max_t) ? 0 : 1;   // decode GEMM1 requantises by itself
  // ... and, behind the fused front kernel, fetches the token rows itself: no gather pass (three launches)
  const int gather = (fused_front && decode_on && T <= kDirectRowsMaxTokens) ? 0 : 1;
  return (fused_front ? 3 : 5) + gather + requant;
}

int b200moe_route(const void* logits, int logits_dtype, const void* bias, int bias_dtype, int T,
                  float routed_scaling_factor, int local_expert_offset, int e_local, int hidden, int inter,
                  int32_t* topk_ids, float* topk_w, void* workspace, size_t workspace_bytes, void* stream) {
  if (!logits || !bias || !topk_ids || !topk_w) return B200MOE_ERR_INVALID_ARGUMENT;
  if ((logits_dtype != B200MOE_F32 && logits_dtype != B200MOE_BF16) ||
      (bias_dtype != B200MOE_F32 && bias_dtype != B200MOE_BF16))
    return B200MOE_ERR_INVALID_ARGUMENT;
  if (local_expert_offset < 0 || local_expert_offset + e_local > kNumExperts) return B200MOE_ERR_INVALID_ARGUMENT;
  Workspace ws;
  int rc = bind_workspace(T, e_local, hidden, inter, workspace, workspace_bytes, &ws);
  if (rc != B200MOE_OK) return rc;
  int num_sms = 0;
  if ((rc = ensure_device(&num_sms)) != B200MOE_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if ((rc = clear_counters(ws, e_local, st)) != B200MOE_OK) return rc;
  CUDA_TRY(launch_route(logits, logits_dtype, bias, bias_dtype, T, routed_scaling_factor, local_expert_offset, e_local,
                        topk_ids, topk_w, ws.at<int>(ws.L.chunk_counts), num_sms, st));
  return B200MOE_OK;
}

int b200moe_count(const int32_t* topk_ids, int64_t ids_row_stride, int T, int local_expert_offset, int e_local,
                  int hidden, int inter, void* workspace, size_t workspace_bytes, void* stream) {
  if (!topk_ids || ids_row_stride < kTopK) return B200MOE_ERR_INVALID_ARGUMENT;
  if (local_expert_offset < 0 || local_expert_offset + e_local > kNumExperts) return B200MOE_ERR_INVALID_ARGUMENT;
  Workspace ws;
  int rc = bind_workspace(T, e_local, hidden, inter, workspace, workspace_bytes, &ws);
  if (rc != B200MOE_OK) return rc;
  int num_sms = 0;
  if ((rc = ensure_device(&num_sms)) != B200MOE_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if ((rc = clear_counters(ws, e_local, st)) != B200MOE_OK) return rc;
  CUDA_TRY(launch_count(topk_ids, ids_row_stride, T, local_expert_offset, e_local, ws.at<int>(ws.L.chunk_counts),
                        num_sms, st));
  return B200MOE_OK;
}

// `placed`: routing, scan and placement of this call already ran as one kernel (front_small.cu).
static int experts_impl(const int32_t* topk_ids, int64_t ids_row_stride, const float* topk_w, int64_t w_row_stride,
                        const uint8_t* hidden_states, int64_t hidden_row_stride, const float* hidden_scale,
                        int64_t scale_stride_t, int64_t scale_stride_kb, const uint8_t* w1, const float* w1_scale,
                        const uint8_t* w2, const float* w2_scale, int T, int e_local, int local_expert_offset,
                        int hidden, int inter, void* workspace, size_t workspace_bytes, void* out_bf16,
                        int64_t out_row_stride, void* stream, bool placed, const RowSegments* segs = nullptr,
                        const RowSegments* segs_dev = nullptr, const int* n_rows_dev = nullptr) {
  // The event pair armed by b200moe_profile_next_gemm1 is for this call only: forget it on every
  // way out (the GEMM1 launch below consumes it first when the call gets that far).
  struct DisarmProfile {
    ~DisarmProfile() { g_prof_start = g_prof_stop = nullptr; }
  } disarm_profile;
  if (!topk_ids || !topk_w || !w1 || !w1_scale || !w2 || !w2_scale) return B200MOE_ERR_INVALID_ARGUMENT;
  if (T > 0 && ((!segs && !segs_dev && (!hidden_states || !hidden_scale)) || !out_bf16))
    return B200MOE_ERR_INVALID_ARGUMENT;
  if (segs || segs_dev) {   // rows are read from the segments: no separate payload / scale arrays
    hidden_row_stride = hidden;
    hidden_states = nullptr;
  }
  if (ids_row_stride < kTopK || w_row_stride < kTopK) return B200MOE_ERR_INVALID_ARGUMENT;
  if (local_expert_offset < 0 || local_expert_offset + e_local > kNumExperts) return B200MOE_ERR_INVALID_ARGUMENT;
  Workspace ws;
  int rc = bind_workspace(T, e_local, hidden, inter, workspace, workspace_bytes, &ws);
  if (rc != B200MOE_OK) return rc;
  if (hidden_row_stride < hidden || hidden_row_stride % 16 != 0 ||
      reinterpret_cast<uintptr_t>(hidden_states) % 16 != 0 || reinterpret_cast<uintptr_t>(w1) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(w2) % 16 != 0 || reinterpret_cast<uintptr_t>(out_bf16) % 16 != 0 ||
      out_row_stride < hidden || out_row_stride % 8 != 0)
    return B200MOE_ERR_MISALIGNED;
  if (T == 0) return B200MOE_OK;
  int num_sms = 0;
  if ((rc = ensure_device(&num_sms)) != B200MOE_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);

  const bool fits = stream_gemm_fits(hidden / kBlockK, ws.L.max_tiles, num_sms) &&
                    stream_gemm_fits(inter / kBlockK, ws.L.max_tiles, num_sms);
  const int nt = fits ? decode_tile(T) : 0;                      // > 0: GEMM1 also requantises
  const int slab_nt = nt ? nt : (fits ? stream_tile(T, e_local) : 0);     // > 0: the streaming kernels (slabs of 128 weight rows)
  // A call of at most 8 tokens that the one-block front kernel routed and placed runs no gather pass: its GEMM1
  // fetches the token rows and their scales where the caller keeps them (and zeroes the output rows).  Measured
  // with inputs cold in HBM: -4 us at 1 token, -2 at 4, but +2..4 at 16 tokens with 4 rows (56 separate 128-byte
  // pieces per row instead of one coalesced pass), hence the limit.
  const bool direct_a = placed && nt == 16 && T <= kDirectRowsMaxTokens && !segs && !segs_dev;
  // The output rows, which GEMM2's epilogue adds into, are zeroed by the gather pass; by GEMM1 without a gather pass, and by
  // the grouped GEMM1 when the output is larger than L2 and in one piece, and more than three experts are local.  Below the size
  // of L2 the zeros stay there until GEMM2 and cost the gather little (901 tokens: gather 223, GEMM1 228 us a call; 8192 rows of
  // an expert-parallel rank 857, 864).  With few local experts GEMM1 is too short to hide 148 CTAs' stores behind its K
  // loops, and a padded row stride takes a division per 16 bytes.  us a call zeroed by the gather pass / GEMM1, output in one piece:
  // 1 expert, 14107 tokens 124.9 / 137.2, 30001 tokens 192.5 / 210.9; 2: 139.3 / 141.3, 204.8 / 213.0; 3: 143.4 / 149.5,
  // 213.0 / 215.2; 4: 249.9 / 245.8, 440.3 / 423.9; 8: 311.3 / 309.3, 591.9 / 583.7; 32: 964.6 / 948.1; 64: 1716 / 1700.
  // Padded rows, 14107 tokens: 1 expert 124.9 / 155.6; 4: 251.9 / 264.2; 32: 950.3 / 956.5; 64: 1718 / 1739.
  const bool zero_in_gemm = !slab_nt && (long long)T * hidden * 2 > kZeroInGemmBytes && e_local >= kZeroInGemmExperts &&
                            out_row_stride == hidden;
  if (!direct_a)
    CUDA_TRY(launch_permute(ws, topk_ids, ids_row_stride, topk_w, w_row_stride, hidden_states, hidden_row_stride,
                            hidden_scale, scale_stride_t, scale_stride_kb, T, e_local, local_expert_offset, hidden,
                            kTileM, num_sms, st, placed, segs, out_bf16, out_row_stride, !zero_in_gemm, segs_dev,
                            n_rows_dev));

  GemmParams g1;
  memset(&g1, 0, sizeof(g1));
  if (direct_a) {   // the caller's rows, one row per box
    if ((rc = make_tmap(&g1.tmap_a, hidden_states, (uint64_t)T, (uint64_t)hidden, (uint64_t)hidden_row_stride, 1)) !=
        B200MOE_OK)
      return rc;
  } else if (!slab_nt && (rc = make_tmap(&g1.tmap_a, ws.base + ws.L.a_packed, (uint64_t)ws.L.m_cap, (uint64_t)hidden,
                                         (uint64_t)hidden, kTileM)) != B200MOE_OK) {
    return rc;
  }
  // one box = 128 gate rows + the matching 128 up rows (streaming kernels: 64 + 64, a group of K blocks)
  rc = slab_nt ? make_tmap_gate_up_kblocks(&g1.tmap_b, w1, (uint64_t)e_local, (uint64_t)inter, (uint64_t)hidden, 64,
                                           group_kblocks(hidden))
               : make_tmap_gate_up(&g1.tmap_b, w1, (uint64_t)e_local, (uint64_t)inter, (uint64_t)hidden, 128);
  if (rc != B200MOE_OK) return rc;
  g1.meta = ws.at<int>(ws.L.meta);
  g1.tile_expert = ws.at<int>(ws.L.tile_expert);
  g1.row_token = ws.at<int>(ws.L.row_token);
  g1.a_scale = ws.at<float>(ws.L.a_scale);
  g1.b_scale = w1_scale;
  g1.m_cap = ws.L.m_cap;
  g1.n_per_expert = 2 * inter;
  g1.kblocks = hidden / kBlockK;
  g1.n_tiles = slab_nt ? inter / 64 : inter / 128;
  g1.expert_count = ws.at<int>(ws.L.expert_count);
  g1.inter = inter;
  g1.hidden = hidden;
  g1.act = ws.at<__half>(ws.L.act);
  g1.row_amax = ws.at<unsigned>(ws.L.row_amax);
  g1.tile_done = nt ? ws.at<int>(ws.L.tile_done) : nullptr;
  g1.act_q_out = ws.at<uint8_t>(ws.L.act_q);
  g1.row_scale_out = ws.at<float>(ws.L.row_scale);
  g1.direct_a = direct_a ? 1 : 0;
  g1.zero_tokens = direct_a || zero_in_gemm ? T : 0;
  g1.zero_rows_dev = n_rows_dev;
  g1.out = reinterpret_cast<__nv_bfloat16*>(out_bf16);
  g1.out_stride = out_row_stride;
  g1.hscale = hidden_scale;
  g1.hs_stride_t = scale_stride_t;
  g1.hs_stride_kb = scale_stride_kb;
  g1.status = ws.at<int>(ws.L.status);
  g1.status_mirror = g_status_mirror;
  g1.splitk_scratch = ws.at<float>(ws.L.splitk_scratch);
  g1.splitk_count = ws.at<int>(ws.L.splitk_count);
  // B200MOE_PROF=1: CTA 0 writes its cycle counters into the padding after `meta` (GEMM1: 10 x u64 at meta+32, GEMM2: at
  // meta+136; the last word tells the streaming kernels' from the grouped ones'); cleared with the counters each call.
  static const bool prof_on = getenv("B200MOE_PROF") != nullptr;
  g1.prof = prof_on ? ws.at<unsigned long long>(ws.L.meta + 32) : nullptr;
  if (g_prof_start) CUDA_TRY(cudaEventRecord(g_prof_start, st));
  {
    cudaError_t le;
    if (slab_nt) {
      StreamParams s1;
      if ((rc = make_stream_params(&s1, g1, ws, ws.L.a_packed, hidden, slab_nt)) != B200MOE_OK) return rc;
      le = launch_stream_gemm(1, slab_nt, s1, ws.L.max_tiles, num_sms, st);
    } else {
      le = launch_grouped_gemm(1, g1, num_sms, st);
    }
    cudaEvent_t stop = g_prof_stop;
    g_prof_start = g_prof_stop = nullptr;   // one shot, whatever happens next
    if (le != cudaSuccess) return cuda_fail(le, "GEMM1 launch");
    if (stop) CUDA_TRY(cudaEventRecord(stop, st));
  }

  // decode sizes requantise inside GEMM1 (the CTA that stores an expert's last weight slab); the 128-row tiles
  // need a pass of their own (see gemm.cu)
  if (!nt) CUDA_TRY(launch_requant(ws, inter, num_sms, st));

  GemmParams g2;
  memset(&g2, 0, sizeof(g2));
  if (!slab_nt &&
      (rc = make_tmap(&g2.tmap_a, ws.base + ws.L.act_q, (uint64_t)ws.L.m_cap, (uint64_t)inter, (uint64_t)inter,
                      kTileM)) != B200MOE_OK)
    return rc;
  // the whole B tile (or the 128-row slab of a group of K blocks) in one box
  rc = slab_nt ? make_tmap_kblocks(&g2.tmap_b, w2, (uint64_t)e_local * hidden, (uint64_t)inter, 128, group_kblocks(inter))
               : make_tmap(&g2.tmap_b, w2, (uint64_t)e_local * hidden, (uint64_t)inter, (uint64_t)inter, 256);
  if (rc != B200MOE_OK) return rc;
  g2.meta = g1.meta;
  g2.tile_expert = g1.tile_expert;
  g2.row_token = g1.row_token;
  g2.b_scale = w2_scale;
  g2.m_cap = ws.L.m_cap;
  g2.n_per_expert = hidden;
  g2.kblocks = inter / kBlockK;
  g2.n_tiles = slab_nt ? hidden / 128 : hidden / 256;
  g2.expert_count = g1.expert_count;
  g2.inter = inter;
  g2.hidden = hidden;
  g2.row_scale = ws.at<float>(ws.L.row_scale);
  g2.row_weight = ws.at<float>(ws.L.row_weight);
  g2.out = reinterpret_cast<__nv_bfloat16*>(out_bf16);
  g2.out_stride = out_row_stride;
  g2.status = g1.status;
  g2.status_mirror = g1.status_mirror;
  g2.splitk_scratch = g1.splitk_scratch;
  g2.splitk_count = g1.splitk_count + kStreamMaxCtas;
  g2.prof = prof_on ? ws.at<unsigned long long>(ws.L.meta + 136) : nullptr;
  if (slab_nt) {
    StreamParams s2;
    if ((rc = make_stream_params(&s2, g2, ws, ws.L.act_q, inter, slab_nt)) != B200MOE_OK) return rc;
    CUDA_TRY(launch_stream_gemm(2, slab_nt, s2, ws.L.max_tiles, num_sms, st));
  } else {
    CUDA_TRY(launch_grouped_gemm(2, g2, num_sms, st));
  }

  // nothing follows GEMM2: its epilogue added every packed row into its token's output row
  return B200MOE_OK;
}

int b200moe_experts(const int32_t* topk_ids, int64_t ids_row_stride, const float* topk_w, int64_t w_row_stride,
                    const uint8_t* hidden_states, int64_t hidden_row_stride, const float* hidden_scale,
                    int64_t scale_stride_t, int64_t scale_stride_kb, const uint8_t* w1, const float* w1_scale,
                    const uint8_t* w2, const float* w2_scale, int T, int e_local, int local_expert_offset,
                    int hidden, int inter, void* workspace, size_t workspace_bytes, void* out_bf16,
                    int64_t out_row_stride, void* stream) {
  return experts_impl(topk_ids, ids_row_stride, topk_w, w_row_stride, hidden_states, hidden_row_stride, hidden_scale,
                      scale_stride_t, scale_stride_kb, w1, w1_scale, w2, w2_scale, T, e_local, local_expert_offset,
                      hidden, inter, workspace, workspace_bytes, out_bf16, out_row_stride, stream, false);
}

int b200moe_run(const void* logits, int logits_dtype, const void* bias, int bias_dtype, const uint8_t* hidden_states,
                int64_t hidden_row_stride, const float* hidden_scale, int64_t scale_stride_t,
                int64_t scale_stride_kb, const uint8_t* w1, const float* w1_scale, const uint8_t* w2,
                const float* w2_scale, int T, int e_local, int local_expert_offset, float routed_scaling_factor,
                int hidden, int inter, void* workspace, size_t workspace_bytes, void* out_bf16,
                int64_t out_row_stride, void* stream) {
  Workspace ws;
  int rc = bind_workspace(T, e_local, hidden, inter, workspace, workspace_bytes, &ws);
  if (rc != B200MOE_OK) return rc;
  if (T == 0) return B200MOE_OK;
  int32_t* ids = ws.at<int32_t>(ws.L.topk_ids);
  float* w = ws.at<float>(ws.L.topk_w);
  // Decode-size calls: routing, scan and placement in one block (B200MOE_FRONT=0: the separate kernels).
  static const bool front_on = [] {
    const char* v = getenv("B200MOE_FRONT");
    return !(v && v[0] == '0');
  }();
  if (front_on && T <= kFrontSmallMaxTokens) {
    if (!logits || !bias) return B200MOE_ERR_INVALID_ARGUMENT;
    if ((logits_dtype != B200MOE_F32 && logits_dtype != B200MOE_BF16) ||
        (bias_dtype != B200MOE_F32 && bias_dtype != B200MOE_BF16))
      return B200MOE_ERR_INVALID_ARGUMENT;
    if (local_expert_offset < 0 || local_expert_offset + e_local > kNumExperts) return B200MOE_ERR_INVALID_ARGUMENT;
    int num_sms = 0;
    if ((rc = ensure_device(&num_sms)) != B200MOE_OK) return rc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // (no memset: this kernel clears the call's counters itself)
    CUDA_TRY(launch_route_place_small(ws, logits, logits_dtype, bias, bias_dtype, T, routed_scaling_factor,
                                      local_expert_offset, e_local, kTileM, st));
    return experts_impl(ids, kTopK, w, kTopK, hidden_states, hidden_row_stride, hidden_scale, scale_stride_t,
                        scale_stride_kb, w1, w1_scale, w2, w2_scale, T, e_local, local_expert_offset, hidden, inter,
                        workspace, workspace_bytes, out_bf16, out_row_stride, stream, true);
  }
  rc = b200moe_route(logits, logits_dtype, bias, bias_dtype, T, routed_scaling_factor, local_expert_offset, e_local,
                     hidden, inter, ids, w, workspace, workspace_bytes, stream);
  if (rc != B200MOE_OK) return rc;
  return b200moe_experts(ids, kTopK, w, kTopK, hidden_states, hidden_row_stride, hidden_scale, scale_stride_t,
                         scale_stride_kb, w1, w1_scale, w2, w2_scale, T, e_local, local_expert_offset, hidden, inter,
                         workspace, workspace_bytes, out_bf16, out_row_stride, stream);
}

int b200moe_read_status(const void* workspace, void* stream, int32_t* detail) {
  if (!workspace) return B200MOE_ERR_INVALID_ARGUMENT;
  int32_t host[4] = {0, 0, 0, 0};
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUDA_TRY(cudaMemcpyAsync(host, workspace, sizeof(host), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(cudaStreamSynchronize(st));
  if (detail) memcpy(detail, host, sizeof(host));
  return host[kStatusCode];
}

int b200moe_selftest_wait_timeout(void* status_int4, void* stream) {
  if (!status_int4) return B200MOE_ERR_INVALID_ARGUMENT;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUDA_TRY(cudaMemsetAsync(status_int4, 0, 16, st));
  CUDA_TRY(launch_wait_timeout_selftest(reinterpret_cast<int*>(status_int4), st));
  return B200MOE_OK;
}

int b200moe_ep_pack(const int32_t* topk_ids, const float* topk_w, const uint8_t* hidden_states,
                    int64_t hidden_row_stride, const float* hidden_scale, int64_t scale_stride_t,
                    int64_t scale_stride_kb, int T, int hidden, int world, uint8_t* send_rows, int32_t* dest_counts,
                    int32_t* send_slot, void* stream) {
  if (!dest_counts || T < 0) return B200MOE_ERR_INVALID_ARGUMENT;
  if (T > 0 && (!topk_ids || !topk_w || !send_rows || !send_slot || !hidden_states || !hidden_scale))
    return B200MOE_ERR_INVALID_ARGUMENT;   // an empty batch may come with null (zero-sized) buffers
  if (world != 1 && world != 2 && world != 4 && world != 8) return B200MOE_ERR_UNSUPPORTED_SHAPE;
  if (hidden < 512 || hidden % 512 != 0) return B200MOE_ERR_UNSUPPORTED_SHAPE;   // keeps send rows 16-byte aligned
  if (hidden_row_stride % 16 != 0 || reinterpret_cast<uintptr_t>(hidden_states) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(send_rows) % 16 != 0)
    return B200MOE_ERR_MISALIGNED;
  int num_sms = 0;
  int rc = ensure_device(&num_sms);
  if (rc != B200MOE_OK) return rc;
  CUDA_TRY(launch_ep_pack(topk_ids, topk_w, hidden_states, hidden_row_stride, hidden_scale, scale_stride_t,
                          scale_stride_kb, T, hidden, world, send_rows, dest_counts, send_slot, num_sms,
                          reinterpret_cast<cudaStream_t>(stream)));
  return B200MOE_OK;
}

int b200moe_ep_local_experts(const void* const* send_base, const int32_t* from_peers, int world, int cap_rows,
                             int64_t row_bytes, const uint8_t* w1, const float* w1_scale, const uint8_t* w2,
                             const float* w2_scale, int e_local, int local_expert_offset, int hidden, int inter,
                             void* workspace, size_t workspace_bytes, void* out_bf16, int64_t out_row_stride,
                             void* stream) {
  if (!send_base || !from_peers || cap_rows < 0) return B200MOE_ERR_INVALID_ARGUMENT;
  if (world != 1 && world != 2 && world != 4 && world != 8) return B200MOE_ERR_UNSUPPORTED_SHAPE;
  if (row_bytes < hidden + 4 * (hidden / kBlockK) + 64 || row_bytes % 16 != 0) return B200MOE_ERR_MISALIGNED;
  if (local_expert_offset < 0 || local_expert_offset + e_local > kNumExperts) return B200MOE_ERR_INVALID_ARGUMENT;
  PeerBases bases;
  memset(&bases, 0, sizeof(bases));
  for (int s = 0; s < world; ++s) {
    if (!send_base[s]) return B200MOE_ERR_INVALID_ARGUMENT;
    if (reinterpret_cast<uintptr_t>(send_base[s]) % 16 != 0) return B200MOE_ERR_MISALIGNED;
    bases.base[s] = reinterpret_cast<const uint8_t*>(send_base[s]);
  }
  Workspace ws;
  int rc = bind_workspace(cap_rows, e_local, hidden, inter, workspace, workspace_bytes, &ws);
  if (rc != B200MOE_OK) return rc;
  if (cap_rows == 0) return B200MOE_OK;
  int num_sms = 0;
  if ((rc = ensure_device(&num_sms)) != B200MOE_OK) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if ((rc = clear_counters(ws, e_local, st)) != B200MOE_OK) return rc;
  RowSegments* segs_dev = ws.at<RowSegments>(ws.L.ep_segments);
  int* n_rows_dev = ws.at<int>(ws.L.ep_segments + 192);
  static_assert(sizeof(RowSegments) <= 192, "the segment table and the row count share 256 bytes");
  int32_t* ids = ws.at<int32_t>(ws.L.topk_ids);
  float* w = ws.at<float>(ws.L.topk_w);
  CUDA_TRY(launch_ep_segments_pull(bases, from_peers, world, row_bytes, cap_rows, hidden, segs_dev, n_rows_dev, ids, w,
                                   num_sms, st));
  CUDA_TRY(launch_count(ids, kTopK, cap_rows, local_expert_offset, e_local, ws.at<int>(ws.L.chunk_counts), num_sms, st,
                        n_rows_dev));
  return experts_impl(ids, kTopK, w, kTopK, nullptr, hidden, nullptr, 0, 0, w1, w1_scale, w2, w2_scale, cap_rows,
                      e_local, local_expert_offset, hidden, inter, workspace, workspace_bytes, out_bf16, out_row_stride,
                      stream, false, nullptr, segs_dev, n_rows_dev);
}

int b200moe_ep_combine_peers(const void* const* partial_bf16, const int32_t* row_start, const int32_t* send_slot,
                             int T, int hidden, int world, void* out_bf16, void* stream) {
  if (T < 0) return B200MOE_ERR_INVALID_ARGUMENT;
  if (T == 0) return B200MOE_OK;
  if (!partial_bf16 || !row_start || !send_slot || !out_bf16) return B200MOE_ERR_INVALID_ARGUMENT;
  if (world != 1 && world != 2 && world != 4 && world != 8) return B200MOE_ERR_UNSUPPORTED_SHAPE;
  if (hidden < 8 || hidden % 8 != 0) return B200MOE_ERR_UNSUPPORTED_SHAPE;
  PeerPartials peers;
  memset(&peers, 0, sizeof(peers));
  for (int d = 0; d < world; ++d) {
    if (!partial_bf16[d] || reinterpret_cast<uintptr_t>(partial_bf16[d]) % 16 != 0) return B200MOE_ERR_MISALIGNED;
    peers.partial[d] = partial_bf16[d];
  }
  if (reinterpret_cast<uintptr_t>(out_bf16) % 16 != 0) return B200MOE_ERR_MISALIGNED;
  int num_sms = 0;
  int rc = ensure_device(&num_sms);
  if (rc != B200MOE_OK) return rc;
  CUDA_TRY(launch_ep_combine_peers(peers, row_start, send_slot, T, hidden, world, out_bf16, num_sms,
                                   reinterpret_cast<cudaStream_t>(stream)));
  return B200MOE_OK;
}

int b200moe_ep_combine(const void* returned_bf16, const int32_t* send_slot, const int32_t* dest_counts, int T,
                       int hidden, int world, void* out_bf16, void* stream) {
  if (T < 0) return B200MOE_ERR_INVALID_ARGUMENT;
  if (T == 0) return B200MOE_OK;
  if (!returned_bf16 || !send_slot || !dest_counts || !out_bf16) return B200MOE_ERR_INVALID_ARGUMENT;
  if (world != 1 && world != 2 && world != 4 && world != 8) return B200MOE_ERR_UNSUPPORTED_SHAPE;
  if (hidden < 8 || hidden % 8 != 0) return B200MOE_ERR_UNSUPPORTED_SHAPE;
  if (reinterpret_cast<uintptr_t>(returned_bf16) % 16 != 0 || reinterpret_cast<uintptr_t>(out_bf16) % 16 != 0)
    return B200MOE_ERR_MISALIGNED;
  int num_sms = 0;
  int rc = ensure_device(&num_sms);
  if (rc != B200MOE_OK) return rc;
  CUDA_TRY(launch_ep_combine(returned_bf16, send_slot, dest_counts, T, hidden, world, out_bf16, num_sms,
                             reinterpret_cast<cudaStream_t>(stream)));
  return B200MOE_OK;
}

}  // extern "C"
