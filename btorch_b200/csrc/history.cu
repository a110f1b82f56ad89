// The spike history of a module (SpikeHistory, btorch/models/history.py:28-358)
// to and from the engine's bitmap ring, and the scatter's edge records: the
// set-up and the hand-over of a multi-step call, one launch each.
#include "common.cuh"

namespace bt {

constexpr int kHistWords = 8;  // words of a warp: 8 coalesced loads or stores in flight

// Which (d, b) row and which words a warp owns; false past the end.
__device__ __forceinline__ bool history_item(int64_t batch, int D, int64_t words, int64_t& d, int64_t& b, int64_t& w0) {
  const int64_t gw = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t per = (words + kHistWords - 1) / kHistWords;
  const int64_t rest = gw / per;
  w0 = (gw - rest * per) * kHistWords;
  d = rest / batch;
  b = rest - d * batch;
  return d < D;
}

__device__ __forceinline__ int64_t history_slot(const int64_t* cursor, int64_t advance, int64_t d, int D) {
  if (!cursor) return d;
  int64_t slot = (*cursor + advance - 1 - d) % D;
  return slot < 0 ? slot + D : slot;
}

// ring[(t0 - 1 - d) mod H][b][w] = the spikes d steps ago, for d < D, from the
// history memory hist[b][slot][n] (slot = (*cursor - 1 - d) mod D in circular
// mode, d when cursor is NULL).  A warp makes 8 words, a ballot each: bound by the
// history's bytes (one word per warp took 219 us for 90 MB).
__global__ void k_history_load(int64_t batch, int D, int64_t n, const float* __restrict__ hist,
                               const int64_t* __restrict__ cursor, int64_t t0, int H, uint32_t* __restrict__ ring) {
  const int64_t words = (n + 31) >> 5;
  int64_t d, b, w0;
  if (!history_item(batch, D, words, d, b, w0)) return;  // whole warps
  const int lane = int(lane_id());
  const float* row = hist + (b * D + history_slot(cursor, 0, d, D)) * n;
  float v[kHistWords];
#pragma unroll
  for (int u = 0; u < kHistWords; ++u) {
    const int64_t i = (w0 + u) * 32 + lane;
    v[u] = i < n ? __ldg(row + i) : 0.0f;
  }
  uint32_t mine = 0u;
#pragma unroll
  for (int u = 0; u < kHistWords; ++u) {
    const uint32_t m = __ballot_sync(0xffffffffu, v[u] != 0.0f);
    if (lane == u) mine = m;
  }
  if (lane < kHistWords && w0 + lane < words) ring[(((t0 - 1 - d) % H) * batch + b) * words + w0 + lane] = mine;
}

// The reverse after `advance` steps: hist[b][slot(d)][n] = the spikes of step
// t_end - 1 - d, slot by the cursor advanced by `advance`.
__global__ void k_history_store(int64_t batch, int D, int64_t n, const uint32_t* __restrict__ ring, int64_t t_end, int H,
                                const int64_t* __restrict__ cursor, int64_t advance, float* __restrict__ hist) {
  const int64_t words = (n + 31) >> 5;
  int64_t d, b, w0;
  if (!history_item(batch, D, words, d, b, w0)) return;
  const int lane = int(lane_id());
  float* row = hist + (b * D + history_slot(cursor, advance, d, D)) * n;
  uint32_t mine = 0u;
  if (lane < kHistWords && w0 + lane < words) mine = __ldg(ring + (((t_end - 1 - d) % H) * batch + b) * words + w0 + lane);
#pragma unroll
  for (int u = 0; u < kHistWords; ++u) {
    const uint32_t m = __shfl_sync(0xffffffffu, mine, u);
    const int64_t i = (w0 + u) * 32 + lane;
    if (i < n) row[i] = float((m >> lane) & 1u);
  }
}

__global__ void k_cursor_advance(int64_t* cursor, int64_t advance, int D) { *cursor = (*cursor + advance) % D; }

// edges[e] = (post, weight) records of the expanded CSR: the weight gathered
// through perm, 0 on the padding.  Bound by its 20 bytes an edge.
__global__ void __launch_bounds__(256) k_pack_edges(int64_t nnz, int64_t padded, const uint32_t* __restrict__ dst,
                                                    const int32_t* __restrict__ perm, const float* __restrict__ w,
                                                    uint2* __restrict__ edges) {
  const int64_t e0 = (int64_t(blockIdx.x) * 256 + threadIdx.x) * 4;
  if (e0 >= padded) return;  // padded % 4 == 0
  const uint4 p = __ldg(reinterpret_cast<const uint4*>(dst + e0));
  float v[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) v[u] = e0 + u < nnz ? __ldg(w + __ldg(perm + e0 + u)) : 0.0f;
  uint4* out = reinterpret_cast<uint4*>(edges + e0);
  out[0] = make_uint4(p.x, __float_as_uint(v[0]), p.y, __float_as_uint(v[1]));
  out[1] = make_uint4(p.z, __float_as_uint(v[2]), p.w, __float_as_uint(v[3]));
}

}  // namespace bt

using namespace bt;

namespace {
int history_check(int64_t batch, int32_t D, int64_t n, int32_t H, int64_t t) {
  BT_CHECK_ARG(batch > 0 && n > 0 && D > 0 && H >= D, "history: batch=%lld D=%d n=%lld H=%d", (long long)batch, D,
               (long long)n, H);
  BT_CHECK_ARG(t >= D, "history: step %lld before the history's first", (long long)t);
  BT_CHECK_ARG(batch * n * D < (int64_t(1) << 38), "history too large");
  return BT_OK;
}
unsigned history_grid(int64_t batch, int32_t D, int64_t n) {
  return unsigned(ceil_div(batch * D * ceil_div((n + 31) / 32, kHistWords), 8));
}
}  // namespace

extern "C" int bt_history_load(int64_t batch, int32_t D, int64_t n, const float* hist, const int64_t* cursor, int64_t t0,
                               int32_t H, uint32_t* ring, void* stream) {
  if (int st = history_check(batch, D, n, H, t0)) return st;
  BT_CHECK_ARG(hist && ring, "null pointer");
  k_history_load<<<history_grid(batch, D, n), 256, 0, static_cast<cudaStream_t>(stream)>>>(batch, D, n, hist, cursor, t0,
                                                                                           H, ring);
  BT_CHECK_LAUNCH("k_history_load");
  return BT_OK;
}

extern "C" int bt_history_store(int64_t batch, int32_t D, int64_t n, const uint32_t* ring, int64_t t_end, int32_t H,
                                int64_t* cursor, int64_t advance, float* hist, void* stream) {
  if (int st = history_check(batch, D, n, H, t_end)) return st;
  BT_CHECK_ARG(hist && ring && advance >= 0, "bad argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  k_history_store<<<history_grid(batch, D, n), 256, 0, s>>>(batch, D, n, ring, t_end, H, cursor, advance, hist);
  BT_CHECK_LAUNCH("k_history_store");
  if (cursor) {
    k_cursor_advance<<<1, 1, 0, s>>>(cursor, advance, D);
    BT_CHECK_LAUNCH("k_cursor_advance");
  }
  return BT_OK;
}

extern "C" int bt_pack_edges(int64_t nnz, int64_t padded, const uint32_t* csr_dst, const int32_t* csr_perm,
                             const float* w, uint32_t* edges, void* stream) {
  BT_CHECK_ARG(nnz >= 0 && padded >= nnz && padded % 4 == 0 && nnz < (int64_t(1) << 31), "bad size");
  if (padded == 0) return BT_OK;
  BT_CHECK_ARG(csr_dst && edges && (nnz == 0 || (csr_perm && w)), "null pointer");
  BT_CHECK_ARG(((reinterpret_cast<uintptr_t>(csr_dst) | reinterpret_cast<uintptr_t>(edges)) & 15) == 0,
               "csr_dst and edges must be 16-byte aligned");
  k_pack_edges<<<unsigned(ceil_div(padded, 1024)), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      nnz, padded, csr_dst, csr_perm, w, reinterpret_cast<uint2*>(edges));
  BT_CHECK_LAUNCH("k_pack_edges");
  return BT_OK;
}
