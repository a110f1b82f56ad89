// Sparse x dense-batch products through the transposed operand:
//   out[b][j] = sum over row j's edges e of w_e * g[b][col_e]
// read from gT = g transposed ([n_cols][pitch]), so that an edge reads one
// contiguous run of samples instead of one scattered word per sample.  Used
// by the backward of SparseConn (rows = sources, columns = posts; the
// reference's torch index-op backward, btorch/models/_sparse_triton.py:389-415).
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace bt {

// out[c][r] = in[r][c] for an rows x cols fp32 matrix, out rows `pitch` apart
// (the columns past `rows` written as zeros), through 32 x 32 shared-memory
// tiles (block 32 x 8: coalesced reads and writes).
__global__ void k_transpose(int64_t rows, int64_t cols, int64_t pitch, const float* __restrict__ in,
                            float* __restrict__ out) {
  __shared__ float tile[32][33];
  const int64_t c0 = int64_t(blockIdx.x) * 32, r0 = int64_t(blockIdx.y) * 32;
#pragma unroll
  for (int k = 0; k < 32; k += 8) {
    const int64_t r = r0 + threadIdx.y + k, c = c0 + threadIdx.x;
    if (c < cols) tile[threadIdx.y + k][threadIdx.x] = r < rows ? in[r * cols + c] : 0.0f;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 32; k += 8) {
    const int64_t c = c0 + threadIdx.y + k, r = r0 + threadIdx.x;
    if (r < pitch && c < cols) out[c * pitch + r] = tile[threadIdx.x][threadIdx.y + k];
  }
}

template <int V>
struct FVec {
  float v[V];
};

// Plain loads: the transposed operand is written by the launches before, which
// may still run when this one's blocks start (launch_step).
template <int V>
__device__ __forceinline__ FVec<V> ld_vec(const float* p) {
  FVec<V> r;
  if constexpr (V == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    r.v[0] = q.x, r.v[1] = q.y, r.v[2] = q.z, r.v[3] = q.w;
  } else {
    static_assert(V == 1, "runs of 4 samples or single ones");
    r.v[0] = *p;
  }
  return r;
}

constexpr int kGatherWarps = 8;
// Runs of gT in flight per lane (8: 4200 rows of 410 edges at batch 128 68 us, 88
// with the 4 the compiler kept in flight; at the 64 registers of four blocks the
// widest instances spill 4 to 24 bytes).
constexpr int kGatherUnroll = 8;

// G lanes (a power of two) cover a block of G V samples at V samples each; the
// S = 32 / G lane groups of a warp and the P warps of a row split its edges,
// their partial sums meet in a butterfly and in shared memory (fixed order:
// deterministic).  Without the lane groups a warp on 16 samples keeps 4 of its
// lanes busy (18.9 us against 8.4 for 2000 rows of 100 edges); without the
// warps per row 1000 rows leave the chip idle (45 against 19 us, 300 edges,
// batch 128).  Bound by the L1-miss path: 4 batch bytes an edge, 14 TB/s at
// batch 128 (8192 rows of 410 edges: 115 us, 142 with a warp per row whose
// results went out as single words).  The CTA's rows are written through
// shared memory, as runs of out[b].  Measured and slower: streaming gT
// through shared memory in column tiles (195 us), narrow sample
// blocks with several rows per warp for reuse in L1 (150 us), and CTAs of 32 rows in
// step over windows of columns (138 us).
// SKIP0: entries of gT that are zero add nothing, whatever the weight.
template <int V, int G, int P, bool SKIP0>
__device__ __forceinline__ void rows_gather(int64_t batch, int64_t pitch, int64_t n_rows, const int32_t* __restrict__ ptr,
                                            const uint32_t* __restrict__ col, const float* __restrict__ wts,
                                            const float* gT, float* out) {
  constexpr int S = 32 / G, R = kGatherWarps / P;  // lane groups of a warp, rows of a CTA
  __shared__ float s_out[kGatherWarps][G * V + 1];
  const int warp = int(threadIdx.x >> 5), lane = int(lane_id());
  const int64_t j0 = int64_t(blockIdx.x) * R;
  const int64_t j = j0 + warp / P;
  const int part = warp % P;
  const int64_t b0 = int64_t(blockIdx.y) * (G * V);
  const int grp = lane / G, gl = lane % G;
  const int64_t bl = b0 + gl * V;  // this lane's first sample
  const bool in = bl < pitch;      // pitch % V == 0
  float acc[V];
#pragma unroll
  for (int v = 0; v < V; ++v) acc[v] = 0.0f;
  if (j < n_rows) {
    const int32_t beg = ptr[j], end = ptr[j + 1];
    for (int32_t base = beg + 32 * part; base < end; base += 32 * P) {
      const int32_t e = base + lane;
      const uint32_t c = e < end ? (__ldg(col + e) & kIdMask) : 0u;
      const float w = e < end ? __ldg(wts + e) : 0.0f;
      const int cnt = end - base < 32 ? end - base : 32;
      const int steps = (cnt + S - 1) / S;
      // kGatherUnroll runs in flight per lane, then their chain
      for (int q0 = 0; q0 < steps; q0 += kGatherUnroll) {
        FVec<V> g[kGatherUnroll];
        float wq[kGatherUnroll];
#pragma unroll
        for (int u = 0; u < kGatherUnroll; ++u) {
          const int k = (q0 + u) * S + grp;
          const uint32_t cq = __shfl_sync(0xffffffffu, c, k & 31);
          wq[u] = __shfl_sync(0xffffffffu, w, k & 31);
#pragma unroll
          for (int v = 0; v < V; ++v) g[u].v[v] = 0.0f;
          if (in && k < cnt) g[u] = ld_vec<V>(gT + int64_t(cq) * pitch + bl);
          else wq[u] = 0.0f;
        }
#pragma unroll
        for (int u = 0; u < kGatherUnroll; ++u)
#pragma unroll
          for (int v = 0; v < V; ++v)
            if (!SKIP0 || g[u].v[v] != 0.0f) acc[v] = fmaf(wq[u], g[u].v[v], acc[v]);
      }
    }
#pragma unroll
    for (int off = G; off < 32; off <<= 1)
#pragma unroll
      for (int v = 0; v < V; ++v) acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], off);
  }
  if (grp == 0) {
#pragma unroll
    for (int v = 0; v < V; ++v) s_out[warp][gl * V + v] = acc[v];
  }
  __syncthreads();
  for (int q = int(threadIdx.x); q < R * G * V; q += kGatherWarps * 32) {
    const int r = q % R, b = q / R;
    if (j0 + r >= n_rows || b0 + b >= batch) continue;
    float sum = s_out[r * P][b];
#pragma unroll
    for (int p = 1; p < P; ++p) sum += s_out[r * P + p][b];
    out[(b0 + b) * n_rows + j0 + r] = sum;
  }
}

template <int V, int G, int P>
__global__ void __launch_bounds__(kGatherWarps * 32, 4) k_rows_gather(int64_t batch, int64_t pitch, int64_t n_rows,
                                                                  const int32_t* __restrict__ ptr,
                                                                  const uint32_t* __restrict__ col,
                                                                  const float* __restrict__ wts, const float* gT,
                                                                  float* out) {
  step_begin();
  rows_gather<V, G, P, false>(batch, pitch, n_rows, ptr, col, wts, gT, out);
}

// Warps per row: enough for about 40 warps per SM over the rows and sample
// blocks (8192 rows: one; 4200 rows: 2, 1000 rows: 8; measured faster
// than one, 8192 rows slower).
template <int V, int G, typename F>
static void pick_parts(int64_t pitch, int64_t n_rows, F&& go) {
  const int64_t ny = ceil_div(pitch, G * V);
  const int64_t warps = n_rows * ny, want = int64_t(device_sms()) * 40;
  using std::integral_constant;
  const integral_constant<int, V> v;
  const integral_constant<int, G> g;
  if (warps >= want) go(v, g, integral_constant<int, 1>(), ny);
  else if (2 * warps >= want) go(v, g, integral_constant<int, 2>(), ny);
  else if (4 * warps >= want) go(v, g, integral_constant<int, 4>(), ny);
  else go(v, g, integral_constant<int, 8>(), ny);
}

// go(V, G, P, sample blocks) for this shape
template <int V, typename F>
static void pick_lanes(int64_t pitch, int64_t n_rows, F&& go) {
  const int64_t nv = pitch / V;  // vectors of a row
  if (nv <= 1) pick_parts<V, 1>(pitch, n_rows, go);
  else if (nv <= 2) pick_parts<V, 2>(pitch, n_rows, go);
  else if (nv <= 4) pick_parts<V, 4>(pitch, n_rows, go);
  else if (nv <= 8) pick_parts<V, 8>(pitch, n_rows, go);
  else if (nv <= 16) pick_parts<V, 16>(pitch, n_rows, go);
  else pick_parts<V, 32>(pitch, n_rows, go);
}

// out [batch][n_rows] from gT [n_cols][pitch] (pitch >= batch, zeros past it).
// first: no launch of the caller's goes before it (launch_step).
int rows_product(bool first, int64_t batch, int64_t pitch, int64_t n_rows, const int32_t* ptr, const uint32_t* col,
                 const float* wts, const float* gT, float* out, cudaStream_t s) {
  auto go = [&](auto v, auto g, auto p, int64_t ny) {
    constexpr int V = decltype(v)::value, G = decltype(g)::value, P = decltype(p)::value;
    launch_step(first, k_rows_gather<V, G, P>, dim3(unsigned(ceil_div(n_rows, kGatherWarps / P)), unsigned(ny)),
                kGatherWarps * 32, 0, s, batch, pitch, n_rows, ptr, col, wts, gT, out);
  };
  // scratch that is not padded to a multiple of 4, or not aligned, is read in words
  if (pitch % 4 == 0 && (reinterpret_cast<uintptr_t>(gT) & 15) == 0) pick_lanes<4>(pitch, n_rows, go);
  else pick_lanes<1>(pitch, n_rows, go);
  BT_CHECK_LAUNCH("k_rows_gather");
  return BT_OK;
}

// ------------------------------------------------- forward, any activity --
//
// out = x @ W in whatever order is faster for this x, as counted on the device:
// few nonzeros are pushed along their sources' out-edges with fp32 reductions
// in L2, many are gathered over every post's in-edges from x transposed.

// Whether the gather is the faster one: 8 + 4 batch bytes an edge at 14 TB/s
// against 145 G reductions/s over nonzeros x mean out-degree (from about 4 % of
// nonzeros at 32 samples and more, 40 % at one).
__device__ __forceinline__ bool push_dense(const int32_t* ctl, int64_t n_in, int64_t pitch) {
  const long long cnt = *reinterpret_cast<const volatile int32_t*>(ctl);
  return cnt * 96 > n_in * (8 + 4 * (pitch > 8 ? pitch : 8));
}

// list[k] = the flat indices of x's nonzeros (order of arrival), ctl[0] their
// count: 8 elements per thread, one atomic per block.
__global__ void __launch_bounds__(256) k_compact(int64_t total, const float* __restrict__ x, int32_t* __restrict__ ctl,
                                                 int32_t* __restrict__ list) {
  __shared__ int s_warp[8], s_base;
  const int lane = int(lane_id()), warp = int(threadIdx.x >> 5);
  const int64_t base = int64_t(blockIdx.x) * 2048 + threadIdx.x;
  uint32_t nz = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u)
    if (base + u * 256 < total && __ldg(x + base + u * 256) != 0.0f) nz |= 1u << u;
  const int cnt = __popc(nz);
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int w = 0; w < 8; ++w) {
      const int c = s_warp[w];
      s_warp[w] = sum;
      sum += c;
    }
    s_base = sum ? atomicAdd(ctl, sum) : 0;
  }
  __syncthreads();
  int at = s_base + s_warp[warp] + incl - cnt;
#pragma unroll
  for (int u = 0; u < 8; ++u)
    if (nz & (1u << u)) list[at++] = int32_t(base + u * 256);
}

// What the chosen path needs: x transposed (rows `pitch` apart, zeros past the
// batch), or out cleared and, unless w_csr was given, the weights in CSR order.
__global__ void __launch_bounds__(256) k_push_prepare(int64_t batch, int64_t n_in, int64_t n_out, int64_t pitch,
                                                      int64_t nnz, const float* __restrict__ x,
                                                      const int32_t* __restrict__ perm, const float* __restrict__ w,
                                                      const int32_t* ctl, float* scratch, float* out) {
  step_begin();
  __shared__ float tile[32][33];
  if (push_dense(ctl, n_in, pitch)) {
    const int tx = int(threadIdx.x) & 31, ty = int(threadIdx.x) >> 5;
    const int64_t nc = (n_in + 31) >> 5, nt = nc * ((pitch + 31) >> 5);
    for (int64_t t = blockIdx.x; t < nt; t += gridDim.x) {
      const int64_t c0 = t % nc * 32, r0 = t / nc * 32;
      __syncthreads();
#pragma unroll
      for (int k = 0; k < 32; k += 8) {
        const int64_t r = r0 + ty + k, c = c0 + tx;
        if (c < n_in) tile[ty + k][tx] = r < batch ? __ldg(x + r * n_in + c) : 0.0f;
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < 32; k += 8) {
        const int64_t c = c0 + ty + k, r = r0 + tx;
        if (r < pitch && c < n_in) scratch[c * pitch + r] = tile[tx][ty + k];
      }
    }
    return;
  }
  const int64_t tid = int64_t(blockIdx.x) * 256 + threadIdx.x, threads = int64_t(gridDim.x) * 256;
  for (int64_t q = tid; q < batch * n_out; q += threads) out[q] = 0.0f;
  if (perm) {
    for (int64_t e = tid; e < nnz; e += 4 * threads) {
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = e + u * threads < nnz ? __ldg(w + __ldg(perm + e + u * threads)) : 0.0f;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (e + u * threads < nnz) scratch[e + u * threads] = v[u];
    }
  }
}

// The product by the chosen path.  The push streams a source's out-edges, 4 per
// lane (two 128-bit loads when the CSR arrays allow, which the host checks).
template <int V, int G, int P>
__global__ void __launch_bounds__(kGatherWarps * 32, 3) k_push_product(
    int64_t batch, int64_t n_in, int64_t n_out, int64_t pitch, const int32_t* __restrict__ csr_ptr,
    const uint32_t* __restrict__ csr_dst, const float* csr_w, const int32_t* __restrict__ csc_ptr,
    const uint32_t* __restrict__ csc_src, const float* __restrict__ w, const float* __restrict__ x, const int32_t* ctl,
    const int32_t* list, const float* xT, float* out) {
  step_begin();
  if (push_dense(ctl, n_in, pitch)) {
    rows_gather<V, G, P, true>(batch, pitch, n_out, csc_ptr, csc_src, w, xT, out);
    return;
  }
  const int32_t count = *reinterpret_cast<const volatile int32_t*>(ctl);
  const int lane = int(lane_id());
  const int64_t blk = int64_t(blockIdx.y) * gridDim.x + blockIdx.x;
  const int64_t warps = int64_t(gridDim.x) * gridDim.y * kGatherWarps;
  for (int64_t it = blk * kGatherWarps + (threadIdx.x >> 5); it < count; it += warps) {
    const int32_t flat = list[it];
    const int64_t b = flat / n_in, j = flat % n_in;
    const float val = __ldg(x + flat);
    const int32_t beg = csr_ptr[j], end = csr_ptr[j + 1];
    float* row = out + b * n_out;
    for (int32_t g = (beg & ~3) + lane * 4; g < end; g += 128) {
      const uint4 d4 = __ldg(reinterpret_cast<const uint4*>(csr_dst + g));
      const float4 w4 = *reinterpret_cast<const float4*>(csr_w + g);
      const uint32_t dd[4] = {d4.x, d4.y, d4.z, d4.w};
      const float ww[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (g + q >= beg && g + q < end) atomicAdd(row + (dd[q] & kIdMask), ww[q] * val);
    }
  }
}

}  // namespace bt

using namespace bt;

namespace {
int grad_input_t(int64_t batch, int64_t pitch, int64_t n_in, int64_t n_out, const int32_t* csr_ptr,
                 const uint32_t* csr_dst, const float* csr_w, const float* grad_out, float* grad_x, float* work,
                 void* stream) {
  BT_CHECK_ARG(batch >= 0 && n_in >= 0 && n_out >= 0, "negative size");
  if (batch == 0 || n_in == 0) return BT_OK;
  BT_CHECK_ARG(csr_ptr && grad_out && grad_x && work, "null pointer");
  BT_CHECK_ARG(batch * n_out < (int64_t(1) << 40), "too large");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (n_out > 0) {
    const dim3 tgrid(unsigned(ceil_div(n_out, 32)), unsigned(ceil_div(pitch, 32)));
    BT_CHECK_ARG(tgrid.y < 65536, "batch too large for the transpose grid");
    k_transpose<<<tgrid, dim3(32, 8), 0, s>>>(batch, n_out, pitch, grad_out, work);
    BT_CHECK_LAUNCH("k_transpose");
  }
  return rows_product(n_out == 0, batch, pitch, n_in, csr_ptr, csr_dst, csr_w, work, grad_x, s);
}
}  // namespace

extern "C" int bt_spmv_grad_input_t(int64_t batch, int64_t n_in, int64_t n_out, const int32_t* csr_ptr,
                                    const uint32_t* csr_dst, const float* csr_w, const float* grad_out,
                                    float* grad_x, float* work, void* stream) {
  return grad_input_t(batch, batch, n_in, n_out, csr_ptr, csr_dst, csr_w, grad_out, grad_x, work, stream);
}

extern "C" int bt_spmv_grad_input_pad(int64_t batch, int64_t n_in, int64_t n_out, const int32_t* csr_ptr,
                                      const uint32_t* csr_dst, const float* csr_w, const float* grad_out,
                                      float* grad_x, float* work, void* stream) {
  return grad_input_t(batch, ceil_div(batch, 4) * 4, n_in, n_out, csr_ptr, csr_dst, csr_w, grad_out, grad_x, work,
                      stream);
}

// Samples of one pass of bt_spmv_push, whose scratch holds two arrays of x's size (the
// list of its nonzeros, and x transposed where the gather runs): all of them while
// an array stays within 256 MB; beyond that as many as keep it there, or half of
// them up to 512, whose two arrays take no more than one of the whole batch.  (A pass
// that pushes packs the weights again, 12 bytes an edge: below 512 samples that
// starts to show.)  Sample blocks are the grid's y: below 2^22 samples.
static int64_t push_samples(int64_t batch, int64_t n_in) {
  constexpr int64_t kWords = int64_t(1) << 26, kSlab = int64_t(1) << 22;
  const int64_t half = std::min<int64_t>(ceil_div(batch, 2), 512);
  const int64_t most = std::min(kSlab, std::max(kWords / std::max<int64_t>(n_in, 1), half));
  return std::min(batch, std::max<int64_t>(4, most & ~int64_t(3)));
}

// work: 8 control words, the list of nonzeros, then x transposed or the packed weights
extern "C" int64_t bt_spmv_push_work_words(int64_t batch, int64_t n_in, int64_t padded) {
  if (batch < 0 || n_in < 0 || padded < 0) return 0;
  const int64_t samples = push_samples(batch, n_in), pitch = ceil_div(samples, 4) * 4;
  return 8 + ceil_div(samples * n_in, 4) * 4 + std::max(pitch * n_in, ceil_div(padded, 4) * 4);
}

namespace {
// One pass, of push_samples samples at most.
int push_pass(int64_t batch, int64_t n_in, int64_t n_out, int64_t nnz, const int32_t* csr_ptr, const uint32_t* csr_dst,
              const int32_t* csr_perm, const float* csr_w, const int32_t* csc_ptr, const uint32_t* csc_src, const float* w,
              const float* x, float* out, int32_t* work, cudaStream_t s) {
  const int64_t pitch = ceil_div(batch, 4) * 4, total = batch * n_in;
  int32_t* list = work + 8;
  float* scratch = reinterpret_cast<float*>(work + 8 + ceil_div(total, 4) * 4);
  if (cudaMemsetAsync(work, 0, sizeof(int32_t) * 4, s) != cudaSuccess)
    return bt_set_error(BT_ERR_CUDA, "memset failed");
  k_compact<<<unsigned(ceil_div(total, 2048)), 256, 0, s>>>(total, x, work, list);
  BT_CHECK_LAUNCH("k_compact");
  const int64_t most = std::max(std::max(ceil_div(batch * n_out, 1024), ceil_div(nnz, 1024)),
                                ceil_div(n_in, 32) * ceil_div(pitch, 32));
  launch_step(false, k_push_prepare, dim3(unsigned(std::min<int64_t>(device_sms() * 8, most))), 256, 0, s, batch, n_in, n_out, pitch, nnz,
              x, csr_w ? nullptr : csr_perm, w, work, scratch, out);
  BT_CHECK_LAUNCH("k_push_prepare");
  const float* packed = csr_w ? csr_w : scratch;
  pick_lanes<4>(pitch, n_out, [&](auto v, auto g, auto p, int64_t ny) {
    constexpr int V = decltype(v)::value, G = decltype(g)::value, P = decltype(p)::value;
    launch_step(false, k_push_product<V, G, P>, dim3(unsigned(ceil_div(n_out, kGatherWarps / P)), unsigned(ny)),
                kGatherWarps * 32, 0, s, batch, n_in, n_out, pitch, csr_ptr, csr_dst, packed, csc_ptr, csc_src, w, x, work,
                list, scratch, out);
  });
  BT_CHECK_LAUNCH("k_push_product");
  return BT_OK;
}
}  // namespace

extern "C" int bt_spmv_push(int64_t batch, int64_t n_in, int64_t n_out, int64_t nnz, const int32_t* csr_ptr,
                            const uint32_t* csr_dst, const int32_t* csr_perm, const float* csr_w, const int32_t* csc_ptr,
                            const uint32_t* csc_src, const float* w, const float* x, float* out, int32_t* work,
                            void* stream) {
  BT_CHECK_ARG(batch >= 0 && n_in >= 0 && n_out >= 0 && nnz >= 0, "negative size");
  BT_CHECK_ARG(batch * n_in < (int64_t(1) << 31), "batch * n_in must be below 2^31");
  if (batch == 0 || n_out == 0) return BT_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  BT_CHECK_ARG(out, "null pointer");
  if (n_in == 0 || nnz == 0) {
    if (cudaMemsetAsync(out, 0, sizeof(float) * size_t(batch * n_out), s) != cudaSuccess)
      return bt_set_error(BT_ERR_CUDA, "memset failed");
    return BT_OK;
  }
  BT_CHECK_ARG(csr_ptr && csr_dst && (csr_perm || csr_w) && csc_ptr && csc_src && w && x && work, "null pointer");
  BT_CHECK_ARG(((reinterpret_cast<uintptr_t>(csr_dst) | reinterpret_cast<uintptr_t>(csr_w) |
                 reinterpret_cast<uintptr_t>(work)) & 15) == 0, "edge arrays and work must be 16-byte aligned");
  const int64_t samples = push_samples(batch, n_in);
  for (int64_t b0 = 0; b0 < batch; b0 += samples)  // one after the other through the same scratch
    if (int st = push_pass(std::min(samples, batch - b0), n_in, n_out, nnz, csr_ptr, csr_dst, csr_perm, csr_w, csc_ptr,
                           csc_src, w, x + b0 * n_in, out + b0 * n_out, work, s))
      return st;
  return BT_OK;
}
