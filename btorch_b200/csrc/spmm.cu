// Sparse x dense-batch products through the transposed operand:
//   out[b][j] = sum over row j's edges e of w_e * g[b][col_e]
// read from gT = g transposed ([n_cols][pitch]), so that an edge reads one
// contiguous run of samples instead of one scattered word per sample.  Used
// by the backward of SparseConn (rows = sources, columns = posts; the
// reference's torch index-op backward, btorch/models/_sparse_triton.py:389-415).
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

template <int V>
__device__ __forceinline__ FVec<V> ld_vec(const float* p) {
  FVec<V> r;
  if constexpr (V == 4) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    r.v[0] = q.x, r.v[1] = q.y, r.v[2] = q.z, r.v[3] = q.w;
  } else if constexpr (V == 2) {
    const float2 q = __ldg(reinterpret_cast<const float2*>(p));
    r.v[0] = q.x, r.v[1] = q.y;
  } else {
    r.v[0] = __ldg(p);
  }
  return r;
}

constexpr int kGatherWarps = 8;

// G lanes (a power of two) cover a block of G V samples at V samples each; the
// S = 32 / G lane groups of a warp and the P warps of a row split its edges,
// their partial sums meet in a butterfly and in shared memory (fixed order:
// deterministic).  Without the lane groups a warp on 16 samples keeps 4 of its
// lanes busy (18.9 us against 8.4 for 2000 rows of 100 edges); without the
// warps per row 1000 rows leave the chip idle (45 against 21 us, 300 edges,
// batch 128).  Bound by the L1-miss path: 4 batch bytes an edge, 14 TB/s at
// batch 128 (8192 rows of 410 edges: 119 us, 142 with a warp per row whose
// results went out as single words).  The CTA's rows are written through
// shared memory, as runs of out[b].  Measured and slower: streaming gT
// through shared memory in column tiles (195 us), and narrow sample blocks
// with several rows per warp for reuse in L1 (150 us).
template <int V, int G, int P>
__global__ void __launch_bounds__(kGatherWarps * 32) k_rows_gather(int64_t batch, int64_t pitch, int64_t n_rows,
                                                                  const int32_t* __restrict__ ptr,
                                                                  const uint32_t* __restrict__ col,
                                                                  const float* __restrict__ wts,
                                                                  const float* __restrict__ gT, float* __restrict__ out) {
  step_begin();
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
#pragma unroll 4
      for (int q = 0; q < steps; ++q) {
        const int k = q * S + grp;
        const uint32_t cq = __shfl_sync(0xffffffffu, c, k);
        const float wq = __shfl_sync(0xffffffffu, w, k);
        if (in && k < cnt) {
          const FVec<V> g = ld_vec<V>(gT + int64_t(cq) * pitch + bl);
#pragma unroll
          for (int v = 0; v < V; ++v) acc[v] = fmaf(wq, g.v[v], acc[v]);
        }
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

// Warps per row: enough for about 40 warps per SM over the rows and sample
// blocks (8192 rows: one; 4200 rows: 2, 1000 rows: 8; measured faster
// than one, 8192 rows slower).
template <int V, int G>
static void launch_gather_g(int64_t batch, int64_t pitch, int64_t n_rows, const int32_t* ptr, const uint32_t* col,
                            const float* wts, const float* gT, float* out, cudaStream_t s) {
  const int64_t ny = ceil_div(pitch, G * V);
  auto go = [&](auto kern, int P) {
    launch_step(kern, dim3(unsigned(ceil_div(n_rows, kGatherWarps / P)), unsigned(ny)), kGatherWarps * 32, 0, s, batch,
                pitch, n_rows, ptr, col, wts, gT, out);
  };
  const int64_t warps = n_rows * ny, want = 148 * 40;
  if (warps >= want) go(k_rows_gather<V, G, 1>, 1);
  else if (2 * warps >= want) go(k_rows_gather<V, G, 2>, 2);
  else if (4 * warps >= want) go(k_rows_gather<V, G, 4>, 4);
  else go(k_rows_gather<V, G, 8>, 8);
}

template <int V>
static void launch_gather(int64_t batch, int64_t pitch, int64_t n_rows, const int32_t* ptr, const uint32_t* col,
                          const float* wts, const float* gT, float* out, cudaStream_t s) {
  const int64_t nv = pitch / V;  // vectors of a row
  if (nv <= 1) launch_gather_g<V, 1>(batch, pitch, n_rows, ptr, col, wts, gT, out, s);
  else if (nv <= 2) launch_gather_g<V, 2>(batch, pitch, n_rows, ptr, col, wts, gT, out, s);
  else if (nv <= 4) launch_gather_g<V, 4>(batch, pitch, n_rows, ptr, col, wts, gT, out, s);
  else if (nv <= 8) launch_gather_g<V, 8>(batch, pitch, n_rows, ptr, col, wts, gT, out, s);
  else if (nv <= 16) launch_gather_g<V, 16>(batch, pitch, n_rows, ptr, col, wts, gT, out, s);
  else launch_gather_g<V, 32>(batch, pitch, n_rows, ptr, col, wts, gT, out, s);
}

// out [batch][n_rows] from gT [n_cols][pitch] (pitch >= batch, zeros past it).
int rows_product(int64_t batch, int64_t pitch, int64_t n_rows, const int32_t* ptr, const uint32_t* col,
                 const float* wts, const float* gT, float* out, cudaStream_t s) {
  // the scratch of one that is not a multiple of 4, or not aligned, takes words
  if (pitch % 4 == 0 && (reinterpret_cast<uintptr_t>(gT) & 15) == 0)
    launch_gather<4>(batch, pitch, n_rows, ptr, col, wts, gT, out, s);
  else
    launch_gather<1>(batch, pitch, n_rows, ptr, col, wts, gT, out, s);
  BT_CHECK_LAUNCH("k_rows_gather");
  return BT_OK;
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
  return rows_product(batch, pitch, n_in, csr_ptr, csr_dst, csr_w, work, grad_x, s);
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
