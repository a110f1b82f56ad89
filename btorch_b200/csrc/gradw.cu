// Weight gradient of SparseConn over stored nonzeros
// (btorch/models/_sparse_triton.py:389-415):
//   grad_w[e = (j -> i)] = sum over rows r with x[r][j] != 0, ascending, of
//   x[r][j] * g[r][i]
// for rows = samples (or steps x samples of a BPTT chunk).
//
// Sparse inputs (spikes): k_active_rows lists each source's nonzero rows once;
// k_grad_weight_lists then keeps the gradient columns of 8 posts in shared
// memory and lets a thread walk its edge's list there.  Dense inputs: a dot
// product of two transposed rows per edge (k_grad_weight_dense).  Which of the
// two runs is decided on the device from the count of nonzeros.
#include "common.cuh"

namespace bt {

constexpr int kGwPosts = 8;         // posts of a CTA
constexpr int kGwThreads = 512;
constexpr int kGwSegment = 4096;    // rows per pass (16 KB of shared memory per post)

__host__ __device__ __forceinline__ int64_t gw_stride(int64_t seg) { return ((seg + 7) / 8 + 1) * 8; }

// ctl[0] nonzeros of x, ctl[1] whether one of them is not 1
__device__ __forceinline__ bool gw_dense(const int32_t* ctl, int64_t rows, int64_t n_in) {
  const unsigned long long cnt = *reinterpret_cast<const volatile unsigned long long*>(ctl);
  const int graded = *reinterpret_cast<const volatile int32_t*>(ctl + 2);
  // per (edge, row): the dot reads 4 bytes of L2 (0.29 ps); a list entry costs
  // a shared-memory read (0.55 ps), with values also a 32-byte sector (2.3 ps)
  return cnt * (graded ? 8 : 2) > (unsigned long long)(rows * n_in);
}

// lists[j] = {count, 4 x each row with x[row][j] != 0, ascending}, uint16, for
// the rows [r0, r0 + seg), padded to whole vectors of 8 with 4 x seg (the zero
// behind each gradient column in k_grad_weight_lists).  CTA = 32 sources: its warps build the 32-row mask words
// (32 coalesced loads in flight each), then a warp writes a source's list
// from them (popcount prefix over the lanes).
__global__ void __launch_bounds__(512) k_active_rows(int64_t r0, int64_t seg, int64_t n_in, int64_t stride,
                                                     const float* __restrict__ x, uint16_t* __restrict__ lists,
                                                     int32_t* __restrict__ ctl) {
  __shared__ uint32_t s_mask[kGwSegment / 32][33];
  __shared__ int s_cnt, s_graded;
  const int warp = int(threadIdx.x >> 5), lane = int(lane_id());
  constexpr int W = 16;
  const int64_t j = int64_t(blockIdx.x) * 32 + lane;
  if (threadIdx.x == 0) s_cnt = s_graded = 0;
  const int words = int((seg + 31) >> 5);
  bool graded = false;
  for (int q = warp; q < words; q += W) {
    float v[32];
#pragma unroll
    for (int l = 0; l < 32; ++l) {
      const int64_t r = int64_t(q) * 32 + l;
      v[l] = (r < seg && j < n_in) ? __ldg(x + (r0 + r) * n_in + j) : 0.0f;
    }
    uint32_t m = 0;
#pragma unroll
    for (int l = 0; l < 32; ++l) {
      m |= (v[l] != 0.0f ? 1u : 0u) << l;
      graded |= v[l] != 0.0f && v[l] != 1.0f;
    }
    s_mask[q][lane] = m;
  }
  __syncthreads();
  if (graded) s_graded = 1;
  for (int c = warp; c < 32; c += W) {
    const int64_t jj = int64_t(blockIdx.x) * 32 + c;
    if (jj >= n_in) break;
    uint16_t* list = lists + jj * stride;
    int total = 0;
    for (int q0 = 0; q0 < words; q0 += 32) {
      const uint32_t m0 = q0 + lane < words ? s_mask[q0 + lane][c] : 0u;
      const int cnt = __popc(m0);
      int incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      int at = 1 + total + incl - cnt;
      for (uint32_t m = m0; m; m &= m - 1) list[at++] = uint16_t(4 * ((q0 + lane) * 32 + __ffs(m) - 1));
      total += __shfl_sync(0xffffffffu, incl, 31);
    }
    // entries total + 1 .. up to the vector's end
    if (lane < 8 && lane > (total & 7)) list[(total & ~7) + lane] = uint16_t(4 * seg);
    if (lane == 0) {
      list[0] = uint16_t(total);
      atomicAdd(&s_cnt, total);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_cnt) atomicAdd(reinterpret_cast<unsigned long long*>(ctl), (unsigned long long)s_cnt);
    if (s_graded) atomicOr(ctl + 2, 1);
  }
}

// CTA = 8 consecutive posts, whose edges are one range of the canonical order;
// thread = edge.  The gradient columns of the posts sit in shared memory
// (row-minor, post stride = 4 mod 32 words: the 32-byte row segments are
// stored without conflicts).  A list's first 16 bytes carry its count and 7
// rows, so a source that is mostly silent costs one sector; byte offsets and
// the padding keep an entry at four instructions (3.3M edges, 2560 rows, 1 %
// spikes: 149 us; a test and an index computation per entry took 1.6 times as
// long, and 1210 us when every edge walked the samples' mask words and read the
// gradient from global memory).  Bound by L1 (84 % of peak): the random
// shared-memory reads (18M wavefronts) and the lists' scattered vectors.
// carry: continue the chain from grad_w (a later row segment); add: add the
// chain's total to grad_w (a later chunk).
__global__ void __launch_bounds__(kGwThreads) k_grad_weight_lists(int64_t r0, int64_t seg, int64_t rows, int64_t n_in,
                                                                  int64_t n_out, int64_t stride,
                                                                  const int32_t* __restrict__ csc_ptr,
                                                                  const uint32_t* __restrict__ csc_src,
                                                                  const float* __restrict__ x,
                                                                  const float* __restrict__ g,
                                                                  const uint16_t* __restrict__ lists,
                                                                  const int32_t* __restrict__ ctl, int has_dense,
                                                                  int carry, int add_to, float* __restrict__ gw) {
  extern __shared__ __align__(16) float s_g[];  // [kGwPosts][pitch]
  if (has_dense && gw_dense(ctl, rows, n_in)) return;  // grid-uniform
  const int pitch = int((seg + 31) / 32 * 32 + 4);
  const int64_t i0 = int64_t(blockIdx.x) * kGwPosts;
  const int cells = int(seg) * kGwPosts;
  for (int q0 = int(threadIdx.x); q0 < cells; q0 += 8 * kGwThreads) {
    float v[8];  // eight loads in flight, then the stores
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int q = q0 + u * kGwThreads;
      const int64_t i = i0 + q % kGwPosts;
      v[u] = (q < cells && i < n_out) ? __ldg(g + (r0 + q / kGwPosts) * n_out + i) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int q = q0 + u * kGwThreads;
      if (q < cells) s_g[(q % kGwPosts) * pitch + q / kGwPosts] = v[u];
    }
  }
  if (threadIdx.x < kGwPosts) s_g[threadIdx.x * pitch + seg] = 0.0f;
  int32_t off[kGwPosts + 1];
#pragma unroll
  for (int p = 0; p <= kGwPosts; ++p) off[p] = csc_ptr[i0 + p < n_out ? i0 + p : n_out];
  __syncthreads();
  const bool graded = *reinterpret_cast<const volatile int32_t*>(ctl + 2) != 0;
  // the source two edges ahead and the head of the next edge's list are in
  // flight while a list is walked
  const int32_t last = off[kGwPosts];
  auto source = [&](int32_t e) { return e < last ? __ldg(csc_src + e) & kIdMask : 0u; };
  auto head = [&](uint32_t j, int32_t e) {
    return e < last ? __ldg(reinterpret_cast<const uint4*>(lists + int64_t(j) * stride)) : make_uint4(0u, 0u, 0u, 0u);
  };
  int32_t e = off[0] + int32_t(threadIdx.x);
  uint32_t j = source(e), j1 = source(e + kGwThreads);
  uint4 v = head(j, e);
  while (e < last) {
    const uint32_t j2 = source(e + 2 * kGwThreads);
    const uint4 v1 = head(j1, e + kGwThreads);
    int p = 0;
#pragma unroll
    for (int k = 1; k < kGwPosts; ++k) p += e >= off[k] ? 1 : 0;
    const uint4* list = reinterpret_cast<const uint4*>(lists + int64_t(j) * stride);
    const char* col = reinterpret_cast<const char*>(s_g + p * pitch);
    const int cnt = int(v.x & 0xffffu);
    const int nv = (cnt + 8) >> 3;  // vectors of the list, its count included
    float acc = carry ? gw[e] : 0.0f;
    auto at = [&](uint32_t off) { return *reinterpret_cast<const float*>(col + off); };
    if (!graded) {
      // fma(1, g, acc) = acc + g, padding adds the column's zero: no test per entry
      const float f1 = at(v.x >> 16), f2 = at(v.y & 0xffffu), f3 = at(v.y >> 16), f4 = at(v.z & 0xffffu),
                  f5 = at(v.z >> 16), f6 = at(v.w & 0xffffu), f7 = at(v.w >> 16);
      acc = add(add(add(add(add(add(add(acc, f1), f2), f3), f4), f5), f6), f7);
      if (nv > 1) v = __ldg(list + 1);
      for (int q = 1; q < nv; ++q) {
        const uint4 u = v;
        if (q + 1 < nv) v = __ldg(list + q + 1);
        const float h0 = at(u.x & 0xffffu), h1 = at(u.x >> 16), h2 = at(u.y & 0xffffu), h3 = at(u.y >> 16),
                    h4 = at(u.z & 0xffffu), h5 = at(u.z >> 16), h6 = at(u.w & 0xffffu), h7 = at(u.w >> 16);
        acc = add(add(add(add(add(add(add(add(acc, h0), h1), h2), h3), h4), h5), h6), h7);
      }
    } else {
      const uint16_t* row = reinterpret_cast<const uint16_t*>(list) + 1;
      for (int k = 0; k < cnt; ++k) {
        const uint32_t off = __ldg(row + k);
        acc = fmaf(__ldg(x + (r0 + (off >> 2)) * n_in + j), at(off), acc);
      }
    }
    gw[e] = add_to ? add(gw[e], acc) : acc;
    e += kGwThreads;
    j = j1, j1 = j2, v = v1;
  }
}

// Dense inputs: warp = post, G lanes hold 4 samples each of the post's gradient
// column and of a source's transposed row, S = 32 / G edges at a time; a
// butterfly over the G lanes closes each dot product (fixed order).  Bound by
// the L2 reads of the transposed input, 4 bytes per (edge, sample).
template <int G>
__global__ void __launch_bounds__(256) k_grad_weight_dense(int64_t rows, int64_t pitch, int64_t n_in, int64_t n_out,
                                                           const int32_t* __restrict__ csc_ptr,
                                                           const uint32_t* __restrict__ csc_src,
                                                           const float* __restrict__ g, const float* __restrict__ xT,
                                                           const int32_t* __restrict__ ctl, int add_to,
                                                           float* __restrict__ gw) {
  if (!gw_dense(ctl, rows, n_in)) return;  // grid-uniform
  constexpr int S = 32 / G;
  const int64_t i = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (i >= n_out) return;
  const int lane = int(lane_id()), grp = lane / G, gl = lane % G;
  const int32_t beg = csc_ptr[i], end = csc_ptr[i + 1];
  for (int64_t b0 = 0; b0 < rows; b0 += G * 4) {
    float gv[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int64_t b = b0 + gl * 4 + v;
      gv[v] = b < rows ? __ldg(g + b * n_out + i) : 0.0f;
    }
    const bool in = b0 + gl * 4 < pitch;
    for (int32_t base = beg; base < end; base += 32) {
      const int32_t e = base + lane;
      const uint32_t src = e < end ? (__ldg(csc_src + e) & kIdMask) : 0u;
      const int cnt = end - base < 32 ? end - base : 32;
      float mine = 0.0f;  // the dot product of edge base + lane
#pragma unroll 4
      for (int q = 0; q < (cnt + S - 1) / S; ++q) {
        const int k = q * S + grp;
        const uint32_t j = __shfl_sync(0xffffffffu, src, k);
        float4 xv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (in && k < cnt) xv = __ldg(reinterpret_cast<const float4*>(xT + int64_t(j) * pitch + b0 + gl * 4));
        // zero inputs are skipped, whatever the gradient there
        float d = xv.x != 0.0f ? xv.x * gv[0] : 0.0f;
        if (xv.y != 0.0f) d = fmaf(xv.y, gv[1], d);
        if (xv.z != 0.0f) d = fmaf(xv.z, gv[2], d);
        if (xv.w != 0.0f) d = fmaf(xv.w, gv[3], d);
#pragma unroll
        for (int off = G >> 1; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
        // lane k of the block of 32 keeps edge k's total: group k % S of step k / S
        const float got = __shfl_sync(0xffffffffu, d, (lane % S) * G);
        if (lane / S == q) mine = got;
      }
      if (e < end) gw[e] = (add_to || b0 > 0) ? gw[e] + mine : mine;
    }
  }
}

// xT[j][r] = x[r][j] (rows `pitch` apart, zeros past the batch) when the dense path runs.
__global__ void k_transpose_dense(int64_t rows, int64_t cols, int64_t pitch, const float* __restrict__ in,
                                  float* __restrict__ out, const int32_t* __restrict__ ctl) {
  if (!gw_dense(ctl, rows, cols)) return;
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

}  // namespace bt

using namespace bt;

// work: 8 control words, the lists of one pass, then the transposed input of a
// batch that fits one pass (longer ones never take the dense path)
extern "C" int64_t bt_grad_weight_work_words(int64_t rows, int64_t n_in, int32_t with_dense) {
  if (rows < 0 || n_in < 0) return 0;
  const int64_t seg = rows < kGwSegment ? rows : kGwSegment;
  int64_t words = 8 + n_in * gw_stride(seg) / 2;
  if (with_dense && rows <= kGwSegment) words += n_in * (ceil_div(rows, 4) * 4);
  return words;
}

extern "C" int bt_spmv_grad_weight_rows(int64_t rows, int64_t n_in, int64_t n_out, const int32_t* csc_ptr,
                                        const uint32_t* csc_src, const float* x, const float* grad_out,
                                        float* grad_w, int32_t accumulate, int32_t with_dense, int32_t* work,
                                        void* stream) {
  BT_CHECK_ARG(rows >= 0 && n_in >= 0 && n_out >= 0, "negative size");
  if (n_out == 0) return BT_OK;
  BT_CHECK_ARG(csc_ptr && grad_w && work && (rows == 0 || n_in == 0 || (x && grad_out)), "null pointer");
  BT_CHECK_ARG((reinterpret_cast<uintptr_t>(work) & 15) == 0, "work must be 16-byte aligned");
  BT_CHECK_ARG(rows * n_in < (int64_t(1) << 40), "too large");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int32_t* ctl = work;
  uint16_t* lists = reinterpret_cast<uint16_t*>(work + 8);
  const int64_t seg_max = rows < kGwSegment ? rows : kGwSegment;
  const int64_t stride = gw_stride(seg_max);
  const int dense = with_dense && rows <= kGwSegment ? 1 : 0;
  const void* kern = reinterpret_cast<const void*>(k_grad_weight_lists);
  const size_t smem_max = sizeof(float) * kGwPosts * (kGwSegment + 4);
  int dev = 0;
  cudaGetDevice(&dev);
  if (!launch_setup_known(kern, dev, smem_max, 1)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem_max)) != cudaSuccess)
      return bt_set_error(BT_ERR_CUDA, "shared memory request of %zu bytes refused", smem_max);
    launch_setup_add(kern, dev, smem_max, 1);
  }
  const unsigned posts = unsigned(ceil_div(n_out, kGwPosts));
  int64_t r0 = 0;
  do {  // one pass even without rows: it writes the zeros
    const int64_t seg = rows - r0 < kGwSegment ? rows - r0 : kGwSegment;
    if (cudaMemsetAsync(ctl, 0, sizeof(int32_t) * 4, s) != cudaSuccess)
      return bt_set_error(BT_ERR_CUDA, "memset failed");
    if (n_in > 0) {
      k_active_rows<<<unsigned(ceil_div(n_in, 32)), 512, 0, s>>>(r0, seg, n_in, stride, x, lists, ctl);
      BT_CHECK_LAUNCH("k_active_rows");
    }
    const size_t smem = sizeof(float) * kGwPosts * size_t((seg + 31) / 32 * 32 + 4);
    k_grad_weight_lists<<<posts, kGwThreads, smem, s>>>(r0, seg, rows, n_in, n_out, stride, csc_ptr, csc_src, x,
                                                        grad_out, lists, ctl, dense, r0 > 0, accumulate && r0 == 0,
                                                        grad_w);
    BT_CHECK_LAUNCH("k_grad_weight_lists");
    r0 += seg;
  } while (r0 < rows);
  if (dense && rows > 0 && n_in > 0) {
    const int64_t pitch = ceil_div(rows, 4) * 4;
    float* xT = reinterpret_cast<float*>(work + 8 + ceil_div(n_in * stride / 2, 4) * 4);
    k_transpose_dense<<<dim3(unsigned(ceil_div(n_in, 32)), unsigned(ceil_div(pitch, 32))), dim3(32, 8), 0, s>>>(
        rows, n_in, pitch, x, xT, ctl);
    const unsigned grid = unsigned(ceil_div(n_out, 8));
    auto go = [&](auto kern_d) {
      kern_d<<<grid, 256, 0, s>>>(rows, pitch, n_in, n_out, csc_ptr, csc_src, grad_out, xT, ctl, accumulate, grad_w);
    };
    if (pitch <= 16) go(k_grad_weight_dense<4>);
    else if (pitch <= 32) go(k_grad_weight_dense<8>);
    else if (pitch <= 64) go(k_grad_weight_dense<16>);
    else go(k_grad_weight_dense<32>);
    BT_CHECK_LAUNCH("k_grad_weight_dense");
  }
  return BT_OK;
}
