// Memory-bound helper kernels around the grouped GEMMs: gathers of token rows and of gradients into the padded,
// expert-sorted layout (by token; by row for expert parallelism) with the zeroing of its padding, the combine of a
// token's K rows, the fp32 -> storage cast, bias-gradient column sums, the last step of a backward pass (cast and
// routing gradients), the rows that expert parallelism sends, and the reference's small sub-operators.
#pragma once
#include "common.cuh"
#include "epilogues.cuh"

namespace yb {

constexpr int kRowWarps = 8;  // rows per CTA in the warp-per-row kernels

// Where the gathers put 16-byte pieces of token rows: rows of T, or three bf16 planes (umma_f32.cuh).
template <typename T>
struct RowDst {
  using Piece = uint4;
  T* p;
  int ld;
  __device__ __forceinline__ Piece piece(const uint4& q) const { return q; }
  __device__ __forceinline__ void put(size_t row, int vec, const Piece& q) const {
    reinterpret_cast<uint4*>(p + row * ld)[vec] = q;
  }
  __device__ __forceinline__ uint4 one() const { return make_uint4(sizeof(T) == 2 ? 0x3f80u : 0x3f800000u, 0u, 0u, 0u); }
};

// The padding among the rows that the weight-gradient GEMMs cover (covered_rows) as zeros.  It lies in the last row tile
// of an expert: CTA `cta` of kPadCtas per expert looks at eight rows of that tile, one to a warp.
constexpr int kPadCtas = kTileM / kRowWarps;
template <class Dst>
__device__ __forceinline__ void zero_padding(const Dst& dst, const RouteTables& rt, int cta, int row_round, int nvec) {
  const int lane = threadIdx.x & 31, e = cta / kPadCtas;
  const int first = rt.pad_off[e], padded = rt.pad_off[e + 1] - first, count = rt.counts[e];
  const int local = padded - kTileM + (cta % kPadCtas) * kRowWarps + (threadIdx.x >> 5);
  if (local < 0 || local >= covered_rows(count, padded, row_round) || rt.row_token[first + local] >= 0) return;
  const typename Dst::Piece zero = dst.piece(make_uint4(0, 0, 0, 0));
  for (int i = lane; i < nvec; i += 32) dst.put((size_t)(first + local), i, zero);
}

// dst[row of assignment (t, k), 0:H] = src[t, :] for every kept assignment (reference: csrc/gather.cu:6-66, which
// fills a padded [E,C,H] buffer).  Rows of dst are dst.ld elements apart; when dst.ld > H the columns behind the copy
// get (1, 0, 0, ...) for token rows and zeros for padding rows: a weight-gradient GEMM that takes dst as its transposed
// operand then yields, in output row H, the column sums of its other operand (the bias gradient,
// reference: csrc/experts_backward.cu:308).
//
// HBM bound, so a token's row is read once and written K times: a warp takes 32 16-byte pieces of one token, the pieces
// of a token side by side in the grid.  Walked by padded row, a warp per row, each token was read K times, from HBM once
// the tokens exceed what L2 keeps.  H = 2880, K = 4, row by row / by token: T = 64 5.4 / 1.7 us, T = 4096 26 / 21,
// T = 16384 120 / 75 (472 MB, 6.3 TB/s).
// The first pad_ctas CTAs zero padding rows (zero_padding); the forward on the tensor cores, where no result depends on
// them, has none.
template <class Dst, int KB>
__global__ void __launch_bounds__(kRowWarps * 32)
gather_tokens_kernel(const void* __restrict__ src, const Dst dst, const RouteTables rt, int64_t Tn, int nvec, int ld_vec,
                     int K, unsigned pad_ctas, int row_round) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  if (blockIdx.x < pad_ctas) {
    zero_padding(dst, rt, (int)blockIdx.x, row_round, ld_vec);
    return;
  }
  const unsigned chunks = (unsigned)(nvec + 31) / 32;
  const unsigned piece = (blockIdx.x - pad_ctas) * kRowWarps + (threadIdx.x >> 5);   // 2^32 pieces are 2 TB
  const int64_t t = piece / chunks;
  const int i = (int)(piece - (unsigned)t * chunks) * 32 + lane;
  if (t >= Tn) return;
  const bool real = i < nvec;
  uint4 q = make_uint4(0, 0, 0, 0);
  if (real) q = __ldg(reinterpret_cast<const uint4*>(src) + t * nvec + i);
  // the columns behind H: the lanes of the last warp once more
  const bool last = ld_vec > nvec && i - lane + 32 >= nvec;
  const int32_t* flat_row = after_wait(rt.flat_row);
  typename Dst::Piece x;
  for (int k0 = 0; k0 < K; k0 += KB) {
    int32_t r[KB];
#pragma unroll
    for (int k = 0; k < KB; ++k) r[k] = k0 + k < K ? flat_row[t * K + k0 + k] : -1;
    if (k0 == 0) x = dst.piece(q);
#pragma unroll
    for (int k = 0; k < KB; ++k)
      if (r[k] >= 0) {
        if (real) dst.put((size_t)r[k], i, x);
        if (last && lane < ld_vec - nvec)
          dst.put((size_t)r[k], nvec + lane, dst.piece(lane == 0 ? dst.one() : make_uint4(0, 0, 0, 0)));
      }
  }
}

template <class Dst>
inline cudaError_t launch_gather_tokens(const void* src, const Dst& dst, const RouteTables& rt, int64_t Tn, int H,
                                        int esize, int E, int K, int row_round, cudaStream_t st) {
  const int nvec = H * esize / 16, ld_vec = dst.ld * esize / 16;
  const int64_t token_ctas = ceil_div(Tn * ceil_div(nvec, 32), kRowWarps), pad_ctas = row_round > 0 ? (int64_t)E * kPadCtas : 0;
  auto kern = K <= 4 ? gather_tokens_kernel<Dst, 4> : gather_tokens_kernel<Dst, 8>;
  return launch_pdl_opt(true, kern, dim3((unsigned)(pad_ctas + token_ctas)), dim3(kRowWarps * 32), 0, st, src, dst, rt, Tn,
                        nvec, ld_vec, K, (unsigned)pad_ctas, row_round);
}

// Backward gather of the expert-parallel path, by row: gys[row, :] = grad_out[token, :]; also seeds the
// routing-weight gradient of the row with <grad_out[token], b_down[e]>, the bias part of <grad_out, y_e>
// (reference: csrc/experts_backward.cu:83-88).
template <typename T>
__global__ void __launch_bounds__(kRowWarps * 32)
gather_grad_kernel(const T* __restrict__ grad_out, const T* __restrict__ down_bias, T* __restrict__ gys,
                   float* __restrict__ gw_row, const int32_t* __restrict__ row_token,
                   const int32_t* __restrict__ tile_expert, const int32_t* __restrict__ header, int H) {
  const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (row >= header[kHdrRowsUsed]) return;
  const int lane = threadIdx.x & 31;
  const int tok = row_token[row];
  constexpr int VE = 16 / (int)sizeof(T);
  const int nvec = H / VE;
  T* d = gys + (size_t)row * H;
  if (tok < 0) {
    for (int i = lane; i < nvec; i += 32) reinterpret_cast<uint4*>(d)[i] = make_uint4(0, 0, 0, 0);
    if (lane == 0) gw_row[row] = 0.f;
    return;
  }
  const int e = tile_expert[row / kTileM];
  const T* b = down_bias + (size_t)e * H;
  float dot = 0.f;
  for (int i = lane; i < nvec; i += 32) {
    float g[VE], bb[VE];
    load_vec<T, VE>(grad_out + (size_t)tok * H + (size_t)i * VE, g);
    store_vec<T, VE>(d + (size_t)i * VE, g);
    load_vec<T, VE>(b + (size_t)i * VE, bb);
#pragma unroll
    for (int j = 0; j < VE; ++j) dot += g[j] * bb[j];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if (lane == 0) gw_row[row] = dot;
}

// The same from the tokens' side (see gather_tokens_kernel), where the gradient may also be the sum of K slot slices
// (reference: csrc/experts_backward.cu:224-228): the K rows of a token take its gradient, which is read once, and the dot products with K experts' biases are accumulated beside each other (T = 8192, H = 2880, K = 4: 101 us
// by row, 79 by token).  `wpt` warps (1, 2, 4 or 8) share a token, so that few tokens also fill the GPU.
// The warps of a token also zero its row of `acc`, the fp32 sums of the hidden states' gradient: stores run at 7 TB/s
// where a memset does 3.9, and a launch is saved (T = 8192, H = 2880: memset 22 us + gather 64, together 77).
template <typename T, class Dst, int KB>
__global__ void __launch_bounds__(kRowWarps * 32)
gather_grad_tokens_kernel(const T* grad_out, int slots, const T* down_bias, const Dst dst, float* __restrict__ gw_row,
                          float* __restrict__ acc, const RouteTables rt, int64_t Tn, int H, int K, int wpt,
                          unsigned pad_ctas, int row_round) {
  pdl_wait();
  pdl_trigger();
  // after a saving forward this is the first kernel of the call: what wrote the caller's tensors may still have been running
  grad_out = after_wait(grad_out);
  down_bias = after_wait(down_bias);
  const int32_t* flat_row = after_wait(rt.flat_row);
  const int32_t* tile_expert = after_wait(rt.tile_expert);
  constexpr int VE = 16 / (int)sizeof(T);
  const int nvec = H / VE;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (blockIdx.x < pad_ctas) {
    zero_padding(dst, rt, (int)blockIdx.x, row_round, nvec);
    return;
  }
  __shared__ float s_dot[kRowWarps][KB];
  const int64_t t = (int64_t)(blockIdx.x - pad_ctas) * (kRowWarps / wpt) + w / wpt;
  const int part = w % wpt;
  for (int k0 = 0; k0 < K; k0 += KB) {
    int32_t r[KB];
    const T* bias[KB];
    float dot[KB];
#pragma unroll
    for (int k = 0; k < KB; ++k) r[k] = t < Tn && k0 + k < K ? flat_row[t * K + k0 + k] : -1;
#pragma unroll
    for (int k = 0; k < KB; ++k) {
      bias[k] = down_bias + (r[k] >= 0 ? (size_t)tile_expert[r[k] / kTileM] * H : 0);
      dot[k] = 0.f;
    }
    if (t < Tn) {
#pragma unroll 2
      for (int i = lane + 32 * part; i < nvec; i += 32 * wpt) {
        float g[VE];
        load_vec<T, VE, true>(grad_out + (size_t)t * slots * H + (size_t)i * VE, g);
        for (int s = 1; s < slots; ++s) {
          float g2[VE];
          load_vec<T, VE, true>(grad_out + ((size_t)t * slots + s) * H + (size_t)i * VE, g2);
#pragma unroll
          for (int j = 0; j < VE; ++j) g[j] += g2[j];
        }
        if (k0 == 0) {
          float* a = acc + (size_t)t * H + (size_t)i * VE;
          if (sizeof(T) == 4 && (reinterpret_cast<uintptr_t>(acc) & 15) != 0) {   // the caller's d_hidden, 8-byte aligned
#pragma unroll
            for (int j = 0; j < VE; j += 2) *reinterpret_cast<float2*>(a + j) = make_float2(0.f, 0.f);
          } else {
#pragma unroll
            for (int j = 0; j < VE; j += 4) *reinterpret_cast<float4*>(a + j) = make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
        uint4 q;
        store_vec<T, VE>(reinterpret_cast<T*>(&q), g);
        const typename Dst::Piece x = dst.piece(q);
#pragma unroll
        for (int k = 0; k < KB; ++k)
          if (r[k] >= 0) {
            dst.put((size_t)r[k], i, x);
            float b[VE];
            load_vec<T, VE, true>(bias[k] + (size_t)i * VE, b);
#pragma unroll
            for (int j = 0; j < VE; ++j) dot[k] = fmaf(g[j], b[j], dot[k]);
          }
      }
    }
#pragma unroll
    for (int k = 0; k < KB; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) dot[k] += __shfl_xor_sync(0xffffffffu, dot[k], o);
      if (lane == 0) s_dot[w][k] = dot[k];
    }
    __syncthreads();
    if (part == 0 && lane < KB) {
      int32_t row = -1;
#pragma unroll
      for (int k = 0; k < KB; ++k) row = lane == k ? r[k] : row;
      if (row >= 0) {
        float sum = 0.f;
        for (int o = 0; o < wpt; ++o) sum += s_dot[w + o][lane];
        gw_row[row] = sum;
      }
    }
    __syncthreads();
  }
}

template <typename T, class Dst>
inline cudaError_t launch_gather_grad_tokens(const T* grad_out, int slots, const T* down_bias, const Dst& dst, float* gw_row,
                                             float* acc, const RouteTables& rt, int64_t Tn, int H, int E, int K,
                                             int row_round, cudaStream_t st) {
  // at least 32 warps per SM, while each has a piece of the row
  int wpt = 1;
  while (wpt < kRowWarps && Tn * wpt < kSMs * 32 && H * (int)sizeof(T) / 16 > 32 * wpt) wpt *= 2;
  const int64_t token_ctas = ceil_div(Tn * wpt, kRowWarps), pad_ctas = (int64_t)E * kPadCtas;
  auto kern = K <= 4 ? gather_grad_tokens_kernel<T, Dst, 4> : gather_grad_tokens_kernel<T, Dst, 8>;
  return launch_pdl_opt(true, kern, dim3((unsigned)(pad_ctas + token_ctas)), dim3(kRowWarps * 32), 0, st, grad_out, slots,
                        down_bias, dst, gw_row, acc, rt, Tn, H, K, wpt, (unsigned)pad_ctas, row_round);
}

// out[i] = (T) acc[i]
template <typename T>
__global__ void cast_kernel(const float* __restrict__ acc, T* __restrict__ out, int64_t n_vec4) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n_vec4; i += stride) {
    float4 q = __ldg(reinterpret_cast<const float4*>(acc) + i);
    const float v[4] = {q.x, q.y, q.z, q.w};
    store_vec<T, 4>(out + i * 4, v);
  }
}

// dst[e, n] = sum over the kept rows r of expert e of  w_r * src[r, n]   (WEIGHTED)
//                                                  or       src[r, n]
// reference: csrc/experts_backward.cu:277 (down bias), :308 (gate_up bias).  fp32 accumulation.
// grid (ceil(N / (32 * elements per 16 bytes)), E); empty experts get exact zeros.
template <typename T, bool WEIGHTED>
__global__ void __launch_bounds__(256)
colsum_kernel(const T* __restrict__ src, const float* __restrict__ row_weight,
              const int32_t* __restrict__ pad_off, const int32_t* __restrict__ counts, int64_t capacity,
              T* __restrict__ dst, int N) {
  // 256 columns per CTA: a lane owns VE adjacent columns (one 16-byte load), the 8 warps take
  // every 8th row, partial sums meet in shared memory.
  constexpr int VE = 16 / (int)sizeof(T);
  constexpr int CPB = 32 * VE;                 // columns per CTA
  __shared__ float part[8][CPB];
  const int e = blockIdx.y;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int n = blockIdx.x * CPB + lane * VE;
  const int r0 = pad_off[e];
  const int c = counts[e];
  const int kept = (int64_t)c < capacity ? c : (int)capacity;
  float acc[VE];
#pragma unroll
  for (int j = 0; j < VE; ++j) acc[j] = 0.f;
  if (n < N) {
    int r = w;
    for (; r + 24 < kept; r += 32) {           // four rows in flight per warp
      float v[4][VE];
#pragma unroll
      for (int u = 0; u < 4; ++u) load_vec<T, VE>(src + (size_t)(r0 + r + 8 * u) * N + n, v[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float wgt = WEIGHTED ? row_weight[r0 + r + 8 * u] : 1.0f;
#pragma unroll
        for (int j = 0; j < VE; ++j) acc[j] = fmaf(wgt, v[u][j], acc[j]);
      }
    }
    for (; r < kept; r += 8) {
      float v[VE];
      load_vec<T, VE>(src + (size_t)(r0 + r) * N + n, v);
      const float wgt = WEIGHTED ? row_weight[r0 + r] : 1.0f;
#pragma unroll
      for (int j = 0; j < VE; ++j) acc[j] = fmaf(wgt, v[j], acc[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < VE; ++j) part[w][lane * VE + j] = acc[j];
  __syncthreads();
  for (int col = threadIdx.x; col < CPB; col += 256) {
    if (blockIdx.x * CPB + col >= N) continue;
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += part[k][col];
    DT<T>::st(dst + (size_t)e * N + blockIdx.x * CPB + col, s);
  }
}

// The last step of a backward pass.  CTAs below cast_ctas: d_hidden = (T) acc (acc null: it is d_hidden itself).  The others:
// d_routing[t, e] (dense) or d_routing[t, slot] = gw_row of the assignment's row, 0 where there is none, a warp per token
// (reference: csrc/experts_backward.cu:266-274, with the sort permutation applied once).  In one launch and by token, so
// that nothing has to be zeroed before: a memset, this scatter by row and the cast were three (T = 1531, E = 64: 18 us,
// now 7).
template <typename T>
__global__ void __launch_bounds__(256)
finish_grads_kernel(const float* acc, T* __restrict__ d_hidden, int64_t n_vec4, unsigned cast_ctas, const float* gw_row,
                    const RouteTables rt, T* __restrict__ d_routing, int64_t Tn, int routing_cols, int E, int K) {
  pdl_wait();
  acc = after_wait(acc);
  gw_row = after_wait(gw_row);
  if (blockIdx.x < cast_ctas) {
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n_vec4; i += (int64_t)cast_ctas * 256) {
      const float4 q = __ldcs(reinterpret_cast<const float4*>(acc) + i);
      const float v[4] = {q.x, q.y, q.z, q.w};
      store_vec<T, 4>(d_hidden + i * 4, v);
    }
    return;
  }
  const int lane = threadIdx.x & 31;
  const int64_t t = (int64_t)(blockIdx.x - cast_ctas) * 8 + (threadIdx.x >> 5);
  if (t >= Tn) return;
  for (int k0 = 0; k0 < K; k0 += 32) {
    const int n = min(32, K - k0);
    const int32_t r = lane < n ? rt.flat_row[t * K + k0 + lane] : -1;
    const float g = r >= 0 ? gw_row[r] : 0.f;
    if (routing_cols != E) {
      if (lane < n) DT<T>::st(d_routing + (size_t)t * K + k0 + lane, g);
      continue;
    }
    const int e = r >= 0 ? rt.tile_expert[r / kTileM] : -1;
    for (int c = lane; c - lane < E; c += 32) {
      float v = 0.f;
      bool set = k0 == 0;                 // columns without an assignment are zero
      for (int k = 0; k < n; ++k) {
        const int ek = __shfl_sync(0xffffffffu, e, k);
        const float gk = __shfl_sync(0xffffffffu, g, k);
        if (ek == c) { v = gk; set = true; }
      }
      if (c < E && set) DT<T>::st(d_routing + (size_t)t * E + c, v);
    }
  }
}

// acc: null where the sums are d_hidden itself
template <typename T>
inline int launch_finish_grads(const float* acc, T* d_hidden, const float* gw_row, const RouteTables& rt, T* d_routing,
                               int64_t Tn, int H, int routing_cols, int E, int K, cudaStream_t st) {
  const int64_t nv = Tn * H / 4;
  const unsigned cast_ctas = acc != nullptr ? (unsigned)std::min<int64_t>(ceil_div(nv, 256), kSMs * 8) : 0u;
  const cudaError_t rc = launch_pdl_opt(true, finish_grads_kernel<T>, dim3(cast_ctas + (unsigned)ceil_div(Tn, 8)), dim3(256), 0,
                                        st, acc, d_hidden, nv, cast_ctas, gw_row, rt, d_routing, Tn, routing_cols, E, K);
  return rc == cudaSuccess && cudaGetLastError() == cudaSuccess ? YAMOE_OK : YAMOE_ERR_CUDA;
}

// the elements of 16 bytes, as fp32
template <typename T>
__device__ __forceinline__ void unpack_vec(const uint4& q, float (&v)[16 / sizeof(T)]) {
  const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if constexpr (sizeof(T) == 4) {
      v[j] = __uint_as_float(u[j]);
    } else {
      v[2 * j] = __uint_as_float(u[j] << 16);
      v[2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u);
    }
  }
}

// out[t, :] = sum over the kept slots k of y[flat_row[t*K + k], :]   (rows already weighted).
// Second half of the combine (reference: csrc/scatter.cu:67-108): fp32 accumulation in slot
// order, one rounding, every output element written exactly once (no zero-fill, no atomics).
// One warp per token and 32 16-byte pieces of its row, with the loads of up to KB slots in flight: latency bounds the
// few-token calls (a warp per token left most SMs idle and walked the columns one after the
// other: 30 us at T = 64 and 512 with H = 2880, now 3 to 5), HBM the others.  The pieces of a row are neighbours in
// the grid, so that its 512-byte parts are read at about the same time (T = 4096 44 us with the tokens as
// neighbours, 30 with the pieces, 24 since the loads wait unconverted; T = 1531, K = 8, H = 2048 23 and 11).
// Rows of another type than the output (fp32 rows of a bf16 call) lie at their flat positions p = t*K + k.
template <typename TY, typename T, int KB>
__global__ void __launch_bounds__(kRowWarps * 32, KB > 4 ? 4 : 5)
combine_padded_kernel(const TY* y, const int32_t* flat_row, T* __restrict__ out, int64_t Tn, int H, int K) {
  pdl_wait();
  y = after_wait(y);
  flat_row = after_wait(flat_row);
  constexpr bool kFlat = !std::is_same<TY, T>::value;
  constexpr int VE = 16 / (int)sizeof(TY);
  const unsigned chunks = (unsigned)(H / VE + 31) / 32;
  const unsigned piece = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  const int64_t t = piece / chunks;
  const int i = (int)(piece - (unsigned)t * chunks) * 32 + (threadIdx.x & 31);
  if (t >= Tn || i >= H / VE) return;
  float acc[VE];
#pragma unroll
  for (int j = 0; j < VE; ++j) acc[j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += KB) {
    int32_t r[KB];
    uint4 q[KB];                           // as loaded: as fp32 they took 105 registers at KB = 8, now 56, and half the warps
#pragma unroll
    for (int k = 0; k < KB; ++k) r[k] = k0 + k < K ? flat_row[t * K + k0 + k] : -1;
#pragma unroll
    for (int k = 0; k < KB; ++k) {
      q[k] = make_uint4(0, 0, 0, 0);
      if (r[k] >= 0)
        q[k] = ld_written(reinterpret_cast<const uint4*>(y + (kFlat ? (size_t)(t * K + k0 + k) : (size_t)r[k]) * H) + i);
    }
#pragma unroll
    for (int k = 0; k < KB; ++k)
      if (r[k] >= 0) {
        float v[VE];
        unpack_vec<TY>(q[k], v);
#pragma unroll
        for (int j = 0; j < VE; ++j) acc[j] += v[j];
      }
  }
  store_vec<T, VE>(out + (size_t)t * H + (size_t)i * VE, acc);
}

template <typename TY, typename T>
inline int launch_combine(const TY* y, const int32_t* flat_row, T* out, int64_t Tn, int H, int K, cudaStream_t st) {
  const dim3 grid((unsigned)ceil_div(Tn * ceil_div(H, 32 * (16 / (int)sizeof(TY))), kRowWarps));
  auto kern = K <= 4 ? combine_padded_kernel<TY, T, 4> : combine_padded_kernel<TY, T, 8>;
  const cudaError_t rc = launch_pdl_opt(true, kern, grid, dim3(kRowWarps * 32), 0, st, y, flat_row, out, Tn, H, K);
  return rc == cudaSuccess && cudaGetLastError() == cudaSuccess ? YAMOE_OK : YAMOE_ERR_CUDA;
}

// ---- expert-parallel helpers ---------------------------------------------------------------
// dst[j, :] = src[sorted_indices[j] / K, :]: rows in expert-sorted order, ready to be sent to
// the ranks that own the experts.  One warp per row, 16-byte accesses.
template <typename T>
__global__ void __launch_bounds__(kRowWarps * 32)
permute_rows_kernel(const T* __restrict__ src, const int32_t* __restrict__ sorted_indices, T* __restrict__ dst,
                    int64_t S, int H, int K, int64_t n_src) {
  const int64_t row = (int64_t)blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (row >= S) return;
  const int lane = threadIdx.x & 31;
  const int flat = sorted_indices[row];
  const int nvec = H * (int)sizeof(T) / 16;
  uint4* d = reinterpret_cast<uint4*>(dst + (size_t)row * H);
  if (flat < 0 || flat / K >= n_src) {          // entry of a dropped assignment (-1): a zero row
    for (int i = lane; i < nvec; i += 32) d[i] = make_uint4(0, 0, 0, 0);
    return;
  }
  const uint4* s = reinterpret_cast<const uint4*>(src + (size_t)(flat / K) * H);
  for (int i = lane; i < nvec; i += 32) d[i] = __ldg(s + i);
}

// inv[sorted_indices[j]] = j; entries outside [0, n_flat) (the -1 tail left for dropped assignments) are skipped
__global__ void invert_perm_kernel(const int32_t* __restrict__ sorted_indices, int32_t* __restrict__ inv, int64_t S,
                                   int64_t n_flat) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= S) return;
  const int32_t p = sorted_indices[j];
  if (p >= 0 && p < n_flat) inv[p] = (int32_t)j;
}

// out[t, :] = sum_k w[t, k] * rows[inv[t*K + k], :]   (fp32 accumulation, fixed order, one rounding).
// The weighted combine of csrc/scatter.cu:67-108 for rows that came back from the expert owners.
template <typename T>
__global__ void __launch_bounds__(kRowWarps * 32)
combine_rows_kernel(const T* __restrict__ rows, const int32_t* __restrict__ inv,
                    const int64_t* __restrict__ router_indices, const T* __restrict__ routing_weights,
                    int routing_cols, T* __restrict__ out, int64_t Tn, int H, int E, int K) {
  const int64_t t = (int64_t)blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (t >= Tn) return;
  const int lane = threadIdx.x & 31;
  constexpr int VE = 16 / (int)sizeof(T);
  const int nvec = H / VE;
  for (int i = lane; i < nvec; i += 32) {
    float acc[VE];
#pragma unroll
    for (int j = 0; j < VE; ++j) acc[j] = 0.f;
    for (int k = 0; k < K; ++k) {
      const int32_t r = inv[t * K + k];
      if (r < 0) continue;
      const int col = (routing_cols == E) ? (int)router_indices[t * K + k] : k;
      const float w = DT<T>::ld(routing_weights + (size_t)t * routing_cols + col);
      float v[VE];
      load_vec<T, VE>(rows + (size_t)r * H + (size_t)i * VE, v);
#pragma unroll
      for (int j = 0; j < VE; ++j) acc[j] = fmaf(w, v[j], acc[j]);
    }
    store_vec<T, VE>(out + (size_t)t * H + (size_t)i * VE, acc);
  }
}

// ---- the reference's three small sub-operators on its padded [E, C, H] layout ------------------
// This library's own path never materialises [E, C, H]; these serve callers of the standalone ops.

// out[e, i, :] = x[indices[bins[e-1] + i] / top_k, :] for i < min(count_e, C), zeros otherwise.
// reference: csrc/gather.cu:7-66.  One warp per (e, i); VEC: 16-byte copies.
template <typename T, bool VEC>
__global__ void __launch_bounds__(kRowWarps * 32)
binned_gather_kernel(const T* __restrict__ x, const int32_t* __restrict__ indices, const int32_t* __restrict__ bins,
                     T* __restrict__ out, int64_t Tn, int H, int E, int C, int top_k) {
  const int64_t r = (int64_t)blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (r >= (int64_t)E * C) return;
  const int lane = threadIdx.x & 31;
  const int e = (int)(r / C), i = (int)(r - (int64_t)e * C);
  const int start = e ? bins[e - 1] : 0;
  int64_t tok = -1;
  if (i < bins[e] - start) {
    tok = indices[start + i] / top_k;
    if (tok < 0 || tok >= Tn) tok = -1;
  }
  T* dst = out + (size_t)r * H;
  if constexpr (VEC) {
    const int nvec = H * (int)sizeof(T) / 16;
    uint4* d = reinterpret_cast<uint4*>(dst);
    if (tok < 0) {
      for (int v = lane; v < nvec; v += 32) d[v] = make_uint4(0, 0, 0, 0);
    } else {
      const uint4* sp = reinterpret_cast<const uint4*>(x + (size_t)tok * H);
      for (int v = lane; v < nvec; v += 32) d[v] = __ldg(sp + v);
    }
  } else {
    for (int h = lane; h < H; h += 32) DT<T>::st(dst + h, tok < 0 ? 0.f : DT<T>::ld(x + (size_t)tok * H + h));
  }
}

__device__ __forceinline__ void atomic_add_elem(float* p, float v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_elem(__nv_bfloat16* p, float v) { atomicAdd(p, __float2bfloat16_rn(v)); }

// y[tok, :] += weights[start + i] * src[e, i, :] for i < min(count_e, C).
// reference: csrc/scatter.cu:67-108: the product is rounded to the storage type, then added
// atomically with one rounding per addition; the order of a token's K additions is not fixed
// there either.  One warp per (e, i).
template <typename T>
__global__ void __launch_bounds__(kRowWarps * 32)
binned_scatter_kernel(const T* __restrict__ src, const int32_t* __restrict__ indices,
                      const int32_t* __restrict__ bins, const T* __restrict__ weights, T* __restrict__ y,
                      int64_t Tn, int H, int E, int C, int top_k) {
  const int64_t r = (int64_t)blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (r >= (int64_t)E * C) return;
  const int lane = threadIdx.x & 31;
  const int e = (int)(r / C), i = (int)(r - (int64_t)e * C);
  const int start = e ? bins[e - 1] : 0;
  if (i >= bins[e] - start) return;
  const int64_t tok = indices[start + i] / top_k;
  if (tok < 0 || tok >= Tn) return;
  const float scale = weights != nullptr ? DT<T>::ld(weights + start + i) : 1.0f;
  const T* sp = src + (size_t)r * H;
  T* yp = y + (size_t)tok * H;
  if constexpr (sizeof(T) == 2) {
    if ((H & 1) == 0 && (reinterpret_cast<uintptr_t>(yp) & 3) == 0 && (reinterpret_cast<uintptr_t>(sp) & 3) == 0) {
      for (int h = 2 * lane; h < H; h += 64) {
        const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(sp + h);
        atomicAdd(reinterpret_cast<__nv_bfloat162*>(yp + h),
                  __floats2bfloat162_rn(__low2float(v) * scale, __high2float(v) * scale));
      }
      return;
    }
  }
  for (int h = lane; h < H; h += 32) {
    float p = DT<T>::ld(sp + h) * scale;
    if constexpr (sizeof(T) == 2) p = __bfloat162float(__float2bfloat16_rn(p));
    atomic_add_elem(yp + h, p);
  }
}

// out[i] = in[idx[i]]    reference: csrc/index_select.cu:7-16
template <typename T>
__global__ void index_select_kernel(const T* __restrict__ in, const int32_t* __restrict__ idx, T* __restrict__ out,
                                    int64_t N) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) out[i] = in[(int64_t)idx[i]];
}

}  // namespace yb
