// fp32 grouped GEMM on the tensor cores (sm_100a): every fp32 operand is the sum of three bf16 parts (split3),
// and six of the nine partial products are multiplied with tcgen05.mma (bf16, fp32 accumulation).  The three that
// are left out amount to at most 2^-24 of the product, of either sign, like the rounding of an FFMA: the
// parts are rounded to nearest.  (Cut off instead, all of one sign, they reached 2^-21 and shrank
// every product.)  Splitting into bf16 parts for the tensor cores: G. Henry, P. T. P. Tang and A. Heinecke,
// "Leveraging the bfloat16 artificial intelligence datatype for higher-precision computations", ARITH 2019.
//
//   arrangement   M operand (256), fp32, split on the way       N operand (up to 160), three bf16 planes
//   kFwd          W[e][k][m]   weight columns                   rows of the expert, K-major
//   kDgrad        W[e][m][k]   weight rows                      rows of the expert, K-major
//   kWgrad        grad[r][m]   columns, k = rows                act[r][n] columns, MN-major
//
// Why this split.  The CUDA cores bound the previous kernel (128 x 128 tile, FFMA) at 33 of 74.5
// TFLOP/s; six bf16 products cost a sixth of the tensor rate, some 270 TFLOP/s.  Splitting costs
// about ten instructions per element, so each side is split where it is cheapest: activations once, by
// the kernel that produces them (three planes instead of one fp32 matrix); weights, which are far
// larger and read by few tiles, by the GEMM itself.  The weight tile arrives as fp32 by TMA, eight
// converter warps read it from shared memory, and write the three parts straight into TMEM, from where
// tcgen05.mma takes its A operand: the parts never touch shared memory, whose bandwidth the B operand
// and the fp32 tile already need.
//
// Precision.  The tensor core adds to an accumulator by truncation, whose errors would add up over a
// long reduction.  Each 64-deep k-block therefore starts a fresh accumulator, takes the small
// products first and the leading one last, and the block's sum is added to a running sum in registers
// with round-to-nearest.  Against 64 bits the README forward is 3.0e-7 off where the FFMA kernel's serial
// sum is 1.6e-6, the gradients of 600 tokens (H = 1024) at most 2.7e-7 against 1.1e-6; at H = 64, where the serial sum
// is short, 2.1e-7 against 2.5e-7.
//
// Measured: gate_up of the README forward (T = 512, H = 2880, E = 8, K = 2) 177 us = 192 TFLOP/s of the
// original product; the whole forward 355 us among others of its kind, 300 to 315 on a cool GPU (the power cap lowers the
// clock), a training step of 600 tokens 366 (CUDA cores: 1797 and 1191).
//
// Infinities and NaN behave as in fp32 arithmetic: see split3_special.
//
// Two CTAs share a tile (cta_group::2), 128 weight columns each: the planes are the larger half of what
// L2 has to deliver (48 KB per 64-deep block against 32 KB of weights), and a pair needs them once.
// With one CTA per tile the README forward took 485 us and the training step 463, by pairs 422 and 405.
//
// A CTA has 24 warps: TMA producer, MMA issuer (of the leader only), two that only complete the
// warpgroup, eight converters (two per TMEM lane quarter, 32 k each) and twelve accumulator / epilogue
// warps (three per lane quarter, which take 16-column chunks in turn).  Shared memory: three stages of weights (32 KB) and
// four of activations (30 KB); TMEM, all 512 columns: two accumulators of 160, two A operands of 96.  Signals between
// the CTAs as in umma_pair.cuh, every wait bounded as in umma_gemm.cuh.
//
// Tiles of up to 160 rows, of a size that the kernel picks for the launch (see s_cost): a tile's weights are converted
// for its rows alone, and with 128 rows at most half of the experts of the README forward (128 rows each on average) took
// two tiles: 276 tiles in four waves of 74 pairs, now 184 in three.  gate_up 216 -> 177 us, the whole forward
// 348 -> 313 (both on a cool GPU), with the waits looked at side by side included: a look at a barrier that is ready takes
// some 120 clocks, of which a k-block had three in the issuer and two in the converters.
#pragma once
#include "misc_kernels.cuh"
#include "umma_pair.cuh"

namespace yb {

constexpr int kF32ConvWarps = 8, kF32AccWarps = 12;
constexpr int kF32Threads = 32 * (4 + kF32ConvWarps + kF32AccWarps);
constexpr int kF32M = 128, kF32K = 64;                   // M per CTA
constexpr int kF32N = 160, kF32WgradN = 128;             // most N of a pair: rows of an expert, columns of the activations
constexpr int kF32Tiles = 6;                             // candidates for the rows of a tile: 160, 144, ... 80
constexpr int kF32WBytes = kF32M * kF32K * 4;            // 32 KB: fp32 tile of the M operand
constexpr int kF32BBytes = 3 * (kF32N / 2) * kF32K * 2;  // 30 KB: this CTA's half of the N operand, three planes
constexpr int kF32WStages = 3, kF32BStages = 4;          // (three of activations where the tables of many experts need room)
constexpr int kF32TmemA = 2 * kF32N;                     // first TMEM column of the A operands
constexpr int kF32TmemAStride = 96;                      // 3 parts x 32 columns (64 bf16)
// Registers of a thread: all warps start with a 768th of the SM's file; issuers give up some, accumulators get them.
constexpr int kF32RegsIssue = 48, kF32RegsConv = 72, kF32RegsAcc = 96;
static_assert(128 * (kF32RegsIssue + 2 * kF32RegsConv + 3 * kF32RegsAcc) <= kF32Threads * 80, "more than the launch brings");
inline int f32_smem(int E, int b_stages) {
  return kF32WStages * kF32WBytes + b_stages * kF32BBytes + 1024 + (3 * E + 2) * 4;
}

// The three parts of a number: a = bf16(x), b = bf16(x - a), c = x - a - b, each rounded to nearest (halves away from
// zero).  They sum to x exactly for |x| >= 2^-110 (below that c falls short of the last bits), with |b| <= 2^-8
// and |c| <= 2^-17 of the power of two below |x|.
//
// Zero parts would turn inf * y into NaN, and parts of mixed signs inf into NaN as well.  So an infinity or NaN is
// (+-1, 0, x): x meets nothing but the leading part of the other factor, and inf * inf stays infinite.
// The finite numbers that bf16 rounds to infinity (the last 0.4 % of the range) are truncated instead.
__device__ __forceinline__ uint32_t round_bf16_bits(float x) { return __float_as_uint(x) + 0x8000u; }   // upper half
__device__ __forceinline__ float upper_half(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

__device__ __forceinline__ uint3 split3_special(float x) {
  const uint32_t u = __float_as_uint(x);
  if (!(fabsf(x) <= 3.402823466e38f)) return make_uint3((u & 0x80000000u) | 0x3f800000u, 0u, x != x ? 0x7fff0000u : u);
  uint32_t a = u + 0x8000u;
  if ((a & 0x7f800000u) == 0x7f800000u) a = u;
  const float r = x - upper_half(a);
  const uint32_t b = round_bf16_bits(r);
  return make_uint3(a, b, __float_as_uint(r - upper_half(b)));
}

// The parts of N numbers as bf16 pairs (the first of a pair in the low half).  Returns NaN where one of them is special;
// the caller then has it done again.  One look at all N: a branch for each pair keeps the loads of the next from
// being issued ahead (README forward of that time 513 us and 412 without; 511 with cvt.rn.bf16x2 instead of integer arithmetic).
template <int N>
__device__ __forceinline__ float split3_finite(const float (&x)[N], uint32_t (&p0)[N / 2], uint32_t (&p1)[N / 2],
                                               uint32_t (&p2)[N / 2]) {
  float bad = 0.f;
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const uint32_t a0 = round_bf16_bits(x[i]), a1 = round_bf16_bits(x[i + 1]);
    const float r0 = x[i] - upper_half(a0), r1 = x[i + 1] - upper_half(a1);
    const uint32_t b0 = round_bf16_bits(r0), b1 = round_bf16_bits(r1);
    const float c0 = r0 - upper_half(b0), c1 = r1 - upper_half(b1);
    p0[i / 2] = __byte_perm(a0, a1, 0x7632);
    p1[i / 2] = __byte_perm(b0, b1, 0x7632);
    p2[i / 2] = __byte_perm(__float_as_uint(c0), __float_as_uint(c1), 0x7632);
    bad += c0 + c1;                          // NaN where a leading part is not finite
  }
  return bad;
}
template <int N>
__device__ __forceinline__ void split3(const float (&x)[N], uint32_t (&p0)[N / 2], uint32_t (&p1)[N / 2], uint32_t (&p2)[N / 2]) {
  const float bad = split3_finite<N>(x, p0, p1, p2);
  if (bad != bad) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      const uint3 s0 = split3_special(x[i]), s1 = split3_special(x[i + 1]);
      p0[i / 2] = __byte_perm(s0.x, s1.x, 0x7632);
      p1[i / 2] = __byte_perm(s0.y, s1.y, 0x7632);
      p2[i / 2] = __byte_perm(s0.z, s1.z, 0x7632);
    }
  }
}

// Where an activation matrix is kept as three bf16 planes: [3][rows][ld].
struct Planes {
  __nv_bfloat16* p;
  int64_t stride;                   // elements between planes
  int ld;
  // four adjacent columns, col a multiple of four
  __device__ __forceinline__ void store4(size_t row, int col, const float (&x)[4]) const {
    uint32_t q0[2], q1[2], q2[2];
    split3<4>(x, q0, q1, q2);
    __nv_bfloat16* d = p + row * ld + col;
    *reinterpret_cast<uint2*>(d) = make_uint2(q0[0], q0[1]);
    *reinterpret_cast<uint2*>(d + stride) = make_uint2(q1[0], q1[1]);
    *reinterpret_cast<uint2*>(d + 2 * stride) = make_uint2(q2[0], q2[1]);
  }
  __device__ __forceinline__ void store1(size_t row, int col, float x) const {        // special or not
    const uint3 s = split3_special(x);
    unsigned short* d = reinterpret_cast<unsigned short*>(p) + row * ld + col;
    d[0] = (unsigned short)(s.x >> 16);
    d[stride] = (unsigned short)(s.y >> 16);
    d[2 * stride] = (unsigned short)(s.z >> 16);
  }
  // For epilogues: what the functions below return is NaN where a number was special; the caller then stores again with
  // store1, from values that it reads back (kept in registers for that, they cost more than the splitting).
  // One column of two adjacent rows, of which `rows` exist
  __device__ __forceinline__ float store_rows2(size_t row, int col, int rows, const float (&x)[2]) const {
    uint32_t q0[1], q1[1], q2[1];
    const float bad = split3_finite<2>(x, q0, q1, q2);
    unsigned short* d = reinterpret_cast<unsigned short*>(p) + row * ld + col;
    if (rows > 0) {
      d[0] = (unsigned short)q0[0];
      d[stride] = (unsigned short)q1[0];
      d[2 * stride] = (unsigned short)q2[0];
    }
    if (rows > 1) {
      d[ld] = (unsigned short)(q0[0] >> 16);
      d[ld + stride] = (unsigned short)(q1[0] >> 16);
      d[ld + 2 * stride] = (unsigned short)(q2[0] >> 16);
    }
    return bad;
  }
  // two adjacent columns, col even
  __device__ __forceinline__ float store2(size_t row, int col, float x0, float x1) const {
    uint32_t q0[1], q1[1], q2[1];
    const float bad = split3_finite<2>({x0, x1}, q0, q1, q2);
    __nv_bfloat16* d = p + row * ld + col;
    *reinterpret_cast<uint32_t*>(d) = q0[0];
    *reinterpret_cast<uint32_t*>(d + stride) = q1[0];
    *reinterpret_cast<uint32_t*>(d + 2 * stride) = q2[0];
    return bad;
  }
};

// The gathers' destinations as planes (see RowDst): a piece, four adjacent columns, is split once for all K rows.  With
// `rows` the fp32 values are written as well, H apart (upstream gradient: M operand of the down weight gradient).
struct PlaneDst {
  struct Piece { uint4 x; uint2 p[3]; };
  Planes planes;
  int ld;
  float* rows;
  __device__ __forceinline__ Piece piece(const uint4& q) const {
    uint32_t p0[2], p1[2], p2[2];
    split3<4>({__uint_as_float(q.x), __uint_as_float(q.y), __uint_as_float(q.z), __uint_as_float(q.w)}, p0, p1, p2);
    return Piece{q, {make_uint2(p0[0], p0[1]), make_uint2(p1[0], p1[1]), make_uint2(p2[0], p2[1])}};
  }
  __device__ __forceinline__ void put(size_t row, int vec, const Piece& q) const {
    __nv_bfloat16* d = planes.p + row * ld + 4 * vec;
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(d + i * planes.stride) = q.p[i];
    if (rows != nullptr) reinterpret_cast<uint4*>(rows + row * ld)[vec] = q.x;
  }
  __device__ __forceinline__ uint4 one() const { return make_uint4(0x3f800000u, 0u, 0u, 0u); }
};

// Between fp32 rows and planes of the same pitch: the buffer of the saving forward holds planes whichever kernels
// fill and read it, and the CUDA-core kernels (weights that TMA cannot address, the validation path) work on rows.
__global__ void __launch_bounds__(kRowWarps * 32)
split_rows_kernel(const float* __restrict__ src, Planes dst, const int32_t* __restrict__ header) {
  const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (row >= header[kHdrRowsUsed]) return;
  for (int i = 4 * (threadIdx.x & 31); i < dst.ld; i += 128) {
    const float4 v = *reinterpret_cast<const float4*>(src + (size_t)row * dst.ld + i);
    dst.store4(row, i, {v.x, v.y, v.z, v.w});
  }
}

__global__ void __launch_bounds__(kRowWarps * 32)
join_rows_kernel(Planes src, float* __restrict__ dst, const int32_t* __restrict__ header) {
  const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5);
  if (row >= header[kHdrRowsUsed]) return;
  for (int i = 4 * (threadIdx.x & 31); i < src.ld; i += 128) {
    const __nv_bfloat16* s = src.p + (size_t)row * src.ld + i;
    float a[4], b[4], c[4];
    load_vec<__nv_bfloat16, 4>(s, a);
    load_vec<__nv_bfloat16, 4>(s + src.stride, b);
    load_vec<__nv_bfloat16, 4>(s + 2 * src.stride, c);
#pragma unroll
    for (int j = 0; j < 4; ++j) a[j] += b[j] + c[j];          // exact: see split3_special
    store_vec<float, 4>(dst + (size_t)row * src.ld + i, a);
  }
}

// ---------------------------------------------------------------------------------------------
// Epilogues: a warp holds 32 consecutive M indices (lane L: m) for 16 consecutive N indices,
//     epi.apply(e, m, row, nvalid, lane, v)      v[i] = C[row + i][m]; only i < nvalid exist
// ---------------------------------------------------------------------------------------------
// Neighbouring columns to one lane: the even lane gets (m, m+1) of rows 0..7, the odd lane
// (m-1, m) of rows 8..15.
__device__ __forceinline__ void pair_columns16(const float (&v)[16], bool odd, float (&lo)[8], float (&hi)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float got = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[8 + i], 1);
    lo[i] = odd ? got : v[i];
    hi[i] = odd ? v[8 + i] : got;
  }
}

// routing weight of row `row + lane` (0 for padding and beyond nvalid) and the ballot of token rows
__device__ __forceinline__ unsigned row_info(const int32_t* row_token, const float* row_weight, int row, int nvalid,
                                             int lane, float& w_lane) {
  bool real = false;
  w_lane = 0.f;
  if (lane < nvalid) {
    real = row_token[row + lane] >= 0;
    if (real && row_weight != nullptr) w_lane = row_weight[row + lane];
  }
  return __ballot_sync(0xffffffffu, real);
}

template <bool TRAIN>
struct F32Glu {                     // see PairGlu
  const float* bias;               // [E, 2H]
  Planes act;                      // [3][rows][H] or null (TRAIN)
  Planes actw;                     // TRAIN: [3][rows][ld]
  float* pre;                      // TRAIN: [rows, 2H]
  const int32_t* row_token;
  const float* row_weight;         // TRAIN
  int H;

  __device__ __forceinline__ void apply(int e, int m, int row, int nvalid, int lane, const float (&v)[16]) const {
    const bool odd = lane & 1;
    const float b = bias[(size_t)e * 2 * H + m];
    float x[16], g[8], u[8];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = v[i] + b;
    pair_columns16(x, odd, g, u);
    const int t0 = odd ? 8 : 0, j = m >> 1;
    float w_lane;
    const unsigned have = row_info(row_token, TRAIN ? row_weight : nullptr, row, nvalid, lane, w_lane);
    float bad = 0.f;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      float a[2], aw[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int t = t0 + i + k;
        const bool ok = (have >> t) & 1u;
        const float w = TRAIN ? __shfl_sync(0xffffffffu, w_lane, t) : 0.f;
        a[k] = ok ? glu_act(g[i + k], u[i + k]) : 0.f;
        aw[k] = a[k] * w;
        if (TRAIN && t < nvalid)
          *reinterpret_cast<float2*>(pre + (size_t)(row + t) * 2 * H + (m & ~1)) =
              ok ? make_float2(g[i + k], u[i + k]) : make_float2(0.f, 0.f);
      }
      if (act.p != nullptr) bad += act.store_rows2(row + t0 + i, j, nvalid - t0 - i, a);
      if constexpr (TRAIN) bad += actw.store_rows2(row + t0 + i, j, nvalid - t0 - i, aw);
    }
    if (bad != bad) {
      if constexpr (TRAIN) {
#pragma unroll 1
        for (int t = t0; t < min(t0 + 8, nvalid); ++t) {
          const float2 q = *reinterpret_cast<const float2*>(pre + (size_t)(row + t) * 2 * H + (m & ~1));
          const float x = glu_act(q.x, q.y);       // 0 for the (0, 0) of a padding row
          if (act.p != nullptr) act.store1(row + t, j, x);
          actw.store1(row + t, j, row_token[row + t] >= 0 ? x * row_weight[row + t] : 0.f);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (t0 + i < nvalid) act.store1(row + t0 + i, j, (have >> (t0 + i)) & 1u ? glu_act(g[i], u[i]) : 0.f);
      }
    }
    if constexpr (TRAIN) {
      if (m - lane < 128) {        // these warps also fill the 64 columns behind H (see PairGlu), four rows each
        const int t = 4 * ((m - lane) >> 5) + (lane >> 3);
        const uint3 s = split3_special(__shfl_sync(0xffffffffu, w_lane, t));
        const bool first = (lane & 7) == 0;
        if (t < nvalid) {
          __nv_bfloat16* d = actw.p + (size_t)(row + t) * actw.ld + H + 8 * (lane & 7);
          *reinterpret_cast<uint4*>(d) = make_uint4(first ? s.x >> 16 : 0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(d + actw.stride) = make_uint4(first ? s.y >> 16 : 0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(d + 2 * actw.stride) = make_uint4(first ? s.z >> 16 : 0u, 0u, 0u, 0u);
        }
      }
    }
  }
};

struct F32WeightedRows {            // see PairWeightedRows
  const float* bias;
  float* y;
  const int32_t* row_token;
  const float* row_weight;
  int N;

  __device__ __forceinline__ void apply(int e, int m, int row, int nvalid, int lane, const float (&v)[16]) const {
    const float b = bias[(size_t)e * N + m];
    float w_lane;
    const unsigned have = row_info(row_token, row_weight, row, nvalid, lane, w_lane);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float w = __shfl_sync(0xffffffffu, w_lane, i);
      if ((have >> i) & 1u) y[(size_t)(row + i) * N + m] = w * (b + v[i]);
    }
  }
};

struct F32ScatterAdd {              // see PairScatterAdd
  float* dst;
  const int32_t* row_token;
  int N;

  __device__ __forceinline__ void apply(int, int m, int row, int nvalid, int lane, const float (&v)[16]) const {
    const bool odd = lane & 1;
    const int tok_lane = lane < nvalid ? row_token[row + lane] : -1;
    float lo[8], hi[8];
    pair_columns16(v, odd, lo, hi);
    const int t0 = odd ? 8 : 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int tok = __shfl_sync(0xffffffffu, tok_lane, t0 + i);
      if (tok >= 0) atomicAdd(reinterpret_cast<float2*>(dst + (size_t)tok * N + (m & ~1)), make_float2(lo[i], hi[i]));
    }
  }
};

struct F32GluBackward {             // see PairGluBackward; the gradient leaves as fp32 rows and as planes
  const float* pre;                // [rows, 2H]
  float* g_pre;                    // [rows, 2H]
  Planes g_planes;                 // [3][rows][2H]
  float* gw_row;
  const int32_t* row_token;
  const float* row_weight;
  int H;

  __device__ __forceinline__ void apply(int, int m, int row, int nvalid, int lane, const float (&v)[16]) const {
    float w_lane, dot[16];
    const unsigned have = row_info(row_token, row_weight, row, nvalid, lane, w_lane);
    const float2* src = reinterpret_cast<const float2*>(pre) + (size_t)row * H + m;
    float2* dst = reinterpret_cast<float2*>(g_pre) + (size_t)row * H + m;
    float bad = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const bool ok = (have >> i) & 1u;
      const float2 q = ok ? ld_written(src + (size_t)i * H) : make_float2(0.f, 0.f);
      const float w = __shfl_sync(0xffffffffu, w_lane, i);
      const float pg = q.x, pu = q.y;
      const float gc = fminf(pg, kLimit);
      const float uc = fminf(fmaxf(pu, -kLimit), kLimit);
      const float s = __fdividef(1.0f, 1.0f + __expf(-kAlpha * gc));
      const float gate_act = gc * s;
      dot[i] = ok ? v[i] * (uc + 1.0f) * gate_act : 0.f;
      const float gi = w * v[i];
      float gu = gi * gate_act;
      float gg = gi * (uc + 1.0f) * (s + gc * s * (1.0f - s) * kAlpha);
      if (pg > kLimit || !ok) gg = 0.f;
      if (pu > kLimit || pu < -kLimit || !ok) gu = 0.f;
      if (i < nvalid) {
        dst[(size_t)i * H] = make_float2(gg, gu);
        bad += g_planes.store2(row + i, 2 * m, gg, gu);
      }
    }
    if (bad != bad) {
#pragma unroll 1
      for (int i = 0; i < nvalid; ++i) {
        const float2 q = dst[(size_t)i * H];
        g_planes.store1(row + i, 2 * m, q.x);
        g_planes.store1(row + i, 2 * m + 1, q.y);
      }
    }
    // lane L ends with half the sum of row L & 15, its partner L ^ 16 with the other half
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < o; ++i) {
        const float got = __shfl_xor_sync(0xffffffffu, up ? dot[i] : dot[i + o], o);
        dot[i] = (up ? dot[i + o] : dot[i]) + got;
      }
    }
    dot[0] += __shfl_xor_sync(0xffffffffu, dot[0], 16);
    if (lane < 16 && ((have >> lane) & 1u)) atomicAdd(gw_row + row + lane, dot[0]);
  }
};

struct F32StoreBias {               // see PairStoreBias
  float* C;
  float* bias_out;
  int H, ld;

  __device__ __forceinline__ void apply(int e, int m, int row, int, int, const float (&v)[16]) const {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int n = row + i;
      if (n < H) C[((size_t)e * H + n) * ld + m] = v[i];
      else if (n == H) bias_out[(size_t)e * ld + m] = v[i];
    }
  }
};

struct F32Params {
  int M, N, K, E;
  int row_round;                   // see PairParams
  const int32_t* pad_off;
  const int32_t* counts;
  int32_t* header;
  int b_stages;
};

// Rows of a tile where an expert's rows (a multiple of 16) are cut into cnt >= 1 tiles; the last one takes the rest.
__device__ __forceinline__ int f32_tile_rows(int rows, int cnt) {
  return cnt == 1 ? rows : (int)(((unsigned)(rows + cnt - 1) / (unsigned)cnt + 15u) & ~15u);
}

// tcgen05.mma with the A operand in TMEM (each CTA of the pair holds its own 128 rows)
__device__ __forceinline__ void tc2_mma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                                uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_st_32x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
               ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tc_st_32x1(uint32_t taddr, uint32_t r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%1], {%0};" ::"r"(r), "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
// whether an mbarrier phase is over, for a first look at several: a look takes some 120 clocks, several side by side no more
__device__ __forceinline__ bool mbar_ready(uint32_t bar, uint32_t parity) { return mbar_try_wait(bar, parity) != 0; }
template <int N> __device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

template <int MODE, class Epi>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kF32Threads, 1)
umma_f32_kernel(const __grid_constant__ CUtensorMap tmM, const __grid_constant__ CUtensorMap tmN,
                const __grid_constant__ CUtensorMap tmN64, const __grid_constant__ CUtensorMap tmN32, const F32Params p,
                const Epi epi) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_w_full[kF32WStages], bar_w_empty[kF32WStages];
  __shared__ __align__(8) uint64_t bar_b_full[kF32BStages], bar_b_empty[kF32BStages];
  __shared__ __align__(8) uint64_t bar_a_full[2], bar_a_empty[2];
  __shared__ __align__(8) uint64_t bar_acc_full[2], bar_acc_empty[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag, s_cost[kF32Tiles];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t smem_b = smem_base + kF32WStages * kF32WBytes;
  int32_t* s_pad = reinterpret_cast<int32_t*>(smem_raw + kF32WStages * kF32WBytes + p.b_stages * kF32BBytes + 1024);
  int32_t* s_first = s_pad + p.E + 1;  // [E + 1] row-tiled: first tile of each expert; s_pad [E + 1]: first padded row
  int32_t* s_rows = s_first + p.E + 1; // [E] rows to cover

  if (threadIdx.x == 0) {
    for (int s = 0; s < kF32WStages; ++s) {
      mbar_init(smem_u32(&bar_w_full[s]), 1);
      mbar_init(smem_u32(&bar_w_empty[s]), kF32ConvWarps);
    }
    for (int s = 0; s < kF32BStages; ++s) {
      mbar_init(smem_u32(&bar_b_full[s]), 2);                    // leader's: both producers
      mbar_init(smem_u32(&bar_b_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&bar_a_full[s]), 2 * kF32ConvWarps);    // leader's
      mbar_init(smem_u32(&bar_a_empty[s]), 1);
      mbar_init(smem_u32(&bar_acc_full[s]), 1);
      mbar_init(smem_u32(&bar_acc_empty[s]), 2 * kF32AccWarps);  // leader's
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // the peer's barriers exist before any remote signal is sent
  tc_fence_after();
  pdl_trigger();
  pdl_wait();
  for (int i = threadIdx.x; i <= p.E; i += kF32Threads) {
    const int p0 = p.pad_off[i];
    s_pad[i] = p0;
    if (i < p.E) {
      s_rows[i] = covered_rows(p.counts[i], p.pad_off[i + 1] - p0, p.row_round);
    }
  }
  __syncthreads();
  const uint32_t tmem_base = tmem_base_slot;

  const int MT = (p.M + 2 * kF32M - 1) / (2 * kF32M);
  const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  if (MODE != kWgrad && warp >= 4 && warp < 4 + kF32Tiles) {
    // Most rows of a tile: the candidate (one to a warp) with the smallest product of waves and clocks of its widest k-block, 12
    // per row on the tensor core (24 instructions) but no less than kConvClocks for the weights' conversion and the chain of
    // signals around it; of equals the one of fewest rows (by most rows, skewed routing, H = 1024, E = 16: T = 600 122 us, now 112;
    // T = 800 128, now 122).  kConvClocks, H = 2880, E = 8, skewed: with 1400 it cuts too finely (T = 333 296 us against 271, T = 1100
    // 688 against 655), with 2000 too coarsely (T = 800 512 against 482); with 1600 H = 2048, E = 16, K = 4, T = 1000 takes 576, now 558.
    // By one warp after the other this stood before the first load of every launch: training step of 600 tokens 379 us, now 364.
    constexpr int kConvClocks = 1800;
    const int cap = kF32N - 16 * (warp - 4);
    int n = 0, widest = 0;
#pragma unroll 1
    for (int e = lane; e < p.E; e += 32) {
      const int rows = s_rows[e], cnt = (int)((unsigned)(rows + cap - 1) / (unsigned)cap);
      n += cnt;
      if (cnt > 0) widest = max(widest, f32_tile_rows(rows, cnt));
    }
    n = __reduce_add_sync(0xffffffffu, n);
    widest = __reduce_max_sync(0xffffffffu, widest);
    if (lane == 0) s_cost[warp - 4] = (n * MT + n_clusters - 1) / n_clusters * max(12 * widest, kConvClocks);
  }
  __syncthreads();
  if (MODE != kWgrad && warp == 4) {
    int tile = kF32N, best = s_cost[0];
#pragma unroll
    for (int i = 1; i < kF32Tiles; ++i)
      if (s_cost[i] <= best) { best = s_cost[i]; tile = kF32N - 16 * i; }
    int before = 0;
#pragma unroll 1
    for (int e0 = 0; e0 < p.E; e0 += 32) {
      const int n = e0 + lane < p.E ? (s_rows[e0 + lane] + tile - 1) / tile : 0;
      int inc = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (e0 + lane < p.E) s_first[e0 + lane] = before + inc - n;
      before += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) s_first[p.E] = before;
  }
  __syncthreads();
  const int NT = (p.N + kF32WgradN - 1) / kF32WgradN;       // kWgrad
  const int total = (MODE == kWgrad ? p.E * NT : s_first[p.E]) * MT;
  // as in umma_pair.cuh; e: expert of an earlier item of the same role, moved on
  auto decode = [&](int id, int& e, int& m0, int& n0, int& width, int& kblocks) {
    if constexpr (MODE == kWgrad) {
      e = id / (MT * NT);
      const int rem = id - e * (MT * NT);
      const int nt = rem / MT;
      m0 = (rem - nt * MT) * 2 * kF32M + (int)rank * kF32M;
      n0 = nt * kF32WgradN;
      const int left = p.N - n0;
      width = left > 64 ? kF32WgradN : (left + 15) & ~15;   // a 64-column box per CTA, or both halves in one box
      kblocks = s_rows[e] / kF32K;
    } else {
      while (s_first[e + 1] * MT <= id) ++e;
      const int cnt = s_first[e + 1] - s_first[e];
      const int local = id - s_first[e] * MT;
      const int mt = cnt == 1 ? local : local / cnt;
      const int rows = s_rows[e];
      const int step = f32_tile_rows(rows, cnt);
      const int off = (local - mt * cnt) * step;
      m0 = mt * 2 * kF32M + (int)rank * kF32M;
      n0 = s_pad[e] + off;
      width = min(step, rows - off);
      kblocks = p.K / kF32K;
    }
  };
  auto give_up = [&](int status) {
    abort_flag = 1;
    atomicMax(p.header + kHdrStatus, status);
  };

  if (warp < 4) {
  fewer_registers<kF32RegsIssue>();
  if (warp == 0) {
    // =========================== TMA producer ================================================
    if (lane == 0) {
      int ws = 0, bs = 0;
      uint32_t wph = 0, bph = 0;
      bool ok = true;
      // weights run one k-block ahead of the activations (they are released earlier)
      int w_id = cluster_id, w_kb = 0;
      int w_e = 0, w_m0 = 0, w_n0 = 0, w_width = 0, w_kblocks = 0;
      auto w_open = [&]() {                         // next work item that has k-blocks
        while (w_id < total) {
          decode(w_id, w_e, w_m0, w_n0, w_width, w_kblocks);
          if (w_kblocks > 0) return;
          w_id += n_clusters;
        }
      };
      auto w_issue = [&]() -> bool {
        if (w_id >= total) return true;
        if (!mbar_wait(smem_u32(&bar_w_empty[ws]), wph ^ 1u, &abort_flag)) return false;
        const uint32_t full = smem_u32(&bar_w_full[ws]);
        const uint32_t sw = smem_base + ws * kF32WBytes;
        const int k0 = w_kb * kF32K;
        mbar_expect_tx(full, kF32WBytes);
        if constexpr (MODE == kFwd) {
          tma_load_3d(sw, &tmM, w_m0, k0, w_e, full);
        } else if constexpr (MODE == kDgrad) {
          tma_load_3d(sw, &tmM, k0, w_m0, w_e, full);
          tma_load_3d(sw + kF32WBytes / 2, &tmM, k0 + 32, w_m0, w_e, full);
        } else {
          tma_load_2d(sw, &tmM, w_m0, s_pad[w_e] + k0, full);
        }
        if (++ws == kF32WStages) { ws = 0; wph ^= 1u; }
        if (++w_kb == w_kblocks) {
          w_kb = 0;
          w_id += n_clusters;
          w_open();
        }
        return true;
      };
      w_open();
      ok = w_issue();
      int e = 0;
      for (int id = cluster_id; id < total && ok; id += n_clusters) {
        int m0, n0, width, kblocks;
        decode(id, e, m0, n0, width, kblocks);
        const int half = width >> 1;
        // this CTA's rows (columns) of the N operand: one box of 80, 64 or 32
        const int box = MODE == kWgrad ? 64 : half > 64 ? 80 : half > 32 ? 64 : 32;
        const uint32_t bytes = (uint32_t)box * (3 * kF32K * 2);
        const int my_n = n0 + (int)rank * half;
        for (int kb = 0; kb < kblocks; ++kb) {
          ok = w_issue() && mbar_wait(smem_u32(&bar_b_empty[bs]), bph ^ 1u, &abort_flag);
          if (!ok) break;
          const uint32_t full = mapa_u32(smem_u32(&bar_b_full[bs]), 0);
          const uint32_t sb = smem_b + bs * kF32BBytes;
          mbar_expect_tx_cluster(full, bytes);
          if constexpr (MODE == kWgrad) tma2_load_4d(sb, &tmN, my_n & 63, s_pad[e] + kb * kF32K, my_n >> 6, 0, full);
          else tma2_load_3d(sb, box == 80 ? &tmN : box == 64 ? &tmN64 : &tmN32, kb * kF32K, my_n, 0, full);
          if (++bs == p.b_stages) { bs = 0; bph ^= 1u; }
        }
      }
      // the commits that free the last stages must have arrived here before this CTA ends
      for (int g = 0; g < p.b_stages && ok; ++g) {
        ok = mbar_wait(smem_u32(&bar_b_empty[bs]), bph ^ 1u, &abort_flag);
        if (++bs == p.b_stages) { bs = 0; bph ^= 1u; }
      }
      if (!ok) give_up(kStatusProducerTimeout);
    }
    __syncwarp();
  } else if (warp == 1) {
    // =========================== MMA issuer (leader CTA only; see umma_pair.cuh) ==============
    if (leader) {
      constexpr bool kBMn = MODE == kWgrad;
      constexpr uint32_t idesc_base = (1u << 4) | (1u << 7) | (1u << 10) | ((kBMn ? 1u : 0u) << 16) |
                                      ((uint32_t)(2 * kF32M >> 4) << 24);
      constexpr uint32_t b_kstep = kBMn ? (16 * 128) >> 4 : 32 >> 4;
      // parts (of M operand, of N operand), smallest products first
      constexpr int kPartA[6] = {0, 2, 1, 0, 1, 0}, kPartB[6] = {2, 0, 1, 1, 0, 0};
      const uint64_t bdesc0 = make_smem_desc(smem_b, kBMn ? 8192 : 16, 1024);
      const bool elected = elect_one();
      int slot = 0, bs = 0;                          // A operand and accumulator: two of each; B stage
      uint32_t phase = 0, bph = 0;
      bool ok = true;
      int e = 0;
      for (int id = cluster_id; id < total && ok; id += n_clusters) {
        int m0, n0, width, kblocks;
        decode(id, e, m0, n0, width, kblocks);
        const uint32_t idesc = idesc_base | ((uint32_t)(width >> 3) << 17);
        const uint32_t plane = (uint32_t)((MODE == kWgrad ? 64 : width > 128 ? 80 : width > 64 ? 64 : 32) * kF32K * 2) >> 4;
        for (int kb = 0; kb < kblocks; ++kb) {
          const bool r0 = mbar_ready(smem_u32(&bar_acc_empty[slot]), phase ^ 1u), r1 = mbar_ready(smem_u32(&bar_b_full[bs]), bph),
                     r2 = mbar_ready(smem_u32(&bar_a_full[slot]), phase);
          ok = (r0 || mbar_wait(smem_u32(&bar_acc_empty[slot]), phase ^ 1u, &abort_flag)) &&
               (r1 || mbar_wait(smem_u32(&bar_b_full[bs]), bph, &abort_flag)) &&
               (r2 || mbar_wait(smem_u32(&bar_a_full[slot]), phase, &abort_flag));
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          if (elected) {
            const uint32_t d = tmem_base + slot * kF32N;
            const uint32_t a0 = tmem_base + kF32TmemA + slot * kF32TmemAStride;
            const uint64_t bdesc = bdesc0 + (uint64_t)(bs * (kF32BBytes >> 4));
#pragma unroll
            for (int q = 0; q < 6; ++q)
#pragma unroll
              for (int k = 0; k < kF32K / 16; ++k)
                tc2_mma_bf16_ts(d, a0 + kPartA[q] * 32 + k * 8, bdesc + (uint64_t)(kPartB[q] * plane + k * b_kstep), idesc,
                                (uint32_t)((q | k) != 0));
            tc2_commit_pair(smem_u32(&bar_a_empty[slot]));
            tc2_commit_pair(smem_u32(&bar_b_empty[bs]));
            tc2_commit_pair(smem_u32(&bar_acc_full[slot]));
          }
          __syncwarp();
          slot ^= 1;
          if (slot == 0) phase ^= 1u;
          if (++bs == p.b_stages) { bs = 0; bph ^= 1u; }
        }
      }
      if (!ok && lane == 0) give_up(kStatusMmaTimeout);
    }
    __syncwarp();
  }
  } else if (warp < 4 + kF32ConvWarps) {
    // =========================== converters: fp32 tile -> three parts in TMEM ================
    fewer_registers<kF32RegsConv>();
    const int q = warp & 3, khalf = (warp - 4) >> 2;
    const int mrow = q * 32 + lane;
    int ws = 0, slot = 0;
    uint32_t wph = 0, phase = 0;
    bool ok = true;
    int e = 0;
    for (int id = cluster_id; id < total && ok; id += n_clusters) {
      int m0, n0, width, kblocks;
      decode(id, e, m0, n0, width, kblocks);
      for (int kb = 0; kb < kblocks; ++kb) {
        const bool r0 = mbar_ready(smem_u32(&bar_w_full[ws]), wph), r1 = mbar_ready(smem_u32(&bar_a_empty[slot]), phase ^ 1u);
        if (!__all_sync(0xffffffffu, r0 && r1)) {
          ok = mbar_wait_warp(smem_u32(&bar_w_full[ws]), wph, &abort_flag) &&
               mbar_wait_warp(smem_u32(&bar_a_empty[slot]), phase ^ 1u, &abort_flag);
          if (!ok) break;
        }
        tc_fence_after();
        const uint8_t* tile = smem_raw + (smem_base - smem_u32(smem_raw)) + ws * kF32WBytes;
        const uint32_t t = tmem_base + kF32TmemA + slot * kF32TmemAStride + khalf * 16 + ((uint32_t)(q * 32) << 16);
        // MODE kDgrad: 32 k of row mrow are 128 bytes, 16-byte pieces swizzled by the row
        const uint8_t* rowp = tile + khalf * (kF32WBytes / 2) + mrow * 128;
        const float* colp = reinterpret_cast<const float*>(tile) + khalf * 32 * kF32M + mrow;
        float bad = 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {                // 16 k at a time
          float x[16];
          if constexpr (MODE == kDgrad) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 f = *reinterpret_cast<const float4*>(rowp + (((h * 4 + i) ^ (mrow & 7)) << 4));
              x[4 * i] = f.x; x[4 * i + 1] = f.y; x[4 * i + 2] = f.z; x[4 * i + 3] = f.w;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i] = colp[(h * 16 + i) * kF32M];
          }
          uint32_t p0[8], p1[8], p2[8];
          bad += split3_finite<16>(x, p0, p1, p2);
          tc_st_32x8(t + h * 8, p0);
          tc_st_32x8(t + h * 8 + 32, p1);
          tc_st_32x8(t + h * 8 + 64, p2);
        }
        if (__any_sync(0xffffffffu, bad != bad)) {
          tc_st_wait();
#pragma unroll 1
          for (int i = 0; i < 16; ++i) {             // rolled, from memory again: rare, and the hot code stays short
            float y0, y1;
            if constexpr (MODE == kDgrad) {
              const uint8_t* piece = rowp + (((i >> 1) ^ (mrow & 7)) << 4) + 8 * (i & 1);
              y0 = *reinterpret_cast<const float*>(piece);
              y1 = *reinterpret_cast<const float*>(piece + 4);
            } else {
              y0 = colp[2 * i * kF32M];
              y1 = colp[(2 * i + 1) * kF32M];
            }
            const uint3 s0 = split3_special(y0), s1 = split3_special(y1);
            tc_st_32x1(t + i, __byte_perm(s0.x, s1.x, 0x7632));
            tc_st_32x1(t + i + 32, __byte_perm(s0.y, s1.y, 0x7632));
            tc_st_32x1(t + i + 64, __byte_perm(s0.z, s1.z, 0x7632));
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_w_empty[ws]));
        if (++ws == kF32WStages) { ws = 0; wph ^= 1u; }
        tc_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&bar_a_full[slot]), 0));
        slot ^= 1;
        if (slot == 0) phase ^= 1u;
      }
    }
    // the commits that free the last operands must have arrived here before this CTA ends
    for (int g = 0; g < 2 && ok; ++g) {
      ok = mbar_wait_warp(smem_u32(&bar_a_empty[slot]), phase ^ 1u, &abort_flag);
      slot ^= 1;
      if (slot == 0) phase ^= 1u;
    }
    if (!ok) give_up(kStatusMmaTimeout);
    __syncwarp();
  } else {
    // =========================== accumulators and epilogue ===================================
    more_registers<kF32RegsAcc>();
    const int q = warp & 3, third = (warp - 4 - kF32ConvWarps) >> 2;   // takes the 16-column chunks third, third + 3, ...
    int slot = 0;
    uint32_t phase = 0;
    bool ok = true;
    int e = 0;
    for (int id = cluster_id; id < total && ok; id += n_clusters) {
      int m0, n0, width, kblocks;
      decode(id, e, m0, n0, width, kblocks);
      float acc[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = 0.f;
      for (int kb = 0; kb < kblocks; ++kb) {
        ok = mbar_wait_warp(smem_u32(&bar_acc_full[slot]), phase, &abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t t = tmem_base + slot * kF32N + third * 16 + ((uint32_t)(q * 32) << 16);
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if ((third + 3 * c) * 16 < width) {
            uint32_t r[16];
            tc_ld_32x16(t + c * 48, r);
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[c * 16 + i] += __uint_as_float(r[i]);
          }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&bar_acc_empty[slot]), 0));
        slot ^= 1;
        if (slot == 0) phase ^= 1u;
      }
      if (!ok) break;
      const int m = m0 + q * 32 + lane;
      if (m - lane < p.M) {                          // M is a multiple of 32
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (const int n = (third + 3 * c) * 16; n < width) {
            float v[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = acc[c * 16 + i];
            epi.apply(e, m, n0 + n, min(16, width - n), lane, v);
          }
      }
    }
    if (!ok) give_up(kStatusEpilogueTimeout);
    __syncwarp();
  }

  // ---- teardown ---------------------------------------------------------------------------
  tc_fence_before();
  __syncthreads();
  if (abort_flag != 0) {
    // give copies that may still be in flight time to land before the shared memory is released
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();          // neither CTA releases shared memory or TMEM the pair may still use
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// Most tiles of at least 80 rows (the smallest candidate) that the padded rows make.
inline int64_t f32_max_tiles(int64_t max_rows, int E) { return max_rows / 80 + E; }

// GemmArgs as for launch_umma_pair: A / lda describe the planes (N operand; `a_plane` elements
// between planes), B / ldb the fp32 operand.  All widths and pitches are multiples of 64.
template <int MODE, class Epi>
inline int launch_umma_f32(const GemmArgs& g, int64_t a_plane, const Epi& epi, int64_t max_rows, int row_round,
                           cudaStream_t stream) {
  if (!umma_available() || g.E > kUmmaMaxExperts) return YAMOE_ERR_UNSUPPORTED;
  CUtensorMap tmM, tmN, tmN64, tmN32;
  bool ok = true;
  if (MODE == kWgrad) {
    const uint64_t dn[4] = {64, (uint64_t)max_rows, (uint64_t)g.lda / 64, 3};
    const uint64_t sn[3] = {(uint64_t)g.lda * 2, 128, (uint64_t)a_plane * 2};
    const uint32_t b1[4] = {64, 64, 1, 3};
    ok = make_map(&tmN, g.A, 4, dn, sn, b1);
    tmN64 = tmN32 = tmN;                 // not used
    const uint64_t dm[2] = {(uint64_t)g.N, (uint64_t)max_rows}, sm[1] = {(uint64_t)g.ldb * 4};
    const uint32_t bm[2] = {kF32M, kF32K};
    ok = ok && make_map(&tmM, g.B, 2, dm, sm, bm, kMapF32);
  } else {
    const uint64_t dn[3] = {(uint64_t)g.K, (uint64_t)max_rows, 3};
    const uint64_t sn[2] = {(uint64_t)g.lda * 2, (uint64_t)a_plane * 2};
    const uint32_t b80[3] = {64, 80, 3}, b64[3] = {64, 64, 3}, b32[3] = {64, 32, 3};
    ok = make_map(&tmN, g.A, 3, dn, sn, b80) && make_map(&tmN64, g.A, 3, dn, sn, b64) && make_map(&tmN32, g.A, 3, dn, sn, b32);
    const uint64_t sm[2] = {(uint64_t)g.ldb * 4, (uint64_t)g.b_expert_stride * 4};
    if (MODE == kFwd) {
      const uint64_t dm[3] = {(uint64_t)g.N, (uint64_t)g.K, (uint64_t)g.E};
      const uint32_t bm[3] = {kF32M, kF32K, 1};
      ok = ok && make_map(&tmM, g.B, 3, dm, sm, bm, kMapF32);
    } else {
      const uint64_t dm[3] = {(uint64_t)g.K, (uint64_t)g.N, (uint64_t)g.E};
      const uint32_t bm[3] = {32, kF32M, 1};
      ok = ok && make_map(&tmM, g.B, 3, dm, sm, bm, kMapF32Swizzled);
    }
  }
  if (!ok) return YAMOE_ERR_CUDA;
  auto kern = umma_f32_kernel<MODE, Epi>;
  static PerDevice<int> resident;    // per template instantiation and device
  const int pairs = resident_pairs(kern, kF32Threads, kMaxDynamicSmem, resident);
  if (pairs <= 0) return YAMOE_ERR_CUDA;
  const int b_stages = f32_smem(g.E, kF32BStages) <= kMaxDynamicSmem ? kF32BStages : kF32BStages - 1;
  const F32Params p{g.N, g.M, g.K, g.E, row_round, g.pad_off, g.counts, const_cast<int32_t*>(g.header), b_stages};
  const int64_t MT = ceil_div(g.N, 2 * kF32M);
  const int64_t total_max = MODE == kWgrad ? (int64_t)g.E * MT * ceil_div(g.M, kF32WgradN) : f32_max_tiles(max_rows, g.E) * MT;
  const int grid = (int)(2 * std::min<int64_t>(total_max, pairs));
  if (grid <= 0) return YAMOE_OK;
  if (launch_pdl_opt(true, kern, dim3(grid), dim3(kF32Threads), f32_smem(g.E, b_stages), stream, tmM, tmN, tmN64, tmN32, p, epi) != cudaSuccess)
    return YAMOE_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? YAMOE_OK : YAMOE_ERR_CUDA;
}

}  // namespace yb
