// Grouped GEMM of CTA pairs (tcgen05 cta_group::2) with the token rows in the N dimension of the
// instruction: the kernel of the single-GPU forward, backward and training paths (bf16 operands,
// fp32 accumulation in TMEM, sm_100a).
//
//   arrangement   M operand (256 per pair)                     N operand (up to 256)
//   kFwd          W[e][k][m]   weight columns, MN-major        rows of the expert, K-major
//   kDgrad        W[e][m][k]   weight rows, K-major            rows of the expert, K-major
//   kWgrad        grad[r][m]   columns, MN-major, k = rows     act[r][n] columns, MN-major
//
// What bounds it: power for the large problems (the SM clock falls to 1.3 - 1.4 GHz), HBM below about 100 rows per
// expert.  Measured against the one-CTA kernel that it replaced, whole calls: T = 512 (E = 32, H = 2880)
// 357 -> 311 us, 64 tokens through the layer 353 -> 291, T = 1531 (E = 64, K = 8, H = 2048) 517 -> 437,
// T = 4096 952 -> 894, T = 16384 (E = 128, skewed) 3840 -> 3560, gradients at T = 8192 5018 -> 4572.
//
// Why this split.  The one-CTA kernel (128 rows x 256 columns) was bound by what L2 delivers to an
// SM: 48 KB per 64-deep k-block are 96 bytes per clock at full tensor rate, where an SM gets about
// 73.  A pair computes 256 x 256 and each CTA stages 128 rows of either operand: 32 KB per k-block,
// 64 bytes per clock.  And M is the dimension that comes in steps of 256 whatever the problem is,
// while N may be any multiple of 16: with the tokens in N, an expert's rows are split into tiles
// of equal width and no instruction is spent on padding beyond 16 rows (the one-CTA kernel padded
// every expert to 128 rows, 12 % of all instructions with 512 rows per expert and half of them with
// 64).  The weights' last M tile may be partly empty: 2880 columns take 12 pairs of which the last
// has 64 columns, 6.7 %; 5760 take 23, 2.2 %.
//
// A CTA has 11 or 19 warps: two TMA producers, MMA issuer (of the leader only), eight or sixteen epilogue warps (two or four
// per TMEM lane quarter, which take 32-column chunks in turn; see pair_16_warps).  A larger item, 512 rows in two accumulators
// that share the weight slab, was no gain: 25 % fewer operand bytes, but the rings that it needs cost the issuer a second
// wait per k-block (7 to 10 % of any launch), and an accumulator must be drained while the other is filled (T = 4096
// 715 -> 768 .. 868 us in four forms).  Six stages of 32 KB; two accumulators of
// 256 TMEM columns, so that the epilogue of a tile overlaps the main loop of the next.  The
// epilogue thread of lane m holds 32 rows' values of ONE weight column: bias and column sums are per
// thread, and the rows of the output are written by the lanes of a warp side by side.
//
// The issuing warps walk their loops as whole warps and elect a lane for the instruction itself: with
// the loop inside `if (lane == 0)` every descriptor moved through per-thread registers, and issuing was
// slower than the tensor core (gate_up at T = 4096 without any loads: 433 us, now 286; the loads
// without any MMA, one producer lane against two producer warps: 422 us and 319).
//
// Signals: both producers post their bytes on the leader's full barrier; one tcgen05.commit
// multicast to both CTAs frees a stage or publishes an accumulator; the epilogue warps of both CTAs
// arrive on the leader's accumulator-empty barrier.  No TMA multicast: each CTA loads its own
// operands.  Every wait is bounded as in umma_gemm.cuh.
#pragma once
#include "umma_gemm.cuh"

namespace yb {

constexpr int kPairM = 256, kPairN = 256;
constexpr int kPairABytes = 128 * 128;     // this CTA's 128 M rows x 64 bf16
constexpr int kPairBBytes = 128 * 128;     // this CTA's half of the N rows (up to 128) x 64 bf16
constexpr int kPairStageBytes = kPairABytes + kPairBBytes;
constexpr int kPairStages = 6;
constexpr int kPairGroups = kPairStages / 2;   // stages are freed two at a time
constexpr int kPairSmem = kPairStages * kPairStageBytes + 1024;   // + slack for 1024-byte alignment
constexpr int kPairParkBytes = 32 * 128 * 2;   // parked output rows of four epilogue warps (PairStoreBias)

__device__ __forceinline__ void mbar_expect_tx_cluster(uint32_t bar_cluster_addr, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(bar_cluster_addr), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ void tma2_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma2_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2,
                                             uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tma2_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                             uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
// arrives on the barrier at this shared-memory offset in both CTAs of the pair once every MMA issued so far is done
__device__ __forceinline__ void tc2_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tc2_mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// true in one lane of the (converged) warp
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r != 0;
}

struct PairParams {
  int M;                        // M dimension of the instruction: weight columns / rows, grad columns
  int N;                        // kWgrad: columns of the activations; otherwise the rows come from the tables
  int K, E;                     // kFwd / kDgrad: reduction length
  int row_round;                // rows of an expert are covered up to this multiple (16 or 64)
  const int32_t* pair_expert;   // expert of every tile of up to 256 rows
  const int32_t* pair_off;      // [E+1] prefix sums of those tiles
  const int32_t* pad_off;
  const int32_t* counts;
  int32_t* header;
  int groups;                   // of four epilogue warps, which take the chunks of a tile in turn
};

// ---------------------------------------------------------------------------------------------
// Epilogues.  A warp holds 32 consecutive M indices (lane L: m) for 32 consecutive N indices:
//     epi.apply(e, m, row, nvalid, lane, v)      v[i] = C[row + i][m];  only i < nvalid exist
// For the row-tiled arrangements `row` is a row of the padded layout, for kWgrad an output row.
// ---------------------------------------------------------------------------------------------

// Neighbouring lanes hold neighbouring columns: after the exchange the even lane has columns (m, m+1)
// of rows 0..15, the odd lane columns (m-1, m) of rows 16..31.
__device__ __forceinline__ void pair_columns(const float (&v)[32], bool odd, float (&lo)[16], float (&hi)[16]) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float got = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[16 + i], 1);
    lo[i] = odd ? got : v[i];
    hi[i] = odd ? v[16 + i] : got;
  }
}

// + bias, clamped SwiGLU of the interleaved (gate, up) columns; reference: csrc/moe.cpp:163-180.
// Outputs: `act` (activation) and, for a backward pass, `pre` (biased pre-activations) and `actw`
// (activation times routing weight, rows actw_ld = H + 64 apart; the columns behind the H activations are
// (w, 0, 0, ...), see EpiGlu).  The backward outputs of padding rows are exact zeros.
template <bool TRAIN>
struct PairGlu {
  const __nv_bfloat16* bias;       // [E, 2H]
  __nv_bfloat16* act;              // [rows, H] or null (TRAIN)
  __nv_bfloat16* actw;             // TRAIN: [rows, actw_ld]
  __nv_bfloat16* pre;              // TRAIN: [rows, 2H]
  const int32_t* row_token;        // TRAIN
  const float* row_weight;         // TRAIN
  int H, actw_ld;

  __device__ __forceinline__ void apply(int e, int m, int row, int nvalid, int lane, const float (&v)[32]) const {
    const bool odd = lane & 1;
    const float b = __bfloat162float(bias[(size_t)e * 2 * H + m]);
    float x[32], g[16], u[16];
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = v[i] + b;
    pair_columns(x, odd, g, u);
    const int t0 = odd ? 16 : 0;
    const int j = m >> 1;
    if constexpr (!TRAIN) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float a = glu_act(g[i], u[i]);
        if (t0 + i < nvalid) act[(size_t)(row + t0 + i) * H + j] = __float2bfloat16_rn(a);
      }
    } else {
      float w_lane = 0.f;
      bool real = false;
      if (lane < nvalid) {
        real = row_token[row + lane] >= 0;
        if (real) w_lane = row_weight[row + lane];
      }
      const unsigned have = __ballot_sync(0xffffffffu, real);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int t = t0 + i;
        const float w = __shfl_sync(0xffffffffu, w_lane, t);
        const bool ok = (have >> t) & 1u;
        const uint32_t packed = ok ? pack_bf16x2(g[i], u[i]) : 0u;
        // the backward pass re-derives the activation from the stored (rounded) pre-activations; 0 for (0, 0)
        const float a = glu_act(__uint_as_float(packed << 16), __uint_as_float(packed & 0xffff0000u));
        if (t < nvalid) {
          const size_t r = row + t;
          *reinterpret_cast<uint32_t*>(pre + r * 2 * H + (m & ~1)) = packed;
          if (act != nullptr) act[r * H + j] = __float2bfloat16_rn(a);
          actw[r * actw_ld + j] = __float2bfloat16_rn(a * w);
        }
      }
      // The warps with columns 0..127 also fill the 64 columns behind H, eight rows each, eight columns to a lane.  As a
      // loop of one warp over all rows with 4 bytes to a lane this was half of the kernel (gate_up at T = 2000,
      // E = 32: H = 512 68 us, now 39; H = 1024 96 and 69), and the backward pass at H <= 512 slower than with the
      // one-CTA kernel.
      if (m - lane < 128) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int t = 8 * ((m - lane) >> 5) + 4 * i + (lane >> 3);
          const float w = __shfl_sync(0xffffffffu, w_lane, t);
          if (t < nvalid)
            *reinterpret_cast<uint4*>(actw + (size_t)(row + t) * actw_ld + H + 8 * (lane & 7)) =
                make_uint4((lane & 7) == 0 ? pack_bf16x2(w, 0.f) : 0u, 0u, 0u, 0u);
        }
      }
    }
  }
};

// y[row] = w_row * (v + bias); the K rows of a token are summed by combine_padded_kernel.
// reference: csrc/moe.cpp:187, csrc/scatter.cu:98-106
struct PairWeightedRows {
  const __nv_bfloat16* bias;       // [E, N]
  __nv_bfloat16* y;                // [rows, N]
  const int32_t* row_token;
  const float* row_weight;
  int N;

  __device__ __forceinline__ void apply(int e, int m, int row, int nvalid, int lane, const float (&v)[32]) const {
    const bool odd = lane & 1;
    const float b = __bfloat162float(bias[(size_t)e * N + m]);
    float w_lane = 0.f;
    bool real = false;
    if (lane < nvalid) {
      real = row_token[row + lane] >= 0;
      if (real) w_lane = row_weight[row + lane];
    }
    const unsigned have = __ballot_sync(0xffffffffu, real);
    float x[32], lo[16], hi[16];
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = b + v[i];
    pair_columns(x, odd, lo, hi);
    const int t0 = odd ? 16 : 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int t = t0 + i;
      const float w = __shfl_sync(0xffffffffu, w_lane, t);
      if ((have >> t) & 1u)
        *reinterpret_cast<uint32_t*>(y + (size_t)(row + t) * N + (m & ~1)) = pack_bf16x2(w * lo[i], w * hi[i]);
    }
  }
};

// The same in fp32, y[flat position of the row] = w_row * (v + bias): decode-sized calls, whose rows the GEMV
// kernels sum in fp32 (decode_sized).  At most 256 rows, so their bytes do not matter; rounded to bf16 first
// they took the error of 16 tokens (E = 128, H = 2880) against 64 bits from 2.3e-3 to 2.9e-3.
struct PairWeightedFlat {
  const __nv_bfloat16* bias;       // [E, N]
  float* y;                        // [S, N]
  const int32_t* row_token;
  const int32_t* row_flat;
  const float* row_weight;
  int N;

  __device__ __forceinline__ void apply(int e, int m, int row, int nvalid, int lane, const float (&v)[32]) const {
    const bool odd = lane & 1;
    const float b = __bfloat162float(bias[(size_t)e * N + m]);
    float w_lane = 0.f;
    int p_lane = -1;
    if (lane < nvalid && row_token[row + lane] >= 0) {
      w_lane = row_weight[row + lane];
      p_lane = row_flat[row + lane];
    }
    float x[32], lo[16], hi[16];
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = b + v[i];
    pair_columns(x, odd, lo, hi);
    const int t0 = odd ? 16 : 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float w = __shfl_sync(0xffffffffu, w_lane, t0 + i);
      const int p = __shfl_sync(0xffffffffu, p_lane, t0 + i);
      if (p >= 0) *reinterpret_cast<float2*>(y + (size_t)p * N + (m & ~1)) = make_float2(w * lo[i], w * hi[i]);
    }
  }
};

// dst[token] += v in fp32 (data gradient of the hidden states; reference: csrc/experts_backward.cu:92-124)
struct PairScatterAdd {
  float* dst;                      // [T, N]
  const int32_t* row_token;
  int N;

  __device__ __forceinline__ void apply(int, int m, int row, int nvalid, int lane, const float (&v)[32]) const {
    const bool odd = lane & 1;
    const int tok_lane = lane < nvalid ? row_token[row + lane] : -1;
    float lo[16], hi[16];
    pair_columns(v, odd, lo, hi);
    const int t0 = odd ? 16 : 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int tok = __shfl_sync(0xffffffffu, tok_lane, t0 + i);
      if (tok >= 0) atomicAdd(reinterpret_cast<float2*>(dst + (size_t)tok * N + (m & ~1)), make_float2(lo[i], hi[i]));
    }
  }
};

// Data gradient of the down projection with the GLU backward (see EpiGluBackward): v is
// (grad_y . W_d^T)[m], the pre-activations of the pair lie side by side, 4 bytes per lane.
struct PairGluBackward {
  static constexpr bool kPrefetchTile = true;
  const __nv_bfloat16* pre;        // [rows, 2H]
  __nv_bfloat16* g_pre;            // [rows, 2H]
  float* gw_row;                   // [rows]
  const int32_t* row_token;
  const float* row_weight;
  int H;

  // asks L2 for the 128 bytes of each of 32 rows that apply() will read: called while the tile's main
  // loop runs, since four dependent trips to HBM are as long as that loop
  __device__ __forceinline__ void prefetch(int m, int row, int nvalid, int lane) const {
    if (lane < nvalid)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(pre + (size_t)(row + lane) * 2 * H + 2 * (m - lane)));
  }

  __device__ __forceinline__ void apply(int, int m, int row, int nvalid, int lane, const float (&v)[32]) const {
    float w_lane = 0.f;
    bool real = false;
    if (lane < nvalid) {
      real = row_token[row + lane] >= 0;
      if (real) w_lane = row_weight[row + lane];
    }
    const unsigned have = __ballot_sync(0xffffffffu, real);
    float dot[32];
    const uint32_t* src = reinterpret_cast<const uint32_t*>(pre) + (size_t)row * H + m;
    uint32_t* dst = reinterpret_cast<uint32_t*>(g_pre) + (size_t)row * H + m;
    uint32_t p[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) p[i] = ((have >> i) & 1u) ? __ldcs(src + (size_t)i * H) : 0u;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const float w = __shfl_sync(0xffffffffu, w_lane, i);
      const float pg = __uint_as_float(p[i] << 16), pu = __uint_as_float(p[i] & 0xffff0000u);
      const float gc = fminf(pg, kLimit);
      const float uc = fminf(fmaxf(pu, -kLimit), kLimit);
      const float s = __fdividef(1.0f, 1.0f + __expf(-kAlpha * gc));
      const float gate_act = gc * s;
      const bool ok = (have >> i) & 1u;
      dot[i] = ok ? v[i] * (uc + 1.0f) * gate_act : 0.f;
      const float gi = w * v[i];
      float gu = gi * gate_act;
      float gg = gi * (uc + 1.0f) * (s + gc * s * (1.0f - s) * kAlpha);
      if (pg > kLimit) gg = 0.f;
      if (pu > kLimit || pu < -kLimit) gu = 0.f;
      if (i < nvalid) dst[(size_t)i * H] = ok ? pack_bf16x2(gg, gu) : 0u;
    }
    // sums over the 32 lanes of all 32 rows at once: after the step of width o a lane keeps the rows
    // whose index agrees with its own in bit o, so that lane L ends with the sum of row L
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < o; ++i) {
        const float got = __shfl_xor_sync(0xffffffffu, up ? dot[i] : dot[i + o], o);
        dot[i] = (up ? dot[i + o] : dot[i]) + got;
      }
    }
    if (real) atomicAdd(gw_row + row + lane, dot[0]);
  }
};

// 32 M indices x 32 N indices of an accumulator: two TMEM loads of 16 lanes x 32 columns leave in a thread pairs of
// neighbouring N of the M indices lane / 4 + 8 i, which is how stmatrix takes the rows of 8 x 8 matrices.
__device__ __forceinline__ void tc_ld_16x256_issue(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr + (16u << 16)) : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};"
               ::"r"(addr), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}

// Weight gradient: output row n = `row` + i of C[e] ([H, ld]); row H is the bias gradient (the operand
// in N carries a column of ones or routing weights behind its H columns), later rows do not exist.
// With few rows per expert this GEMM is bound by its output (3 H^2 values per expert for as little
// as one k-block), so the tile leaves by TMA: four warps park 32 rows of 128 columns in shared memory (two boxes of 64
// columns, swizzled so that the eight rows of a matrix fall on different banks), and copies clipped at the matrix edge
// store them while the warps go on.  The transposition is stmatrix's: with shuffles and 4-byte stores the epilogue of a
// tile took longer still.  192 rows per expert (E = 64, H = 2048): gate_up 395 us with shuffles, 360 by stmatrix, 306 with
// sixteen epilogue warps instead of eight; down 205, 190, 160 (1.07 and 0.54 GB of output, 145 and 73 us at the rate of a
// fill).  Eight warps with two buffers each took 350 and 185, meeting once for two chunks 363.
struct PairStoreBias {
  static constexpr bool kTmaStore = true;
  __nv_bfloat16* C;                // [E, H, ld]
  __nv_bfloat16* bias_out;         // [E, ld]
  int H, ld;

  // accumulator values (tc_ld_16x256_issue) as bf16 pairs along N: p[4 j + h] holds N 8 j .. 8 j + 7 of M 8 h .. 8 h + 7
  static __device__ __forceinline__ void pack(const uint32_t (&r)[32], uint32_t (&p)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int i = 16 * (h >> 1) + 4 * j + 2 * (h & 1);
        p[4 * j + h] = pack_bf16x2(__uint_as_float(r[i]), __uint_as_float(r[i + 1]));
      }
  }
  static __device__ __forceinline__ void park(const uint32_t (&p)[16], int q, int lane, uint32_t buf) {
    const uint32_t row = lane & 7, piece = 4 * (q & 1) + (lane >> 3);
    const uint32_t dst = buf + (q >> 1) * (kPairParkBytes / 2) + row * 128 + ((piece ^ row) << 4);
#pragma unroll
    for (int j = 0; j < 4; ++j) stmatrix_x4_trans(dst + j * 8 * 128, p[4 * j], p[4 * j + 1], p[4 * j + 2], p[4 * j + 3]);
  }
  // parked row i is the bias gradient: one column to a thread of the group
  __device__ __forceinline__ void bias_row(int e, int cta_m, int i, int q, int lane, const uint8_t* buf) const {
    const int col = q * 32 + lane, c = col & 63;
    if (cta_m + col < ld)
      bias_out[(size_t)e * ld + cta_m + col] = *reinterpret_cast<const __nv_bfloat16*>(
          buf + (q >> 1) * (kPairParkBytes / 2) + i * 128 + (((c >> 3) ^ (i & 7)) << 4) + 2 * (c & 7));
  }
};

template <class E, class = void>
struct epi_tma_store : std::false_type {};
template <class E>
struct epi_tma_store<E, std::enable_if_t<E::kTmaStore>> : std::true_type {};

// Shared memory: ring, parking space for each group of four epilogue warps (kTmaStore), expert tables.  Beside the tables of
// more than some 140 experts there is space for two groups; the others then have no chunks.
constexpr int kMaxDynamicSmem = 227 * 1024 - 256;               // the barriers are static
inline int pair_smem(int park_groups, int E) { return kPairSmem + park_groups * kPairParkBytes + (3 * E + 2) * 4; }

// Epilogue warps: eight, or sixteen where the epilogue of a tile is long beside its main loop, as hidden behind the next
// tile it is not, or where the last one of a CTA counts; else the additional warps only wait and take power (T = 4096,
// H = 2880: 735 us with eight, 755 with sixteen).
// Weight gradients: up to some 512 rows per expert (8 / 16 warps: 192 rows, H = 2048 gate_up 359 / 306 us, down 190 / 160;
// 1024 rows, H = 2880 788 / 806 and 396 / 407; a whole backward of 16 experts, H = 2048: 100 rows 340 / 297, 320 460 / 439, 400
// 507 / 492, 512 585 / 583, 600 663 / 669, 700 767 / 783; H = 1024: 100 rows 146 / 135, 512 237 / 236, 600 253 / 254).
inline bool pair_wgrad_16_warps(int64_t S, int E) { return S <= 512 * (int64_t)E; }
// The others: main loops of up to 16 k-blocks (a forward of 16 experts, H = 1024: 192 rows 51.4 / 48.1 us, 1000 rows 115 / 110;
// 24 k-blocks, H = 1536: 192 rows 78.5 / 76.0, 512 126.1 / 126.5, 1000 201.7 / 203.9; 32, H = 2048: 192 rows 112 / 108, 512 202.0 / 202.6),
// with the longer epilogue of the GLU's backward up to 32 (192 rows, H = 2048 180 / 168; a whole backward of 1024 rows 1000 / 974).
inline bool pair_16_warps(int kblocks, bool glu_backward) { return kblocks <= (glu_backward ? 32 : 16); }

__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, int c0, int c1, int c2, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void group_sync(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }

// One outcome for the four warps of a group: they meet in group_sync for every chunk, where a warp whose wait gave
// up would be missing for good.
__device__ __forceinline__ bool group_all(int id, bool ok) {
  uint32_t all;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %2, 0;\n\tbar.red.and.pred q, %1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(all) : "r"(id), "r"((uint32_t)ok) : "memory");
  return all != 0;
}

template <int MODE, class Epi, int kEpiWarps>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(32 * (3 + kEpiWarps), 1)
umma_pair_kernel(const __grid_constant__ CUtensorMap tmM, const __grid_constant__ CUtensorMap tmN,
                 const __grid_constant__ CUtensorMap tmNsmall, const __grid_constant__ CUtensorMap tmOut,
                 const PairParams p, const Epi epi) {
  constexpr bool kStore = epi_tma_store<Epi>::value;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kPairStages];       // used in the leader CTA
  __shared__ __align__(8) uint64_t bar_empty[kPairGroups];      // per CTA
  __shared__ __align__(8) uint64_t bar_tmem_full[2];            // per CTA
  __shared__ __align__(8) uint64_t bar_tmem_empty[2];           // used in the leader CTA
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  int32_t* s_pad = reinterpret_cast<int32_t*>(smem_raw + kPairSmem + (kStore ? p.groups * kPairParkBytes : 0));
  int32_t* s_pair = s_pad + p.E + 1;   // [E + 1] row-tiled: first 256-row tile of each expert; s_pad [E + 1]: first padded row
  int32_t* s_rows = s_pair + p.E + 1;  // [E] rows to cover

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairStages; ++s) mbar_init(smem_u32(&bar_full[s]), 2);   // arrive.expect_tx of both producers
    for (int s = 0; s < kPairGroups; ++s) mbar_init(smem_u32(&bar_empty[s]), 1);
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&bar_tmem_full[a]), 1);
      mbar_init(smem_u32(&bar_tmem_empty[a]), 2 * kEpiWarps);
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
  const uint32_t tmem_base = tmem_base_slot;
  pdl_trigger();
  pdl_wait();
  for (int i = threadIdx.x; i <= p.E; i += 32 * (3 + kEpiWarps)) {
    const int p0 = p.pad_off[i];
    s_pad[i] = p0;
    if (MODE != kWgrad) s_pair[i] = p.pair_off[i];
    if (i < p.E) {
      s_rows[i] = covered_rows(p.counts[i], p.pad_off[i + 1] - p0, p.row_round);
    }
  }
  __syncthreads();

  const int MT = (p.M + kPairM - 1) / kPairM;
  const int NT = (p.N + kPairN - 1) / kPairN;     // kWgrad
  const int total = MODE == kWgrad ? p.E * MT * NT : p.header[kHdrPairs] * MT;
  const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
  // expert of a work item: the one entry that comes from global memory, asked for one item ahead
  auto expert_of = [&](int id) -> int {
    if constexpr (MODE == kWgrad) return 0;
    return id < total ? p.pair_expert[id / MT] : 0;
  };
  // work item -> expert, first M index, first N index (row or column), width (multiple of 16), k-blocks.
  // The tiles of one M slab follow each other: the CTAs running at any moment share the weight slab in L2.
  auto decode = [&](int id, int e_hint, int& e, int& m0, int& n0, int& width, int& kblocks) {
    if constexpr (MODE == kWgrad) {
      e = id / (MT * NT);
      const int rem = id - e * (MT * NT);
      const int nt = rem / MT;
      m0 = (rem - nt * MT) * kPairM;
      n0 = nt * kPairN;
      const int left = p.N - n0;
      // widths above 64 come in whole 64-column boxes per CTA; a narrower rest fits into one box
      width = left > 128 ? 256 : left > 64 ? 128 : (left + 15) & ~15;
      kblocks = s_rows[e] / kUmmaBK;
    } else {
      e = e_hint;
      const int first = s_pair[e];
      const int cnt = s_pair[e + 1] - first;
      const int local = id - first * MT;
      const int mt = local / cnt;
      const int rows = s_rows[e];
      const int step = ((rows + cnt - 1) / cnt + 63) & ~63;     // whole 32-row boxes per CTA; the last tile takes the rest
      const int off = (local - mt * cnt) * step;
      m0 = mt * kPairM;
      n0 = s_pad[e] + off;
      width = min(step, rows - off);
      kblocks = p.K / kUmmaBK;
    }
  };

  if (warp == 0 || warp == 2 + kEpiWarps) {
    // =========================== TMA producers (both CTAs) ===================================
    // One warp for the M operand, which also announces the bytes of both, and one for the N operand: a
    // warp that issues everything is slower than the tensor core.  The whole warp walks the loop (see
    // the MMA issuer); a stage cannot be filled early, both warps wait for it to be free.
    const bool for_m = warp == 0;
    const bool elected = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int e_next = expert_of(cluster_id);
    for (int id = cluster_id; id < total && ok; id += n_clusters) {
      int e, m0, n0, width, kblocks;
      decode(id, e_next, e, m0, n0, width, kblocks);
      e_next = expert_of(id + n_clusters);
      const int half = width >> 1;
      const int my_m = m0 + (int)rank * 128, my_n = n0 + (int)rank * half;
      const bool load_m = my_m < p.M;      // nothing of this CTA's M rows exists: its results are not read
      // N operand: one copy of 128 rows, or up to three of 32 (row-tiled); one copy of two or one
      // 64-column boxes (kWgrad)
      const bool big = MODE == kWgrad ? half > 64 : half > 96;
      const int small = MODE == kWgrad ? 1 : (half + 31) >> 5;
      const uint32_t bytes = (load_m ? kPairABytes : 0) + (big ? kPairBBytes : MODE == kWgrad ? 8192 : small * 4096);
      const int row_k = MODE == kWgrad ? s_pad[e] : 0;
      for (int kb = 0; kb < kblocks; ++kb) {
        if ((stage & 1) == 0) {
          ok = mbar_wait_warp(smem_u32(&bar_empty[stage >> 1]), phase ^ 1u, &abort_flag);
          if (!ok) break;
        }
        if (elected) {
          const uint32_t full = mapa_u32(smem_u32(&bar_full[stage]), 0);
          const uint32_t sa = smem_base + stage * kPairStageBytes;
          const int k0 = kb * kUmmaBK;
          if (for_m) {
            mbar_expect_tx_cluster(full, bytes);
            if (load_m) {
              if constexpr (MODE == kWgrad) tma2_load_3d(sa, &tmM, 0, row_k + k0, my_m >> 6, full);
              else if constexpr (MODE == kFwd) tma2_load_4d(sa, &tmM, 0, k0, my_m >> 6, e, full);
              else tma2_load_3d(sa, &tmM, k0, my_m, e, full);
            }
          } else {
            const uint32_t sb = sa + kPairABytes;
            if constexpr (MODE == kWgrad) {
              if (big) tma2_load_3d(sb, &tmN, 0, row_k + k0, my_n >> 6, full);
              else tma2_load_3d(sb, &tmNsmall, my_n & 63, row_k + k0, my_n >> 6, full);
            } else if (big) {
              tma2_load_2d(sb, &tmN, k0, my_n, full);
            } else {
              for (int i = 0; i < small; ++i) tma2_load_2d(sb + i * 4096, &tmNsmall, k0, my_n + 32 * i, full);
            }
          }
        }
        __syncwarp();
        if (++stage == kPairStages) { stage = 0; phase ^= 1u; }
      }
    }
    // the commits that free the last stages must have arrived here before this CTA ends
    for (int g = 0; g < kPairGroups && ok; ++g)
      ok = mbar_wait_warp(smem_u32(&bar_empty[g]), 2 * g < stage ? phase : phase ^ 1u, &abort_flag);
    if (!ok && lane == 0) {
      abort_flag = 1;
      atomicMax(p.header + kHdrStatus, (int)kStatusProducerTimeout);
    }
    __syncwarp();
  } else if (warp == 1) {
    // =========================== MMA issuer (leader CTA only) ================================
    // The whole warp walks the loop, so that descriptors and addresses stay in uniform registers; one
    // elected lane issues.
    if (leader) {
      constexpr bool kAMn = MODE != kDgrad, kBMn = MODE == kWgrad;
      // instruction descriptor without its N field (bits 17..22 = N / 8), which depends on the tile
      constexpr uint32_t idesc_base = (1u << 4) | (1u << 7) | (1u << 10) | ((kAMn ? 1u : 0u) << 15) |
                                      ((kBMn ? 1u : 0u) << 16) | ((uint32_t)(kPairM >> 4) << 24);
      constexpr uint32_t a_kstep = kAMn ? (16 * 128) >> 4 : 32 >> 4;   // descriptor units of 16 bytes
      constexpr uint32_t b_kstep = kBMn ? (16 * 128) >> 4 : 32 >> 4;
      const uint64_t adesc0 = make_smem_desc(smem_base, kAMn ? 8192 : 16, 1024);
      const uint64_t bdesc0 = make_smem_desc(smem_base + kPairABytes, kBMn ? 8192 : 16, 1024);
      const bool elected = elect_one();
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      int e_next = expert_of(cluster_id);
      for (int id = cluster_id; id < total && ok; id += n_clusters) {
        int e, m0, n0, width, kblocks;
        decode(id, e_next, e, m0, n0, width, kblocks);
        e_next = expert_of(id + n_clusters);
        if (kblocks == 0) continue;
        const uint32_t idesc = idesc_base | ((uint32_t)(width >> 3) << 17);
        ok = mbar_wait_warp(smem_u32(&bar_tmem_empty[acc]), acc_phase ^ 1u, &abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * kUmmaAccStride;
        for (int kb = 0; kb < kblocks; ++kb) {
          ok = mbar_wait_warp(smem_u32(&bar_full[stage]), phase, &abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (elected) {
            const uint64_t adesc = adesc0 + (uint64_t)(stage * (kPairStageBytes >> 4));
            const uint64_t bdesc = bdesc0 + (uint64_t)(stage * (kPairStageBytes >> 4));
#pragma unroll
            for (int k = 0; k < kUmmaBK / 16; ++k)
              tc2_mma_bf16(d_tmem, adesc + (uint64_t)(k * a_kstep), bdesc + (uint64_t)(k * b_kstep), idesc,
                           (uint32_t)((kb | k) != 0));
            if (stage & 1) tc2_commit_pair(smem_u32(&bar_empty[stage >> 1]));
            if (kb == kblocks - 1) tc2_commit_pair(smem_u32(&bar_tmem_full[acc]));
          }
          __syncwarp();
          if (++stage == kPairStages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
      if (ok && (stage & 1) && elected) tc2_commit_pair(smem_u32(&bar_empty[stage >> 1]));   // a group that is half used
      if (!ok && lane == 0) {
        abort_flag = 1;
        atomicMax(p.header + kHdrStatus, (int)kStatusMmaTimeout);
      }
    }
    __syncwarp();
  } else {
    // =========================== epilogue (warps 2 .. 1 + kEpiWarps of both CTAs) ============
    const int q = warp & 3;                    // TMEM lane quarter this warp may read
    const int turn = (warp - 2) >> 2;          // takes the 32-column chunks turn, turn + groups, ...
    const int groups = kStore ? p.groups : kEpiWarps / 4;
    [[maybe_unused]] const uint32_t park = smem_base + kPairStages * kPairStageBytes + turn * kPairParkBytes;
    int acc = 0;
    uint32_t acc_phase = 0;
    int e_next = expert_of(cluster_id);
    for (int id = cluster_id; id < total; id += n_clusters) {
      int e, m0, n0, width, kblocks;
      decode(id, e_next, e, m0, n0, width, kblocks);
      e_next = expert_of(id + n_clusters);
      const int cta_m = m0 + (int)rank * 128;
      const int m = cta_m + q * 32 + lane;
      // M is a multiple of 32.  (Stored by TMA, the four warps of a group stay together and the copy clips.)
      const bool mine = kStore ? cta_m < p.M && turn < groups : m - lane < p.M;
      const int nchunks = (width + 31) >> 5;
      // 32 columns of the accumulator: as fp32 by M index, or (kStore) packed for stmatrix
      auto emit = [&](int c, const auto& v) {
        const int row = n0 + c * 32;
        if constexpr (kStore) {
          const bool issuer = q == 0 && lane == 0;
          if (issuer) tma_store_wait_read();
          group_sync(1 + turn);
          epi.park(v, q, lane, park);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the parked rows are read by the copy
          group_sync(1 + turn);
          if (issuer) {
            if (row < epi.H) {
              tma_store_3d(&tmOut, cta_m, row, e, park);
              if (cta_m + 64 < epi.ld) tma_store_3d(&tmOut, cta_m + 64, row, e, park + kPairParkBytes / 2);
            }
            tma_store_commit();
          }
          if (row <= epi.H && epi.H < row + 32)
            epi.bias_row(e, cta_m, epi.H - row, q, lane, smem_raw + (park - smem_u32(smem_raw)));
        } else {
          epi.apply(e, m, row, min(32, width - c * 32), lane, v);
        }
      };
      if (kblocks == 0) {                      // kWgrad of an expert without rows
        if constexpr (kStore) {
          const uint32_t z[16] = {};
          if (mine)
            for (int c = turn; c < nchunks; c += groups) emit(c, z);
        }
        continue;
      }
      if constexpr (epi_prefetches<Epi>::value) {
        if (mine)
          for (int c = turn; c < nchunks; c += groups) epi.prefetch(m, n0 + c * 32, min(32, width - c * 32), lane);
      }
      bool ok = mbar_wait_warp(smem_u32(&bar_tmem_full[acc]), acc_phase, &abort_flag);
      if constexpr (kStore) ok = group_all(1 + turn, ok);
      if (!ok) {
        abort_flag = 1;
        atomicMax(p.header + kHdrStatus, (int)kStatusEpilogueTimeout);
        break;
      }
      tc_fence_after();
      if (mine) {
        const uint32_t t_row = tmem_base + acc * kUmmaAccStride + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
        for (int c = turn; c < nchunks; c += groups) {
          uint32_t r[32];
          if constexpr (kStore) {
            tc_ld_16x256_issue(t_row + c * 32, r);
            tc_ld_wait(r);
            uint32_t v[16];
            epi.pack(r, v);
            emit(c, v);
          } else {
            tc_ld_32x32_issue(t_row + c * 32, r);
            tc_ld_wait(r);
            float v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
            emit(c, v);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&bar_tmem_empty[acc]), 0));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
    if constexpr (kStore) {
      if (q == 0 && lane == 0) tma_store_wait_all();
    }
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

// Number of CTA pairs of `kern` that run at the same time on the current device (asked once per kernel
// and device, with its shared memory set up).
template <typename... KArgs>
inline int resident_pairs(void (*kern)(KArgs...), int threads, int smem, PerDevice<int>& known) {
  const int dev = current_device_index();
  int n = known.get(dev);
  if (n > 0) return n;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(umma_sm_count() & ~1);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
    (void)cudaGetLastError();
    n = umma_sm_count() / 2;
  }
  known.set(dev, n);
  return n;
}

// Same operand description as launch_umma_gemm (GemmArgs), with the tile-pair tables and counts.
// H % 64 == 0 holds on every path here: all pitches and widths are multiples of 64.
// `row_round`: 16 where rows beyond an expert's own are never read again, 64 where a weight-gradient
// GEMM will reduce over them (its k-blocks).
template <int MODE, int kEpiWarps, class Epi>
inline int launch_umma_pair_warps(const GemmArgs& g, const Epi& epi, int64_t max_rows, int64_t max_tiles, int row_round,
                                  cudaStream_t stream) {
  if (!umma_available() || g.E > kUmmaMaxExperts) return YAMOE_ERR_UNSUPPORTED;
  CUtensorMap tmM, tmN, tmNs;
  bool ok = true;
  if (MODE == kWgrad) {
    const uint64_t dm[3] = {64, (uint64_t)max_rows, (uint64_t)g.ldb / 64}, sm[2] = {(uint64_t)g.ldb * 2, 128};
    const uint64_t dn[3] = {64, (uint64_t)max_rows, (uint64_t)g.lda / 64}, sn[2] = {(uint64_t)g.lda * 2, 128};
    const uint32_t b2[3] = {64, 64, 2}, b1[3] = {64, 64, 1};
    ok = make_map(&tmM, g.B, 3, dm, sm, b2) && make_map(&tmN, g.A, 3, dn, sn, b2) && make_map(&tmNs, g.A, 3, dn, sn, b1);
  } else {
    const uint64_t dn[2] = {(uint64_t)g.K, (uint64_t)max_rows}, sn[1] = {(uint64_t)g.lda * 2};
    const uint32_t b128[2] = {64, 128}, b32[2] = {64, 32};
    ok = make_map(&tmN, g.A, 2, dn, sn, b128) && make_map(&tmNs, g.A, 2, dn, sn, b32);
    if (MODE == kFwd) {
      const uint64_t dm[4] = {64, (uint64_t)g.K, (uint64_t)g.N / 64, (uint64_t)g.E};
      const uint64_t sm[3] = {(uint64_t)g.ldb * 2, 128, (uint64_t)g.b_expert_stride * 2};
      const uint32_t bm[4] = {64, 64, 2, 1};
      ok = ok && make_map(&tmM, g.B, 4, dm, sm, bm);
    } else {
      const uint64_t dm[3] = {(uint64_t)g.K, (uint64_t)g.N, (uint64_t)g.E};
      const uint64_t sm[2] = {(uint64_t)g.ldb * 2, (uint64_t)g.b_expert_stride * 2};
      const uint32_t bm[3] = {64, 128, 1};
      ok = ok && make_map(&tmM, g.B, 3, dm, sm, bm);
    }
  }
  constexpr bool kStore = epi_tma_store<Epi>::value;
  constexpr int kThreads = 32 * (3 + kEpiWarps);
  const int groups = !kStore || pair_smem(kEpiWarps / 4, g.E) <= kMaxDynamicSmem ? kEpiWarps / 4 : 2;
  const int smem = pair_smem(kStore ? groups : 0, g.E);
  CUtensorMap tmOut = tmM;               // not used
  if constexpr (kStore) {
    const uint64_t d[3] = {(uint64_t)epi.ld, (uint64_t)epi.H, (uint64_t)g.E};
    const uint64_t st[2] = {(uint64_t)epi.ld * 2, (uint64_t)epi.ld * epi.H * 2};
    const uint32_t b[3] = {64, 32, 1};
    ok = ok && make_map(&tmOut, epi.C, 3, d, st, b);
  }
  if (!ok) return YAMOE_ERR_CUDA;
  auto kern = umma_pair_kernel<MODE, Epi, kEpiWarps>;
  static PerDevice<int> resident;    // per template instantiation and device
  const int pairs = resident_pairs(kern, kThreads, kMaxDynamicSmem, resident);
  if (pairs <= 0) return YAMOE_ERR_CUDA;
  const PairParams p{g.N, g.M, g.K, g.E, row_round, g.pair_expert, g.pair_off, g.pad_off, g.counts,
                     const_cast<int32_t*>(g.header), groups};
  const int64_t MT = ceil_div(g.N, kPairM);
  // the tables bound the number of row tiles by max_tiles (128-row tiles)
  const int64_t total_max = MODE == kWgrad ? (int64_t)g.E * MT * ceil_div(g.M, kPairN) : max_tiles * MT;
  const int grid = (int)(2 * std::min<int64_t>(total_max, pairs));
  if (grid <= 0) return YAMOE_OK;
  if (launch_pdl_opt(true, kern, dim3(grid), dim3(kThreads), smem, stream, tmM, tmN, tmNs, tmOut, p, epi) != cudaSuccess)
    return YAMOE_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? YAMOE_OK : YAMOE_ERR_CUDA;
}

template <int MODE, class Epi>
inline int launch_umma_pair(const GemmArgs& g, const Epi& epi, int64_t max_rows, int64_t max_tiles, int row_round,
                            bool sixteen, cudaStream_t stream) {
  return sixteen ? launch_umma_pair_warps<MODE, 16>(g, epi, max_rows, max_tiles, row_round, stream)
                 : launch_umma_pair_warps<MODE, 8>(g, epi, max_rows, max_tiles, row_round, stream);
}

}  // namespace yb
