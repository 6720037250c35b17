// Routing: per-expert histogram, prefix sums and a stable counting sort of the S = T*K
// (token, slot) assignments, in two launches and without any device-wide spin wait.
//
// Replaces, bit for bit, what the reference computes with a CUB radix sort
// (csrc/sort.cu:17-59: ascending expert id, ties by ascending flat position) followed by
// bincount_cumsum (csrc/bincount_cumsum.cu:7-56: inclusive scan, slot E left at 0), the
// routing-weight gather (csrc/moe.cpp:199-203) and index_select (csrc/index_select.cu:7-16).
//
// Launch 1  route_count_kernel   one CTA per 2048 assignments: shared-memory histogram ->
//           block_counts[blk][e].  The CTA that takes the last ticket turns block_counts into
//           exclusive prefixes over blocks and derives counts, bins, the padded row offsets
//           and the tile -> expert table.
// Launch 2  route_place_kernel   same partition; every warp ranks its 256 assignments with
//           __match_any_sync ballots (stable within the warp), warps are chained through a
//           shared-memory prefix, blocks through block_counts; each assignment is written to
//           its sorted slot and to its row of the padded, expert-sorted layout.
#pragma once
#include "common.cuh"

namespace yb {

constexpr int kRouteThreads = 256;
constexpr int kRouteWarps = kRouteThreads / 32;
constexpr int kRouteRounds = 8;                                   // assignments per lane
constexpr int kRouteItems = kRouteThreads * kRouteRounds;         // assignments per CTA

__global__ void __launch_bounds__(kRouteThreads)
route_count_kernel(const int64_t* __restrict__ router_indices, int S, int E, int64_t capacity,
                   RouteTables rt, int nblk) {
  extern __shared__ int32_t smem_i[];
  int32_t* hist = smem_i;            // [E]
  int32_t* poff = smem_i + E;        // [E+1]
  int32_t* qoff = smem_i + 2 * E + 1;  // [E+1]
  __shared__ int is_last;
  const int tid = threadIdx.x;
  for (int e = tid; e < E; e += kRouteThreads) hist[e] = 0;
  __syncthreads();
  const int base = blockIdx.x * kRouteItems;
#pragma unroll
  for (int i = 0; i < kRouteRounds; ++i) {
    int j = base + i * kRouteThreads + tid;
    if (j < S) {
      int64_t e = router_indices[j];
      if (e >= 0 && e < E) atomicAdd(&hist[(int)e], 1);
    }
  }
  __syncthreads();
  for (int e = tid; e < E; e += kRouteThreads) rt.block_counts[(size_t)blockIdx.x * E + e] = hist[e];
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    int t = atomicAdd(&rt.header[kHdrTicket], 1);
    is_last = (t == nblk - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  for (int e = tid; e < E; e += kRouteThreads) {
    int run = 0;
    for (int b = 0; b < nblk; ++b) {
      volatile int32_t* p = rt.block_counts + (size_t)b * E + e;
      int c = *p;
      *p = run;
      run += c;
    }
    rt.counts[e] = run;
    hist[e] = run;
  }
  __syncthreads();
  if (tid == 0) {
    int cum = 0, rows = 0, dropped = 0, pairs = 0;
    for (int e = 0; e < E; ++e) {
      int c = hist[e];
      cum += c;
      rt.bins[e] = cum;
      int kept = (int64_t)c < capacity ? c : (int)capacity;
      dropped += c - kept;
      poff[e] = rows;
      rt.pad_off[e] = rows;
      qoff[e] = pairs;
      if (rt.pair_off != nullptr) rt.pair_off[e] = pairs;
      const int tiles = (kept + kTileM - 1) / kTileM;
      rows += tiles * kTileM;
      pairs += (tiles + 1) / 2;
    }
    poff[E] = rows;
    qoff[E] = pairs;
    if (rt.pair_off != nullptr) rt.pair_off[E] = pairs;
    rt.header[kHdrPairs] = pairs;
    rt.bins[E] = 0;
    rt.pad_off[E] = rows;
    rt.header[kHdrRowTiles] = rows / kTileM;
    rt.header[kHdrRowsUsed] = rows;
    rt.header[kHdrDropped] = dropped;
    rt.header[kHdrTicket] = 0;
  }
  __syncthreads();
  if (rt.tile_expert != nullptr) {
    for (int e = tid; e < E; e += kRouteThreads)
      for (int t = poff[e] / kTileM; t < poff[e + 1] / kTileM; ++t) rt.tile_expert[t] = e;
  }
  if (rt.pair_expert != nullptr) {
    for (int e = tid; e < E; e += kRouteThreads)
      for (int t = qoff[e]; t < qoff[e + 1]; ++t) rt.pair_expert[t] = e;
  }
}

template <typename T>
__global__ void __launch_bounds__(kRouteThreads)
route_place_kernel(const int64_t* __restrict__ router_indices, const T* __restrict__ routing_weights,
                   int routing_cols, int S, int E, int K, int64_t capacity, RouteTables rt) {
  extern __shared__ int32_t smem_i[];
  int32_t* wcnt = smem_i;  // [kRouteWarps][E]
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int i = tid; i < kRouteWarps * E; i += kRouteThreads) wcnt[i] = 0;
  __syncthreads();
  const int base = blockIdx.x * kRouteItems + w * (32 * kRouteRounds);
  int ex[kRouteRounds];
#pragma unroll
  for (int i = 0; i < kRouteRounds; ++i) {
    int j = base + i * 32 + lane;
    int e = -1 - lane;  // unique negative key: never matches another lane
    if (j < S) {
      int64_t v = router_indices[j];
      if (v >= 0 && v < E) e = (int)v;
    }
    ex[i] = e;
  }
  int32_t* mine = wcnt + w * E;
#pragma unroll
  for (int i = 0; i < kRouteRounds; ++i) {
    unsigned mask = __match_any_sync(0xffffffffu, ex[i]);
    if (ex[i] >= 0 && (__ffs(mask) - 1) == lane) mine[ex[i]] += __popc(mask);
    __syncwarp();
  }
  __syncthreads();
  for (int e = tid; e < E; e += kRouteThreads) {
    int run = rt.block_counts[(size_t)blockIdx.x * E + e];
    for (int ww = 0; ww < kRouteWarps; ++ww) {
      int c = wcnt[ww * E + e];
      wcnt[ww * E + e] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kRouteRounds; ++i) {
    const int e = ex[i];
    unsigned mask = __match_any_sync(0xffffffffu, e);
    int pos = 0;
    if (e >= 0) pos = mine[e] + __popc(mask & ((1u << lane) - 1u));
    __syncwarp();
    if (e >= 0 && (__ffs(mask) - 1) == lane) mine[e] += __popc(mask);
    __syncwarp();
    if (e >= 0) {
      const int p = base + i * 32 + lane;
      const int start = e ? rt.bins[e - 1] : 0;
      rt.sorted_values[start + pos] = e;
      rt.sorted_indices[start + pos] = p;
      if (rt.flat_pos != nullptr) rt.flat_pos[p] = start + pos;
      if (rt.row_token != nullptr && (int64_t)pos < capacity) {
        const int r = rt.pad_off[e] + pos;
        const int t = p / K;
        rt.row_token[r] = t;
        rt.row_flat[r] = p;
        rt.flat_row[p] = r;
        const int col = (routing_cols == E) ? e : (p - t * K);
        rt.row_weight[r] = DT<T>::ld(routing_weights + (size_t)t * routing_cols + col);
      }
    }
  }
}

// Host-side launcher.  `rt` must point into zero-initialised header memory for the ticket
// (the caller memsets the header) and, when row tables are requested, row_token / row_flat
// must have been filled with -1.
template <typename T>
inline int launch_route(const int64_t* router_indices, const T* routing_weights, int routing_cols,
                        int64_t T_tokens, int E, int K, int64_t capacity, const RouteTables& rt,
                        cudaStream_t stream) {
  const int S = (int)(T_tokens * K);
  const int nblk = (int)ceil_div(S, kRouteItems);
  size_t smem1 = (size_t)(3 * E + 2) * sizeof(int32_t);
  size_t smem2 = (size_t)kRouteWarps * E * sizeof(int32_t);
  route_count_kernel<<<nblk, kRouteThreads, smem1, stream>>>(router_indices, S, E, capacity, rt, nblk);
  route_place_kernel<T><<<nblk, kRouteThreads, smem2, stream>>>(router_indices, routing_weights,
                                                               routing_cols, S, E, K, capacity, rt);
  return cudaGetLastError() == cudaSuccess ? YAMOE_OK : YAMOE_ERR_CUDA;
}

// ---- one launch for everything ------------------------------------------------------------------
// Up to kRouteClusterMaxS assignments: a cluster of eight CTAs counts, exchanges its histograms
// through distributed shared memory, scans and places, and also writes what the two-launch form has
// the caller fill beforehand (the header, -1 for padding rows and dropped assignments).  What bounds
// this step is latency: four launches (two memsets, count, place) and the round trips between them took
// some 28 us at S = 65536 and little less below; one takes 6.5 us up to S = 4096, 12 us at 16384.  It does not write sorted_values / sorted_indices, which the expert pass never reads.
// The limit: above it eight SMs place more slowly (about five scattered accesses per assignment) than
// the two-launch form, which spreads over S / 2048 CTAs.
constexpr int kRouteCluster = 8;
constexpr int kRouteClusterThreads = 1024;
constexpr int kRouteClusterWarps = kRouteClusterThreads / 32;
constexpr int kRouteClusterMaxRounds = 4;
constexpr int kRouteClusterMaxS = kRouteCluster * kRouteClusterThreads * kRouteClusterMaxRounds;

inline size_t route_cluster_smem(int E) {
  return (size_t)E * 3 * sizeof(int32_t) + (size_t)kRouteClusterWarps * E * sizeof(uint16_t);
}

template <typename T>
__global__ void __cluster_dims__(kRouteCluster, 1, 1) __launch_bounds__(kRouteClusterThreads, 1)
route_cluster_kernel(const int64_t* __restrict__ router_indices, const T* __restrict__ routing_weights,
                     int routing_cols, int S, int E, int K, int rounds, int64_t capacity, RouteTables rt) {
  extern __shared__ int32_t smem_i[];
  int32_t* hist = smem_i;                  // [E] this CTA's counts, read by the others
  int32_t* first = smem_i + E;             // [E] first padded row of the expert
  int32_t* before = smem_i + 2 * E;        // [E] assignments of the expert in lower CTAs
  uint16_t* wcnt = reinterpret_cast<uint16_t*>(smem_i + 3 * E);   // [warps][E] counts, then prefixes over warps
  __shared__ int s_warp[3][kRouteClusterWarps];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  pdl_trigger();                           // the next kernel may set up (it waits for this one's end)
  const int rank = (int)cluster_ctarank();
  const int base = (rank * kRouteClusterWarps + w) * 32 * rounds;
  int ex[kRouteClusterMaxRounds];
#pragma unroll
  for (int i = 0; i < kRouteClusterMaxRounds; ++i) {
    const int j = base + i * 32 + lane;
    int e = -1 - lane;                     // unique negative key: never matches another lane
    if (i < rounds && j < S) {
      const int64_t v = router_indices[j];
      if (v >= 0 && v < E) e = (int)v;
    }
    ex[i] = e;
  }
  for (int i = tid; i < kRouteClusterWarps * E / 2; i += kRouteClusterThreads) reinterpret_cast<uint32_t*>(wcnt)[i] = 0;
  __syncthreads();
  uint16_t* mine = wcnt + w * E;
#pragma unroll
  for (int i = 0; i < kRouteClusterMaxRounds; ++i)
    if (i < rounds) {
      const unsigned mask = __match_any_sync(0xffffffffu, ex[i]);
      if (ex[i] >= 0 && (__ffs(mask) - 1) == lane) mine[ex[i]] += (uint16_t)__popc(mask);
      __syncwarp();
    }
  __syncthreads();
  const int e = tid;                       // E <= 1024 = threads of the CTA
  if (e < E) {
    int run = 0;
#pragma unroll 8
    for (int ww = 0; ww < kRouteClusterWarps; ++ww) {
      const int c = wcnt[ww * E + e];
      wcnt[ww * E + e] = (uint16_t)run;
      run += c;
    }
    hist[e] = run;
  }
  cluster_sync_all();
  int total = 0, lower = 0;
  if (e < E) {
    const uint32_t addr = smem_addr_u32(hist + e);
#pragma unroll
    for (int c = 0; c < kRouteCluster; ++c) {
      const int v = __float_as_int(ld_shared_cluster_f32(mapa_u32(addr, (uint32_t)c)));
      total += v;
      if (c < rank) lower += v;
    }
  }
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");   // done with the others' shared memory (wait: at the end)
  // inclusive scans over the experts: assignments, 128-row tiles, pairs of tiles
  const int kept = (int64_t)total < capacity ? total : (int)capacity;
  const int tiles = (kept + kTileM - 1) / kTileM, pairs = (tiles + 1) / 2;
  int inc[3] = {total, tiles, pairs};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc[q], o);
      if (lane >= o) inc[q] += v;
    }
    if (lane == 31) s_warp[q][w] = inc[q];
  }
  __syncthreads();
  if (w < 3) {
    int v = s_warp[w][lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    s_warp[w][lane] = v;
  }
  __syncthreads();
  if (w > 0) {
#pragma unroll
    for (int q = 0; q < 3; ++q) inc[q] += s_warp[q][w - 1];
  }
  const int tile0 = inc[1] - tiles, pair0 = inc[2] - pairs;
  if (e < E) {
    first[e] = tile0 * kTileM;
    before[e] = lower;
  }
  __syncthreads();
  if (rank == 0) {
    if (e < E) {
      rt.counts[e] = total;
      rt.bins[e] = inc[0];
      rt.pad_off[e] = tile0 * kTileM;
      rt.pair_off[e] = pair0;
      for (int t = 0; t < tiles; ++t) rt.tile_expert[tile0 + t] = e;
      for (int t = 0; t < pairs; ++t) rt.pair_expert[pair0 + t] = e;
    }
    const int dropped = __reduce_add_sync(0xffffffffu, total - kept);
    if (lane == 0) s_warp[0][w] = dropped;
    __syncthreads();
    if (tid == kRouteClusterThreads - 1) {         // its inclusive sums are the totals
      int d = 0;
      for (int i = 0; i < kRouteClusterWarps; ++i) d += s_warp[0][i];
      for (int i = 0; i < 16; ++i) rt.header[i] = 0;
      rt.header[kHdrRowTiles] = inc[1];
      rt.header[kHdrRowsUsed] = inc[1] * kTileM;
      rt.header[kHdrDropped] = d;
      rt.header[kHdrPairs] = inc[2];
      rt.bins[E] = 0;
      rt.pad_off[E] = inc[1] * kTileM;
      rt.pair_off[E] = inc[2];
    }
  } else if (e < E && e % (kRouteCluster - 1) == rank - 1) {
    // padding rows of the experts, shared out among the CTAs that do not write the tables
    for (int r = kept; r < tiles * kTileM; ++r) rt.row_token[tile0 * kTileM + r] = -1;
  }
#pragma unroll
  for (int i = 0; i < kRouteClusterMaxRounds; ++i)
    if (i < rounds) {
      const int x = ex[i];
      const unsigned mask = __match_any_sync(0xffffffffu, x);
      int pos = 0;
      if (x >= 0) pos = before[x] + mine[x] + __popc(mask & ((1u << lane) - 1u));
      __syncwarp();
      if (x >= 0 && (__ffs(mask) - 1) == lane) mine[x] += (uint16_t)__popc(mask);
      __syncwarp();
      const int p = base + i * 32 + lane;
      if (p < S) {
        int r = -1;
        if (x >= 0 && (int64_t)pos < capacity) {
          r = first[x] + pos;
          const int t = p / K;
          rt.row_token[r] = t;
          rt.row_flat[r] = p;
          const int col = (routing_cols == E) ? x : (p - t * K);
          rt.row_weight[r] = DT<T>::ld(routing_weights + (size_t)t * routing_cols + col);
        }
        rt.flat_row[p] = r;
      }
    }
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

// Routing of the expert pass: all tables, row tables included, from uninitialised memory.
template <typename T>
inline int launch_route_rows(const int64_t* router_indices, const T* routing_weights, int routing_cols,
                             int64_t T_tokens, int E, int K, int64_t capacity, const RouteTables& rt,
                             size_t row_tables_bytes, cudaStream_t stream) {
  const int64_t S = T_tokens * K;
  if (S <= kRouteClusterMaxS) {
    auto kern = route_cluster_kernel<T>;
    const size_t smem = route_cluster_smem(E);
    static PerDevice<size_t> configured;   // per template instantiation and device
    const int dev = current_device_index();
    if (smem > configured.get(dev)) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return YAMOE_ERR_CUDA;
      configured.set(dev, smem);
    }
    const int rounds = (int)ceil_div(S, kRouteCluster * kRouteClusterThreads);
    kern<<<kRouteCluster, kRouteClusterThreads, smem, stream>>>(router_indices, routing_weights, routing_cols, (int)S, E,
                                                                K, rounds, capacity, rt);
    return cudaGetLastError() == cudaSuccess ? YAMOE_OK : YAMOE_ERR_CUDA;
  }
  YB_CUDA_OK(cudaMemsetAsync(rt.header, 0, 16 * sizeof(int32_t), stream));
  YB_CUDA_OK(cudaMemsetAsync(rt.row_token, 0xFF, row_tables_bytes, stream));
  return launch_route<T>(router_indices, routing_weights, routing_cols, T_tokens, E, K, capacity, rt, stream);
}

inline int route_blocks(int64_t S) { return (int)ceil_div(S, kRouteItems); }

}  // namespace yb
