// MoE routing and token permutation kernels.
//
//   router_topk        : softmax over E experts, top-k (k <= 8), optional renormalisation; with a replay
//                        table the expert choice comes from the rollout engine (rollout routing replay)
//                        and only the gate weights are recomputed from the current logits.
//   build_permutation  : deterministic counting sort of (token, slot) pairs by expert; each expert's rows
//                        are padded to a multiple of `align` (64 for training so that the weight-gradient
//                        contraction blocks stay inside one expert, 1 for inference) and cut into GEMM row
//                        tiles of at most 128 rows that never straddle experts.
//   permute / combine  : gather rows into expert order / weighted gather-sum back to token order, with
//                        their backward passes. All gathers are index-driven (no atomics), so results are
//                        bitwise reproducible.
//
// Reference counterparts: Megatron TopKRouter + token dispatcher (scripts/models/qwen3-30B-A3B.py:29-41),
// the replay hook in miles/utils/replay_base.py:14-237 and the Triton fused-MoE align/sort stage in
// miles/backends/fsdp_utils/kernels/fused_experts.py:15-379.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "launchers.h"
#include "pdl.cuh"

namespace mb {
namespace {

using bf16 = __nv_bfloat16;
constexpr int kMaxK = 16;

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One warp per token, E <= 256 (8 values per lane).
__global__ void router_topk_kernel(const float* __restrict__ logits, const int* __restrict__ replay_ids,
                                   int* __restrict__ topk_ids, float* __restrict__ topk_w,
                                   float* __restrict__ probs_out, int T, int E, int K, int renorm) {
  pdl_enter();
  const int wpb = blockDim.x >> 5;
  const int t = blockIdx.x * wpb + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  float p[8];
  float mx = -FLT_MAX;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int e = lane + 32 * i;
    p[i] = e < E ? logits[static_cast<long long>(t) * E + e] : -FLT_MAX;
    mx = fmaxf(mx, p[i]);
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int e = lane + 32 * i;
    p[i] = e < E ? __expf(p[i] - mx) : 0.f;
    sum += p[i];
  }
  sum = warp_sum(sum);
  const float inv = 1.f / sum;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    p[i] *= inv;
    const int e = lane + 32 * i;
    if (probs_out && e < E) probs_out[static_cast<long long>(t) * E + e] = p[i];
  }
  int ids[kMaxK];
  float ws[kMaxK];
  if (replay_ids) {
    for (int k = 0; k < K; ++k) {
      int e = replay_ids[static_cast<long long>(t) * K + k];
      e = (e < 0 || e >= E) ? 0 : e;
      // fetch p[e] from the owning lane
      const int owner = e & 31, slot = e >> 5;
      float v = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (slot == i) v = p[i];
      ids[k] = e;
      ws[k] = __shfl_sync(0xffffffffu, v, owner);
    }
  } else {
    float q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = (lane + 32 * i) < E ? p[i] : -1.f;
    for (int k = 0; k < K; ++k) {
      float best = -1.f;
      int best_e = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int e = lane + 32 * i;
        if (q[i] > best || (q[i] == best && e < best_e)) {
          best = q[i];
          best_e = e;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oe = __shfl_xor_sync(0xffffffffu, best_e, o);
        if (ob > best || (ob == best && oe < best_e)) {
          best = ob;
          best_e = oe;
        }
      }
      ids[k] = best_e;
      ws[k] = best;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (lane + 32 * i == best_e) q[i] = -2.f;
    }
  }
  if (renorm) {
    float s = 0.f;
    for (int k = 0; k < K; ++k) s += ws[k];
    const float r = 1.f / fmaxf(s, 1e-20f);
    for (int k = 0; k < K; ++k) ws[k] *= r;
  }
  if (lane == 0) {
    for (int k = 0; k < K; ++k) {
      topk_ids[static_cast<long long>(t) * K + k] = ids[k];
      topk_w[static_cast<long long>(t) * K + k] = ws[k];
    }
  }
}

// dlogits for: p = softmax(logits); w_k = p[id_k] (/ sum_j p[id_j] when renorm).
__global__ void router_bwd_kernel(const float* __restrict__ probs, const int* __restrict__ topk_ids,
                                  const float* __restrict__ topk_w, const float* __restrict__ dtopk_w,
                                  float* __restrict__ dlogits, int T, int E, int K, int renorm) {
  const int wpb = blockDim.x >> 5;
  const int t = blockIdx.x * wpb + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  // dL/dp[e] for the selected experts
  float dp[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  float s_sel = 1.f, dot = 0.f;
  if (renorm) {
    s_sel = 0.f;
    for (int k = 0; k < K; ++k) {
      const int e = topk_ids[static_cast<long long>(t) * K + k];
      s_sel += probs[static_cast<long long>(t) * E + e];
      dot += dtopk_w[static_cast<long long>(t) * K + k] * topk_w[static_cast<long long>(t) * K + k];
    }
    s_sel = fmaxf(s_sel, 1e-20f);
  }
  for (int k = 0; k < K; ++k) {
    const int e = topk_ids[static_cast<long long>(t) * K + k];
    const float g = dtopk_w[static_cast<long long>(t) * K + k];
    const float v = renorm ? (g - dot) / s_sel : g;  // d w_k / d p_j = (delta_kj - w_k) / s
    if ((e & 31) == lane) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if ((e >> 5) == i) dp[i] += v;
    }
  }
  // softmax backward: dlogit = p * (dp - sum_j p_j dp_j)
  float pv[8];
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int e = lane + 32 * i;
    pv[i] = e < E ? probs[static_cast<long long>(t) * E + e] : 0.f;
    acc += pv[i] * dp[i];
  }
  acc = warp_sum(acc);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int e = lane + 32 * i;
    if (e < E) dlogits[static_cast<long long>(t) * E + e] = pv[i] * (dp[i] - acc);
  }
}

// ---------------------------------------------------------------- permutation
// A stable counting sort of the n = T * K entries by expert. The entries are dealt to warps in contiguous runs; a warp
// walks over its run 32 entries at a time, and the lanes that hold the same expert find one another with a match
// instruction, so an entry's rank among the warp's earlier entries of its expert costs one shared-memory read. The
// ranks become rows once every warp's counts are summed over the warps (and blocks) before it. What bounds it is latency:
// 131072 ids are half a megabyte. (One block per expert that reads every id, which this replaced, read them 2 E times:
// 131072 entries over 128 experts took 282 us in three kernels, these take 20 us; 128 entries 10.7 us, now 3.2 us.)
constexpr int SORT_ROUNDS = 16;  // entries per lane and warp at most
constexpr int SORT_WARPS = 4;    // warps per block of the many-block variant: counts and scans fit shared memory up to 14500 experts

// One warp: `rank[r]` of entry first + 32 r + lane among the warp's entries of the same expert, the warp's counts in
// `hist` (shared memory, zeroed by the caller). Ids outside [0, E) get no rank. The last entry is `last` - 1.
template <int ROUNDS>
__device__ __forceinline__ void warp_ranks(const int* __restrict__ ids, int first, int last, int E, int* hist, int (&id)[ROUNDS],
                                           int (&rank)[ROUNDS]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const int i = first + 32 * r + lane;
    const int e = i < last ? ids[i] : -1;
    id[r] = (e >= 0 && e < E) ? e : -1;
  }
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    rank[r] = 0;
    if (first + 32 * r >= last) continue;  // warp-uniform
    const unsigned same = __match_any_sync(0xffffffffu, id[r]);
    const unsigned below = same & ((1u << lane) - 1u);
    const int before = id[r] >= 0 ? hist[id[r]] : 0;
    rank[r] = before + __popc(below);
    __syncwarp();
    if (id[r] >= 0 && below == 0) hist[id[r]] = before + __popc(same);
    __syncwarp();
  }
}

// One warp: exclusive scans over the experts. First the row offsets, every expert's rows padded to `align` and clamped to
// the capacity (offsets are multiples of `align`, so clamping both ends of an expert's range equals shrinking the expert
// that overflows and giving the later ones nothing), then the starts of the 128-row tiles of the clamped ranges; lane l
// owns experts [l*per, (l+1)*per). off[0..E], tstart[0..E]; totals = {number of tiles, live rows}.
__device__ __forceinline__ void scan_experts(const int* cnt, int E, int max_rows, int max_tiles, int align, int* off, int* tstart,
                                             int* __restrict__ totals) {
  const int lane = threadIdx.x & 31;
  const int per = (E + 31) / 32;
  const int e0 = min(E, lane * per), e1 = min(E, e0 + per);
  const int cap = (max_rows / align) * align;
  int local = 0;
  for (int e = e0; e < e1; ++e) local += ((cnt[e] + align - 1) / align) * align;
  int incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  int run = incl - local;
  int tl = 0;
  for (int e = e0; e < e1; ++e) {
    const int s0 = min(run, cap);
    run += ((cnt[e] + align - 1) / align) * align;
    const int s1 = min(run, cap);
    off[e] = s0;
    tl += (s1 - s0 + 127) / 128;
    tstart[e] = s1 - s0;  // rows of the expert for now; turned into a tile start below
  }
  const int total_rows = min(__shfl_sync(0xffffffffu, incl, 31), cap);
  int tincl = tl;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, tincl, o);
    if (lane >= o) tincl += v;
  }
  int trun = tincl - tl;
  for (int e = e0; e < e1; ++e) {
    const int rows = tstart[e];
    tstart[e] = trun;
    trun += (rows + 127) / 128;
  }
  const int total_tiles = __shfl_sync(0xffffffffu, tincl, 31);
  if (lane == 0) {
    off[E] = total_rows;
    tstart[E] = total_tiles < max_tiles ? total_tiles : max_tiles;
    totals[0] = tstart[E];
    totals[1] = total_rows;
  }
}

// The tile list: tile t of an expert covers its rows 128 j .. 128 j + 127; tiles[t] = {expert, first row, rows, 0}.
__device__ __forceinline__ void write_tiles(const int* off, const int* tstart, int E, int max_tiles, int* __restrict__ tiles) {
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const int rows_e = off[e + 1] - off[e];
    for (int j = 0; tstart[e] + j < tstart[e + 1] && tstart[e] + j < max_tiles; ++j)
      reinterpret_cast<int4*>(tiles)[tstart[e] + j] = make_int4(e, off[e] + 128 * j, min(128, rows_e - 128 * j), 0);
  }
}

// Small problems (decode steps) in one block: ranks, scans, tile list and rows, with nothing to initialise beforehand.
template <int ROUNDS>
__global__ void __launch_bounds__(512)
build_small_kernel(const int* __restrict__ ids, int n, int E, int max_rows, int max_tiles, int align,
                   int* __restrict__ counts_out, int* __restrict__ offsets, int* __restrict__ dest_row,
                   int* __restrict__ row_src, int* __restrict__ tiles, int* __restrict__ totals) {
  pdl_enter();
  extern __shared__ int sm[];  // cnt[E], off[E+1], tstart[E+1], hist[warps][E]
  int* cnt = sm;
  int* off = cnt + E;
  int* tstart = off + E + 1;
  int* hist = tstart + E + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int i = threadIdx.x; i < nwarps * E; i += blockDim.x) hist[i] = 0;
  for (int i = threadIdx.x; i < max_rows; i += blockDim.x) row_src[i] = -1;
  __syncthreads();
  const int first = warp * ROUNDS * 32;
  int id[ROUNDS], rank[ROUNDS];
  warp_ranks<ROUNDS>(ids, first, min(n, first + ROUNDS * 32), E, hist + warp * E, id, rank);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int run = 0;
    for (int w = 0; w < nwarps; ++w) {
      const int v = hist[w * E + e];
      hist[w * E + e] = run;
      run += v;
    }
    cnt[e] = run;
    counts_out[e] = run;
  }
  __syncthreads();
  if (warp == 0) scan_experts(cnt, E, max_rows, max_tiles, align, off, tstart, totals);
  __syncthreads();
  for (int e = threadIdx.x; e <= E; e += blockDim.x) offsets[e] = off[e];
  write_tiles(off, tstart, E, max_tiles, tiles);
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const int i = first + 32 * r + lane;
    if (i >= n) continue;
    const int e = id[r];
    int row = -1;  // an id outside the experts, or no room for it
    if (e >= 0) {
      const int k = hist[warp * E + e] + rank[r];
      if (k < off[e + 1] - off[e]) {
        row = off[e] + k;
        row_src[row] = i;
      }
    }
    dest_row[i] = row;
  }
}

// Larger problems, pass 1: every block counts its SORT_WARPS * SORT_ROUNDS * 32 entries by expert.
__global__ void __launch_bounds__(SORT_WARPS * 32)
count_kernel(const int* __restrict__ ids, int n, int E, int* __restrict__ block_hist) {
  extern __shared__ int hist[];  // [E]
  for (int e = threadIdx.x; e < E; e += blockDim.x) hist[e] = 0;
  __syncthreads();
  const int first = blockIdx.x * SORT_WARPS * SORT_ROUNDS * 32;
  const int last = min(n, first + SORT_WARPS * SORT_ROUNDS * 32);
#pragma unroll 4
  for (int i = first + threadIdx.x; i < last; i += SORT_WARPS * 32) {
    const int e = ids[i];
    if (e >= 0 && e < E) atomicAdd(&hist[e], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) block_hist[static_cast<long long>(blockIdx.x) * E + e] = hist[e];
}

// Pass 2, one block: block_hist becomes the number of an expert's entries in the blocks before each; scans and tile list.
__global__ void __launch_bounds__(1024)
scan_kernel(int* __restrict__ block_hist, int blocks, int parts, int E, int max_rows, int max_tiles, int align, int* __restrict__ counts,
            int* __restrict__ offsets, int* __restrict__ tiles, int* __restrict__ totals) {
  extern __shared__ int sm[];  // cnt[E], off[E+1], tstart[E+1], part[parts][E]
  int* cnt = sm;
  int* off = cnt + E;
  int* tstart = off + E + 1;
  int* part = tstart + E + 1;
  const int run_len = (blocks + parts - 1) / parts;  // the blocks in several runs: as many chains of loads per expert are in flight
  for (int i = threadIdx.x; i < parts * E; i += blockDim.x) {
    const int p = i / E, e = i - p * E;
    const int b1 = min(blocks, (p + 1) * run_len);
    int sum = 0;
#pragma unroll 8
    for (int b = p * run_len; b < b1; ++b) sum += block_hist[static_cast<long long>(b) * E + e];
    part[i] = sum;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int run = 0;
    for (int p = 0; p < parts; ++p) {
      const int v = part[p * E + e];
      part[p * E + e] = run;
      run += v;
    }
    cnt[e] = run;
    counts[e] = run;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < parts * E; i += blockDim.x) {
    const int p = i / E, e = i - p * E;
    const int b1 = min(blocks, (p + 1) * run_len);
    int run = part[i];
#pragma unroll 8
    for (int b = p * run_len; b < b1; ++b) {
      int* h = block_hist + static_cast<long long>(b) * E + e;
      const int v = *h;
      *h = run;
      run += v;
    }
  }
  if (threadIdx.x < 32) scan_experts(cnt, E, max_rows, max_tiles, align, off, tstart, totals);
  __syncthreads();
  for (int e = threadIdx.x; e <= E; e += blockDim.x) offsets[e] = off[e];
  write_tiles(off, tstart, E, max_tiles, tiles);
}

// Pass 3: the rows of a block's entries.
__global__ void __launch_bounds__(SORT_WARPS * 32)
assign_kernel(const int* __restrict__ ids, int n, int E, const int* __restrict__ block_hist, const int* __restrict__ offsets,
              int* __restrict__ dest_row, int* __restrict__ row_src) {
  extern __shared__ int hist[];  // [SORT_WARPS][E]
  for (int i = threadIdx.x; i < SORT_WARPS * E; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int first = (blockIdx.x * SORT_WARPS + warp) * SORT_ROUNDS * 32;
  int id[SORT_ROUNDS], rank[SORT_ROUNDS];
  warp_ranks<SORT_ROUNDS>(ids, first, min(n, first + SORT_ROUNDS * 32), E, hist + warp * E, id, rank);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int run = block_hist[static_cast<long long>(blockIdx.x) * E + e];
#pragma unroll
    for (int w = 0; w < SORT_WARPS; ++w) {
      const int v = hist[w * E + e];
      hist[w * E + e] = run;
      run += v;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < SORT_ROUNDS; ++r) {
    const int i = first + 32 * r + lane;
    if (i >= n) continue;
    const int e = id[r];
    int row = -1;  // an id outside the experts, or no room for it (only if max_rows was under-provisioned)
    if (e >= 0) {
      const int k = hist[warp * E + e] + rank[r];
      const int o = offsets[e];
      if (k < offsets[e + 1] - o) {
        row = o + k;
        row_src[row] = i;
      }
    }
    dest_row[i] = row;
  }
}

// Permuted rows are written by one kernel and read by the next. Up to half of L2 (126 MB) they are still there when they are read; beyond
// that they only push out what is (weights, the rows of the tokens), and go first (PASSING). us with / without, 8 choices of 128 experts,
// 2048 columns: 16384 tokens (537 MB) permute 164 / 169, combine 135 / 148; 8192 tokens (268 MB) 67 / 73 and 66 / 75; at 2048 and 777 tokens
// (67 and 58 MB), alone or with the products behind, the two differ by less than their runs do. 24 decode steps of 16 rows (0.5 MB)
// 85.2 / 84.1 ms, in another run 86.4 / 86.1.
constexpr long long PASSING_BYTES = 64ll << 20;
template <bool PASSING>
__device__ __forceinline__ void put_row(uint4* p, const uint4& v) {
  if constexpr (PASSING) __stcs(p, v);
  else *p = v;
}
template <bool PASSING>
__device__ __forceinline__ uint4 take_row(const uint4* p) {
  if constexpr (PASSING) return __ldcs(p);
  else return *p;
}

// x_perm[row] = x[row_src[row] / K] or zeros for padding rows. One warp per row, four 16-byte loads of it in flight per lane
// (131072 rows of 2048: 158 us when every thread placed its own 16 bytes after a 64-bit division, 148 us now; the copy alone
// is 604 MB).
template <bool PASSING>
__global__ void permute_kernel(const bf16* __restrict__ x, const int* __restrict__ row_src,
                               const int* __restrict__ num_m_tiles, bf16* __restrict__ x_perm, int max_rows, int H,
                               int K) {
  pdl_enter();
  const int live_rows = min(num_m_tiles[1], max_rows);
  const int vec_per_row = H / 8;
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < live_rows; row += gridDim.x * wpb) {
    const int src = row_src[row];
    const uint4* from = reinterpret_cast<const uint4*>(x + static_cast<long long>(src < 0 ? 0 : src / K) * H);
    uint4* to = reinterpret_cast<uint4*>(x_perm + static_cast<long long>(row) * H);
    for (int c0 = lane; c0 < vec_per_row; c0 += 128) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = (src >= 0 && c0 + 32 * u < vec_per_row) ? from[c0 + 32 * u] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c0 + 32 * u < vec_per_row) put_row<PASSING>(to + c0 + 32 * u, v[u]);
    }
  }
}

__device__ __forceinline__ void acc8(const uint4& raw, float w, float (&a)[8]) {
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(b[i]);
    a[2 * i] += w * f.x;
    a[2 * i + 1] += w * f.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&a)[8]) {
  uint4 r;
  __nv_bfloat162 t;
  t = __floats2bfloat162_rn(a[0], a[1]); r.x = *reinterpret_cast<uint32_t*>(&t);
  t = __floats2bfloat162_rn(a[2], a[3]); r.y = *reinterpret_cast<uint32_t*>(&t);
  t = __floats2bfloat162_rn(a[4], a[5]); r.z = *reinterpret_cast<uint32_t*>(&t);
  t = __floats2bfloat162_rn(a[6], a[7]); r.w = *reinterpret_cast<uint32_t*>(&t);
  return r;
}

// out[t] = sum_k w[t,k] * y_perm[dest_row[t,k]]; with w == nullptr the weights are 1 (permute backward). A block takes 128
// 16-byte columns of one token after another; the rows of up to eight choices are asked for together and added in order
// (16384 tokens, 8 choices, 2048 columns: 185 us with one load in flight per thread, 128 us with eight; 671 MB move).
constexpr int COMBINE_THREADS = 128;
template <bool PASSING>
__global__ void __launch_bounds__(COMBINE_THREADS)
combine_kernel(const bf16* __restrict__ y_perm, const int* __restrict__ dest_row, const float* __restrict__ topk_w,
               const bf16* __restrict__ residual, bf16* __restrict__ out, int T, int K, int H) {
  pdl_enter();
  const int vec_per_row = H / 8;
  const int c = blockIdx.y * COMBINE_THREADS + threadIdx.x;
  if (c >= vec_per_row) return;
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (residual) acc8(reinterpret_cast<const uint4*>(residual + static_cast<long long>(t) * H)[c], 1.f, a);
    for (int k0 = 0; k0 < K; k0 += 8) {
      const long long at = static_cast<long long>(t) * K + k0;
      int row[8];
      float w[8];
      uint4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const bool has = k0 + k < K;
        row[k] = has ? dest_row[at + k] : -1;
        w[k] = (has && topk_w) ? topk_w[at + k] : 1.f;
      }
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (row[k] >= 0) v[k] = take_row<PASSING>(reinterpret_cast<const uint4*>(y_perm + static_cast<long long>(row[k]) * H) + c);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (row[k] >= 0) acc8(v[k], w[k], a);
    }
    reinterpret_cast<uint4*>(out + static_cast<long long>(t) * H)[c] = pack8(a);
  }
}

// One warp per permuted row: dy_perm[row] = w * dout[token]; dw[entry] = <dout[token], y_perm[row]>.
template <bool PASSING>
__global__ void combine_bwd_kernel(const bf16* __restrict__ dout, const bf16* __restrict__ y_perm,
                                   const int* __restrict__ row_src, const int* __restrict__ num_m_tiles,
                                   const float* __restrict__ topk_w, bf16* __restrict__ dy_perm,
                                   float* __restrict__ dtopk_w, int max_rows, int K, int H) {
  const int live_rows = min(num_m_tiles[1], max_rows);
  const int wpb = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < live_rows; row += gridDim.x * wpb) {
    const int src = row_src[row];
    uint4* dst = reinterpret_cast<uint4*>(dy_perm + static_cast<long long>(row) * H);
    if (src < 0) {
      for (int c = lane; c < H / 8; c += 32) dst[c] = make_uint4(0, 0, 0, 0);
      continue;
    }
    const float w = topk_w[src];
    const uint4* g = reinterpret_cast<const uint4*>(dout + static_cast<long long>(src / K) * H);
    const uint4* y = reinterpret_cast<const uint4*>(y_perm + static_cast<long long>(row) * H);
    float dot = 0.f;
    const int vec_per_row = H / 8;
    for (int c0 = lane; c0 < vec_per_row; c0 += 128) {  // four columns of both rows in flight
      uint4 gr[4], yr[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        gr[u] = yr[u] = make_uint4(0, 0, 0, 0);
        if (c0 + 32 * u < vec_per_row) {
          gr[u] = g[c0 + 32 * u];
          if (dtopk_w) yr[u] = take_row<PASSING>(y + c0 + 32 * u);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (c0 + 32 * u >= vec_per_row) break;
        float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        acc8(gr[u], w, a);
        put_row<PASSING>(dst + c0 + 32 * u, pack8(a));
        if (dtopk_w) {
          const __nv_bfloat162* gb = reinterpret_cast<const __nv_bfloat162*>(&gr[u]);
          const __nv_bfloat162* yb = reinterpret_cast<const __nv_bfloat162*>(&yr[u]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 gf = __bfloat1622float2(gb[i]), yf = __bfloat1622float2(yb[i]);
            dot += gf.x * yf.x + gf.y * yf.y;
          }
        }
      }
    }
    if (dtopk_w) {
      dot = warp_sum(dot);
      if (lane == 0) dtopk_w[src] = dot;
    }
  }
}

bool passing(long long rows, int H) { return rows * H * 2 > PASSING_BYTES; }

int grid_for(long long items, int threads, int cap = 148 * 8) {
  long long b = (items + threads - 1) / threads;
  if (b < 1) b = 1;
  return static_cast<int>(b < cap ? b : cap);
}

}  // namespace

void moe_router_topk(const float* logits, const int* replay_ids, int* topk_ids, float* topk_w, float* probs_out,
                     int T, int E, int K, bool renorm, cudaStream_t s) {
  if (T <= 0) return;
  const int wpb = 4;
  pdl_launch(router_topk_kernel, (T + wpb - 1) / wpb, wpb * 32, 0, s, logits, replay_ids, topk_ids, topk_w, probs_out, T, E, K,
                                                              renorm ? 1 : 0);
}

void moe_router_bwd(const float* probs, const int* topk_ids, const float* topk_w, const float* dtopk_w, float* dlogits,
                    int T, int E, int K, bool renorm, cudaStream_t s) {
  if (T <= 0) return;
  const int wpb = 4;
  router_bwd_kernel<<<(T + wpb - 1) / wpb, wpb * 32, 0, s>>>(probs, topk_ids, topk_w, dtopk_w, dlogits, T, E, K,
                                                             renorm ? 1 : 0);
}

// Blocks of the many-block variant; their counts are its scratch, ints [blocks][E].
static int sort_blocks(int n) { return n > 0 ? (n + SORT_WARPS * SORT_ROUNDS * 32 - 1) / (SORT_WARPS * SORT_ROUNDS * 32) : 1; }
// One block up to 4096 entries (16 warps of 8 rounds; its counts per warp need 4 (16 + 3) E bytes of shared memory).
static bool sort_in_one_block(int n, int max_rows, int E) { return n <= 4096 && max_rows <= 16384 && E <= 512; }

int moe_permutation_launches(int T, int K, int max_rows, int E) { return sort_in_one_block(T * K, max_rows, E) ? 1 : 3; }

long long moe_permutation_scratch(int T, int K, int max_rows, int E) {
  return sort_in_one_block(T * K, max_rows, E) ? 0 : static_cast<long long>(sort_blocks(T * K)) * E;
}

cudaError_t moe_build_permutation(const int* topk_ids, int T, int K, int E, int max_rows, int max_tiles, int align,
                                  int* expert_counts, int* expert_offsets, int* dest_row, int* row_src, int* tile_group,
                                  int* num_m_tiles, int* scratch, cudaStream_t s) {
  const int n = T * K;
  if (sort_in_one_block(n, max_rows, E)) {
    const auto smem = [&](int warps) { return static_cast<size_t>((warps + 3) * E + 2) * sizeof(int); };
    const int warps = n <= 128 ? 4 : 16;  // (four also fill row_src and the tile list quickly enough)
    return pdl_launch(n <= 512 ? build_small_kernel<1> : build_small_kernel<8>, 1, 32 * warps, smem(warps), s, topk_ids, n, E, max_rows,
                      max_tiles, align, expert_counts, expert_offsets, dest_row, row_src, tile_group, num_m_tiles);
  }
  const int blocks = sort_blocks(n);
  const int parts = E <= 1024 ? 8 : 1;  // (more experts: enough threads have one to follow, and shared memory holds their counts once)
  const size_t count_smem = static_cast<size_t>(E) * sizeof(int), assign_smem = SORT_WARPS * count_smem;
  const size_t scan_smem = static_cast<size_t>((3 + parts) * E + 2) * sizeof(int);
  // All three get their shared memory before the first is launched: a pass without the one before it would follow counts
  // that nobody wrote. Too many experts for it are refused here.
  const auto allow = [](auto kernel, size_t bytes) {
    return bytes <= 48 * 1024 ? cudaSuccess : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  };
  cudaError_t e = allow(count_kernel, count_smem);
  if (e == cudaSuccess) e = allow(scan_kernel, scan_smem);
  if (e == cudaSuccess) e = allow(assign_kernel, assign_smem);
  if (e == cudaSuccess) e = cudaMemsetAsync(row_src, 0xff, sizeof(int) * static_cast<size_t>(max_rows), s);
  if (e != cudaSuccess) return e;
  const auto launch = [s](auto kernel, int grid, int threads, size_t smem, auto... args) {  // its own result, not what others left
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
  };
  e = launch(count_kernel, blocks, SORT_WARPS * 32, count_smem, topk_ids, n, E, scratch);
  if (e == cudaSuccess)
    e = launch(scan_kernel, 1, 1024, scan_smem, scratch, blocks, parts, E, max_rows, max_tiles, align, expert_counts, expert_offsets,
               tile_group, num_m_tiles);
  if (e == cudaSuccess)
    e = launch(assign_kernel, blocks, SORT_WARPS * 32, assign_smem, topk_ids, n, E, scratch, expert_offsets, dest_row, row_src);
  return e;
}

void moe_permute(const void* x, const int* row_src, const int* num_m_tiles, void* x_perm, int max_rows, int H, int K,
                 cudaStream_t s) {
  if (max_rows <= 0) return;
  pdl_launch(passing(max_rows, H) ? permute_kernel<true> : permute_kernel<false>, grid_for(max_rows, 8), 256, 0, s, static_cast<const bf16*>(x), row_src, num_m_tiles,
                                                       static_cast<bf16*>(x_perm), max_rows, H, K);
}

void moe_combine(const void* y_perm, const int* dest_row, const float* topk_w, const void* residual, void* out, int T,
                 int K, int H, cudaStream_t s) {
  if (T <= 0) return;
  const dim3 grid(T, (H / 8 + COMBINE_THREADS - 1) / COMBINE_THREADS);
  pdl_launch(passing(static_cast<long long>(T) * K, H) ? combine_kernel<true> : combine_kernel<false>, grid, COMBINE_THREADS, 0, s, static_cast<const bf16*>(y_perm), dest_row, topk_w,
                                                  static_cast<const bf16*>(residual), static_cast<bf16*>(out), T, K, H);
}

void moe_unpermute_sum(const void* dx_perm, const int* dest_row, void* dx, int T, int K, int H, cudaStream_t s) {
  moe_combine(dx_perm, dest_row, nullptr, nullptr, dx, T, K, H, s);
}

void moe_combine_bwd(const void* dout, const void* y_perm, const int* row_src, const int* num_m_tiles,
                     const float* topk_w, void* dy_perm, float* dtopk_w, int max_rows, int K, int H, cudaStream_t s) {
  if (max_rows <= 0) return;
  const int wpb = 8;
  const auto kernel = passing(max_rows, H) ? combine_bwd_kernel<true> : combine_bwd_kernel<false>;
  kernel<<<grid_for(max_rows, wpb), wpb * 32, 0, s>>>(
      static_cast<const bf16*>(dout), static_cast<const bf16*>(y_perm), row_src, num_m_tiles, topk_w,
      static_cast<bf16*>(dy_perm), dtopk_w, max_rows, K, H);
}

}  // namespace mb
