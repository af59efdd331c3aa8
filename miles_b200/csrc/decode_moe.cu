// The experts of a decode step of at most 8 tokens: routing, gate and up projections with SwiGLU, down projection with the
// weighted combination and the residual. Three launches, between which nothing travels but the plan of the step, the activated
// rows of the chosen experts and the sum.
//
// All three are bound by latency at one token and by the bytes of the chosen experts at eight. The weights go through a ring of
// shared-memory stages filled by bulk asynchronous copies; two CTAs share an SM, so that one's start, end and reductions are
// covered by the other's copies. The token columns of an MMA (N = 8 of mma.m16n8k16, 16 weight rows as M, k permuted so that a lane
// reads 16 contiguous bytes) are the tokens of the step themselves: what a column multiplies does not change from expert to
// expert, and a token that did not choose the expert is left out when results are stored or summed.
//
//   router_decode    the product of small_gemv.cuh over a cluster of a CTA per 16 experts, whose first one routes
//   moe_decode_up    act[pair, I] = silu(gate) * up for the experts in use; a tile is eight gate rows and their eight up rows,
//                    whose sums, rounded to bf16, meet in the epilogue
//   moe_decode_down  y[t] = residual[t] + sum over the token's experts of w * W2[e] act[pair]
//
// Plan (int32): [0] experts in use; from [4] on 20 values for each of them, in the order of their ids: id, three unused, the
// pair (token * top_k + choice) of each of the eight tokens or -1, the tokens' weights as fp32 bits.
//
// Sums run in the order, and are rounded where, the kernels of decode_stream.cu and moe_combine have it: the values are theirs bit for bit,
// and a row's do not depend on the other rows of the step.
//
// Measured, us in a captured chain over 128 experts of 768 x 2048, against six launches (product, routing, up, down with SwiGLU,
// combination; one CTA per SM with items of 64 KB): 1 token 31.7 -> 26.4, 2 tokens 50.9 -> 37.6, 4 tokens 71.6 -> 57.7, 8 tokens
// 107 -> 87.8. Alone, 1 and 8 tokens (8 and some 52 experts): up 12.0 and 54.2 (their bytes at 6.5 TB/s: 7.7 and 50), down and
// combination 8.9 and 28.4 (3.9 and 25).
//
// Experts too many or too wide for this (`moe_decode_fits`) take decode_small.cu and decode_stream.cu.
//
// Reference counterpart: SGLang's fused-MoE decode kernels (miles/backends/sglang_utils/sglang_engine.py:73-152 launches them).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include <string>

#include "gemm.h"
#include "launchers.h"
#include "pdl.cuh"
#include "ptx.cuh"
#include "small_gemv.cuh"

namespace mb {
namespace {

constexpr int MAX_E = 128;          // a cluster of eight CTAs routes
constexpr int PLAN_HEAD = 4, PLAN_REC = 20, REC_PAIR = 4, REC_W = 12;
constexpr int ROWS = 16;            // weight rows of an MMA
constexpr int CWARPS = 8;           // consumer warps, each with an eighth of k
constexpr int THREADS = 32 * (1 + CWARPS);
constexpr int RING = 100 * 1024;    // of one of two CTAs on an SM
constexpr int RING_ALONE = 200 * 1024;
constexpr int MAX_STAGES = 6;
constexpr int MAX_REGS = 112;       // of a thread: two CTAs on an SM

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ uint4 lds16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * CWARPS) : "memory"); }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The first CTA's counterpart of an address in this CTA's shared memory, and stores to it.
__device__ __forceinline__ uint32_t of_first(const void* local) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(0u));
  return a;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void st_cluster(uint32_t addr, bf16 v) {
  asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(addr), "h"(__bfloat16_as_ushort(v)) : "memory");
}
// Copies in flight get a bounded chance to land before shared memory is released.
__device__ __forceinline__ void let_copies_land() {
  const unsigned long long t0 = globaltimer_ns();
  while (globaltimer_ns() - t0 < 2000000ull) {
  }
}
// Expert ids of all records, four per lane, asked for together with their count.
struct Experts {
  int id[MAX_E / 32];
  __device__ __forceinline__ Experts(const int* plan, int E, int lane) {
#pragma unroll
    for (int k = 0; k < MAX_E / 32; ++k) id[k] = lane + 32 * k < E ? plan[PLAN_HEAD + (lane + 32 * k) * PLAN_REC] : 0;
  }
  __device__ __forceinline__ int operator()(int i) const {  // warp-uniform i
    int v = id[0];
#pragma unroll
    for (int k = 1; k < MAX_E / 32; ++k) v = i >> 5 == k ? id[k] : v;
    return __shfl_sync(0xffffffffu, v, i & 31);
  }
};

// ---------------------------------------------------------------------------------------------- routing
// Order of floats as unsigned integers, -0 as +0; what can never be chosen (NaN, -infinity) is 0.
__device__ __forceinline__ unsigned order_key(float v) {
  if (!(v >= -FLT_MAX)) return 0u;
  const unsigned b = __float_as_uint(v + 0.f);
  return b & 0x80000000u ? ~b : b | 0x80000000u;
}

// Softmax, top-k (ties to the lower id) and the plan, by the first CTA: a warp per token, its logits in registers.
__device__ __forceinline__ void route(const float* lg, int T, int E, int K, int renorm, int* __restrict__ topk_ids,
                                      float* __restrict__ topk_w, int* __restrict__ plan) {
  constexpr int VALS = MAX_E / 32;
  __shared__ unsigned mask_s[MAX_E];  // tokens that chose the expert
  __shared__ int rec_s[MAX_E];        // its record
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < E; e += blockDim.x) mask_s[e] = 0u;
  __syncthreads();
  const bool has = warp < T;
  float my_w = 0.f;
  int my_id = MAX_E;
  if (has) {
    float v[VALS], m = -FLT_MAX;
    unsigned key[VALS];
#pragma unroll
    for (int i = 0; i < VALS; ++i) {
      const int e = lane + 32 * i;
      v[i] = e < E ? lg[warp * E + e] : -FLT_MAX;
      key[i] = e < E ? order_key(v[i]) : 0u;
      m = fmaxf(m, v[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < VALS; ++i)
      if (lane + 32 * i < E) s += __expf(v[i] - m);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float inv = 1.f / s;
    float wsum = 0.f;
    for (int k = 0; k < K; ++k) {
      unsigned best = 0u;
#pragma unroll
      for (int i = 0; i < VALS; ++i) best = max(best, key[i]);
      best = __reduce_max_sync(0xffffffffu, best);
      int bi = MAX_E;
#pragma unroll
      for (int i = VALS - 1; i >= 0; --i)
        if (key[i] == best) bi = lane + 32 * i;
      bi = best == 0u ? MAX_E : static_cast<int>(__reduce_min_sync(0xffffffffu, static_cast<unsigned>(bi)));
      float bv = 0.f;
#pragma unroll
      for (int i = 0; i < VALS; ++i)
        if (bi == lane + 32 * i) {
          bv = v[i];
          key[i] = 0u;
        }
      bv = __shfl_sync(0xffffffffu, bv, bi & 31);
      const float pw = __expf((best == 0u ? -FLT_MAX : bv) - m) * inv;
      wsum += pw;
      if (lane == k) {
        my_w = pw;
        my_id = bi;
      }
    }
    if (lane < K) {
      my_w = renorm ? my_w / wsum : my_w;
      topk_ids[warp * K + lane] = my_id < E ? my_id : 0x7fffffff;
      topk_w[warp * K + lane] = my_w;
      if (my_id < E) atomicOr(&mask_s[my_id], 1u << warp);
    }
  }
  __syncthreads();
  if (warp == 0) {  // the experts in use, in order
    int n = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const bool on = e0 + lane < E && mask_s[e0 + lane] != 0u;
      const unsigned b = __ballot_sync(0xffffffffu, on);
      if (on) rec_s[e0 + lane] = n + __popc(b & ((1u << lane) - 1u));
      n += __popc(b);
    }
    if (lane == 0) plan[0] = n;
  }
  __syncthreads();
  if (has && lane < K && my_id < E) {
    int* rec = plan + PLAN_HEAD + rec_s[my_id] * PLAN_REC;
    rec[REC_PAIR + warp] = warp * K + lane;
    rec[REC_W + warp] = __float_as_int(my_w);
  }
  for (int i = threadIdx.x; i < E * TOK; i += blockDim.x) {
    const int e = i / TOK, t = i % TOK;
    if (mask_s[e] == 0u) continue;
    int* rec = plan + PLAN_HEAD + rec_s[e] * PLAN_REC;
    if (t == 0) rec[0] = e;
    if (!((mask_s[e] >> t) & 1u)) rec[REC_PAIR + t] = -1;
  }
}

__global__ void __launch_bounds__(1024)
router_decode_kernel(const bf16* __restrict__ x, int T, const bf16* __restrict__ g, float eps, const bf16* __restrict__ W, int E, int H, int K,
                     int renorm, int* __restrict__ topk_ids, float* __restrict__ topk_w, int* __restrict__ plan) {
  __shared__ float lg[TOK * MAX_E];
  cluster_sync();  // (all CTAs run before one stores into another's shared memory; the predecessor is still busy)
  gemv_tile<true>(x, T, g, eps, W, H, [&](int t, int n, float v) { st_cluster(of_first(lg + t * E + n), v); });
  cluster_sync();
  if (blockIdx.x == 0) route(lg, T, E, K, renorm, topk_ids, topk_w, plan);
}

// ---------------------------------------------------------------------------------------------- gate and up
struct UpArgs {
  const bf16* W;       // [E, 2I, K]
  const bf16* x;       // [T, K]
  const bf16* norm_w;
  const int* plan;
  bf16* out;           // [pairs, I]
  float eps;
  int T, E, I, stages;
  int* status;
};

constexpr int UP_STAGE = 4;  // 256-wide k slices in a stage

// K = NCH * 256. Items are (expert, eight columns of I), in contiguous runs. A warp sums the slice of k that a warp of
// decode_stream.cu sums (`SL` 32-wide chunks of every 2048), in its order, so the values are the same. A stage holds whole slices: of a
// contraction of several stages the first four warps multiply one, the other four the next (and all wait for every stage: a warp that
// left one out could take the phase before the last for the one that it waits for).
template <int NCH>
__global__ void __maxnreg__(MAX_REGS) moe_up_kernel(const UpArgs a) {
  constexpr int K = NCH * 256;
  constexpr int CS = NCH < UP_STAGE ? NCH : UP_STAGE;
  constexpr int PARTS = (NCH + CS - 1) / CS;
  constexpr int LAST = NCH - (PARTS - 1) * CS;  // slices of the last stage
  constexpr int SL = PARTS == 1 ? NCH : 8, BLOCKS = (NCH + 7) / 8;
  constexpr int PITCH = CS * 512 + 64;  // (skewed: a warp's sixteen-byte reads touch every bank once)
  constexpr int STAGE = ROWS * PITCH;
  extern __shared__ uint8_t smem_raw[];
  __shared__ float red[2][CWARPS][ROWS][TOK];
  __shared__ float ssq[CWARPS][TOK];
  __shared__ __align__(8) unsigned long long bars[2 * MAX_STAGES];
  __shared__ int abort_s;
  volatile int* abort_flag = &abort_s;
  const uint32_t base = (smem_u32(smem_raw) + 127u) & ~127u;
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (MAX_STAGES + s); };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), CWARPS);
    }
    fence_barrier_init();
  }
  __syncthreads();
  pdl_enter();
  const int tiles = a.I / 8;
  int stage = 0;
  uint32_t phase = 0;
  auto advance = [&] {
    if (++stage == a.stages) {
      stage = 0;
      phase ^= 1u;
    }
  };
  auto run = [&](int& begin, int& end) {
    const int total = min(a.plan[0], a.E) * tiles;
    begin = static_cast<int>(static_cast<long long>(total) * blockIdx.x / gridDim.x);
    end = static_cast<int>(static_cast<long long>(total) * (blockIdx.x + 1) / gridDim.x);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer: a row per lane
    const Experts experts(a.plan, a.E, lane);
    int begin, end;
    run(begin, end);
    int g = begin / tiles, t = begin - g * tiles;
    bool ok = true;
    for (int item = begin; ok && item < end; ++item) {
      const int e = experts(g);
      const long long row = static_cast<long long>(e) * 2 * a.I + (lane < 8 ? 0 : a.I) + t * 8 + (lane & 7);
      const bf16* src = a.W + row * K;
#pragma unroll
      for (int p = 0; p < PARTS; ++p) {
        const uint32_t bytes = (p == PARTS - 1 ? LAST : CS) * 512u;
        ok = __all_sync(0xffffffffu, ok && mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, a.status, ERR_WAIT_EMPTY));
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(full_bar(stage), ROWS * bytes);
        __syncwarp();
        if (lane < ROWS) bulk_g2s(base + stage * STAGE + lane * PITCH, src + p * CS * 256, bytes, full_bar(stage));
        advance();
      }
      if (++t == tiles) {
        t = 0;
        ++g;
      }
    }
    if (!ok) let_copies_land();
  } else {
    // ------------------------------------------------------------------ consumers
    const int cw = warp - 1, ct = threadIdx.x - 32;
    const int r = lane >> 2, c = lane & 3;
    // this lane's share of its token's row, scaled by the norm's weights
    uint4 xa[BLOCKS * SL];
    float ss = 0.f;
#pragma unroll
    for (int u = 0; u < BLOCKS * SL; ++u) {
      const int k = u / SL * 2048 + (cw * SL + u % SL) * 32;
      xa[u] = make_uint4(0u, 0u, 0u, 0u);
      if (k < K) xa[u] = load_act<true>(a.x + static_cast<long long>(r) * K, a.norm_w, k + c * 8, r < a.T, ss);  // (warp-uniform)
    }
    int begin, end;
    run(begin, end);
    int g = begin / tiles, t = begin - g * tiles;
    // epilogue: thread (i, h, j) sums gate (h = 0) or up row i of token j
    const int ei = ct >> 4, eh = (ct >> 3) & 1, ej = ct & 7;
    ss = quad_sum(ss);
    if (c == 0) ssq[cw][r] = ss;
    float rs = 0.f;
    int pair = -1, par = 0;
    bool ok = true;
    for (int item = begin; item < end; ++item) {
      if (ct < 128 && (item == begin || t == 0)) pair = a.plan[PLAN_HEAD + g * PLAN_REC + REC_PAIR + ej];
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int p = 0; p < PARTS; ++p) {
        const int slice = PARTS == 1 ? cw : cw & 3;
        ok = ok && mbar_wait(full_bar(stage), phase, abort_flag, a.status, ERR_WAIT_FULL);
        if (ok) {
          if (PARTS == 1 || ((p & 1) == cw >> 2 && slice < (p == PARTS - 1 ? LAST : CS))) {  // (this warp's)
            const uint32_t sa = base + stage * STAGE + r * PITCH + (slice * SL * 32 + c * 8) * 2, sb = sa + 8 * PITCH;
#pragma unroll
            for (int u = 0; u < SL; ++u) {
              const uint4 w0 = lds16(sa + u * 64), w1 = lds16(sb + u * 64), xv = xa[p / 2 * SL + u];
              mma16816(acc, w0.x, w1.x, w0.y, w1.y, xv.x, xv.y);
              mma16816(acc, w0.z, w1.z, w0.w, w1.w, xv.z, xv.w);
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(empty_bar(stage));
        }
        advance();
      }
      red[par][cw][r][2 * c] = acc[0];
      red[par][cw][r][2 * c + 1] = acc[1];
      red[par][cw][r + 8][2 * c] = acc[2];
      red[par][cw][r + 8][2 * c + 1] = acc[3];
      consumer_sync();
      if (item == begin) {
        float q = 0.f;
#pragma unroll
        for (int w = 0; w < CWARPS; ++w) q += ssq[w][ej];
        rs = rsqrtf(q / static_cast<float>(K) + a.eps);
      }
      if (ct < 128) {  // (the other buffer is written next, so nobody has to wait for this)
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < CWARPS; ++w) v += red[par][w][ei + 8 * eh][ej];
        v = __bfloat162float(__float2bfloat16(v * rs));  // gate and up are bf16 everywhere else, too
        const float up = __shfl_xor_sync(0xffffffffu, v, 8);
        if (ok && eh == 0 && pair >= 0) a.out[static_cast<long long>(pair) * a.I + t * 8 + ei] = __float2bfloat16(v / (1.f + __expf(-v)) * up);
      }
      par ^= 1;
      if (++t == tiles) {
        t = 0;
        ++g;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------- down
// A CTA owns 16 rows of the output, for all tokens, and walks over the experts in use (a cluster of two deals them out alternately);
// an expert's tile is one contiguous copy. Its product, summed over the warps' k slices (those of decode_stream.cu) and rounded to bf16,
// waits in the first CTA's shared memory for the end, where a token's pairs are added in the order of its choices: neither the other tokens'
// experts nor the CTA that had an expert show in a sum, and the values are those of a product per pair and `moe_combine`. A lane's
// activations of the next expert are asked for while it multiplies this one.
struct DownArgs {
  const bf16* W;         // [E, H, I]
  const bf16* act;       // [pairs, I]
  const int* plan;
  const bf16* residual;  // [T, H]
  bf16* out;             // [T, H]
  int T, K, E, H, I, stages;
  int* status;
};

constexpr int MAX_PAIRS = TOK * 32;

// CPW: 32-wide k chunks of a warp: contiguous up to four, else eight of every 2048 (warps behind the end of k have fewer).
template <int CPW>
__global__ void __maxnreg__(MAX_REGS) moe_down_kernel(const DownArgs a) {
  constexpr int SL = CPW <= 4 ? CPW : 8;
  extern __shared__ uint8_t smem_raw[];
  __shared__ float red[2][CWARPS][ROWS][TOK];
  __shared__ short pair_s[MAX_E][TOK];  // [expert of this CTA][token] -> pair, or -1
  __shared__ float w_s[MAX_PAIRS];      // the pairs' weights (the first CTA's copy is used, as with their products)
  __shared__ __align__(8) unsigned long long bars[2 * MAX_STAGES];
  __shared__ int abort_s;
  volatile int* abort_flag = &abort_s;
  const uint32_t base = (smem_u32(smem_raw) + 127u) & ~127u;
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (MAX_STAGES + s); };
  const int pitch = a.I * 2, stage_bytes = ROWS * pitch, pairs = a.T * a.K;
  bf16* y_s = reinterpret_cast<bf16*>(smem_raw + (base - smem_u32(smem_raw)) + a.stages * stage_bytes);  // [pairs][ROWS]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), CWARPS);
    }
    fence_barrier_init();
  }
  for (int i = threadIdx.x; i < pairs; i += THREADS) {  // (a choice without an expert adds nothing)
    w_s[i] = 0.f;
    reinterpret_cast<uint4*>(y_s)[2 * i] = reinterpret_cast<uint4*>(y_s)[2 * i + 1] = make_uint4(0u, 0u, 0u, 0u);
  }
  __syncwarp();
  cluster_sync();  // (the other CTA runs before one stores into its shared memory; the predecessor is still busy)
  pdl_enter();
  const int rank = blockIdx.x, ranks = gridDim.x;  // (the cluster spans the grid's first dimension)
  const int row0 = blockIdx.y * ROWS;
  const int ot = threadIdx.x / ROWS, orow = threadIdx.x % ROWS;  // output of the first threads of rank 0
  const long long at = static_cast<long long>(ot) * a.H + row0 + orow;
  const bool writes = rank == 0 && threadIdx.x < ROWS * TOK && ot < a.T;
  const float res = writes ? __bfloat162float(a.residual[at]) : 0.f;
  int stage = 0;
  uint32_t phase = 0;
  auto advance = [&] {
    if (++stage == a.stages) {
      stage = 0;
      phase ^= 1u;
    }
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    const Experts experts(a.plan, a.E, lane);
    const int n = min(a.plan[0], a.E);
    bool ok = true;
    for (int i = rank; ok && i < n; i += ranks) {
      const int e = experts(i);
      ok = __all_sync(0xffffffffu, mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, a.status, ERR_WAIT_EMPTY));
      if (!ok) break;
      if (lane == 0) {
        mbar_expect_tx(full_bar(stage), stage_bytes);
        bulk_g2s(base + stage * stage_bytes, a.W + (static_cast<long long>(e) * a.H + row0) * a.I, stage_bytes, full_bar(stage));
      }
      advance();
    }
    if (!ok) let_copies_land();
  } else {
    // ------------------------------------------------------------------ consumers
    const int cw = warp - 1, ct = threadIdx.x - 32;
    const int r = lane >> 2, c = lane & 3;
    const int n = min(a.plan[0], a.E);
    const int mine = n > rank ? (n - rank + ranks - 1) / ranks : 0;
    for (int i = ct; rank + i / TOK * ranks < a.E; i += 32 * CWARPS) {  // (records behind the last one are not used)
      const int* rec = a.plan + PLAN_HEAD + (rank + i / TOK * ranks) * PLAN_REC;
      const int pair = rec[REC_PAIR + i % TOK];
      const float w = __int_as_float(rec[REC_W + i % TOK]);
      const bool has = i / TOK < mine && pair >= 0 && pair < pairs;
      pair_s[i / TOK][i % TOK] = static_cast<short>(has ? pair : -1);
      if (has) st_cluster(of_first(w_s + pair), w);
    }
    consumer_sync();
    const auto k_of = [&](int u) { return u / SL * 2048 + (cw * SL + u % SL) * 32; };  // chunks that lie beyond I are skipped (warp-uniform)
    auto load = [&](int i, uint4 (&x)[CPW]) {
      const int pair = pair_s[i][r];
#pragma unroll
      for (int u = 0; u < CPW; ++u) {
        x[u] = make_uint4(0u, 0u, 0u, 0u);
        if (pair >= 0 && k_of(u) < a.I) x[u] = ldg16(a.act + static_cast<long long>(pair) * a.I + k_of(u) + c * 8);
      }
    };
    uint4 xa[CPW], xn[CPW];
    if (mine > 0) load(0, xa);
    bool ok = true;
    for (int i = 0; i < mine; ++i) {
      if (i + 1 < mine) load(i + 1, xn);
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      ok = ok && mbar_wait(full_bar(stage), phase, abort_flag, a.status, ERR_WAIT_FULL);
      if (ok) {
        const uint32_t sa = base + stage * stage_bytes + r * pitch + c * 16, sb = sa + 8 * pitch;
#pragma unroll
        for (int u = 0; u < CPW; ++u) {
          if (k_of(u) < a.I) {
            const uint4 w0 = lds16(sa + k_of(u) * 2), w1 = lds16(sb + k_of(u) * 2);
            mma16816(acc, w0.x, w1.x, w0.y, w1.y, xa[u].x, xa[u].y);
            mma16816(acc, w0.z, w1.z, w0.w, w1.w, xa[u].z, xa[u].w);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty_bar(stage));
      }
      float(&part)[CWARPS][ROWS][TOK] = red[i & 1];
      part[cw][r][2 * c] = acc[0];
      part[cw][r][2 * c + 1] = acc[1];
      part[cw][r + 8][2 * c] = acc[2];
      part[cw][r + 8][2 * c + 1] = acc[3];
      consumer_sync();
      if (ct >> 7 == (i & 1)) {  // half of the threads sum an expert's slices, the other half the next one's (the buffers alternate, too)
        const int row = (ct & 127) >> 3, t = ct & 7, pair = pair_s[i][t];
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < CWARPS; ++w) v += part[w][row][t];
        if (ok && pair >= 0) st_cluster(of_first(y_s + pair * ROWS + row), __float2bfloat16(v));
      }
#pragma unroll
      for (int u = 0; u < CPW; ++u) xa[u] = xn[u];
      advance();
    }
  }
  // every thread of every CTA of the cluster arrives, whatever happened before
  __syncthreads();
  cluster_sync();
  if (writes) {
    float v = res + 0.f;
    for (int k0 = 0; k0 < a.K; k0 += 8) {
      float w[8], y[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int pair = ot * a.K + min(k0 + k, a.K - 1);
        w[k] = w_s[pair];
        y[k] = __bfloat162float(y_s[pair * ROWS + orow]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k0 + k < a.K) v = fmaf(w[k], y[k], v);
    }
    a.out[at] = __float2bfloat16(v);
  }
}

// ---------------------------------------------------------------------------------------------- host side
template <typename... P, typename... A>
cudaError_t launch_cluster(void (*kernel)(P...), dim3 grid, int threads, size_t smem, unsigned cluster, cudaStream_t s, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <int NCH>
cudaError_t launch_up(UpArgs a, int max_active, cudaStream_t s) {
  constexpr int CS = NCH < UP_STAGE ? NCH : UP_STAGE;
  constexpr int STAGE = ROWS * (CS * 512 + 64);
  a.stages = RING / STAGE < MAX_STAGES ? RING / STAGE : MAX_STAGES;
  const int smem = a.stages * STAGE + 128;
  auto kern = moe_up_kernel<NCH>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const long long items = static_cast<long long>(max_active) * (a.I / 8);
  return pdl_launch(kern, static_cast<int>(items < 2 * 148 ? items : 2 * 148), THREADS, smem, s, a);
}

template <int CPW>
cudaError_t launch_down(DownArgs a, cudaStream_t s) {
  const int stage = ROWS * a.I * 2, outs = a.T * a.K * ROWS * 2;
  const bool two = 3 * stage + outs <= RING;  // CTAs on an SM
  a.stages = ((two ? RING : RING_ALONE) - outs) / stage;
  if (a.stages > MAX_STAGES) a.stages = MAX_STAGES;
  const int smem = a.stages * stage + outs + 128;
  auto kern = moe_down_kernel<CPW>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const int tiles = a.H / ROWS;
  const unsigned split = tiles * 2 <= (two ? 2 : 1) * 148 ? 2 : 1;  // two CTAs per tile while the SMs hold all of them at once
  return launch_cluster(kern, dim3(split, tiles), THREADS, smem, split, s, a);
}

int launched(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return 0;
  cudaGetLastError();  // (reported here)
  return gemm_fail(std::string(what) + " launch failed: " + cudaGetErrorString(e));
}

}  // namespace

int moe_decode_plan_size(int E) { return PLAN_HEAD + E * PLAN_REC; }

// Rows of whole k slices in registers (H), three stages of a down tile in the largest ring (I).
bool moe_decode_fits(int E, int K, int H, int I) {
  return E >= 16 && E <= MAX_E && E % 16 == 0 && K >= 1 && K <= 32 && K <= E && H % 256 == 0 && H <= 4096 && I >= 32 && I % 32 == 0 &&
         3 * ROWS * I * 2 <= RING_ALONE;
}

int router_decode(const void* x, int T, const void* norm_w, float eps, const void* W, int E, int H, int K, bool renorm, int* topk_ids,
                  float* topk_w, int* plan, cudaStream_t s) {
  const int warps = gemv_warps(H) < TOK ? TOK : gemv_warps(H);  // (the routing takes a warp per token)
  return launched(launch_cluster(router_decode_kernel, dim3(E / 16), 32 * warps, 0, E / 16, s, static_cast<const bf16*>(x), T,
                                 static_cast<const bf16*>(norm_w), eps, static_cast<const bf16*>(W), E, H, K, renorm ? 1 : 0, topk_ids,
                                 topk_w, plan),
                  "router_decode");
}

int moe_decode_up(const void* x, int T, const void* norm_w, float eps, const void* W1, const int* plan, int max_active, int E, int H, int I,
                  void* act, int* status, cudaStream_t s) {
  UpArgs a = {};
  a.W = static_cast<const bf16*>(W1);
  a.x = static_cast<const bf16*>(x);
  a.norm_w = static_cast<const bf16*>(norm_w);
  a.plan = plan;
  a.out = static_cast<bf16*>(act);
  a.eps = eps;
  a.T = T;
  a.E = E;
  a.I = I;
  a.status = status;
#define MB_UP(N) \
  case N: return launched(launch_up<N>(a, max_active, s), "moe_decode_up")
  switch (H / 256) {
    MB_UP(1); MB_UP(2); MB_UP(3); MB_UP(4); MB_UP(5); MB_UP(6); MB_UP(7); MB_UP(8);
    MB_UP(9); MB_UP(10); MB_UP(11); MB_UP(12); MB_UP(13); MB_UP(14); MB_UP(15); MB_UP(16);
  }
#undef MB_UP
  return gemm_fail("moe_decode_up: unsupported width");
}

int moe_decode_down(const void* act, const void* W2, const int* plan, const void* residual, int T, int K, int E, int H, int I, void* y, int* status,
                    cudaStream_t s) {
  DownArgs a = {};
  a.W = static_cast<const bf16*>(W2);
  a.act = static_cast<const bf16*>(act);
  a.plan = plan;
  a.residual = static_cast<const bf16*>(residual);
  a.out = static_cast<bf16*>(y);
  a.T = T;
  a.K = K;
  a.E = E;
  a.H = H;
  a.I = I;
  a.status = status;
#define MB_DOWN(N) \
  case N: return launched(launch_down<N>(a, s), "moe_decode_down")
  // chunks of a warp as launch_stream of decode_stream.cu deals them
  switch (I % 256 == 0 && I <= 1024 ? I / 256 : I <= 2048 ? 8 : 10) {
    MB_DOWN(1); MB_DOWN(2); MB_DOWN(3); MB_DOWN(4); MB_DOWN(8); MB_DOWN(10);
  }
#undef MB_DOWN
  return gemm_fail("moe_decode_down: unsupported width");
}

}  // namespace mb
