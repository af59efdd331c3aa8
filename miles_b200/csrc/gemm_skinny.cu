// y[T, N] = x[T, K] W[N, K]^T (+ residual) for at most 128 rows of x: decode steps and short prompts of the engine.
//
// Such a product is bound by the bytes of W, and what decides its speed is how many of them are in flight, from how many
// SMs, how soon after the launch. The weights are therefore the 128-row operand of the tensor-core tile and the tokens its
// narrow one (16, 32, 64 or 128 columns), so that no part of a tile is padding that has to be streamed, and the contraction
// of one 128-row tile is split over a cluster of up to eight CTAs, each of which accumulates its share in TMEM. The shares
// meet in shared memory: every CTA stores its partial tile there, and after a cluster barrier each sums its part of the
// tokens over the cluster (distributed shared memory, in rank order, so results do not depend on timing) and stores it.
// Two or three CTAs share an SM, each with a ring of TMA stages as deep as its k range or its share of the SM allows: which
// SM holds how many does not matter, since all wait for the same HBM.
//
//   warp 0     : TMA producer (weights and activations, 128-byte swizzle, no multicast)
//   warp 1     : TMEM allocator, single-thread tcgen05.mma issuer
//   warps 2..5 : TMEM -> shared memory, cluster sum, store
//
// Measured, us per launch over weights that do not stay in L2 (before: 16-row mma.sync blocks up to 32 rows, tiles of 128
// token rows above; the weights' bytes alone at 6.5 TB/s): 23 tokens 19456 x 2560 41 -> 21.9 (15.3), 2560 x 9728 35 -> 13.8
// (7.7), 6144 x 2560 18 -> 10.8 (4.8), 128 x 2048 7 -> 5.0; 93 tokens 2560 x 9728 46 -> 17.5, 2560 x 4096 21 -> 11.8.
//
// Counterpart in the reference stack: the decode GEMMs of the serving engines (miles/backends/sglang_utils/sglang_engine.py:73-152).
#include <cuda.h>
#include <string.h>

#include <string>

#include "gemm.h"
#include "pdl.cuh"
#include "ptx.cuh"

namespace mb {
namespace {

constexpr int BM = 128, BK = 64;
constexpr int W_STAGE = BM * BK * 2;
constexpr int SK_THREADS = 192;
constexpr int MAX_SK_STAGES = 12;

struct SkinnyArgs {
  int T, N;
  int k_blocks, per_rank;  // 64-wide blocks of the contraction, and of each CTA of the cluster
  int stages;
  void* out;
  long long ldc;
  int out_fp32, vec_ok;
  const __nv_bfloat16* residual;  // same layout as out
  int* status;
};

__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t local_addr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

template <int NT>
__global__ void __launch_bounds__(SK_THREADS)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const SkinnyArgs p) {
  constexpr int X_STAGE = NT * BK * 2;
  constexpr int STAGE = W_STAGE + X_STAGE;
  constexpr uint32_t TMEM_COLS = NT < 32 ? 32 : NT;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  __shared__ __align__(8) unsigned long long bars[2 * MAX_SK_STAGES + 1];
  __shared__ uint32_t tmem_slot_s;
  __shared__ int abort_s;
  volatile int* abort_flag = &abort_s;
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (MAX_SK_STAGES + s); };
  const uint32_t done_bar = bar0 + 8u * (2 * MAX_SK_STAGES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank(), ranks = cluster_size();
  const int n0 = blockIdx.y * BM;
  const int kb0 = min(p.k_blocks, static_cast<int>(rank) * p.per_rank);
  const int k_iters = min(p.k_blocks, kb0 + p.per_rank) - kb0;

  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(done_bar, 1);
    fence_barrier_init();
    prefetch_tensormap(&map_w);
    prefetch_tensormap(&map_x);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot_s), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot_s);

  // the first ring of weights on its way into L2 while the predecessor finishes
  if (warp == 0 && lane == 0)
    for (int kb = 0; kb < min(k_iters, p.stages); ++kb) tma_prefetch_2d(&map_w, (kb0 + kb) * BK, n0);
  pdl_enter();

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < k_iters; ++kb) {
        if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.status, ERR_WAIT_EMPTY)) {
          ok = false;
          break;
        }
        mbar_expect_tx(full_bar(stage), STAGE);
        const uint32_t dst = base + stage * STAGE;
        tma_load_2d(dst, &map_w, full_bar(stage), (kb0 + kb) * BK, n0);
        tma_load_2d(dst + W_STAGE, &map_x, full_bar(stage), (kb0 + kb) * BK, 0);
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!ok) {  // give copies in flight a bounded chance to land before shared memory is released
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(BM, NT, false, false);
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = 0; kb < k_iters; ++kb) {
      if (!mbar_wait(full_bar(stage), phase, abort_flag, p.status, ERR_WAIT_FULL)) {
        ok = false;
        break;
      }
      tc_fence_after();
      if (lane == 0) {
        const uint32_t w = base + stage * STAGE, x = w + W_STAGE;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          umma_f16(tmem, make_smem_desc(w + k * 32, 16, 1024), make_smem_desc(x + k * 32, 16, 1024), idesc, (kb > 0 || k > 0) ? 1u : 0u);
        umma_commit(empty_bar(stage));
      }
      __syncwarp();
      if (++stage == p.stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (ok && lane == 0 && k_iters > 0) umma_commit(done_bar);
    __syncwarp();
  } else {
    // this CTA's share of the tile -> shared memory [token][row], over the ring (every stage has been consumed by now)
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const bool ok = k_iters == 0 || mbar_wait(done_bar, 0, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after();
      const uint32_t t_addr = tmem + (static_cast<uint32_t>(quad * 32) << 16);
      const uint32_t dst = base + row * 4;
#pragma unroll
      for (int c = 0; c < NT; c += 16) {
        if (c >= p.T) break;
        uint32_t r[16];
        if (k_iters > 0) {
          tmem_ld_32x16(t_addr + c, r);
          tmem_ld_wait();
        } else {  // (a rank past the end of the contraction)
#pragma unroll
          for (int i = 0; i < 16; ++i) r[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + (c + i) * (BM * 4)), "r"(r[i]) : "memory");
      }
      tc_fence_before();
    }
  }
  // every thread of every CTA of the cluster arrives, whatever happened before
  __syncthreads();
  cluster_sync_all();
  if (warp >= 2) {
    const int et = threadIdx.x - 64;  // 0..127
    const int col4 = et & 31;         // four rows of W
    const int n = n0 + col4 * 4;
    for (int t = static_cast<int>(rank) + static_cast<int>(ranks) * (et >> 5); t < p.T; t += static_cast<int>(ranks) * 4) {
      const uint32_t src = base + t * (BM * 4) + col4 * 16;
      float4 part[8];
#pragma unroll
      for (uint32_t r = 0; r < 8; ++r)
        if (r < ranks) part[r] = ld_cluster_f4(src, r);
      float4 v = part[0];
#pragma unroll
      for (uint32_t r = 1; r < 8; ++r)
        if (r < ranks) {
          v.x += part[r].x;
          v.y += part[r].y;
          v.z += part[r].z;
          v.w += part[r].w;
        }
      const long long o = static_cast<long long>(t) * p.ldc + n;
      float f[4] = {v.x, v.y, v.z, v.w};
      if (p.vec_ok && n + 4 <= p.N) {
        if (p.residual) {
          const uint2 raw = *reinterpret_cast<const uint2*>(p.residual + o);
          const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
          const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
          f[0] += a.x;
          f[1] += a.y;
          f[2] += b.x;
          f[3] += b.y;
        }
        if (p.out_fp32) *reinterpret_cast<float4*>(static_cast<float*>(p.out) + o) = make_float4(f[0], f[1], f[2], f[3]);
        else *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.out) + o) = make_uint2(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]));
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (n + i >= p.N) break;
          if (p.residual) f[i] += __bfloat162float(p.residual[o + i]);
          if (p.out_fp32) static_cast<float*>(p.out)[o + i] = f[i];
          else static_cast<__nv_bfloat16*>(p.out)[o + i] = __float2bfloat16(f[i]);
        }
      }
    }
  }
  __syncwarp();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
  cluster_sync_all();  // no CTA leaves while another still reads its shared memory
}

template <int NT>
int launch_skinny(const GemmProblem& g, const __nv_bfloat16* residual, cudaStream_t stream) {
  constexpr int STAGE = W_STAGE + NT * BK * 2;
  CUtensorMap mw, mx;
  if (gemm_make_map(&mw, g.b, BM)) return -1;
  if (gemm_make_map(&mx, g.a, NT)) return -1;
  SkinnyArgs p;
  memset(&p, 0, sizeof(p));
  p.T = g.M;
  p.N = g.N;
  p.k_blocks = (g.K + BK - 1) / BK;
  const int tiles = (g.N + BM - 1) / BM;
  // Split the contraction while every CTA keeps four blocks of it and the SMs hold all CTAs at once: three each, or two of
  // the wider token tiles once the split is two (measured, us with split 8 | 4 | 2: 5120 x 2048, 64 tokens 11.1 | 10.0 | 13;
  // 16 tokens 8.0 | 9.1 | 11; 24576 x 4096, 64 tokens, 2 at three per SM against 1 at two: 39.1 | 44.6).
  int split = 1;
  while (split < 8 && tiles * split * 2 <= 148 * (NT >= 64 && split >= 2 ? 2 : 3) && p.k_blocks >= split * 2 * 4) split *= 2;
  p.per_rank = (p.k_blocks + split - 1) / split;
  // The ring: as deep as the k range, or as the CTA's share of the SM's shared memory, a half or a third of it. (One CTA per
  // SM with all of it is slower even for 128 CTAs: sixteen clusters of eight do not fit the eight GPCs at one per SM. At
  // least two stages hold the [NT][128] fp32 partial tile that overlays the ring.)
  const int budget = (tiles * split <= 2 * 148 ? 100 : 73) * 1024;
  int stages = budget / STAGE;
  if (stages > MAX_SK_STAGES) stages = MAX_SK_STAGES;
  if (stages > p.per_rank) stages = p.per_rank;
  if (stages < 2) stages = 2;
  p.stages = stages;
  p.out = g.c;
  p.ldc = g.ldc;
  p.out_fp32 = g.out_fp32 ? 1 : 0;
  p.residual = residual;
  p.status = g.status;
  p.vec_ok = (g.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(g.c) & (g.out_fp32 ? 15 : 7)) == 0 &&
              (reinterpret_cast<uintptr_t>(residual) & 7) == 0) ? 1 : 0;
  const int smem = stages * STAGE + 1024;
  auto kern = gemm_skinny_kernel<NT>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 102 * 1024) != cudaSuccess)
    return gemm_fail("cudaFuncSetAttribute(MaxDynamicSharedMemorySize) failed");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(split, tiles);
  cfg.blockDim = dim3(SK_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, mw, mx, p);
  if (e != cudaSuccess) {
    cudaGetLastError();  // (reported here)
    return gemm_fail(std::string("skinny gemm launch failed: ") + cudaGetErrorString(e));
  }
  return 0;
}

}  // namespace

// N: beyond three tiles per SM (an LM head) the persistent kernel of gemm.cu streams the weights as fast (151936 x 2048:
// 100 us, 95 at 6.5 TB/s).
bool gemm_is_skinny(const GemmProblem& p) {
  return p.mode == GEMM_DENSE && p.M <= 128 && !p.a.mn_major && !p.b.mn_major && !p.accumulate && !p.row_ptrs && p.n_dest == 0 &&
         p.max_ctas == 0 && !p.whole_k && p.N <= 148 * 3 * BM;
}

int gemm_skinny_launch(const GemmProblem& g, const void* residual, cudaStream_t stream) {
  const __nv_bfloat16* r = static_cast<const __nv_bfloat16*>(residual);
  if (g.M <= 16) return launch_skinny<16>(g, r, stream);
  if (g.M <= 32) return launch_skinny<32>(g, r, stream);
  if (g.M <= 64) return launch_skinny<64>(g, r, stream);
  return launch_skinny<128>(g, r, stream);
}

}  // namespace mb
