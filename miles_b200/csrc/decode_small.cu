// Light kernels for decode steps of at most 8 tokens.
//
// small_gemv_direct: y[T,N] = (norm?)(x) W^T (+ residual) for weight matrices of a few tens of MB (qkv, o, router):
// one CTA per 16 weight rows, k split across up to 32 warps so that every load of the CTA is issued before the
// first MMA. It starts faster than the persistent streaming kernel of decode_stream.cu (no ring to fill), which
// wins once the matrix is large enough to keep that ring busy. Same MMA scheme: 8 tokens = N of mma.m16n8k16, k
// permuted so that a lane reads 16 contiguous bytes per row, RMSNorm folded in.
//
// router_small: softmax -> top-k (+renorm) over the fp32 router logits and the per-expert (token, slot) lists that
// the weight-streaming MoE kernels consume instead of a sorted permutation.
//
// Reference counterpart: the top-k softmax routing inside SGLang's fused MoE
// (miles/backends/sglang_utils/sglang_engine.py:73-152 launches those engines).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "launchers.h"
#include "pdl.cuh"
#include "small_gemv.cuh"

namespace mb {
namespace {

template <bool NORM>
__global__ void __launch_bounds__(1024) small_gemv_kernel(const bf16* __restrict__ x, int T, const bf16* __restrict__ g,
                                                          float eps, const bf16* __restrict__ W, int N, int K,
                                                          const bf16* __restrict__ residual, void* __restrict__ out,
                                                          int out_fp32) {
  gemv_tile<NORM>(x, T, g, eps, W, K, [&](int t, int n, float v) {
    const long long o = static_cast<long long>(t) * N + n;
    if (residual) v += __bfloat162float(residual[o]);
    if (out_fp32)
      static_cast<float*>(out)[o] = v;
    else
      static_cast<bf16*>(out)[o] = __float2bfloat16(v);
  });
}


// ---------------------------------------------------------------------------------------------- router_small
// One CTA of 8 warps over the fp32 router logits [T, E] (a small_gemv with the norm folded in produces them).
// Outputs: topk_ids[T,K], topk_w[T,K], and for the MoE kernels the compact list of active experts with, per
// expert, the (token, slot) pairs routed to it: active[0] = count, active[1..] = expert ids, pair_count[E],
// pair_list[E][TOK] (pair = t*K + k; a token picks an expert at most once).
// A token's warp keeps its logits in registers (VALS per lane) and takes one maximum after another; the lists come from one
// mask of token bits per expert and a ballot over each 32 experts. One row over 128 experts: 4.0 us, 11.4 us when the logits
// and the experts already taken were read again for every choice and one thread collected the active experts.
template <int VALS>
__global__ void __launch_bounds__(256) router_small_kernel(const float* __restrict__ logits, int T, int E, int K,
                                                           int renorm, int* __restrict__ topk_ids,
                                                           float* __restrict__ topk_w, int* __restrict__ active,
                                                           int* __restrict__ pair_count, int* __restrict__ pair_list) {
  pdl_enter();
  __shared__ unsigned mask_s[32 * VALS];  // tokens that chose the expert
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < E; e += blockDim.x) mask_s[e] = 0u;
  float v[VALS];
  float m = -FLT_MAX;
  const bool has = warp < T;
  if (has) {
#pragma unroll
    for (int i = 0; i < VALS; ++i) {
      const int e = lane + 32 * i;
      v[i] = e < E ? logits[static_cast<long long>(warp) * E + e] : -FLT_MAX;
      m = fmaxf(m, v[i]);
    }
  }
  __syncthreads();
  float my_w = 0.f;
  int my_id = 0;
  if (has) {
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
    unsigned taken = 0u;  // this lane's experts among the choices so far
    for (int k = 0; k < K; ++k) {
      float best = -FLT_MAX;
      int bi = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < VALS; ++i) {
        const int e = lane + 32 * i;
        if (e < E && !((taken >> i) & 1u) && (v[i] > best || (v[i] == best && e < bi))) {
          best = v[i];
          bi = e;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) {
          best = ob;
          bi = oi;
        }
      }
      if ((bi & 31) == lane) taken |= 1u << (bi >> 5 & 31);
      const float pw = __expf(best - m) * inv;
      wsum += pw;
      if (lane == k) {
        my_w = pw;
        my_id = bi;
      }
    }
    if (lane < K) {
      topk_ids[warp * K + lane] = my_id;
      topk_w[warp * K + lane] = renorm ? my_w / wsum : my_w;
      if (my_id < E) atomicOr(&mask_s[my_id], 1u << warp);
    }
  }
  __syncthreads();
  // a token picks an expert at most once, so its place in the expert's list is the number of earlier tokens in the mask
  if (has && lane < K && my_id < E)
    pair_list[my_id * TOK + __popc(mask_s[my_id] & ((1u << warp) - 1u))] = warp * K + lane;
  for (int e = threadIdx.x; e < E; e += blockDim.x) pair_count[e] = __popc(mask_s[e]);
  if (warp == 7) {  // the experts in use, in order
    int n = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const bool on = e0 + lane < E && mask_s[e0 + lane] != 0u;
      const unsigned b = __ballot_sync(0xffffffffu, on);
      if (on) active[1 + n + __popc(b & ((1u << lane) - 1u))] = e0 + lane;
      n += __popc(b);
    }
    if (lane == 0) active[0] = n;
  }
}

}  // namespace

cudaError_t small_gemv_direct(const void* x, int T, const void* norm_w, float eps, const void* W, int N, int K,
                              const void* residual, void* out, bool out_fp32, cudaStream_t s) {
  return pdl_launch(norm_w ? small_gemv_kernel<true> : small_gemv_kernel<false>, N / 16, 32 * gemv_warps(K), 0, s, static_cast<const bf16*>(x), T,
                    static_cast<const bf16*>(norm_w), eps, static_cast<const bf16*>(W), N, K, static_cast<const bf16*>(residual), out,
                    out_fp32 ? 1 : 0);
}

void router_small(const float* logits, int T, int E, int K, bool renorm, int* topk_ids, float* topk_w, int* active,
                  int* pair_count, int* pair_list, cudaStream_t s) {
  if (E <= 128)
    pdl_launch(router_small_kernel<4>, 1, 256, 0, s, logits, T, E, K, renorm ? 1 : 0, topk_ids, topk_w, active, pair_count, pair_list);
  else  // up to 1024 experts (checked by the caller)
    pdl_launch(router_small_kernel<32>, 1, 256, 0, s, logits, T, E, K, renorm ? 1 : 0, topk_ids, topk_w, active, pair_count, pair_list);
}

}  // namespace mb
