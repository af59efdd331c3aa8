// Fused log-probability + entropy over a row of vocabulary logits, forward and backward.
//
// One CTA per row computes, in a single online-softmax sweep over the (bf16 or fp32) logits scaled by
// 1/temperature: log-sum-exp, sum_v p_v x_v, the target's log-probability and the entropy
// H = lse - sum_v p_v x_v. The [T, V] fp32 probabilities are never materialised. The backward pass
// writes dL/dlogits as bf16 (in place for bf16 logits) so the LM-head GEMMs can consume it directly.
//
// Reference counterparts: Megatron fused_vocab_parallel_cross_entropy and _VocabParallelEntropy
// (miles/backends/training_utils/loss_hub/math_utils.py:280-299,397-433).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "launchers.h"

namespace mb {
namespace {

using bf16 = __nv_bfloat16;

struct Stat {
  float m, s, sx;  // running max, sum exp(x-m), sum exp(x-m)*x
};

__device__ __forceinline__ void stat_add(Stat& a, float x) {
  if (x > a.m) {
    const float c = __expf(a.m - x);
    a.s = a.s * c + 1.f;
    a.sx = a.sx * c + x;
    a.m = x;
  } else {
    const float e = __expf(x - a.m);
    a.s += e;
    a.sx += e * x;
  }
}
__device__ __forceinline__ Stat stat_merge(const Stat& a, const Stat& b) {
  Stat r;
  r.m = fmaxf(a.m, b.m);
  const float ca = a.m == -FLT_MAX ? 0.f : __expf(a.m - r.m);
  const float cb = b.m == -FLT_MAX ? 0.f : __expf(b.m - r.m);
  r.s = a.s * ca + b.s * cb;
  r.sx = a.sx * ca + b.sx * cb;
  return r;
}

template <typename T>
__device__ __forceinline__ float ld(const T* p, long long i);
template <>
__device__ __forceinline__ float ld<float>(const float* p, long long i) { return p[i]; }
template <>
__device__ __forceinline__ float ld<bf16>(const bf16* p, long long i) { return __bfloat162float(p[i]); }

template <typename T, int THREADS>
__global__ void logprob_fwd_kernel(const T* __restrict__ logits, const int* __restrict__ targets,
                                   float* __restrict__ logprob, float* __restrict__ entropy, float* __restrict__ lse_out,
                                   float* __restrict__ psumx_out, int V, long long ld_, float inv_temp) {
  __shared__ Stat red[THREADS / 32];
  const long long row = blockIdx.x;
  const T* x = logits + row * ld_;
  Stat st{-FLT_MAX, 0.f, 0.f};
  constexpr int VEC = 16 / sizeof(T);
  const bool aligned = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  int v0 = 0;
  if (aligned) {
    const int nvec = V / VEC;
    for (int i = threadIdx.x; i < nvec; i += THREADS) {
      const uint4 raw = reinterpret_cast<const uint4*>(x)[i];
      if constexpr (sizeof(T) == 2) {
        const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __bfloat1622float2(b[j]);
          stat_add(st, f.x * inv_temp);
          stat_add(st, f.y * inv_temp);
        }
      } else {
        const float* f = reinterpret_cast<const float*>(&raw);
#pragma unroll
        for (int j = 0; j < 4; ++j) stat_add(st, f[j] * inv_temp);
      }
    }
    v0 = nvec * VEC;
  }
  for (int i = v0 + threadIdx.x; i < V; i += THREADS) stat_add(st, ld<T>(x, i) * inv_temp);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Stat other;
    other.m = __shfl_xor_sync(0xffffffffu, st.m, o);
    other.s = __shfl_xor_sync(0xffffffffu, st.s, o);
    other.sx = __shfl_xor_sync(0xffffffffu, st.sx, o);
    st = stat_merge(st, other);
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = st;
  __syncthreads();
  if (threadIdx.x == 0) {
    Stat tot = red[0];
    for (int w = 1; w < THREADS / 32; ++w) tot = stat_merge(tot, red[w]);
    const float lse = tot.m + logf(tot.s);
    const float px = tot.sx / tot.s;
    if (lse_out) lse_out[row] = lse;
    if (psumx_out) psumx_out[row] = px;
    if (entropy) entropy[row] = lse - px;
    if (logprob) {
      const int t = targets[row];
      logprob[row] = (t >= 0 && t < V) ? ld<T>(x, t) * inv_temp - lse : 0.f;
    }
  }
}

// The end of it where the product already left (maximum, sum, moment about the maximum) for every 128 columns (EPI_SCORES of gemm.cu): part
// [pieces][T], row_target[T] the targets' scaled logits. A lane per row, the pieces dealt to the warps in turn.
constexpr int MERGE_WARPS = 16;
__global__ void __launch_bounds__(32 * MERGE_WARPS)
logprob_merge_kernel(const float4* __restrict__ part, const float* __restrict__ row_target, const int* __restrict__ targets,
                     float* __restrict__ logprob, float* __restrict__ entropy, float* __restrict__ lse_out, float* __restrict__ psumx_out, int T,
                     int V, int pieces) {
  __shared__ Stat red[MERGE_WARPS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = blockIdx.x * 32 + lane;
  const auto merge = [](const Stat& a, const Stat& b) {
    const float m = fmaxf(a.m, b.m), ca = __expf(a.m - m), cb = __expf(b.m - m);
    Stat r{m, a.s * ca + b.s * cb, 0.f};
    if (ca > 0.f) r.sx = ca * (a.sx + a.s * (a.m - m));
    if (cb > 0.f) r.sx += cb * (b.sx + b.s * (b.m - m));
    return r;
  };
  Stat st{-FLT_MAX, 0.f, 0.f};
  if (row < T) {
#pragma unroll 8
    for (int i = warp; i < pieces; i += MERGE_WARPS) {
      const float4 v = part[static_cast<long long>(i) * T + row];
      st = merge(st, Stat{v.x, v.y, v.z});
    }
  }
  red[warp][lane] = st;
  __syncthreads();
  if (warp > 0 || row >= T) return;
  for (int w = 1; w < MERGE_WARPS; ++w) st = merge(st, red[w][lane]);
  const float ls = logf(st.s), mean = st.sx / st.s, lse = st.m + ls;
  lse_out[row] = lse;
  psumx_out[row] = st.m + mean;
  entropy[row] = ls - mean;  // (about the maximum: what the two have in common does not have to cancel)
  const int t = targets[row];
  logprob[row] = (t >= 0 && t < V) ? row_target[row] - lse : 0.f;
}

// VEC values per thread and step (16-byte loads of both types, 8- or 16-byte stores) where rows and pointers allow, else one.
// In place over bf16 logits every value is read and written by the same thread. 2048 rows of 151936 fp32 logits: 622 us with
// 4-byte loads and 2-byte stores, 277 us now (1.87 GB move).
template <typename T, int THREADS, int VEC>
__global__ void logprob_bwd_kernel(const T* __restrict__ logits, const int* __restrict__ targets,
                                   const float* __restrict__ lse, const float* __restrict__ psumx,
                                   const float* __restrict__ dlogprob, const float* __restrict__ dentropy,
                                   bf16* __restrict__ dlogits, int V, long long ld_, long long ld_out, float inv_temp) {
  const long long row = blockIdx.x;
  const T* x = logits + row * ld_;
  bf16* dx = dlogits + row * ld_out;
  const float l = lse[row];
  const float px = psumx[row];
  const float dlp = dlogprob ? dlogprob[row] : 0.f;
  const float dh = dentropy ? dentropy[row] : 0.f;
  const int t = targets[row];
  for (int i = (blockIdx.y * THREADS + threadIdx.x) * VEC; i < V; i += gridDim.y * THREADS * VEC) {
    float f[VEC];
    if constexpr (VEC == 1) {
      f[0] = ld<T>(x, i);
    } else {
      const uint4 raw = *reinterpret_cast<const uint4*>(x + i);
      if constexpr (sizeof(T) == 2) {
        const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int j = 0; j < VEC / 2; ++j) {
          const float2 v = __bfloat1622float2(b[j]);
          f[2 * j] = v.x;
          f[2 * j + 1] = v.y;
        }
      } else {
#pragma unroll
        for (int j = 0; j < VEC; ++j) f[j] = reinterpret_cast<const float*>(&raw)[j];
      }
    }
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      const float xs = f[j] * inv_temp;
      const float p = __expf(xs - l);
      float g = -dlp * p - dh * p * (xs - px);
      if (i + j == t) g += dlp;
      f[j] = g * inv_temp;
    }
    if constexpr (VEC == 1) {
      dx[i] = __float2bfloat16(f[0]);
    } else {
      __nv_bfloat162 o[VEC / 2];
#pragma unroll
      for (int j = 0; j < VEC / 2; ++j) o[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
      if constexpr (VEC == 8) *reinterpret_cast<uint4*>(dx + i) = *reinterpret_cast<const uint4*>(o);
      else *reinterpret_cast<uint2*>(dx + i) = *reinterpret_cast<const uint2*>(o);
    }
  }
}

template <typename T, int VEC>
void launch_bwd(const T* logits, const int* targets, const float* lse, const float* psumx, const float* dlogprob,
                const float* dentropy, bf16* dlogits, int rows, int V, long long ld, long long ld_out, float inv_temp, cudaStream_t s) {
  constexpr int PER_BLOCK = 256 * VEC * (VEC == 1 ? 8 : 4);  // a few steps per thread
  const dim3 grid(rows, (V + PER_BLOCK - 1) / PER_BLOCK > 0 ? (V + PER_BLOCK - 1) / PER_BLOCK : 1);
  logprob_bwd_kernel<T, 256, VEC><<<grid, 256, 0, s>>>(logits, targets, lse, psumx, dlogprob, dentropy, dlogits, V, ld, ld_out, inv_temp);
}

}  // namespace

void logprob_entropy_fwd(const void* logits, bool fp32, const int* targets, float* logprob, float* entropy, float* lse,
                         float* psum_x, int T, int V, long long ld, float inv_temp, cudaStream_t s) {
  if (T <= 0) return;
  if (fp32)
    logprob_fwd_kernel<float, 512><<<T, 512, 0, s>>>(static_cast<const float*>(logits), targets, logprob, entropy, lse,
                                                     psum_x, V, ld, inv_temp);
  else
    logprob_fwd_kernel<bf16, 512><<<T, 512, 0, s>>>(static_cast<const bf16*>(logits), targets, logprob, entropy, lse,
                                                    psum_x, V, ld, inv_temp);
}

void logprob_entropy_merge(const float* part, const float* row_target, const int* targets, float* logprob, float* entropy, float* lse, float* psum_x,
                           int T, int V, cudaStream_t s) {
  if (T <= 0) return;
  logprob_merge_kernel<<<(T + 31) / 32, 32 * MERGE_WARPS, 0, s>>>(reinterpret_cast<const float4*>(part), row_target, targets, logprob, entropy, lse,
                                                                  psum_x, T, V, (V + 127) / 128);
}

void logprob_entropy_bwd(const void* logits, bool fp32, const int* targets, const float* lse, const float* psum_x,
                         const float* dlogprob, const float* dentropy, void* dlogits, int T, int V, long long ld,
                         long long ld_out, float inv_temp, cudaStream_t s) {
  if (T <= 0) return;
  bf16* out = static_cast<bf16*>(dlogits);
  const auto even = [&](int vec) {  // whole vectors, aligned in every row
    return V % vec == 0 && ld % vec == 0 && ld_out % vec == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0 &&
           (reinterpret_cast<uintptr_t>(dlogits) & (2 * vec - 1)) == 0;
  };
#define MB_BWD(T, VEC) \
  launch_bwd<T, VEC>(static_cast<const T*>(logits), targets, lse, psum_x, dlogprob, dentropy, out, T_, V, ld, ld_out, inv_temp, s)
  const int T_ = T;
  if (fp32) {
    if (even(4)) MB_BWD(float, 4);
    else MB_BWD(float, 1);
  } else {
    if (even(8)) MB_BWD(bf16, 8);
    else MB_BWD(bf16, 1);
  }
#undef MB_BWD
}

}  // namespace mb
