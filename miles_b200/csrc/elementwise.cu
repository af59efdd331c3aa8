// Bandwidth-bound fused kernels of the transformer block: RMSNorm (fwd/bwd), per-head QK-RMSNorm +
// rotary embedding (fwd/bwd, optionally scattering K/V into a paged cache), SwiGLU (fwd/bwd) and the
// fused Adam update. All rows are processed with 128-bit loads/stores and fp32 arithmetic.
//
// Reference counterparts: TransformerEngine RMSNorm / fused RoPE / bias-SwiGLU and FusedAdam as used
// by the Megatron trainer (miles/backends/megatron_utils/model.py:125-210, 560-570).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launchers.h"
#include "pdl.cuh"

namespace mb {
namespace {

using bf16 = __nv_bfloat16;

struct alignas(16) BF8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void load8(const bf16* p, float (&f)[8]) {
  const BF8 r = *reinterpret_cast<const BF8*>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(r.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(bf16* p, const float (&f)[8]) {
  BF8 r;
#pragma unroll
  for (int i = 0; i < 4; ++i) r.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<BF8*>(p) = r;
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&t);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (threadIdx.x < THREADS / 32) ? red[threadIdx.x] : 0.f;
  if (w == 0) {
    t = warp_sum(t);
    if (l == 0) red[0] = t;
  }
  __syncthreads();
  const float r = red[0];
  __syncthreads();
  return r;
}

// ------------------------------------------------------------------ RMSNorm
// One CTA per row; H % 8 == 0. Optionally adds a residual first: h = x + res, writes h to res_out.
// VPT: 16-byte pieces of the row that a thread holds in registers from the first pass to the second, together with the norm's
// weights (0: rows too wide for that are read again). 16384 rows of 2048 with a residual: 65.5 ->
// 57.3 us (268 MB), without 49.1 -> 38.9.
template <int THREADS, int VPT>
__global__ void __launch_bounds__(THREADS)
rmsnorm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res, const bf16* __restrict__ w, bf16* __restrict__ y,
                   bf16* __restrict__ res_out, float* __restrict__ rstd, int H, float eps) {
  pdl_enter();
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const bf16* xr = x + row * H;
  float ss = 0.f;
  if constexpr (VPT > 0) {
    float f[VPT][8];
    BF8 wv[VPT];
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int c = (v * THREADS + threadIdx.x) * 8;
      if (c >= H) break;
      load8(xr + c, f[v]);
      wv[v] = *reinterpret_cast<const BF8*>(w + c);
      if (res) {
        float g[8];
        load8(res + row * H + c, g);
        // round through bf16 so that the statistics match what is stored
#pragma unroll
        for (int i = 0; i < 8; ++i) f[v][i] = __bfloat162float(__float2bfloat16(f[v][i] + g[i]));
        store8(res_out + row * H + c, f[v]);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += f[v][i] * f[v][i];
    }
    const float tot = block_sum<THREADS>(ss, red);
    const float r = rsqrtf(tot / H + eps);
    if (threadIdx.x == 0 && rstd) rstd[row] = r;
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int c = (v * THREADS + threadIdx.x) * 8;
      if (c >= H) break;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 g = __bfloat1622float2(wv[v].v[i]);
        f[v][2 * i] = f[v][2 * i] * r * g.x;
        f[v][2 * i + 1] = f[v][2 * i + 1] * r * g.y;
      }
      store8(y + row * H + c, f[v]);
    }
    return;
  }
  for (int c = threadIdx.x * 8; c < H; c += THREADS * 8) {
    float f[8];
    load8(xr + c, f);
    if (res) {
      float g[8];
      load8(res + row * H + c, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] += g[i];
      // round through bf16 so that the statistics match what is stored
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = __bfloat162float(__float2bfloat16(f[i]));
      store8(res_out + row * H + c, f);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += f[i] * f[i];
  }
  const float tot = block_sum<THREADS>(ss, red);
  const float r = rsqrtf(tot / H + eps);
  if (threadIdx.x == 0 && rstd) rstd[row] = r;
  const bf16* src = res ? res_out + row * H : xr;
  for (int c = threadIdx.x * 8; c < H; c += THREADS * 8) {
    float f[8], g[8];
    load8(src + c, f);
    load8(w + c, g);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = f[i] * r * g[i];
    store8(y + row * H + c, f);
  }
}

// dx = rstd * (dy*w - xhat * mean(dy*w*xhat)); dw partials are accumulated per CTA over a strip of rows.
// VPT as above: a thread keeps its columns of a row, of the weights and of dw in registers, and asks for its columns of the next row
// before it sums this one (0: wide rows are read twice and dw lives in shared memory). 16384 rows of 2048:
// 124 -> 87 us, with a residual's gradient 152 -> 93 (268 MB).
template <int THREADS, int VPT>
__global__ void __launch_bounds__(THREADS)
rmsnorm_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w, const float* __restrict__ rstd,
                   const bf16* __restrict__ dres, bf16* __restrict__ dx, float* __restrict__ dw_partial, int T, int H) {
  __shared__ float red[32];
  if constexpr (VPT > 0) {
    float acc[VPT][8], g[VPT][8];
    BF8 na[VPT], nb[VPT], ne[VPT];
    float nr = 0.f;
    const auto fetch = [&](long long row) {
      nr = rstd[row];
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int c = (v * THREADS + threadIdx.x) * 8;
        if (c >= H) break;
        na[v] = *reinterpret_cast<const BF8*>(dy + row * H + c);
        nb[v] = *reinterpret_cast<const BF8*>(x + row * H + c);
        if (dres) ne[v] = *reinterpret_cast<const BF8*>(dres + row * H + c);
      }
    };
    const auto unpack = [](const BF8& r, float (&f)[8]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 t = __bfloat1622float2(r.v[i]);
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
      }
    };
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int c = (v * THREADS + threadIdx.x) * 8;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[v][i] = g[v][i] = 0.f;
      if (c < H) load8(w + c, g[v]);
    }
    if (blockIdx.x < T) fetch(blockIdx.x);
    for (long long row = blockIdx.x; row < T; row += gridDim.x) {
      const float r = nr;
      BF8 ca[VPT], cb[VPT], ce[VPT];
      float dot = 0.f;
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        if ((v * THREADS + threadIdx.x) * 8 >= H) break;
        ca[v] = na[v];
        cb[v] = nb[v];
        ce[v] = ne[v];
        float a[8], b[8];
        unpack(ca[v], a);
        unpack(cb[v], b);
#pragma unroll
        for (int i = 0; i < 8; ++i) dot += a[i] * g[v][i] * b[i] * r;
      }
      if (row + gridDim.x < T) fetch(row + gridDim.x);
      const float mean = block_sum<THREADS>(dot, red) / H;
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int c = (v * THREADS + threadIdx.x) * 8;
        if (c >= H) break;
        float a[8], b[8], o[8];
        unpack(ca[v], a);
        unpack(cb[v], b);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xhat = b[i] * r;
          o[i] = r * (a[i] * g[v][i] - xhat * mean);
          acc[v][i] += a[i] * xhat;
        }
        if (dres) {
          float e[8];
          unpack(ce[v], e);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += e[i];
        }
        store8(dx + row * H + c, o);
      }
    }
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int c = (v * THREADS + threadIdx.x) * 8;
      if (c >= H) break;
      float* to = dw_partial + static_cast<long long>(blockIdx.x) * H + c;
      *reinterpret_cast<float4*>(to) = make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
      *reinterpret_cast<float4*>(to + 4) = make_float4(acc[v][4], acc[v][5], acc[v][6], acc[v][7]);
    }
    return;
  }
  extern __shared__ float dw_acc[];  // [H]
  for (int c = threadIdx.x; c < H; c += THREADS) dw_acc[c] = 0.f;
  __syncthreads();
  for (long long row = blockIdx.x; row < T; row += gridDim.x) {
    const float r = rstd[row];
    float dot = 0.f;
    for (int c = threadIdx.x * 8; c < H; c += THREADS * 8) {
      float a[8], b[8], g[8];
      load8(dy + row * H + c, a);
      load8(x + row * H + c, b);
      load8(w + c, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) dot += a[i] * g[i] * b[i] * r;
    }
    const float mean = block_sum<THREADS>(dot, red) / H;
    for (int c = threadIdx.x * 8; c < H; c += THREADS * 8) {
      float a[8], b[8], g[8], o[8];
      load8(dy + row * H + c, a);
      load8(x + row * H + c, b);
      load8(w + c, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float xhat = b[i] * r;
        o[i] = r * (a[i] * g[i] - xhat * mean);
        dw_acc[c + i] += a[i] * xhat;
      }
      if (dres) {
        float e[8];
        load8(dres + row * H + c, e);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] += e[i];
      }
      store8(dx + row * H + c, o);
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < H; c += THREADS) dw_partial[static_cast<long long>(blockIdx.x) * H + c] = dw_acc[c];
}

__global__ void colsum_kernel(const float* __restrict__ part, float* __restrict__ out, int rows, int H, int accumulate) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= H) return;
  float s = 0.f;
  for (int r = 0; r < rows; ++r) s += part[static_cast<long long>(r) * H + c];
  out[c] = accumulate ? out[c] + s : s;
}

// ------------------------------------------------------------------ QK-norm + RoPE
// qkv: [T, (Hq + 2*Hk) * D] as produced by the fused QKV projection (q heads, then k heads, then v heads).
// Outputs: q_out [T, Hq, D], k_out [T, Hk, D] (v is consumed in place by the attention kernels).
// When kv_cache pointers are given, K and V rows are also scattered to slot_mapping[t] of the paged cache.
// inv_freq_tab (64 floats, or null): inverse frequencies of a model with scaled rotary embeddings (Llama-3.1 style or
// linear scaling); null means theta^(-d/64).
//
// Bound by memory once the trigonometry is shared: a half-warp owns a head and a warp walks over the heads of ONE token, so that
// sines and cosines are taken once per token instead of once per head, and the powf behind them once per warp (one warp per
// (token, head) had spent its time in powf and sincosf). A lane holds four values of the first half of the rotated dimensions and
// the four they pair with, so a rotation needs no exchange; the four angles of a lane are shared with the other half-warp,
// each takes two. A token's heads are dealt to `chunks` warps: few tokens (decoding) need the parallelism, many do not.
// 16384 tokens, 32 query + 4 key heads: forward 363 -> 125 us, 111 with two pairs of heads ahead and four blocks per SM (four pairs
// 116), backward 416 -> 172 us (302 and 453 MB moved): the instructions of norms and roundings are what bounds it now;
// one token (in a captured graph): 2.9 -> 2.6 us.
constexpr int ROPE_D = 128;
constexpr int ROPE_AHEAD = 2;  // pairs of heads in flight, forward

struct Four {
  float v[4];
};
__device__ __forceinline__ Four unpack4(const uint2& r) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
  return {{a.x, a.y, b.x, b.y}};
}
__device__ __forceinline__ uint2 pack4(const Four& f) { return make_uint2(pack2(f.v[0], f.v[1]), pack2(f.v[2], f.v[3])); }
__device__ __forceinline__ uint2 ld8b(const bf16* p) { return *reinterpret_cast<const uint2*>(p); }
__device__ __forceinline__ void st8b(bf16* p, const uint2& v) { *reinterpret_cast<uint2*>(p) = v; }
// Sum over a head from a lane's two sums of four. The order is fixed, whatever rot_half and the lanes' share of a head: sums of
// four consecutive dimensions, to which the ones 64, 32, 16, 8 and 4 dimensions further are added in turn. (Another order, or
// another place of the fused multiply-add in the rotation, rounds one value in 10^5 differently; through the layers that became
// 1 % of a short pack's gradients, and single values of sparse ones by more than their root mean square.)
__device__ __forceinline__ float head_sum(float a, float b, int rot_half) {
  if (rot_half == 64) {  // (b lies 64 dimensions after a, the lane 8 further 32)
    a += b;
    a += __shfl_xor_sync(0xffffffffu, a, 8);
  } else {  // (the other way round)
    a += __shfl_xor_sync(0xffffffffu, a, 8);
    b += __shfl_xor_sync(0xffffffffu, b, 8);
    a += b;
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  return a;
}

// Where lane l of a half-warp finds its values in a head, and the angles it rotates them by. rot_half = 64: dimension d pairs with
// d + 64 and all of them rotate. rot_half = 32: only the first 64 dimensions do (d pairs with d + 32), lanes 8..15 hold the
// rest, which passes through.
struct RopeLane {
  int a, b;        // first of the four dimensions, and of the four they pair with
  bool rotated;
  float freq[2];   // inverse frequencies of this lane's two of its four angles (half-warp 0: the first two)
};
__device__ __forceinline__ RopeLane rope_lane(int l, int half, int rot_half, float theta, const float* tab) {
  RopeLane r;
  r.rotated = l * 4 < rot_half;
  r.a = r.rotated ? l * 4 : rot_half + l * 4;  // (rot_half = 32, l >= 8: 64, 68, .. 92)
  r.b = r.rotated ? r.a + rot_half : r.a + 32;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int d = (l * 4 + half * 2 + j) & (rot_half - 1);
    r.freq[j] = tab ? tab[d] : powf(theta, -static_cast<float>(d) / static_cast<float>(rot_half));
  }
  return r;
}
__device__ __forceinline__ void rope_angles(const RopeLane& r, float p, int half, Four& cs, Four& sn) {
  float c[2], s[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) sincosf(p * r.freq[j], &s[j], &c[j]);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float oc = __shfl_xor_sync(0xffffffffu, c[j], 16), os = __shfl_xor_sync(0xffffffffu, s[j], 16);
    cs.v[j] = half ? oc : c[j];
    sn.v[j] = half ? os : s[j];
    cs.v[2 + j] = half ? c[j] : oc;
    sn.v[2 + j] = half ? s[j] : os;
  }
  if (!r.rotated) cs = {{1.f, 1.f, 1.f, 1.f}}, sn = {{0.f, 0.f, 0.f, 0.f}};
}

__global__ void __launch_bounds__(256, 4)
qk_norm_rope_fwd_kernel(const bf16* __restrict__ qkv, const bf16* __restrict__ qw, const bf16* __restrict__ kw,
                        const int* __restrict__ pos, bf16* __restrict__ q_out, bf16* __restrict__ k_out,
                        float* __restrict__ q_rstd, float* __restrict__ k_rstd, bf16* __restrict__ k_cache,
                        bf16* __restrict__ v_cache, const int* __restrict__ slot_mapping, int T, int Hq, int Hk, float theta,
                        float eps, int use_norm, const float* __restrict__ inv_freq_tab, int rot_half, int chunks, int per) {
  pdl_enter();
  constexpr int D = ROPE_D;
  const int lane = threadIdx.x & 31, half = lane >> 4, l = lane & 15;
  const int heads = Hq + 2 * Hk;
  const RopeLane rl = rope_lane(l, half, rot_half, theta, inv_freq_tab);
  uint2 wqa = make_uint2(0u, 0u), wqb = wqa, wka = wqa, wkb = wqa;
  if (use_norm) wqa = ld8b(qw + rl.a), wqb = ld8b(qw + rl.b), wka = ld8b(kw + rl.a), wkb = ld8b(kw + rl.b);
  const long long items = static_cast<long long>(T) * chunks;
  const long long stride = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  for (long long it = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); it < items; it += stride) {
    const int t = static_cast<int>(it / chunks);
    const int h0 = static_cast<int>(it - static_cast<long long>(t) * chunks) * per, h1 = min(heads, h0 + per);
    const int slot = (k_cache || v_cache) ? slot_mapping[t] : -1;
    Four cs, sn;
    rope_angles(rl, static_cast<float>(pos[t]), half, cs, sn);
    const bf16* row = qkv + static_cast<long long>(t) * heads * D;
    // both pairs of heads are asked for before the first is used (the branches below keep the compiler from doing so)
    for (int hb = h0; hb < h1; hb += 2 * ROPE_AHEAD) {
      uint2 raw_a[ROPE_AHEAD], raw_b[ROPE_AHEAD];
#pragma unroll
      for (int n = 0; n < ROPE_AHEAD; ++n) {
        const int h = hb + 2 * n + half;
        raw_a[n] = raw_b[n] = make_uint2(0u, 0u);
        if (h < h1 && (h < Hq + Hk || v_cache)) raw_a[n] = ld8b(row + h * D + rl.a), raw_b[n] = ld8b(row + h * D + rl.b);
      }
#pragma unroll
      for (int n = 0; n < ROPE_AHEAD; ++n) {
        const int hp = hb + 2 * n;
        if (hp >= h1) break;  // warp-uniform
        const int h = hp + half;
        const bool act = h < h1 && (h < Hq + Hk || v_cache), is_q = h < Hq;
        const uint2 ra = raw_a[n], rb = raw_b[n];
        Four x = unpack4(ra), y = unpack4(rb);
        if (use_norm) {
          float sx = 0.f, sy = 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            sx += x.v[i] * x.v[i];
            sy += y.v[i] * y.v[i];
          }
          const float ss = head_sum(sx, sy, rot_half);
          const float r = rsqrtf(ss / D + eps);
          const Four wa = unpack4(is_q ? wqa : wka), wb = unpack4(is_q ? wqb : wkb);
          // match the unfused path: the normalised value is rounded to bf16 before the rotation
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            x.v[i] = __bfloat162float(__float2bfloat16(x.v[i] * r * wa.v[i]));
            y.v[i] = __bfloat162float(__float2bfloat16(y.v[i] * r * wb.v[i]));
          }
          if (act && l == 0) {
            if (is_q && q_rstd) q_rstd[static_cast<long long>(t) * Hq + h] = r;
            if (!is_q && h < Hq + Hk && k_rstd) k_rstd[static_cast<long long>(t) * Hk + (h - Hq)] = r;
          }
        }
        if (!act) continue;
        if (h >= Hq + Hk) {  // V head: only the cache scatter
          if (slot >= 0) {
            bf16* dst = v_cache + (static_cast<long long>(slot) * Hk + (h - Hq - Hk)) * D;
            st8b(dst + rl.a, ra);
            st8b(dst + rl.b, rb);
          }
          continue;
        }
        // rotate-half RoPE: out[d] = x[d]*cos - x[d+64]*sin (d<64); out[d+64] = x[d+64]*cos + x[d]*sin, each with the first
        // dimension's product fused and the other one rounded, whatever the compiler would choose
        Four u, w;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          u.v[i] = __fmaf_rn(x.v[i], cs.v[i], -__fmul_rn(y.v[i], sn.v[i]));
          w.v[i] = __fmaf_rn(x.v[i], sn.v[i], __fmul_rn(y.v[i], cs.v[i]));
        }
        if (!rl.rotated) u = x, w = y;
        const uint2 oa = pack4(u), ob = pack4(w);
        if (is_q) {
          bf16* dst = q_out + (static_cast<long long>(t) * Hq + h) * D;
          st8b(dst + rl.a, oa);
          st8b(dst + rl.b, ob);
        } else {
          const int hk = h - Hq;
          if (k_out) {
            bf16* dst = k_out + (static_cast<long long>(t) * Hk + hk) * D;
            st8b(dst + rl.a, oa);
            st8b(dst + rl.b, ob);
          }
          if (k_cache && slot >= 0) {
            bf16* dst = k_cache + (static_cast<long long>(slot) * Hk + hk) * D;
            st8b(dst + rl.a, oa);
            st8b(dst + rl.b, ob);
          }
        }
      }
    }
    __syncwarp();
  }
}

// Backward of the kernel above. dq [T,Hq,D], dk [T,Hk,D], dv [T,Hk,D] -> dqkv [T, heads*D]; weight gradients of the head
// norms are summed in registers over all heads and tokens of a lane, then over the block in shared memory, and added
// to the fp32 [D] buffers with one atomic per value and block.
__global__ void __launch_bounds__(256)
qk_norm_rope_bwd_kernel(const bf16* __restrict__ dq, const bf16* __restrict__ dk, const bf16* __restrict__ dv,
                        const bf16* __restrict__ qkv, const bf16* __restrict__ qw, const bf16* __restrict__ kw,
                        const int* __restrict__ pos, const float* __restrict__ q_rstd, const float* __restrict__ k_rstd,
                        bf16* __restrict__ dqkv, float* __restrict__ dqw, float* __restrict__ dkw, int T, int Hq, int Hk,
                        float theta, int use_norm, const float* __restrict__ inv_freq_tab, int rot_half, int chunks, int per) {
  constexpr int D = ROPE_D;
  __shared__ float wacc[2][D];
  for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) (&wacc[0][0])[i] = 0.f;
  __syncthreads();
  const int lane = threadIdx.x & 31, half = lane >> 4, l = lane & 15;
  const int heads = Hq + 2 * Hk;
  const RopeLane rl = rope_lane(l, half, rot_half, theta, inv_freq_tab);
  Four aqa = {{0.f, 0.f, 0.f, 0.f}}, aqb = aqa, aka = aqa, akb = aqa;
  uint2 wqa = make_uint2(0u, 0u), wqb = wqa, wka = wqa, wkb = wqa;
  if (use_norm) wqa = ld8b(qw + rl.a), wqb = ld8b(qw + rl.b), wka = ld8b(kw + rl.a), wkb = ld8b(kw + rl.b);
  const long long items = static_cast<long long>(T) * chunks;
  const long long stride = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  for (long long it = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); it < items; it += stride) {
    const int t = static_cast<int>(it / chunks);
    const int h0 = static_cast<int>(it - static_cast<long long>(t) * chunks) * per, h1 = min(heads, h0 + per);
    Four cs, sn;
    rope_angles(rl, static_cast<float>(pos[t]), half, cs, sn);
    const long long row = static_cast<long long>(t) * heads * D;
#pragma unroll 2
    for (int hp = h0; hp < h1; hp += 2) {
      const int h = hp + half;
      const bool act = h < h1, is_q = h < Hq, is_v = h >= Hq + Hk;
      uint2 ga = make_uint2(0u, 0u), gb = ga, xa = ga, xb = ga;
      float r = 0.f;
      if (act) {
        const bf16* src = is_q ? dq + (static_cast<long long>(t) * Hq + h) * D
                               : (is_v ? dv + (static_cast<long long>(t) * Hk + (h - Hq - Hk)) * D
                                       : dk + (static_cast<long long>(t) * Hk + (h - Hq)) * D);
        ga = ld8b(src + rl.a);
        gb = ld8b(src + rl.b);
        if (use_norm && !is_v) {
          xa = ld8b(qkv + row + h * D + rl.a);
          xb = ld8b(qkv + row + h * D + rl.b);
          r = is_q ? q_rstd[static_cast<long long>(t) * Hq + h] : k_rstd[static_cast<long long>(t) * Hk + (h - Hq)];
        }
      }
      const Four g = unpack4(ga), e = unpack4(gb);
      // inverse rotation: dx[d] = g[d]*cos + g[d+64]*sin ; dx[d+64] = g[d+64]*cos - g[d]*sin (the second one's product fused)
      Four u, w;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        u.v[i] = __fmaf_rn(e.v[i], sn.v[i], __fmul_rn(g.v[i], cs.v[i]));
        w.v[i] = __fmaf_rn(e.v[i], cs.v[i], -__fmul_rn(g.v[i], sn.v[i]));
      }
      if (!rl.rotated) u = g, w = e;
      if (use_norm) {
        const Four x = unpack4(xa), y = unpack4(xb);
        const Four wa = unpack4(is_q ? wqa : wka), wb = unpack4(is_q ? wqb : wkb);
        float dx = 0.f, dy = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          dx = __fmaf_rn(__fmul_rn(__fmul_rn(u.v[i], wa.v[i]), x.v[i]), r, dx);
          dy = __fmaf_rn(__fmul_rn(__fmul_rn(w.v[i], wb.v[i]), y.v[i]), r, dy);
        }
        const float dot = head_sum(dx, dy, rot_half) / D;
        const bool to_k = !is_q && !is_v;  // (a V head's lanes hold nothing that a sum may see)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float xh = x.v[i] * r, yh = y.v[i] * r, da = u.v[i] * xh, db = w.v[i] * yh;
          aqa.v[i] += is_q ? da : 0.f;
          aqb.v[i] += is_q ? db : 0.f;
          aka.v[i] += to_k ? da : 0.f;
          akb.v[i] += to_k ? db : 0.f;
          u.v[i] = __fmul_rn(r, __fmaf_rn(-xh, dot, __fmul_rn(u.v[i], wa.v[i])));
          w.v[i] = __fmul_rn(r, __fmaf_rn(-yh, dot, __fmul_rn(w.v[i], wb.v[i])));
        }
      }
      if (act) {
        st8b(dqkv + row + h * D + rl.a, is_v ? ga : pack4(u));
        st8b(dqkv + row + h * D + rl.b, is_v ? gb : pack4(w));
      }
    }
    __syncwarp();
  }
  if (use_norm) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      atomicAdd(&wacc[0][rl.a + i], aqa.v[i]);
      atomicAdd(&wacc[0][rl.b + i], aqb.v[i]);
      atomicAdd(&wacc[1][rl.a + i], aka.v[i]);
      atomicAdd(&wacc[1][rl.b + i], akb.v[i]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < D; i += blockDim.x) {
      if (dqw) atomicAdd(dqw + i, wacc[0][i]);
      if (dkw) atomicAdd(dkw + i, wacc[1][i]);
    }
  }
}

// ------------------------------------------------------------------ SwiGLU
// in: [T, 2I] = [gate | up]; out: [T, I] = silu(gate) * up.
// Eight values per thread and iteration. `Index` is 32 bits wide wherever the item count allows (up to 64 GB of input): a 64-bit division per item
// had bound these kernels (131072 rows of 2 x 768: forward 150 -> 132 us, backward of 139264 rows 211 -> 187 us), as had a grid of a few
// blocks per SM, whose threads wait for one item's loads before they ask for the next.
template <typename Index>
__global__ void swiglu_fwd_kernel(const bf16* __restrict__ in, bf16* __restrict__ out, Index n8, Index per_row) {
  pdl_enter();
  for (Index idx = static_cast<Index>(blockIdx.x) * blockDim.x + threadIdx.x; idx < n8;
       idx += static_cast<Index>(gridDim.x) * blockDim.x) {
    const Index row = idx / per_row;
    const bf16* src = in + (static_cast<long long>(row) * per_row + idx) * 8;  // row * 2I + column
    float g[8], u[8], o[8];
    load8(src, g);
    load8(src + static_cast<long long>(per_row) * 8, u);
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] = g[i] / (1.f + __expf(-g[i])) * u[i];
    store8(out + static_cast<long long>(idx) * 8, o);
  }
}

template <typename Index>
__global__ void swiglu_bwd_kernel(const bf16* __restrict__ dout, const bf16* __restrict__ in, bf16* __restrict__ din, Index n8,
                                  Index per_row) {
  for (Index idx = static_cast<Index>(blockIdx.x) * blockDim.x + threadIdx.x; idx < n8;
       idx += static_cast<Index>(gridDim.x) * blockDim.x) {
    const Index row = idx / per_row;
    const long long at = (static_cast<long long>(row) * per_row + idx) * 8, half = static_cast<long long>(per_row) * 8;
    float g[8], u[8], d[8], dg[8], du[8];
    load8(in + at, g);
    load8(in + at + half, u);
    load8(dout + static_cast<long long>(idx) * 8, d);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float s = 1.f / (1.f + __expf(-g[i]));
      const float silu = g[i] * s;
      du[i] = d[i] * silu;
      dg[i] = d[i] * u[i] * (s + silu * (1.f - s));
    }
    store8(din + at, dg);
    store8(din + at + half, du);
  }
}

// ------------------------------------------------------------------ fused Adam(W)
// One flat buffer per call. The parameter is bf16; its fp32 master copy is kept in one of two forms:
//   * `master` (fp32 array), or
//   * `lo` (16-bit array): the master is split over the bf16 weight itself and a signed 16-bit remainder,
//         master_bits = (weight_bits << 16) + lo,     weight_bits = (master_bits + 0x8000) >> 16,
//     so the weight the GEMMs read is the master rounded to nearest (ties away from zero) and the pair
//     reconstructs every fp32 bit. An update far below half a bf16 ulp therefore accumulates in `lo`
//     instead of being rounded away; memory per parameter is 4 bytes instead of 6.
// With neither, the update is applied to the bf16 value itself (only sensible for large learning rates).
// The gradient is bf16 or fp32; moments are fp32 or bf16. `skip_flag` / `grad_scale` are read from device
// memory so that the clip coefficient computed by a previous kernel never travels through the host.
// Eight elements per thread, 128-bit loads and stores; the host launcher handles a ragged tail.
template <typename T>
__device__ __forceinline__ void adam_load8(const T* p, float (&o)[8]);
template <>
__device__ __forceinline__ void adam_load8<bf16>(const bf16* p, float (&o)[8]) {
  load8(p, o);
}
template <>
__device__ __forceinline__ void adam_load8<float>(const float* p, float (&o)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
  o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}
template <typename T>
__device__ __forceinline__ void adam_store8(T* p, const float (&o)[8]);
template <>
__device__ __forceinline__ void adam_store8<bf16>(bf16* p, const float (&o)[8]) {
  store8(p, o);
}
template <>
__device__ __forceinline__ void adam_store8<float>(float* p, const float (&o)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(o[4], o[5], o[6], o[7]);
}

// The bias corrections 1 - b1^t and 1 - b2^t come folded into one factor under the root and one on eps:
//   (m / c1) / (sqrt(v / c2) + eps) = m / (sqrt(v * c1^2 / c2) + c1 * eps),
// one division and one root per element instead of three and one, and one rounding fewer. With a thread per eight elements
// (instead of a grid of eight blocks per SM that walks over them) the update is bound by memory: 641 M weights with fp32
// gradients and bf16 moments, 12.8 GB: 2.76 -> 2.50 ms; 604 M with bf16 gradients: 2.49 -> 1.97 ms.
struct AdamScalars {
  float lr, b1, b2, wd, v_scale, eps;
};

__device__ __forceinline__ float adam_update(float w, float grad, float& mi, float& vi, const AdamScalars& a) {
  mi = a.b1 * mi + (1.f - a.b1) * grad;
  vi = a.b2 * vi + (1.f - a.b2) * grad * grad;
  const float upd = mi / (sqrtf(vi * a.v_scale) + a.eps);
  return w - a.lr * (upd + a.wd * w);
}

__device__ __forceinline__ float split_join(unsigned short hi, short lo) {
  return __uint_as_float((static_cast<unsigned>(hi) << 16) + static_cast<unsigned>(static_cast<int>(lo)));
}
__device__ __forceinline__ void split_cut(float w, unsigned short& hi, short& lo) {
  const unsigned bits = __float_as_uint(w);
  const unsigned h = (bits + 0x8000u) >> 16;
  hi = static_cast<unsigned short>(h);
  lo = static_cast<short>(static_cast<int>(bits - (h << 16)));
}

template <typename GT, typename MT>
__global__ void adam_kernel(bf16* __restrict__ p, float* __restrict__ master, short* __restrict__ lo,
                            const GT* __restrict__ g, MT* __restrict__ m, MT* __restrict__ v, long long n,
                            AdamScalars a, const float* __restrict__ grad_scale, const float* __restrict__ skip_flag) {
  if (skip_flag && *skip_flag != 0.f) return;
  const float gs = grad_scale ? *grad_scale : 1.f;
  const long long n8 = n / 8;
  for (long long i8 = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i8 < n8;
       i8 += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long i = i8 * 8;
    float gr[8], mi[8], vi[8], w[8];
    adam_load8<GT>(g + i, gr);
    adam_load8<MT>(m + i, mi);
    adam_load8<MT>(v + i, vi);
    uint4 pw = *reinterpret_cast<const uint4*>(p + i);
    unsigned short* ph = reinterpret_cast<unsigned short*>(&pw);
    uint4 lw;
    short* pl = reinterpret_cast<short*>(&lw);
    if (master) {
      adam_load8<float>(master + i, w);
    } else if (lo) {
      lw = *reinterpret_cast<const uint4*>(lo + i);
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = split_join(ph[j], pl[j]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = __uint_as_float(static_cast<unsigned>(ph[j]) << 16);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = adam_update(w[j], gr[j] * gs, mi[j], vi[j], a);
    adam_store8<MT>(m + i, mi);
    adam_store8<MT>(v + i, vi);
    if (master) {
      adam_store8<float>(master + i, w);
      store8(p + i, w);
    } else if (lo) {
#pragma unroll
      for (int j = 0; j < 8; ++j) split_cut(w[j], ph[j], pl[j]);
      *reinterpret_cast<uint4*>(p + i) = pw;
      *reinterpret_cast<uint4*>(lo + i) = lw;
    } else {
      store8(p + i, w);
    }
  }
  // ragged tail (fewer than eight elements): first threads of block 0
  if (blockIdx.x == 0 && threadIdx.x < n - n8 * 8) {
    const long long i = n8 * 8 + threadIdx.x;
    float mi = static_cast<float>(m[i]), vi = static_cast<float>(v[i]);
    unsigned short hi = reinterpret_cast<unsigned short*>(p)[i];
    float w = master ? master[i] : (lo ? split_join(hi, lo[i]) : __uint_as_float(static_cast<unsigned>(hi) << 16));
    w = adam_update(w, static_cast<float>(g[i]) * gs, mi, vi, a);
    m[i] = static_cast<MT>(mi);
    v[i] = static_cast<MT>(vi);
    if (master) {
      master[i] = w;
      p[i] = __float2bfloat16(w);
    } else if (lo) {
      short l;
      split_cut(w, hi, l);
      reinterpret_cast<unsigned short*>(p)[i] = hi;
      lo[i] = l;
    } else {
      p[i] = __float2bfloat16(w);
    }
  }
}

// master[i] = join(p[i], lo[i]) (fp32 view of a split master, for checkpoints and checks)
__global__ void split_master_join_kernel(const bf16* __restrict__ p, const short* __restrict__ lo, float* __restrict__ out,
                                         long long n) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    out[i] = split_join(reinterpret_cast<const unsigned short*>(p)[i], lo[i]);
}
// (p[i], lo[i]) = cut(master[i])
__global__ void split_master_cut_kernel(const float* __restrict__ master, bf16* __restrict__ p, short* __restrict__ lo,
                                        long long n) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    unsigned short hi;
    short l;
    split_cut(master[i], hi, l);
    reinterpret_cast<unsigned short*>(p)[i] = hi;
    lo[i] = l;
  }
}

// ------------------------------------------------------------------ counter-based normal initialisation
// out[i] = std * N(key, first + i): Philox4x32-10 keyed by `key`, counter = element index / 4, Box-Muller on the four
// 32-bit outputs. The value of an element depends only on (key, its index in the logical tensor), so any sharding
// of the tensor (expert parallel, tensor parallel, pipeline stages) draws the same model, and a 30 B parameter
// model is filled at memory speed instead of through thousands of generator calls.
__device__ __forceinline__ void philox4x32_10(unsigned long long key, unsigned long long ctr, unsigned (&r)[4]) {
  unsigned c0 = static_cast<unsigned>(ctr), c1 = static_cast<unsigned>(ctr >> 32), c2 = 0x9E3779B9u, c3 = 0xBB67AE85u;
  unsigned k0 = static_cast<unsigned>(key), k1 = static_cast<unsigned>(key >> 32);
#pragma unroll
  for (int i = 0; i < 10; ++i) {
    const unsigned hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    const unsigned hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    const unsigned n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  r[0] = c0; r[1] = c1; r[2] = c2; r[3] = c3;
}
__device__ __forceinline__ void normal4(unsigned long long key, unsigned long long ctr, float std, float (&o)[4]) {
  unsigned r[4];
  philox4x32_10(key, ctr, r);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float u1 = (static_cast<float>(r[2 * j] >> 8) + 1.0f) * (1.0f / 16777216.0f);  // (0, 1]
    const float u2 = static_cast<float>(r[2 * j + 1] >> 8) * (1.0f / 16777216.0f);       // [0, 1)
    const float rad = std * sqrtf(-2.0f * __logf(u1));
    float sn, cs;
    __sincosf(6.283185307179586f * u2, &sn, &cs);
    o[2 * j] = rad * cs;
    o[2 * j + 1] = rad * sn;
  }
}
template <typename T>
__global__ void init_normal_kernel(T* __restrict__ out, long long n, unsigned long long key, long long first, float std) {
  // one thread per group of four consecutive logical elements (aligned to four in the logical index space)
  const long long g0 = first / 4, g1 = (first + n + 3) / 4;
  for (long long g = g0 + static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; g < g1;
       g += static_cast<long long>(gridDim.x) * blockDim.x) {
    float v[4];
    normal4(key, static_cast<unsigned long long>(g), std, v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long i = g * 4 + j - first;
      if (i >= 0 && i < n) out[i] = static_cast<T>(v[j]);
    }
  }
}

// Sum of squares of a flat buffer, added to a single fp32 accumulator (for the global grad norm), in two
// stages with a fixed summation order: every block writes its partial sum, one block adds the partials in index
// order. The same gradients therefore always give the same norm bits (an atomicAdd per block would not), which
// keeps the clip coefficient, and with it a whole training step, reproducible.
template <typename GT>
__global__ void sumsq_partial_kernel(const GT* __restrict__ g, long long n, float* __restrict__ partial) {
  __shared__ float red[32];
  float s = 0.f;
  const long long n8 = n / 8;
  for (long long i8 = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i8 < n8;
       i8 += static_cast<long long>(gridDim.x) * blockDim.x) {
    float x[8];
    adam_load8<GT>(g + i8 * 8, x);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += x[j] * x[j];
  }
  if (blockIdx.x == 0 && threadIdx.x < n - n8 * 8) {
    const float x = static_cast<float>(g[n8 * 8 + threadIdx.x]);
    s += x * x;
  }
  s = block_sum<256>(s, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}
__global__ void sumsq_final_kernel(const float* __restrict__ partial, int n, float* __restrict__ out) {
  __shared__ float red[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += 256) s += partial[i];
  s = block_sum<256>(s, red);
  if (threadIdx.x == 0) *out += s;
}

int grid_for(long long work_items, int threads, int cap = 148 * 8) {
  long long b = (work_items + threads - 1) / threads;
  if (b < 1) b = 1;
  return static_cast<int>(b < cap ? b : cap);
}

}  // namespace

void rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* res_out, float* rstd, int T, int H,
                 float eps, cudaStream_t s) {
  if (T <= 0) return;
  const int pieces = (H + 256 * 8 - 1) / (256 * 8);  // of a thread
  const auto kern = pieces == 1 ? rmsnorm_fwd_kernel<256, 1> : pieces == 2 ? rmsnorm_fwd_kernel<256, 2> : pieces <= 4 ? rmsnorm_fwd_kernel<256, 4>
                                                                                                                    : rmsnorm_fwd_kernel<256, 0>;
  pdl_launch(kern, T, 256, 0, s, static_cast<const bf16*>(x), static_cast<const bf16*>(res), static_cast<const bf16*>(w), static_cast<bf16*>(y),
             static_cast<bf16*>(res_out), rstd, H, eps);
}

int rmsnorm_bwd_num_partials(int T) { return T < 296 ? (T < 1 ? 1 : T) : 296; }

void rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx,
                 float* dw_partial, float* dw, bool accumulate_dw, int T, int H, cudaStream_t s) {
  if (T <= 0) return;
  const int blocks = rmsnorm_bwd_num_partials(T);
  const int pieces = (H + 256 * 8 - 1) / (256 * 8);  // of a thread
  const auto kern = pieces == 1 ? rmsnorm_bwd_kernel<256, 1> : pieces == 2 ? rmsnorm_bwd_kernel<256, 2> : rmsnorm_bwd_kernel<256, 0>;
  kern<<<blocks, 256, pieces <= 2 ? 0 : H * sizeof(float), s>>>(
      static_cast<const bf16*>(dy), static_cast<const bf16*>(x), static_cast<const bf16*>(w), rstd,
      static_cast<const bf16*>(dres), static_cast<bf16*>(dx), dw_partial, T, H);
  colsum_kernel<<<(H + 127) / 128, 128, 0, s>>>(dw_partial, dw, blocks, H, accumulate_dw ? 1 : 0);
}

namespace {
// How a token's heads are dealt to warps: every head in one warp when the tokens alone fill the device twice (9472 warps are
// resident at eight blocks of eight warps), else in as many pieces as it takes, down to one pair of heads each.
struct RopeSplit {
  int chunks, per, blocks;
};
RopeSplit rope_split(int T, int heads, int block_cap) {
  const long long want = (2 * 9472 + T - 1) / T;
  const int pairs = (heads + 1) / 2;
  const int c = static_cast<int>(want < 1 ? 1 : (want > pairs ? pairs : want));
  const int per = (pairs + c - 1) / c * 2;
  const int chunks = (heads + per - 1) / per;
  const long long blocks = (static_cast<long long>(T) * chunks + 7) / 8;
  return {chunks, per, static_cast<int>(blocks < block_cap ? blocks : block_cap)};
}
}  // namespace

void qk_norm_rope_fwd(const void* qkv, const void* qw, const void* kw, const int* pos, void* q_out, void* k_out,
                      float* q_rstd, float* k_rstd, void* k_cache, void* v_cache, const int* slot_mapping, int T,
                      int Hq, int Hk, float theta, float eps, bool use_norm, cudaStream_t s, const float* inv_freq,
                      int rotary_dim) {
  if (T <= 0) return;
  const RopeSplit sp = rope_split(T, Hq + 2 * Hk, 148 * 8);
  pdl_launch(qk_norm_rope_fwd_kernel, sp.blocks, 256, 0, s, 
      static_cast<const bf16*>(qkv), static_cast<const bf16*>(qw), static_cast<const bf16*>(kw), pos,
      static_cast<bf16*>(q_out), static_cast<bf16*>(k_out), q_rstd, k_rstd, static_cast<bf16*>(k_cache),
      static_cast<bf16*>(v_cache), slot_mapping, T, Hq, Hk, theta, eps, use_norm ? 1 : 0, inv_freq, rotary_dim / 2, sp.chunks, sp.per);
}

void qk_norm_rope_bwd(const void* dq, const void* dk, const void* dv, const void* qkv, const void* qw, const void* kw,
                      const int* pos, const float* q_rstd, const float* k_rstd, void* dqkv, float* dqw, float* dkw,
                      int T, int Hq, int Hk, float theta, bool use_norm, cudaStream_t s, const float* inv_freq,
                      int rotary_dim) {
  if (T <= 0) return;
  const RopeSplit sp = rope_split(T, Hq + 2 * Hk, 148 * 4);
  qk_norm_rope_bwd_kernel<<<sp.blocks, 256, 0, s>>>(
      static_cast<const bf16*>(dq), static_cast<const bf16*>(dk), static_cast<const bf16*>(dv),
      static_cast<const bf16*>(qkv), static_cast<const bf16*>(qw), static_cast<const bf16*>(kw), pos, q_rstd, k_rstd,
      static_cast<bf16*>(dqkv), dqw, dkw, T, Hq, Hk, theta, use_norm ? 1 : 0, inv_freq, rotary_dim / 2, sp.chunks, sp.per);
}

void swiglu_fwd(const void* in, void* out, long long T, int I, cudaStream_t s) {
  if (T <= 0) return;
  const long long n8 = T * (I / 8);
  const int grid = grid_for(n8, 256, 1 << 24);
  const bf16* src = static_cast<const bf16*>(in);
  bf16* dst = static_cast<bf16*>(out);
  if (n8 < (1ll << 31)) pdl_launch(swiglu_fwd_kernel<unsigned>, grid, 256, 0, s, src, dst, static_cast<unsigned>(n8), static_cast<unsigned>(I / 8));
  else pdl_launch(swiglu_fwd_kernel<long long>, grid, 256, 0, s, src, dst, n8, I / 8);
}

void swiglu_bwd(const void* dout, const void* in, void* din, long long T, int I, cudaStream_t s) {
  if (T <= 0) return;
  const long long n8 = T * (I / 8);
  const int grid = grid_for(n8, 256, 1 << 24);
  const bf16 *d = static_cast<const bf16*>(dout), *src = static_cast<const bf16*>(in);
  bf16* dst = static_cast<bf16*>(din);
  if (n8 < (1ll << 31)) swiglu_bwd_kernel<unsigned><<<grid, 256, 0, s>>>(d, src, dst, static_cast<unsigned>(n8), static_cast<unsigned>(I / 8));
  else swiglu_bwd_kernel<long long><<<grid, 256, 0, s>>>(d, src, dst, n8, I / 8);
}

void adam_step(void* p, float* master, void* lo, const void* g, bool g_fp32, void* m, void* v, bool mv_bf16, long long n,
               float lr, float b1, float b2, float eps, float wd, float bc1, float bc2, const float* grad_scale,
               const float* skip_flag, cudaStream_t s) {
  if (n <= 0) return;
  const int grid = grid_for((n + 7) / 8, 256, 1 << 24);
  bf16* pp = static_cast<bf16*>(p);
  const AdamScalars a{lr, b1, b2, wd, static_cast<float>(static_cast<double>(bc1) * bc1 / bc2),
                      static_cast<float>(static_cast<double>(bc1) * eps)};
#define MB_ADAM(GT, MT)                                                                                            \
  adam_kernel<GT, MT><<<grid, 256, 0, s>>>(pp, master, static_cast<short*>(lo), static_cast<const GT*>(g),          \
                                           static_cast<MT*>(m), static_cast<MT*>(v), n, a, grad_scale, skip_flag)
  if (g_fp32 && !mv_bf16) MB_ADAM(float, float);
  else if (g_fp32 && mv_bf16) MB_ADAM(float, bf16);
  else if (!g_fp32 && !mv_bf16) MB_ADAM(bf16, float);
  else MB_ADAM(bf16, bf16);
#undef MB_ADAM
}

void split_master_join(const void* p, const void* lo, float* out, long long n, cudaStream_t s) {
  if (n <= 0) return;
  split_master_join_kernel<<<grid_for(n, 256), 256, 0, s>>>(static_cast<const bf16*>(p), static_cast<const short*>(lo), out, n);
}
void split_master_cut(const float* master, void* p, void* lo, long long n, cudaStream_t s) {
  if (n <= 0) return;
  split_master_cut_kernel<<<grid_for(n, 256), 256, 0, s>>>(master, static_cast<bf16*>(p), static_cast<short*>(lo), n);
}

void init_normal(void* out, bool fp32, long long n, unsigned long long key, long long first, float std, cudaStream_t s) {
  if (n <= 0) return;
  const int grid = grid_for((n + 3) / 4 + 1, 256, 148 * 16);
  if (fp32) init_normal_kernel<float><<<grid, 256, 0, s>>>(static_cast<float*>(out), n, key, first, std);
  else init_normal_kernel<bf16><<<grid, 256, 0, s>>>(static_cast<bf16*>(out), n, key, first, std);
}

int sumsq_num_partials(long long n) { return grid_for((n + 7) / 8, 256, 148 * 4); }

// `partial`: fp32 scratch of sumsq_num_partials(n) elements; g must be 16-byte aligned.
void sumsq(const void* g, bool g_fp32, long long n, float* partial, float* out, cudaStream_t s) {
  if (n <= 0) return;
  const int grid = sumsq_num_partials(n);
  if (g_fp32) sumsq_partial_kernel<float><<<grid, 256, 0, s>>>(static_cast<const float*>(g), n, partial);
  else sumsq_partial_kernel<bf16><<<grid, 256, 0, s>>>(static_cast<const bf16*>(g), n, partial);
  sumsq_final_kernel<<<1, 256, 0, s>>>(partial, grid, out);
}

}  // namespace mb
