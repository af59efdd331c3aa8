// Paged-KV decode attention (one query token per sequence, GQA), split over the KV length.
//
// Cache layout: k_cache / v_cache are [num_slots, Hk, 128] bf16 where slot = page * page_size + offset
// and block_table[b, i] is the i-th page of sequence b. Grid = (B, Hk, splits); every CTA serves all
// G = Hq/Hk query heads of one KV head over its slice of the context so that each K/V row is read from
// HBM exactly once. Up to 16 splits of one (sequence, KV head) form a cluster and merge their partial (max, sum, out)
// triples through distributed shared memory; more splits go through scratch and a second kernel.
//
// Reference counterpart: flashinfer's trtllm_mha decode backend selected by the B200 recipe
// (scripts/run_qwen3_30b_a3b.py:311-324).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "launchers.h"
#include "pdl.cuh"

namespace mb {
namespace {

using bf16 = __nv_bfloat16;
constexpr int D = 128;
constexpr int WARPS = 4;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void decode_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                    bf16* __restrict__ out, int num_splits) {
  const long long bh = blockIdx.x;  // b * Hq + head
  const int d = threadIdx.x;
  pdl_enter();
  float gm = -FLT_MAX;
  for (int s = 0; s < num_splits; ++s) gm = fmaxf(gm, part_ml[(bh * num_splits + s) * 2]);
  float gl = 0.f, go = 0.f;
  for (int s = 0; s < num_splits; ++s) {
    const float mm = part_ml[(bh * num_splits + s) * 2];
    const float c = mm == -FLT_MAX ? 0.f : __expf(mm - gm);
    gl += part_ml[(bh * num_splits + s) * 2 + 1] * c;
    go += part_o[(bh * num_splits + s) * D + d] * c;
  }
  out[bh * D + d] = __float2bfloat16(gl > 0.f ? go / gl : 0.f);
}


// ---------------------------------------------------------------------------------------------------
// K/V pages are staged through shared memory with cp.async (three stages of 64 tokens, so that two are in flight while
// one is used: what bounds the kernel is how much of the cache each SM has asked for) and the G query heads of one KV head form the (zero padded) 16-row A operand of
// mma.sync m16n8k16, so the work per K/V byte is a handful of instructions and the kernel runs at the
// speed of the cache stream. Each of the 4 warps owns 16 tokens of a stage and keeps its own running
// (max, sum, out); warps are merged through shared memory at the end.
constexpr int TOK = 64;          // tokens per stage
constexpr int LDS = D + 8;       // padded row (272 B) -> conflict-free ldmatrix
constexpr int STAGE_ELEMS = TOK * LDS;
constexpr int DSTAGES = 3;       // 104 KB: two CTAs per SM
constexpr int MAX_CLUSTER_SPLITS = 16;
// Measured (us a launch, pages of 64, caches larger than L2; before: two stages behind a CTA barrier and one page lookup per
// row, merged by a second kernel; the keys' and values' bytes alone): 64 sequences of 1500 tokens, 4 KV heads 63 -> 37 (27);
// 23 of 2300, 8 heads 58 -> 43 (30); 4 of 7900, 4 heads 28 -> 19.5 (9); 1 of 3000, 4 heads 13.8 -> 9.1 (0.8).

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&t);
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t local_addr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// CLUSTER: the splits of one (b, h) are the CTAs of one cluster (rank = split) and merge here; `part_*` is not used.
template <int G, bool CLUSTER>
__global__ void __launch_bounds__(WARPS * 32)
decode_mma_kernel(const bf16* __restrict__ q, const bf16* __restrict__ k_cache, const bf16* __restrict__ v_cache,
                  const int* __restrict__ block_table, const int* __restrict__ seq_lens, float* __restrict__ part_o,
                  float* __restrict__ part_ml, bf16* __restrict__ out, int Hq, int Hk, int page_size, int max_pages,
                  int num_splits, float scale, long long num_slots, int* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char dsm[];
  bf16* Ks = reinterpret_cast<bf16*>(dsm);            // [DSTAGES][TOK][LDS]
  bf16* Vs = Ks + DSTAGES * STAGE_ELEMS;              // [DSTAGES][TOK][LDS]
  const int b = blockIdx.x, h = blockIdx.y, split = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_enter();
  // The length and the page ids come from device memory the caller filled: a length beyond the block-table row is
  // clamped, and a page outside the cache is read as zeros (status 9) instead of being dereferenced.
  int len = seq_lens[b];
  const long long row_cap = static_cast<long long>(max_pages) * page_size;
  if (len < 0 || len > row_cap) {
    if (threadIdx.x == 0 && status) atomicCAS(status, 0, 8);
    len = len < 0 ? 0 : static_cast<int>(row_cap);
  }
  int per = (len + num_splits - 1) / num_splits;
  per = (per + TOK - 1) / TOK * TOK;
  const int t_lo = split * per;
  const int t_hi = min(len, t_lo + per);
  const int n_chunks = t_hi > t_lo ? (t_hi - t_lo + TOK - 1) / TOK : 0;
  const int* table = block_table + static_cast<long long>(b) * max_pages;

  // Q fragments: rows >= G are zero padding
  uint32_t qa[8][4];
  {
    const int r0 = lane >> 2, c = (lane & 3) * 2;
    const bf16* q0 = q + (static_cast<long long>(b) * Hq + h * G + r0) * D;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      qa[ks][0] = r0 < G ? *reinterpret_cast<const uint32_t*>(q0 + ks * 16 + c) : 0u;
      qa[ks][2] = r0 < G ? *reinterpret_cast<const uint32_t*>(q0 + ks * 16 + c + 8) : 0u;
      qa[ks][1] = 0u;  // rows 8..15 exist only as padding (G <= 8)
      qa[ks][3] = 0u;
    }
  }
  float m_run = -FLT_MAX, l_run = 0.f;  // row lane/4
  float o[16][4];
#pragma unroll
  for (int j = 0; j < 16; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;

  // Every warp fetches the 16 tokens of a chunk that it multiplies itself, so warps wait for their own copies only and a
  // stall of one is covered by the others. A chunk starts on a multiple of 64 tokens, so with pages of whole chunks it lies
  // in one page; the page of the chunk after the next is looked up while this one is copied, since the lookup is a dependent
  // access that would otherwise stand before every copy.
  const bool whole = page_size % TOK == 0;
  const int lrow = lane >> 4, c16 = lane & 15;
  const uint32_t dk0 = static_cast<uint32_t>(__cvta_generic_to_shared(Ks + (warp * 16 + lrow) * LDS + c16 * 8));
  const uint32_t dv0 = static_cast<uint32_t>(__cvta_generic_to_shared(Vs + (warp * 16 + lrow) * LDS + c16 * 8));
  const long long row_elems = static_cast<long long>(Hk) * D;
  int next_page = (whole && n_chunks > 0) ? table[t_lo / page_size] : 0;
  int in_page = whole ? t_lo % page_size : 0, page_at = whole ? t_lo / page_size : 0;
  auto valid = [&](long long page) {
    const bool ok = !(page < 0 || (num_slots > 0 && (page + 1) * page_size > num_slots));
    if (!ok && c16 == 0 && status) atomicCAS(status, 0, 9);
    return ok;
  };
  auto issue = [&](int chunk) {  // called for chunks 0, 1, 2, .. in order
    const int stage = chunk % DSTAGES;
    const int t0 = t_lo + chunk * TOK + warp * 16 + lrow;
    const uint32_t dk = dk0 + stage * (STAGE_ELEMS * 2), dv = dv0 + stage * (STAGE_ELEMS * 2);
    if (whole) {
      const long long page = next_page;
      const bool ok = valid(page);
      const long long off = ((ok ? page * page_size + in_page : 0) + warp * 16 + lrow) * row_elems + h * D + c16 * 8;
      const bf16 *ks = k_cache + off, *vs = v_cache + off;
      in_page += TOK;
      if (in_page == page_size) {
        in_page = 0;
        ++page_at;
      }
      if (chunk + 1 < n_chunks) next_page = table[page_at];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const bool live = ok && t0 + 2 * i < t_hi;  // (nothing is read where the size is 0; the address stays in the cache all the same)
        const long long step = live ? 2 * i * row_elems : 0;
        cp_async16(dk + i * (2 * LDS * 2), live ? ks + step : k_cache, live ? 16 : 0);
        cp_async16(dv + i * (2 * LDS * 2), live ? vs + step : v_cache, live ? 16 : 0);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int t = t0 + 2 * i;
        bool ok = t < t_hi;
        long long slot = 0;
        if (ok) {
          const long long page = table[t / page_size];
          ok = valid(page);
          if (ok) slot = page * page_size + t % page_size;
        }
        const long long off = slot * row_elems + h * D + c16 * 8;
        cp_async16(dk + i * (2 * LDS * 2), k_cache + off, ok ? 16 : 0);
        cp_async16(dv + i * (2 * LDS * 2), v_cache + off, ok ? 16 : 0);
      }
    }
  };
  auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };

#pragma unroll
  for (int ch = 0; ch < DSTAGES - 1; ++ch) {
    if (ch < n_chunks) issue(ch);
    commit();
  }
  for (int ch = 0; ch < n_chunks; ++ch) {
    const int stage = ch % DSTAGES;
    asm volatile("cp.async.wait_group %0;" ::"n"(DSTAGES - 2) : "memory");
    __syncwarp();  // the chunk has landed for every lane, and every lane is done with the previous one, whose stage is refilled
    if (ch + DSTAGES - 1 < n_chunks) issue(ch + DSTAGES - 1);
    commit();  // (empty at the end, so that the group count stays)
    const bf16* Kst = Ks + stage * STAGE_ELEMS + (warp * 16) * LDS;
    const bf16* Vst = Vs + stage * STAGE_ELEMS + (warp * 16) * LDS;
    // ---- S = Q K^T for this warp's 16 tokens (two 8-token n-tiles)
    float sacc[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      sacc[nt][0] = sacc[nt][1] = sacc[nt][2] = sacc[nt][3] = 0.f;
#pragma unroll
      for (int kp = 0; kp < 4; ++kp) {  // 32 dims per ldmatrix.x4
        uint32_t b0, b1, b2, b3;
        const bf16* addr = Kst + (nt * 8 + (lane & 7)) * LDS + kp * 32 + (lane >> 3) * 8;
        ldsm_x4(static_cast<uint32_t>(__cvta_generic_to_shared(addr)), b0, b1, b2, b3);
        mma16816(sacc[nt], qa[2 * kp], b0, b1);
        mma16816(sacc[nt], qa[2 * kp + 1], b2, b3);
      }
    }
    // ---- online softmax on row lane/4 (values c0, c1 of both n-tiles)
    const int tok0 = t_lo + ch * TOK + warp * 16 + (lane & 3) * 2;
    float sv[4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = tok0 + nt * 8 + e;
        sv[nt * 2 + e] = t < t_hi ? sacc[nt][e] * scale : -FLT_MAX;
      }
    float mx = fmaxf(fmaxf(sv[0], sv[1]), fmaxf(sv[2], sv[3]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float m_new = fmaxf(m_run, mx);
    const float corr = m_new == -FLT_MAX ? 1.f : __expf(m_run - m_new);
    float pv[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) pv[e] = sv[e] == -FLT_MAX ? 0.f : __expf(sv[e] - m_new);
    l_run = l_run * corr + (pv[0] + pv[1] + pv[2] + pv[3]);
    m_run = m_new;
    uint32_t pa[4];
    pa[0] = pack_bf16x2(pv[0], pv[1]);
    pa[1] = 0u;
    pa[2] = pack_bf16x2(pv[2], pv[3]);
    pa[3] = 0u;
    // ---- O = O * corr + P V
#pragma unroll
    for (int jp = 0; jp < 8; ++jp) {  // two 8-dim n-tiles per ldmatrix.x4.trans
      uint32_t b0, b1, b2, b3;
      const bf16* addr = Vst + (((lane >> 3) & 1) * 8 + (lane & 7)) * LDS + (2 * jp + (lane >> 4)) * 8;
      ldsm_x4_t(static_cast<uint32_t>(__cvta_generic_to_shared(addr)), b0, b1, b2, b3);
      o[2 * jp][0] *= corr; o[2 * jp][1] *= corr;
      o[2 * jp + 1][0] *= corr; o[2 * jp + 1][1] *= corr;
      mma16816(o[2 * jp], pa, b0, b1);
      mma16816(o[2 * jp + 1], pa, b2, b3);
    }
  }
  __syncthreads();  // everyone is done with the stages, which the merge overlays
  // ---- merge the four warps (rows < G only) and write this split's partial
  float lsum = l_run;
  lsum += __shfl_xor_sync(0xffffffffu, lsum, 1);
  lsum += __shfl_xor_sync(0xffffffffu, lsum, 2);
  float* sm_o = reinterpret_cast<float*>(dsm);              // [WARPS][8][D]
  float* sm_m = sm_o + WARPS * 8 * D;                        // [WARPS][8]
  float* sm_l = sm_m + WARPS * 8;
  float* cl_o = sm_l + WARPS * 8;                            // [8][D] this CTA's sums, for the cluster
  float* cl_m = cl_o + 8 * D;                                // [8] maximum, [8] sum
  const int r0 = lane >> 2;
  if (r0 < G) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      sm_o[(warp * 8 + r0) * D + j * 8 + (lane & 3) * 2] = o[j][0];
      sm_o[(warp * 8 + r0) * D + j * 8 + (lane & 3) * 2 + 1] = o[j][1];
    }
    if ((lane & 3) == 0) {
      sm_m[warp * 8 + r0] = m_run;
      sm_l[warp * 8 + r0] = lsum;
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * D; idx += WARPS * 32) {
    const int g = idx / D, d = idx - g * D;
    float gm = -FLT_MAX;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) gm = fmaxf(gm, sm_m[w * 8 + g]);
    float gl = 0.f, go = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float mw = sm_m[w * 8 + g];
      const float c = mw == -FLT_MAX ? 0.f : __expf(mw - gm);
      gl += sm_l[w * 8 + g] * c;
      go += sm_o[(w * 8 + g) * D + d] * c;
    }
    if constexpr (CLUSTER) {
      cl_o[idx] = go;
      if (d == 0) {
        cl_m[g] = gm;
        cl_m[8 + g] = gl;
      }
      continue;
    }
    if (num_splits == 1) {  // nothing to merge: write the normalised output directly
      out[(static_cast<long long>(b) * Hq + h * G + g) * D + d] = __float2bfloat16(gl > 0.f ? go / gl : 0.f);
      continue;
    }
    const long long base = ((static_cast<long long>(b) * Hq + h * G + g) * num_splits + split);
    part_o[base * D + d] = go;
    if (d == 0) {
      part_ml[base * 2] = gm;
      part_ml[base * 2 + 1] = gl;
    }
  }
  if constexpr (CLUSTER) {
    // every CTA arrives, also one whose slice is empty; each then merges a share of the outputs in split order
    cluster_sync_all();
    const uint32_t o_addr = static_cast<uint32_t>(__cvta_generic_to_shared(cl_o));
    const uint32_t m_addr = static_cast<uint32_t>(__cvta_generic_to_shared(cl_m));
    for (int idx = split * (WARPS * 32) + threadIdx.x; idx < G * D; idx += num_splits * WARPS * 32) {
      const int g = idx / D;
      float m[MAX_CLUSTER_SPLITS], l[MAX_CLUSTER_SPLITS], v[MAX_CLUSTER_SPLITS];
      float gm = -FLT_MAX;
#pragma unroll
      for (int sp = 0; sp < MAX_CLUSTER_SPLITS; ++sp)
        if (sp < num_splits) {
          m[sp] = ld_cluster_f32(m_addr + g * 4, sp);
          l[sp] = ld_cluster_f32(m_addr + (8 + g) * 4, sp);
          v[sp] = ld_cluster_f32(o_addr + idx * 4, sp);
        }
#pragma unroll
      for (int sp = 0; sp < MAX_CLUSTER_SPLITS; ++sp)
        if (sp < num_splits) gm = fmaxf(gm, m[sp]);
      float gl = 0.f, go = 0.f;
#pragma unroll
      for (int sp = 0; sp < MAX_CLUSTER_SPLITS; ++sp)
        if (sp < num_splits) {
          const float c = m[sp] == -FLT_MAX ? 0.f : __expf(m[sp] - gm);
          gl += l[sp] * c;
          go += v[sp] * c;
        }
      out[(static_cast<long long>(b) * Hq + h * G) * D + idx] = __float2bfloat16(gl > 0.f ? go / gl : 0.f);
    }
    cluster_sync_all();  // no CTA leaves while another still reads its shared memory
  }
}

}  // namespace

// scratch: fp32 [B*Hq*num_splits*(128+2)]. `num_slots` = rows of the cache (0: page ids are not range-checked);
// `status` (may be null) receives 8 for a length beyond the block-table row, 9 for a page outside the cache.
// Returns the error of this call's own launches (cudaSuccess = 0), not whatever an earlier call left behind.
int paged_decode_attention(const void* q, const void* k_cache, const void* v_cache, const int* block_table,
                           const int* seq_lens, void* out, float* scratch, int B, int Hq, int Hk, int page_size,
                           int max_pages, int num_splits, float scale, cudaStream_t s, long long num_slots, int* status) {
  if (B <= 0) return 0;
  float* part_o = scratch;
  float* part_ml = scratch + static_cast<long long>(B) * Hq * num_splits * D;
  const dim3 grid(B, Hk, num_splits);
  const int G = Hq / Hk;
  constexpr int SMEM = DSTAGES * 2 * STAGE_ELEMS * 2;
  static_assert(SMEM >= ((WARPS + 1) * 8 * (D + 2)) * 4, "the merge overlays the stages");
  const bf16 *qp = static_cast<const bf16*>(q), *kp = static_cast<const bf16*>(k_cache), *vp = static_cast<const bf16*>(v_cache);
  bf16* op = static_cast<bf16*>(out);
  void* args[] = {&qp, &kp, &vp, &block_table, &seq_lens, &part_o, &part_ml, &op, &Hq, &Hk, &page_size, &max_pages,
                  &num_splits, &scale, &num_slots, &status};
  const bool cluster = num_splits > 1 && num_splits <= MAX_CLUSTER_SPLITS;
  const void* fn = nullptr;
#define MB_DECODE(G) fn = cluster ? reinterpret_cast<const void*>(&decode_mma_kernel<G, true>) : reinterpret_cast<const void*>(&decode_mma_kernel<G, false>)
  switch (G) {
    case 1: MB_DECODE(1); break;
    case 2: MB_DECODE(2); break;
    case 4: MB_DECODE(4); break;
    case 8: MB_DECODE(8); break;
    default: return static_cast<int>(cudaErrorInvalidValue);
  }
#undef MB_DECODE
  // The attribute belongs to the (function, device) pair; setting it costs a table lookup, so it is set on every
  // call rather than remembered per process (a second device would otherwise launch with the 48 KB default).
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (e != cudaSuccess) return static_cast<int>(e);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(WARPS * 32);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cluster) {
    if (num_splits > 8) {  // beyond the portable cluster size
      e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e != cudaSuccess) return static_cast<int>(e);
    }
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = num_splits;
    cfg.numAttrs = 2;
  }
  e = cudaLaunchKernelExC(&cfg, fn, args);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (num_splits > 1 && !cluster) {
    e = pdl_launch(decode_merge_kernel, dim3(B * Hq), dim3(D), 0, s, part_o, part_ml, op, num_splits);
  }
  return static_cast<int>(e);
}

}  // namespace mb

// ---------------------------------------------------------------------------------------------------
// Allocation-free variant (declared in noalloc.h): same kernels, split-KV partials in a fixed array that
// is part of the library image instead of a caller-provided scratch tensor.
#include <stdio.h>

#include <mutex>

#include "noalloc.h"

namespace {

// Partial outputs [B*Hq*splits][128] followed by partial (max, sum) pairs [B*Hq*splits][2].
static __device__ __align__(256) float g_noalloc_scratch[MB_NOALLOC_SCRATCH_FLOATS];

constexpr int kMaxDevices = 64;
float* g_scratch_addr[kMaxDevices] = {nullptr};  // device address of the array, per device
std::mutex g_scratch_mutex;
thread_local char g_noalloc_err[256] = "";

int noalloc_fail(int code, const char* msg) {
  snprintf(g_noalloc_err, sizeof(g_noalloc_err), "%s", msg);
  return code;
}

// In host code `g_noalloc_scratch` is only a handle of the symbol; the address kernels may use has to
// be asked from the runtime, once per device, with that device current.
int noalloc_scratch_for_current_device(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) return noalloc_fail(MB_NOALLOC_ERR_CUDA, "cudaGetDevice failed");
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_addr[dev] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) {
      snprintf(g_noalloc_err, sizeof(g_noalloc_err), "cudaGetSymbolAddress(scratch) failed: %s", cudaGetErrorString(e));
      return MB_NOALLOC_ERR_CUDA;
    }
    g_scratch_addr[dev] = p;
  }
  *out = g_scratch_addr[dev];
  return MB_NOALLOC_OK;
}

}  // namespace

extern "C" const char* mb_noalloc_last_error(void) { return g_noalloc_err; }

extern "C" int mb_paged_decode_attention_noalloc(const void* q, const void* k_cache, const void* v_cache,
                                                 const int* block_table, const int* seq_lens, void* out, int B, int Hq,
                                                 int Hk, int page_size, int max_pages, int num_splits, float scale,
                                                 long long num_slots, int* status, cudaStream_t stream) {
  if (!q || !k_cache || !v_cache || !block_table || !seq_lens || !out)
    return noalloc_fail(MB_NOALLOC_ERR_BAD_ARG, "null pointer argument");
  if (B <= 0 || Hq <= 0 || Hk <= 0 || page_size <= 0 || max_pages <= 0 || num_splits <= 0 || num_slots <= 0)
    return noalloc_fail(MB_NOALLOC_ERR_BAD_ARG, "extents must be positive");
  if (Hq % Hk != 0) return noalloc_fail(MB_NOALLOC_ERR_BAD_ARG, "Hq must be a multiple of Hk");
  const int G = Hq / Hk;
  if (G != 1 && G != 2 && G != 4 && G != 8)
    return noalloc_fail(MB_NOALLOC_ERR_BAD_ARG, "Hq / Hk must be 1, 2, 4 or 8");
  const unsigned long long need = 130ull * static_cast<unsigned long long>(B) * Hq * num_splits;
  if (need > MB_NOALLOC_SCRATCH_FLOATS) {
    snprintf(g_noalloc_err, sizeof(g_noalloc_err),
             "B*Hq*num_splits*130 = %llu floats exceed the built-in scratch of %u floats; lower num_splits or the batch",
             need, MB_NOALLOC_SCRATCH_FLOATS);
    return MB_NOALLOC_ERR_TOO_LARGE;
  }
  float* scratch = nullptr;
  const int rc = noalloc_scratch_for_current_device(&scratch);
  if (rc != MB_NOALLOC_OK) return rc;
  // the launcher reports the result of its own launches; an error some earlier, unrelated call left in the
  // runtime's "last error" slot is neither read nor cleared here
  const int e = mb::paged_decode_attention(q, k_cache, v_cache, block_table, seq_lens, out, scratch, B, Hq, Hk, page_size,
                                           max_pages, num_splits, scale, stream, num_slots, status);
  if (e != 0) {
    snprintf(g_noalloc_err, sizeof(g_noalloc_err), "kernel launch failed: %s", cudaGetErrorString(static_cast<cudaError_t>(e)));
    return MB_NOALLOC_ERR_CUDA;
  }
  return MB_NOALLOC_OK;
}
