// Causal variable-length flash attention backward on tcgen05 (training).
//
// One CTA owns one block of 128 keys of one sequence and one KV head. Its dK / dV accumulate in TMEM over every
// query tile (64 rows) at or after the block and over the G = Hq / Hk query heads that share the KV head, so K, V
// stay in shared memory for the whole CTA and dK / dV leave the chip once. Everything is computed transposed
// (keys on the TMEM lanes), which makes P^T and dS^T row-per-thread:
//
//   S^T  = K Q^T            [128 keys x 64 q]   A = K (K-major over d),  B = Q  (K-major over d)
//   dP^T = V dO^T           [128 keys x 64 q]   A = V,                   B = dO
//   P^T  = exp2(S^T * scale*log2e - lse*log2e), dS^T = P^T o (dP^T - D)        (256 threads, two per key row)
//   dV  += P^T  dO          [128 keys x 128 d]  A = P^T  (smem, K-major over q), B = dO (smem, d contiguous)
//   dK  += dS^T Q           [128 keys x 128 d]  A = dS^T (smem, K-major over q), B = Q  (smem, d contiguous)
//   dQ^T = K^T dS^T         [128 d x 64 q]      A = K (d contiguous),           B = dS^T (q contiguous)
//
// dQ is accumulated across key blocks by bulk copies that add (`cp.reduce.async.bulk.tensor`, one per tile of 64 x 128 fp32) into a
// scratch tensor and converted to bf16 by a second kernel; D = rowsum(dO o O) and lse * log2e come from a first one.
//
//   warp 0      : TMA producer: K, V once; then (Q, dO) tiles into a 3-stage ring, with the tile's lse / D rows
//   warp 1      : TMEM allocator + MMA issuer (one thread)
//   warps 2..9  : P^T / dS^T math, two threads per key row (32 query columns each); dK / dV epilogue
//   warps 10..13: dQ^T read-out (one thread per d), transposed into shared memory
//   warp 14     : the copies that add dQ (a thread that waits for a copy reads out nothing meanwhile)
//
// Two tiles are in flight: S^T / dP^T have two buffers in TMEM and P^T / dS^T two in shared memory, so the tensor core runs
// dV, dK, dQ^T of one tile and S^T, dP^T of the tile after the next while the threads work on the tile between. dQ^T of a
// tile goes where its S^T was (read by then), and the S^T after the next waits for the dQ^T to be read out. In shared memory it
// takes the place of the tile's P^T and dS^T once dV and dK have read them; the threads write the next P^T there when the copy has.
//
// TMEM columns: S^T / dQ^T 0..63 and 64..127, dP^T 128..191 and 192..255, dV 256..383, dK 384..511. Every mbarrier wait is
// bounded (ptx.cuh): on expiry the CTA records a status code, leaves its loops, frees TMEM and returns.
//
// Measured with the kernels around it, 32 heads, before (sums into dQ by `red.global.add.f32`, 64 instructions a thread and tile,
// which the read-out warps could not issue faster than one in some 80 clocks; a warp issuing the products) -> now: 9216 tokens in one
// sequence, 8 KV heads, 3.07 -> 2.10 ms (567 -> 828 TFLOP/s); 16384 in six sequences, 4 KV heads, 1.89 -> 1.41 (485 -> 649); with the
// read-out waiting for its own copies 2.28 and 1.48. A tile takes some 3300 clocks, its products 1664.
//
// Reference counterpart: the flash-attention backward behind `--attention-backend flash`
// (scripts/run_qwen3_30b_a3b.py:203).
#include <cuda.h>
#include <float.h>

#include <mutex>
#include <string>

#include "launchers.h"
#include "ptx.cuh"

namespace mb {
namespace {

constexpr int BQ = 64;    // query rows per tile
constexpr int BK = 128;   // keys per CTA
constexpr int HD = 128;
constexpr int ATOM_K = BK * 128;     // 128 rows x 128 B
constexpr int ATOM_Q = BQ * 128;     // 64 rows x 128 B
constexpr int KTILE = 2 * ATOM_K;    // K or V block
constexpr int QTILE = 2 * ATOM_Q;    // Q or dO tile
constexpr int PTILE = ATOM_K;        // P^T or dS^T: 128 keys x 64 q
constexpr int STAGES = 3;
constexpr int SMS = 148;
constexpr int BWD_THREADS = 15 * 32;
constexpr int BWD_SMEM = 2 * KTILE + 4 * PTILE + STAGES * 2 * QTILE + STAGES * 2 * BQ * 4 + 256 + 1024;

struct FaBwdArgs {
  const int4* blocks;  // {kv_row0 (global token index of the block's first key), kv_rows, kv_pos0 (its position in the
                       //  sequence), seq_end (global token index one past the sequence)}
  int Hq, Hk;
  const float* lse2;   // [Hq, T] log-sum-exp * log2(e)
  const float* dsum;   // [Hq, T] rowsum(dO o O)
  __nv_bfloat16* dk;   // [T, Hk, 128]
  __nv_bfloat16* dv;
  long long T;
  float scale, scale_log2;
  int split;           // CTAs, in a cluster, that share the query heads of a key block (a power of two that divides Hq / Hk)
  int* status;
};

__device__ __forceinline__ uint32_t swz_off(int row, int chunk16) {
  return static_cast<uint32_t>(row * 128 + ((chunk16 ^ (row & 7)) << 4));
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// SPLIT: p.split CTAs, a cluster, share a key block's query heads; each sums dV and dK of its own in TMEM, and at the end every CTA
// adds up a part of the rows from all of them, in the order of their heads. One sequence of 4096, 32 query and 4 KV heads: 964 -> 519 us
// (two CTAs), 389 + 388: 130 -> 62 (four); who gains from it is in bwd_split of ops/attention.py.
template <bool SPLIT>
__global__ void __launch_bounds__(BWD_THREADS, 1)
fa_bwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
              const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
              const __grid_constant__ CUtensorMap map_dq, const FaBwdArgs p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t k_s = base;
  const uint32_t v_s = k_s + KTILE;
  const uint32_t pt_s = v_s + KTILE;
  const uint32_t ds_s = pt_s + PTILE;
  const uint32_t ring = pt_s + 4 * PTILE;                  // (P^T, dS^T) twice; per stage: Q tile, dO tile
  const uint32_t stats = ring + STAGES * 2 * QTILE;        // per stage: lse2[64], dsum[64]
  const uint32_t bars = stats + STAGES * 2 * BQ * 4;
  auto BAR = [&](int i) { return bars + 8u * i; };
  constexpr int B_KVF = 0, B_QF = 1, B_QE = 4, B_SF = 7, B_PF = 9, B_DQF = 11, B_DQE = 12, B_FIN = 13;
  constexpr int B_PD = 14, B_ST = 16, B_PB = 18;  // by buffer of P^T / dS^T: read by its products; dQ^T staged in it; copied from it
  const uint32_t tmem_slot = bars + 8u * 20;
  __shared__ int abort_s;
  __shared__ uint32_t tmem_base_s;
  volatile int* abort_flag = &abort_s;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));   // generic pointer to the aligned base
  float* stats_g = reinterpret_cast<float*>(gen + (stats - base));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Heads vary fastest: the list starts with the blocks that have the most queries after them, and all heads' long blocks have
  // to start before anyone's short ones (one head after another left SMs with 1.4 times the average work at the end).
  const int split = SPLIT ? p.split : 1;
  const int job = blockIdx.x / split;
  const int4 blk = p.blocks[job / p.Hk];
  const int hk = job % p.Hk;
  const int G = p.Hq / p.Hk / split;       // this CTA's query heads
  const int hq0 = (hk * split + blockIdx.x % split) * G;
  const int kv_row0 = blk.x, kv_rows = blk.y, seq_end = blk.w;
  // query rows at or after the block's first key: global rows kv_row0 .. seq_end - 1
  const int q_total = seq_end - kv_row0;
  const int n_qt = (q_total + BQ - 1) / BQ;
  const int n_it = n_qt * G;

  if (threadIdx.x == 0) {
    abort_s = 0;
    mbar_init(BAR(B_KVF), 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(BAR(B_QF + s), 1);
      mbar_init(BAR(B_QE + s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(BAR(B_SF + b), 1);
      mbar_init(BAR(B_PF + b), 8);
      mbar_init(BAR(B_PD + b), 1);
      mbar_init(BAR(B_ST + b), 4);
      mbar_init(BAR(B_PB + b), 1);
    }
    mbar_init(BAR(B_DQF), 1);
    mbar_init(BAR(B_DQE), 4);
    mbar_init(BAR(B_FIN), 1);
    fence_barrier_init();
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_do);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    prefetch_tensormap(&map_dq);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x == 0) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(tmem_slot));
    tmem_base_s = v;
  }
  __syncthreads();
  const uint32_t tmem = tmem_base_s;
  const uint32_t t_S = tmem, t_dP = tmem + 128, t_dV = tmem + 256, t_dK = tmem + 384;  // t_S, t_dP: + 64 for odd tiles

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    bool ok = true;
    if (lane == 0) {
      mbar_expect_tx(BAR(B_KVF), 2 * KTILE);
      tma_load_2d(k_s, &map_k, BAR(B_KVF), hk * HD, kv_row0);
      tma_load_2d(k_s + ATOM_K, &map_k, BAR(B_KVF), hk * HD + 64, kv_row0);
      tma_load_2d(v_s, &map_v, BAR(B_KVF), hk * HD, kv_row0);
      tma_load_2d(v_s + ATOM_K, &map_v, BAR(B_KVF), hk * HD + 64, kv_row0);
    }
    for (int it = 0; ok && it < n_it; ++it) {
      const int st = it % STAGES;
      const int g = it / n_qt, qt = it - g * n_qt;
      const int hq = hq0 + g;
      const int q_row0 = kv_row0 + qt * BQ;
      if (!mbar_wait(BAR(B_QE + st), ((it / STAGES) & 1) ^ 1, abort_flag, p.status, ERR_WAIT_EMPTY)) {
        ok = false;
        break;
      }
      // the tile's softmax statistics (rows past the sequence read a clamped row and are masked by the consumers)
      float* sp = stats_g + st * 2 * BQ;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = min(q_row0 + h * 32 + lane, seq_end - 1);
        sp[h * 32 + lane] = p.lse2[static_cast<long long>(hq) * p.T + r];
        sp[BQ + h * 32 + lane] = p.dsum[static_cast<long long>(hq) * p.T + r];
      }
      __syncwarp();
      if (lane == 0) {
        mbar_expect_tx(BAR(B_QF + st), 2 * QTILE);
        const uint32_t qd = ring + st * 2 * QTILE, dd = qd + QTILE;
        tma_load_2d(qd, &map_q, BAR(B_QF + st), hq * HD, q_row0);
        tma_load_2d(qd + ATOM_Q, &map_q, BAR(B_QF + st), hq * HD + 64, q_row0);
        tma_load_2d(dd, &map_do, BAR(B_QF + st), hq * HD, q_row0);
        tma_load_2d(dd + ATOM_Q, &map_do, BAR(B_QF + st), hq * HD + 64, q_row0);
      }
    }
    if (!ok && lane == 0) {  // give copies in flight a bounded chance to land before shared memory is released
      const unsigned long long t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 2000000ull) {
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t id_s = make_idesc_bf16(BK, BQ, false, false);    // S^T, dP^T
      constexpr uint32_t id_acc = make_idesc_bf16(BK, HD, false, true);   // dV, dK: A K-major (q), B d-contiguous
      constexpr uint32_t id_dq = make_idesc_bf16(HD, BQ, true, true);     // dQ^T: A d-contiguous, B q-contiguous
      const uint64_t kd = make_smem_desc(k_s, 16, 1024), vd = make_smem_desc(v_s, 16, 1024);
      const uint64_t kt = make_smem_desc(k_s, ATOM_K, 1024);  // K as an operand that is contiguous along d
      bool ok = true;
      auto wait = [&](uint32_t bar, int n, int code) {
        ok = ok && mbar_wait(bar, n & 1, abort_flag, p.status, code);
        tc_fence_after();
        return ok;
      };
      auto issue_s = [&](int it, int st, int round) {
        if (!wait(BAR(B_QF + st), round, ERR_WAIT_FULL)) return;
        const uint64_t qd = make_smem_desc(ring + st * 2 * QTILE, 16, 1024), dd = make_smem_desc(ring + st * 2 * QTILE + QTILE, 16, 1024);
        const uint32_t buf = (it & 1) * 64;
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t ka = ((k >> 2) * ATOM_K + (k & 3) * 32) >> 4, qa = ((k >> 2) * ATOM_Q + (k & 3) * 32) >> 4;
          umma_f16(t_S + buf, kd + ka, qd + qa, id_s, k > 0 ? 1u : 0u);
        }
#pragma unroll
        for (int k = 0; k < HD / 16; ++k) {
          const uint32_t ka = ((k >> 2) * ATOM_K + (k & 3) * 32) >> 4, qa = ((k >> 2) * ATOM_Q + (k & 3) * 32) >> 4;
          umma_f16(t_dP + buf, vd + ka, dd + qa, id_s, k > 0 ? 1u : 0u);
        }
        umma_commit(BAR(B_SF + (it & 1)));
      };
      wait(BAR(B_KVF), 0, ERR_WAIT_FULL);
      int s_st = 0, s_round = 0;  // ring stage of the next S^T and the times the ring has gone round
      auto next_s = [&](int it) {
        issue_s(it, s_st, s_round);
        if (++s_st == STAGES) {
          s_st = 0;
          ++s_round;
        }
      };
      if (ok && n_it > 0) next_s(0);
      if (ok && n_it > 1) next_s(1);
      int st = 0;
      for (int it = 0; ok && it < n_it; ++it) {
        const int b = it & 1;
        if (!wait(BAR(B_PF + b), it >> 1, ERR_WAIT_TMEM_EMPTY)) break;
        const uint32_t pt = pt_s + b * 2 * PTILE, ds = ds_s + b * 2 * PTILE;
        const uint64_t dst = make_smem_desc(ds, ATOM_K, 1024);
        const uint64_t pa = make_smem_desc(pt, 16, 1024), da = make_smem_desc(ds, 16, 1024);
        const uint64_t qt = make_smem_desc(ring + st * 2 * QTILE, ATOM_Q, 1024), dt = make_smem_desc(ring + st * 2 * QTILE + QTILE, ATOM_Q, 1024);
        // dQ^T first, since its read-out is the longest way to the next S^T; it overwrites this tile's S^T, which has been read
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)  // contraction over the 128 keys
          umma_f16(t_S + b * 64, kt + k * (2048 >> 4), dst + k * (2048 >> 4), id_dq, k > 0 ? 1u : 0u);
        umma_commit(BAR(B_DQF));
#pragma unroll
        for (int k = 0; k < BQ / 16; ++k)  // contraction over the 64 queries of the tile
          umma_f16(t_dV, pa + k * (32 >> 4), dt + k * (2048 >> 4), id_acc, (it > 0 || k > 0) ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < BQ / 16; ++k)
          umma_f16(t_dK, da + k * (32 >> 4), qt + k * (2048 >> 4), id_acc, (it > 0 || k > 0) ? 1u : 0u);
        umma_commit(BAR(B_QE + st));  // the (Q, dO) stage is free once these have run,
        umma_commit(BAR(B_PD + b));   // and so are P^T and dS^T
        if (++st == STAGES) st = 0;
        // dQ^T of this tile is out before the next one's is announced, and before an S^T takes its place
        if (it + 1 < n_it && !wait(BAR(B_DQE), it, ERR_WAIT_TMEM_EMPTY)) break;
        if (it + 2 < n_it) next_s(it + 2);
      }
      if (ok) umma_commit(BAR(B_FIN));
    }
    __syncwarp();
  } else if (warp < 10) {
    // ------------------------------------------------------------------ P^T / dS^T (two threads per key row)
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = quad * 32 + lane;                   // key row inside the block
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const bool key_ok = row < kv_rows;
    bool ok = true;
    for (int it = 0; it < n_it; ++it) {
      const int st = it % STAGES;
      const int g = it / n_qt, qt = it - g * n_qt;
      if (!mbar_wait(BAR(B_SF + (it & 1)), (it >> 1) & 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL)) {
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t s[32], d[32];
      const uint32_t buf = (it & 1) * 64;
      tmem_ld_32x32(t_S + buf + lane_addr + half * 32, s);
      tmem_ld_32x32(t_dP + buf + lane_addr + half * 32, d);
      tmem_ld_wait();
      const float* sp = stats_g + st * 2 * BQ + half * 32;
      // query j of this thread sits at sequence offset qt*64 + half*32 + j from the block's first key
      const int q_off0 = qt * BQ + half * 32;
      const int q_left = q_total - q_off0;              // queries of the tile half that exist
      uint32_t pp[16], dd[16];
      // tiles whose every key precedes every query, all of them there, need no mask (decided per warp)
      const bool masked = kv_rows < BK || q_left < 32 || q_off0 < BK - 1;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        float pv[2], dv[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = 2 * j + e;
          const float x = __uint_as_float(s[c]) * p.scale_log2 - sp[c];
          float pe = ex2(x), de = pe * (__uint_as_float(d[c]) - sp[BQ + c]);
          if (masked) {
            const bool live = key_ok && c < q_left && row <= q_off0 + c;   // causal: key position <= query position
            pe = live ? pe : 0.f;
            de = live ? de : 0.f;
          }
          pv[e] = pe;
          dv[e] = de;
        }
        pp[j] = pack_bf16(pv[0], pv[1]);
        dd[j] = pack_bf16(dv[0], dv[1]);
      }
      if (it >= 2 && !mbar_wait(BAR(B_PB + (it & 1)), ((it >> 1) - 1) & 1, abort_flag, p.status, ERR_WAIT_TMEM_EMPTY)) {
        ok = false;
        break;
      }
      // (this buffer's dQ^T of the tile before the last has been copied, and so its products have run)
      const uint32_t pt = pt_s + (it & 1) * 2 * PTILE, ds = ds_s + (it & 1) * 2 * PTILE;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t o = swz_off(row, half * 4 + c);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(pt + o), "r"(pp[4 * c]), "r"(pp[4 * c + 1]),
                     "r"(pp[4 * c + 2]), "r"(pp[4 * c + 3])
                     : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(ds + o), "r"(dd[4 * c]), "r"(dd[4 * c + 1]),
                     "r"(dd[4 * c + 2]), "r"(dd[4 * c + 3])
                     : "memory");
      }
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR(B_PF + (it & 1)));
    }
    // ---- epilogue: dV, dK (scaled) -> bf16
    if (ok) ok = mbar_wait(BAR(B_FIN), 0, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
    if (!SPLIT && ok) {
      tc_fence_after();
      const long long orow = (static_cast<long long>(kv_row0 + row) * p.Hk + hk) * HD + half * 64;
      uint32_t o[32];
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        const uint32_t src = (which == 0 ? t_dV : t_dK) + lane_addr + half * 64;
        __nv_bfloat16* dst = (which == 0 ? p.dv : p.dk) + orow;
        const float sc = which == 0 ? 1.f : p.scale;
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          tmem_ld_32x32(src + c * 32, o);
          tmem_ld_wait();
          if (key_ok) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint4 v;
              v.x = pack_bf16(__uint_as_float(o[8 * i]) * sc, __uint_as_float(o[8 * i + 1]) * sc);
              v.y = pack_bf16(__uint_as_float(o[8 * i + 2]) * sc, __uint_as_float(o[8 * i + 3]) * sc);
              v.z = pack_bf16(__uint_as_float(o[8 * i + 4]) * sc, __uint_as_float(o[8 * i + 5]) * sc);
              v.w = pack_bf16(__uint_as_float(o[8 * i + 6]) * sc, __uint_as_float(o[8 * i + 7]) * sc);
              *reinterpret_cast<uint4*>(dst + c * 32 + i * 8) = v;
            }
          }
        }
      }
    }
  } else if (warp < 14) {
    // ------------------------------------------------------------------ dQ^T read-out (one thread per d)
    const int quad = warp & 3;
    const int drow = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    for (int it = 0; it < n_it; ++it) {
      const int qt = it % n_qt, buf = it & 1;
      if (!mbar_wait(BAR(B_DQF), it & 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL)) break;
      tc_fence_after();
      uint32_t a[64];
      tmem_ld_32x32(t_S + buf * 64 + lane_addr, *reinterpret_cast<uint32_t(*)[32]>(&a[0]));
      tmem_ld_32x32(t_S + buf * 64 + lane_addr + 32, *reinterpret_cast<uint32_t(*)[32]>(&a[32]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR(B_DQE));
      const int q_row0 = kv_row0 + qt * BQ;
      const int q_left = seq_end - q_row0;  // (rows past the sequence may be another one's: they receive nothing)
      if (!mbar_wait(BAR(B_PD + buf), (it >> 1) & 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL)) break;
      const uint32_t dst = pt_s + buf * 2 * PTILE + drow * 4;  // [64 q][128 d] over P^T and dS^T
#pragma unroll
      for (int c = 0; c < 64; ++c) {
        const float v = c < q_left ? __uint_as_float(a[c]) * p.scale : 0.f;
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst + c * (HD * 4)), "f"(v) : "memory");
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR(B_ST + buf));
    }
  } else if (lane == 0) {
    // ------------------------------------------------------------------ dQ: shared memory added to global memory
    for (int it = 0; it < n_it; ++it) {
      const int g = it / n_qt, qt = it - g * n_qt, buf = it & 1;
      if (!mbar_wait(BAR(B_ST + buf), (it >> 1) & 1, abort_flag, p.status, ERR_WAIT_FULL)) break;
      tma_reduce_add_2d(&map_dq, pt_s + buf * 2 * PTILE, (hq0 + g) * HD, kv_row0 + qt * BQ);
      tma_store_commit();
      tma_store_wait_read<0>();
      mbar_arrive(BAR(B_PB + buf));
    }
    tma_store_wait<0>();
  }
  __syncwarp();

  tc_fence_before();
  __syncthreads();
  if constexpr (SPLIT) {
    // ------------------------------------------------------------------ dV, dK of the cluster's heads added up, CTA by CTA
    // (every thread of every CTA comes here, whatever happened before; a CTA that gave up has set the status, and its sums are void)
    if (warp >= 2 && warp < 10) {
      const int quad = warp & 3, half = (warp - 2) >> 2, row = quad * 32 + lane;
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {  // dV's two quarters of this half row, then dK's: over K, V, P^T and dS^T, which are done with
        uint32_t o[32];
        tmem_ld_32x32((c < 2 ? t_dV : t_dK) + (static_cast<uint32_t>(quad * 32) << 16) + half * 64 + (c & 1) * 32, o);
        tmem_ld_wait();
        const uint32_t dst = base + (c >> 1) * (BK * HD * 4) + row * (HD * 4);
#pragma unroll
        for (int i = 0; i < 8; ++i)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (((half * 16 + (c & 1) * 8 + i) ^ lane) << 4)), "r"(o[4 * i]),
                       "r"(o[4 * i + 1]), "r"(o[4 * i + 2]), "r"(o[4 * i + 3])
                       : "memory");
      }
      tc_fence_before();
    }
    cluster_sync_all();
    const int rank = blockIdx.x % split, rows = BK / split;  // of the block, which this CTA adds up: eight values a thread and turn
    for (int i = threadIdx.x; i < 2 * rows * (HD / 8); i += BWD_THREADS) {
      const int which = i / (rows * (HD / 8)), row = rank * rows + i / (HD / 8) % rows, c = i % (HD / 8);
      const uint32_t src = base + which * (BK * HD * 4) + row * (HD * 4);
      const uint32_t src0 = src + (((2 * c) ^ (row & 31)) << 4), src1 = src + (((2 * c + 1) ^ (row & 31)) << 4);
      float v[8] = {};
      for (int r = 0; r < split; ++r) {
        const float4 x = ld_cluster_f4(map_to_rank(src0, r)), y = ld_cluster_f4(map_to_rank(src1, r));
        v[0] += x.x, v[1] += x.y, v[2] += x.z, v[3] += x.w;
        v[4] += y.x, v[5] += y.y, v[6] += y.z, v[7] += y.w;
      }
      if (row < kv_rows) {
        const float sc = which == 0 ? 1.f : p.scale;
        __nv_bfloat16* dst = (which == 0 ? p.dv : p.dk) + (static_cast<long long>(kv_row0 + row) * p.Hk + hk) * HD + c * 8;
        *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(v[0] * sc, v[1] * sc), pack_bf16(v[2] * sc, v[3] * sc),
                                                    pack_bf16(v[4] * sc, v[5] * sc), pack_bf16(v[6] * sc, v[7] * sc));
      }
    }
    __syncwarp();
    cluster_sync_all();  // no CTA leaves while another still reads its shared memory
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// D[h, t] = sum_d dO[t, h, d] * O[t, h, d];  lse2[h, t] = lse[h, t] * log2(e). Bound by reading O and dO: a half-warp takes a head's
// PREP_ROWS tokens, asked for together with 16 bytes a lane, so that a sector of D and of lse2 leaves as one.
// 16384 tokens of 32 heads, 270 MB: 97 -> 54 us (a warp a row, eight bytes a lane, before; 82 with four rows of neighbouring heads,
// whose results leave as single floats).
constexpr int PREP_ROWS = 8;
__global__ void __launch_bounds__(256, 2)
fa_bwd_prep_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o, const float* __restrict__ lse,
                   float* __restrict__ dsum, float* __restrict__ lse2, long long T, int Hq) {
  const int l = threadIdx.x & 15;
  const long long w = static_cast<long long>(blockIdx.x) * 16 + (threadIdx.x >> 4);
  const long long t0 = w / Hq * PREP_ROWS;
  const int h = static_cast<int>(w % Hq);
  const int n_rows = static_cast<int>(T - t0 < PREP_ROWS ? T - t0 : PREP_ROWS);  // (<= 0 in half-warps past the last token)
  uint4 a[PREP_ROWS], b[PREP_ROWS];
#pragma unroll
  for (int n = 0; n < PREP_ROWS; ++n) {
    a[n] = b[n] = make_uint4(0u, 0u, 0u, 0u);
    if (n < n_rows) {
      a[n] = reinterpret_cast<const uint4*>(o + ((t0 + n) * Hq + h) * HD)[l];
      b[n] = reinterpret_cast<const uint4*>(d_o + ((t0 + n) * Hq + h) * HD)[l];
    }
  }
  float mine = 0.f;  // lane n's row is n
#pragma unroll
  for (int n = 0; n < PREP_ROWS; ++n) {
    const __nv_bfloat162* ab = reinterpret_cast<const __nv_bfloat162*>(&a[n]);
    const __nv_bfloat162* bb = reinterpret_cast<const __nv_bfloat162*>(&b[n]);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = __bfloat1622float2(ab[i]), y = __bfloat1622float2(bb[i]);
      s += x.x * y.x + x.y * y.y;
    }
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (l == n) mine = s;
  }
  if (l < n_rows) {
    const long long at = h * T + t0 + l;
    dsum[at] = mine;
    lse2[at] = lse[at] * 1.4426950408889634f;
  }
}

__global__ void f32_to_bf16_kernel(const float4* __restrict__ in, uint2* __restrict__ out, long long n4) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float4 v = in[i];
    uint2 o;
    o.x = pack_bf16(v.x, v.y);
    o.y = pack_bf16(v.z, v.w);
    out[i] = o;
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
std::string g_err;
EncodeTiledFn g_encode = nullptr;
std::once_flag g_once;

int fail(const std::string& m) {
  g_err = m;
  return -1;
}

// The fp32 accumulator of dQ: [T, Hq * 128], box = one head of 64 rows.
int make_dq_map(CUtensorMap* map, float* ptr, long long T, int Hq) {
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0) return fail("attention scratch must be 16-byte aligned");
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(Hq) * HD, static_cast<cuuint64_t>(T)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(Hq) * HD * 4};
  cuuint32_t box[2] = {HD, BQ};
  cuuint32_t estr[2] = {1u, 1u};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail("cuTensorMapEncodeTiled failed with code " + std::to_string(int(r)));
  return 0;
}

// bf16 [rows, heads*128] view with row pitch `ld` elements; box = 64 columns x `box_rows` rows, 128-byte swizzle.
int make_map(CUtensorMap* map, const void* ptr, long long rows, long long cols, long long ld, unsigned box_rows) {
  std::call_once(g_once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  });
  if (!g_encode) return fail("cuTensorMapEncodeTiled is not available");
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0) return fail("attention operand base must be 16-byte aligned");
  if ((ld * 2) % 16 != 0) return fail("attention operand row pitch must be a multiple of 16 bytes");
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  cuuint32_t box[2] = {64u, box_rows};
  cuuint32_t estr[2] = {1u, 1u};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail("cuTensorMapEncodeTiled failed with code " + std::to_string(int(r)));
  return 0;
}

}  // namespace

const char* flash_attn_bwd_last_error() { return g_err.c_str(); }

// q, d_o, o: [T, Hq, 128] (q and d_o with row pitches q_ld / do_ld elements, o contiguous); k, v: [T, Hk, 128] with
// pitches; lse [Hq, T]; blocks int32 [n, 4]; scratch fp32: dq_acc [T*Hq*128] (zeroed here) then dsum [Hq*T], lse2 [Hq*T].
int flash_attn_bwd(const void* q, long long q_ld, const void* k, long long k_ld, const void* v, long long v_ld, const void* o,
                   const void* d_o, long long do_ld, const float* lse, const int* blocks, int num_blocks, long long T, int Hq,
                   int Hk, int head_dim, float scale, int split, float* scratch, void* dq, void* dk, void* dv, int* status,
                   cudaStream_t stream) {
  if (head_dim != HD) return fail("flash_attn_bwd supports head_dim 128 only");
  if (Hq % Hk != 0) return fail("query heads must be a multiple of kv heads");
  const int heads = Hq / Hk;
  if ((split != 1 && split != 2 && split != 4) || heads % split != 0)
    return fail("split must be 1, 2 or 4 and divide the query heads of a kv head");
  if (T <= 0 || num_blocks <= 0) return 0;
  float* dq_acc = scratch;
  float* dsum = scratch + T * Hq * HD;
  float* lse2 = dsum + T * Hq;
  // the operands' alignment is checked here, before anything reads them
  CUtensorMap mq, mdo, mk, mv, mdq;
  if (make_map(&mq, q, T, static_cast<long long>(Hq) * HD, q_ld, BQ)) return -1;
  if (make_map(&mdo, d_o, T, static_cast<long long>(Hq) * HD, do_ld, BQ)) return -1;
  if (make_map(&mk, k, T, static_cast<long long>(Hk) * HD, k_ld, BK)) return -1;
  if (make_map(&mv, v, T, static_cast<long long>(Hk) * HD, v_ld, BK)) return -1;
  if (make_dq_map(&mdq, dq_acc, T, Hq)) return -1;
  if ((reinterpret_cast<uintptr_t>(o) & 15) != 0) return fail("attention operand base must be 16-byte aligned");
  cudaError_t e = cudaMemsetAsync(dq_acc, 0, sizeof(float) * T * Hq * HD, stream);
  if (e != cudaSuccess) return fail("cudaMemsetAsync failed for the dQ accumulator");
  {
    const long long blocks_n = ((T + PREP_ROWS - 1) / PREP_ROWS * Hq + 15) / 16;
    fa_bwd_prep_kernel<<<static_cast<unsigned>(blocks_n), 256, 0, stream>>>(
        static_cast<const __nv_bfloat16*>(o), static_cast<const __nv_bfloat16*>(d_o), lse, dsum, lse2, T, Hq);
  }
  auto kernel = split > 1 ? fa_bwd_kernel<true> : fa_bwd_kernel<false>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM) != cudaSuccess)
    return fail("cudaFuncSetAttribute(MaxDynamicSharedMemorySize) failed for the attention backward");
  FaBwdArgs a;
  a.blocks = reinterpret_cast<const int4*>(blocks);
  a.Hq = Hq;
  a.Hk = Hk;
  a.lse2 = lse2;
  a.dsum = dsum;
  a.dk = static_cast<__nv_bfloat16*>(dk);
  a.dv = static_cast<__nv_bfloat16*>(dv);
  a.T = T;
  a.scale = scale;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.split = split;
  a.status = status;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(split);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(num_blocks) * Hk * split);
  cfg.blockDim = dim3(BWD_THREADS);
  cfg.dynamicSmemBytes = BWD_SMEM;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, kernel, mq, mdo, mk, mv, mdq, a);
  if (e != cudaSuccess) {
    cudaGetLastError();  // (reported here)
    return fail(std::string("attention backward launch failed: ") + cudaGetErrorString(e));
  }
  const long long n4 = T * Hq * HD / 4;
  long long cb = (n4 + 255) / 256;
  if (cb > SMS * 8) cb = SMS * 8;
  f32_to_bf16_kernel<<<static_cast<unsigned>(cb), 256, 0, stream>>>(reinterpret_cast<const float4*>(dq_acc),
                                                                   reinterpret_cast<uint2*>(dq), n4);
  return 0;
}

}  // namespace mb
