// Persistent, warp-specialised bf16 GEMM for sm_100a.
//
//   warp 0      : TMA producer (cp.async.bulk.tensor, 128B swizzle, no multicast)
//   warp 1      : TMEM allocator + single-thread tcgen05.mma issuer
//   warps 2..9  : epilogue (tcgen05.ld -> registers -> shared memory -> global), two per TMEM lane quadrant, half the columns each
//
// The accumulator is double-buffered in TMEM (2 x BLOCK_N fp32 columns) so the epilogue of tile
// i overlaps the main loop of tile i+1. One kernel covers dense GEMMs, the MoE grouped GEMMs
// (row tiles tagged with an expert id) and the MoE weight-gradient GEMM (contraction over the rows
// of each expert); both operands may be K-major or MN-major, which gives forward (x.W^T), dgrad
// (dy.W) and wgrad (dy^T.x) without materialising a transpose.
//
// Counterpart in the reference stack: TransformerEngine's cuBLASLt GEMM and TEGroupedLinear used by
// the Megatron trainer (miles/backends/megatron_utils/model.py:560-570).
#include "gemm.h"

#include <cuda.h>
#include <stdio.h>
#include <string.h>

#include <mutex>
#include <string>

#include "pdl.cuh"
#include "ptx.cuh"

namespace mb {

namespace {

constexpr int BLOCK_M = 128;
constexpr int BLOCK_K = 64;  // 64 bf16 = 128 B = one swizzle row
constexpr int UMMA_K = 16;
constexpr int kThreads = 320;
constexpr int A_STAGE_BYTES = BLOCK_M * BLOCK_K * 2;

struct KArgs {
  int mode;
  int M, N, K;
  int num_groups;
  int max_tiles;
  const int* tile_group;
  const int* num_m_tiles;
  const int* group_offsets;
  void* c;
  long long ldc;
  long long c_group_stride;
  int accumulate;
  int out_fp32;
  int vec_ok;
  int* status;
  const unsigned long long* row_ptrs;
  unsigned long long* sig_ctrl;
  unsigned long long* sig_flags[8];
  int sig_nranks, sig_me;
  void* dest[8];
  int n_dest;
  void* gu;
  long long gu_ld;
  float4* score_part;
  const int* targets;
  float* score_target;
  float inv_temp;
};

enum Epilogue : int { EPI_PLAIN = 0, EPI_GLU = 1, EPI_SCORES = 2, EPI_ADD = 3 };

struct Tile {
  int a_mn0, b_mn0;  // M/N coordinates in the operand tensors
  int a_k0, b_k0;    // first contraction coordinate in each operand tensor
  int k_iters;
  int c_row0, c_col0;
  int row_end;  // rows >= row_end are not stored
  long long c_base;
};

// CG: CTAs that share a tile (BLOCK_M rows each). EPI_GLU: a tile is BLOCK_N / 2 gate columns and the up columns that go with them.
template <int BLOCK_N, bool B_MN, int CG, int EPI>
__device__ __forceinline__ int num_tiles_of(const KArgs& p) {
  const int n_tiles = (p.N + BLOCK_N - 1) / BLOCK_N;  // (of N / 2 by BLOCK_N / 2 as many)
  constexpr int TILE_M = BLOCK_M * CG;
  if (p.mode == GEMM_DENSE) return ((p.M + TILE_M - 1) / TILE_M) * n_tiles;
  if (p.mode == GEMM_GROUPED_ROWS) {
    int live = *p.num_m_tiles;
    const int cap = p.max_tiles;
    live = live < 0 ? 0 : (live > cap ? cap : live);
    return live * n_tiles;
  }
  return p.num_groups * ((p.M + TILE_M - 1) / TILE_M) * n_tiles;
}

// `rank`: of the CTA among those that share the tile; rows are its own, columns the whole tile's.
template <int BLOCK_N, bool B_MN, int CG, int EPI>
__device__ __forceinline__ Tile decode_tile(const KArgs& p, int t, int rank) {
  Tile r;
  constexpr int TILE_M = BLOCK_M * CG;
  constexpr int TILE_N = EPI == EPI_GLU ? BLOCK_N / 2 : BLOCK_N;  // columns of the output
  const int n_tiles = (p.N + BLOCK_N - 1) / BLOCK_N;
  const int m_tiles = (p.M + TILE_M - 1) / TILE_M;
  if (p.mode == GEMM_DENSE) {
    // Rasterise in bands of 8 row tiles so that concurrently running CTAs share B tiles in L2.
    constexpr int BAND = 8;
    const int per_band = BAND * n_tiles;
    const int band = t / per_band;
    const int first_m = band * BAND;
    const int band_rows = (m_tiles - first_m) < BAND ? (m_tiles - first_m) : BAND;
    const int in_band = t - band * per_band;
    const int mt = first_m + in_band % band_rows;
    const int nt = in_band / band_rows;
    r.a_mn0 = mt * TILE_M + rank * BLOCK_M;
    r.b_mn0 = nt * TILE_N;
    r.a_k0 = 0;
    r.b_k0 = 0;
    r.k_iters = (p.K + BLOCK_K - 1) / BLOCK_K;
    r.c_row0 = r.a_mn0;
    r.c_col0 = r.b_mn0;
    r.row_end = p.M;
    r.c_base = 0;
  } else if (p.mode == GEMM_GROUPED_ROWS) {
    const int mt = t / n_tiles;
    const int nt = t - mt * n_tiles;
    const int4 td = reinterpret_cast<const int4*>(p.tile_group)[mt];
    int g = td.x;
    g = g < 0 ? 0 : (g >= p.num_groups ? p.num_groups - 1 : g);
    r.a_mn0 = td.y < 0 ? 0 : td.y;
    r.row_end = min(p.M, r.a_mn0 + max(0, min(td.z, BLOCK_M)));
    r.a_k0 = 0;
    if (B_MN) {
      r.b_mn0 = nt * BLOCK_N;
      r.b_k0 = g * p.K;
    } else {
      r.b_mn0 = g * p.N + nt * TILE_N;
      r.b_k0 = 0;
    }
    r.k_iters = (p.K + BLOCK_K - 1) / BLOCK_K;
    r.c_row0 = r.a_mn0;
    r.c_col0 = nt * TILE_N;
    r.c_base = 0;
  } else {
    const int per_group = m_tiles * n_tiles;
    const int g = t / per_group;
    const int rem = t - g * per_group;
    const int mt = rem / n_tiles;
    const int nt = rem - mt * n_tiles;
    const int k_lo = p.group_offsets[g];
    const int k_hi = p.group_offsets[g + 1];
    r.a_mn0 = mt * TILE_M + rank * BLOCK_M;
    r.b_mn0 = nt * BLOCK_N;
    r.a_k0 = k_lo;
    r.b_k0 = k_lo;
    r.k_iters = k_hi > k_lo ? (k_hi - k_lo + BLOCK_K - 1) / BLOCK_K : 0;
    r.c_row0 = r.a_mn0;
    r.c_col0 = r.b_mn0;
    r.row_end = p.M;
    r.c_base = static_cast<long long>(g) * p.c_group_stride;
  }
  return r;
}

__device__ __forceinline__ void store_chunk(const KArgs& p, const Tile& t, int row, int col,
                                            const uint32_t (&acc)[32], bool zero) {
  if (row >= t.row_end) return;
  if (p.row_ptrs) {
    // scattered bf16 rows (possibly in a peer GPU's memory): N % 8 == 0 and 16-byte aligned rows are checked on the host
    const unsigned long long base = p.row_ptrs[row];
    if (base == 0ull) return;
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(base) + col;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (col + 8 * i + 8 <= p.N) {
        uint4 v;
        v.x = zero ? 0u : pack_bf16(__uint_as_float(acc[8 * i + 0]), __uint_as_float(acc[8 * i + 1]));
        v.y = zero ? 0u : pack_bf16(__uint_as_float(acc[8 * i + 2]), __uint_as_float(acc[8 * i + 3]));
        v.z = zero ? 0u : pack_bf16(__uint_as_float(acc[8 * i + 4]), __uint_as_float(acc[8 * i + 5]));
        v.w = zero ? 0u : pack_bf16(__uint_as_float(acc[8 * i + 6]), __uint_as_float(acc[8 * i + 7]));
        *reinterpret_cast<uint4*>(dst + 8 * i) = v;
      }
    }
    return;
  }
  const long long off = t.c_base + static_cast<long long>(row) * p.ldc + col;
  const bool full = (col + 32 <= p.N) && p.vec_ok;
  if (p.out_fp32) {
    float* dst = reinterpret_cast<float*>(p.c) + off;
    if (full) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float4 v;
        v.x = zero ? 0.f : __uint_as_float(acc[4 * i + 0]);
        v.y = zero ? 0.f : __uint_as_float(acc[4 * i + 1]);
        v.z = zero ? 0.f : __uint_as_float(acc[4 * i + 2]);
        v.w = zero ? 0.f : __uint_as_float(acc[4 * i + 3]);
        if (p.accumulate) {
          const float4 o = *reinterpret_cast<const float4*>(dst + 4 * i);
          v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
        *reinterpret_cast<float4*>(dst + 4 * i) = v;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (col + i < p.N) {
          float v = zero ? 0.f : __uint_as_float(acc[i]);
          if (p.accumulate) v += dst[i];
          dst[i] = v;
        }
      }
    }
  } else {
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.c) + off;
    if (full) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float f[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = zero ? 0.f : __uint_as_float(acc[8 * i + j]);
        if (p.accumulate) {
          const uint4 o = *reinterpret_cast<const uint4*>(dst + 8 * i);
          const __nv_bfloat162* ob = reinterpret_cast<const __nv_bfloat162*>(&o);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 of = __bfloat1622float2(ob[j]);
            f[2 * j] += of.x;
            f[2 * j + 1] += of.y;
          }
        }
        uint4 v;
        v.x = pack_bf16(f[0], f[1]);
        v.y = pack_bf16(f[2], f[3]);
        v.z = pack_bf16(f[4], f[5]);
        v.w = pack_bf16(f[6], f[7]);
        *reinterpret_cast<uint4*>(dst + 8 * i) = v;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (col + i < p.N) {
          float v = zero ? 0.f : __uint_as_float(acc[i]);
          if (p.accumulate) v += __bfloat162float(dst[i]);
          dst[i] = __float2bfloat16(v);
        }
      }
    }
  }
}

// ---- staged epilogue: a warp's 32 x (128 bytes) chunks pass through shared memory, so that every global access covers whole
// 128-byte (accumulating bf16: 64-byte) row segments instead of 32 pieces of 16 bytes, each its own wavefront, and so that the
// rows that are added to can be asked for several chunks ahead, the first ones while the tile is still being multiplied (weight
// gradients of few tokens, nothing but that read-modify-write, take the adding epilogue below). Without adding: 2048 x
// 151936 x 2048 to fp32 1122 -> 1014 us, 131072 expert rows of 768 x 2048 427 -> 376 us.
// `stg`: 4 KB of shared memory of this warp; 16-byte piece i of row r lies at piece i ^ (r & 7) (conflict-free both ways).
__device__ __forceinline__ void sts16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint4 lds16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}

// Columns of a chunk; instructions and rows per instruction of its global accesses.
template <bool FP32, bool ACC>
struct Chunk {
  static constexpr int COLS = (FP32 || ACC) ? 32 : 64;
  static constexpr int LANES = (FP32 || !ACC) ? 8 : 4;  // lanes that share a row, 16 bytes each
  static constexpr int INSTR = LANES;                   // 32 rows / (32 / LANES rows per instruction)
  static constexpr int AHEAD = FP32 ? 2 : 4;            // chunks whose old values are in flight (8 KB per warp)
};

// Old values of one chunk (rows past the end and columns past N read nothing).
template <bool FP32, bool ACC>
__device__ __forceinline__ void load_old(const KArgs& p, const Tile& t, int row0, int col, int lane, uint4 (&old)[Chunk<FP32, ACC>::INSTR]) {
  using C = Chunk<FP32, ACC>;
  constexpr int ESZ = FP32 ? 4 : 2;
  const int rows = t.row_end - row0 - lane / C::LANES;  // of this lane's rows: those it * (32 / LANES) below this exist
  const uint8_t* at = static_cast<const uint8_t*>(p.c) + (t.c_base + (row0 + lane / C::LANES) * p.ldc + col) * ESZ + (lane % C::LANES) * 16;
  const long long step = (32 / C::LANES) * p.ldc * ESZ;
#pragma unroll
  for (int it = 0; it < C::INSTR; ++it, at += step)
    if (it * (32 / C::LANES) < rows) old[it] = *reinterpret_cast<const uint4*>(at);
}

// Sixty-four bf16 columns of a warp's 32 rows, staged by its lanes, to global memory.
__device__ __forceinline__ void store_rows64(void* c, long long ld, int row0, int row_end, int col, int col_end, int lane, uint32_t stg) {
  __syncwarp();
  const int rows = row_end - row0 - lane / 8;
  uint8_t* at = static_cast<uint8_t*>(c) + ((row0 + lane / 8) * ld + col) * 2 + (lane & 7) * 16;
  const bool in = col + (lane & 7) * 8 + 8 <= col_end;
#pragma unroll
  for (int it = 0; it < 8; ++it, at += 8 * ld) {
    const int r = it * 4 + lane / 8;
    const uint4 v = lds16(stg + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
    if (in && it * 4 < rows) *reinterpret_cast<uint4*>(at) = v;
  }
  __syncwarp();
}

template <int BLOCK_N, bool FP32, bool ACC>
struct StagedEpilogue {
  using C = Chunk<FP32, ACC>;
  static constexpr int CHUNKS = BLOCK_N / C::COLS > 1 ? BLOCK_N / C::COLS / 2 : 1;  // of one warp: half a tile's
  static constexpr int AHEAD = CHUNKS < C::AHEAD ? CHUNKS : C::AHEAD;
  uint4 old[ACC ? AHEAD : 1][C::INSTR];

  __device__ __forceinline__ void begin(const KArgs& p, const Tile& t, int row0, int lane, int half) {
    if constexpr (ACC) {
      const int col0 = t.c_col0 + half * (CHUNKS * C::COLS);
#pragma unroll
      for (int c = 0; c < AHEAD; ++c)
        if (col0 + (c + 1) * C::COLS <= p.N) load_old<FP32, ACC>(p, t, row0, col0 + c * C::COLS, lane, old[c]);
    }
  }

  // Accumulating, the registers of a chunk that is done take the old values of the one AHEAD of it, be it of this tile or, if
  // `more`, of the next: the loads never drain between tiles. Returns whether the next tile's first AHEAD chunks are on their way.
  __device__ __forceinline__ bool run(const KArgs& p, const Tile& t, const Tile& next, bool more, int row0, int next_row0, int lane, int half,
                                      uint32_t t_addr, uint32_t stg) {
    constexpr int ESZ = FP32 ? 4 : 2;
    static_assert(CHUNKS % AHEAD == 0, "a chunk's registers are the same in every tile");
    if (half * CHUNKS * C::COLS >= BLOCK_N) return false;  // (a tile of one chunk)
    t_addr += half * (CHUNKS * C::COLS);
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int col = t.c_col0 + (half * CHUNKS + c) * C::COLS;
      if (col >= p.N) return false;  // warp-uniform
      if (col + C::COLS > p.N) {  // the last, partial chunk
#pragma unroll
        for (int h = 0; h < C::COLS; h += 32)
          if (col + h < p.N) {
            uint32_t acc[32];
            tmem_ld_32x32(t_addr + c * C::COLS + h, acc);
            tmem_ld_wait();
            store_chunk(p, t, row0 + lane, col + h, acc, false);
          }
        return false;
      }
      const uint32_t mine = stg + lane * 128, x = lane & 7;
      if constexpr (FP32 || ACC) {
        uint32_t acc[32];
        tmem_ld_32x32(t_addr + c * 32, acc);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) sts16(mine + ((i ^ x) << 4), acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
      } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t acc[32];
          tmem_ld_32x32(t_addr + c * 64 + h * 32, acc);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float* f = reinterpret_cast<const float*>(acc) + 8 * i;
            sts16(mine + (((h * 4 + i) ^ x) << 4), pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
          }
        }
      }
      __syncwarp();
      const int rows = t.row_end - row0 - lane / C::LANES;
      uint8_t* at = static_cast<uint8_t*>(p.c) + (t.c_base + (row0 + lane / C::LANES) * p.ldc + col) * ESZ + (lane % C::LANES) * 16;
      const long long step = (32 / C::LANES) * p.ldc * ESZ;
#pragma unroll
      for (int it = 0; it < C::INSTR; ++it, at += step) {
        const int r = it * (32 / C::LANES) + lane / C::LANES;
        const uint32_t from = stg + r * 128, sx = r & 7;
        uint4 v;
        if constexpr (FP32 || !ACC) {
          v = lds16(from + (((lane & 7) ^ sx) << 4));
          if constexpr (ACC) {
            const uint4 o = old[c % AHEAD][it];
            v.x = __float_as_uint(__uint_as_float(v.x) + __uint_as_float(o.x));
            v.y = __float_as_uint(__uint_as_float(v.y) + __uint_as_float(o.y));
            v.z = __float_as_uint(__uint_as_float(v.z) + __uint_as_float(o.z));
            v.w = __float_as_uint(__uint_as_float(v.w) + __uint_as_float(o.w));
          }
        } else {  // eight fp32 sums and eight old bf16 values: added in fp32, rounded once
          const uint4 a = lds16(from + (((2 * (lane & 3)) ^ sx) << 4)), b = lds16(from + (((2 * (lane & 3) + 1) ^ sx) << 4));
          const uint4 o = old[c % AHEAD][it];
          const __nv_bfloat162* ob = reinterpret_cast<const __nv_bfloat162*>(&o);
          const float2 o0 = __bfloat1622float2(ob[0]), o1 = __bfloat1622float2(ob[1]), o2 = __bfloat1622float2(ob[2]), o3 = __bfloat1622float2(ob[3]);
          v.x = pack_bf16(__uint_as_float(a.x) + o0.x, __uint_as_float(a.y) + o0.y);
          v.y = pack_bf16(__uint_as_float(a.z) + o1.x, __uint_as_float(a.w) + o1.y);
          v.z = pack_bf16(__uint_as_float(b.x) + o2.x, __uint_as_float(b.y) + o2.y);
          v.w = pack_bf16(__uint_as_float(b.z) + o3.x, __uint_as_float(b.w) + o3.y);
        }
        if (it * (32 / C::LANES) < rows) *reinterpret_cast<uint4*>(at) = v;
      }
      if constexpr (ACC) {
        if (c + AHEAD < CHUNKS) {
          if (col + (AHEAD + 1) * C::COLS <= p.N) load_old<FP32, ACC>(p, t, row0, col + AHEAD * C::COLS, lane, old[c % AHEAD]);
        } else if (more) {
          const int ncol = next.c_col0 + (half * CHUNKS + c + AHEAD - CHUNKS) * C::COLS;
          if (ncol + C::COLS <= p.N) load_old<FP32, ACC>(p, next, next_row0, ncol, lane, old[c % AHEAD]);
        }
      }
      __syncwarp();
    }
    return more;
  }
};

// ---- adding epilogue (EPI_ADD): the rows that are added to come by `cp.async` into the buffers in which they are added to and from
// which they leave, a piece of 32 rows x 128 bytes each, one or two of them a warp; a piece that has left makes room for the next one
// without a buffer, of this tile or the next. Bound by reading and writing C where the contraction is short. Old values in registers
// (StagedEpilogue) are asked for as early, but a warp has to wait for all of its loads to have the first of them: 128 experts of
// 1536 x 2048 in bf16, 777 tokens over them with eight experts each 463 -> 281 us (1.6 GB: 5.7 TB/s), 4096 tokens 428 -> 340, 8192 527 -> 465;
// in fp32, by pairs, 151936 x 2048 with 776 tokens 652 -> 561 us (2.5 GB), 5120 x 2048 with 16384 333 -> 316, 24576 x 4096 with 9216 1256 -> 1201.

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Buffers of a warp: one beside the four stages of a 256-wide tile of one CTA, which take the room of the second.
constexpr int add_buffers(int block_n, int stages, int cg) { return block_n == 256 && cg == 1 && stages == 4 ? 1 : 2; }

template <int BLOCK_N, bool FP32, int BUFFERS>
struct AddEpilogue {
  static constexpr int ESZ = FP32 ? 4 : 2;
  static constexpr int COLS = 128 / ESZ;                // of a piece
  static constexpr int PIECES = BLOCK_N / 2 / COLS;     // of one warp: half a tile's
  static constexpr int AHEAD = PIECES < BUFFERS ? PIECES : BUFFERS;
  static_assert(PIECES % AHEAD == 0, "a piece's buffer is the same in every tile");

  // Asks for piece c of the warp's half of a tile (rows past the end and pieces past column N, a multiple of COLS, read nothing) and closes the group.
  static __device__ __forceinline__ void ask(const KArgs& p, const Tile& t, int row0, int c, int lane, int half, uint32_t stg) {
    const int col = t.c_col0 + (half * PIECES + c) * COLS;
    if (col < p.N) {
      const int rows = t.row_end - row0 - lane / 8;
      const uint8_t* at = static_cast<const uint8_t*>(p.c) + (t.c_base + (row0 + lane / 8) * p.ldc + col) * ESZ + (lane & 7) * 16;
      const long long step = 4 * p.ldc * ESZ;
#pragma unroll
      for (int it = 0; it < 8; ++it, at += step) {
        const int r = it * 4 + lane / 8;
        if (it * 4 < rows) cp_async16(stg + r * 128 + (((lane & 7) ^ (r & 7)) << 4), at);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // The tile's first AHEAD pieces have been asked for; afterwards those of `next` have, if `more`.
  static __device__ __forceinline__ void run(const KArgs& p, const Tile& t, const Tile& next, bool more, int row0, int next_row0, int lane,
                                             int half, uint32_t t_addr, uint32_t stg0) {
    t_addr += half * (BLOCK_N / 2);
#pragma unroll 1
    for (int c = 0; c < PIECES; ++c) {
      const int col = t.c_col0 + (half * PIECES + c) * COLS;
      const uint32_t stg = stg0 + (c % AHEAD) * 4096;
      asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD - 1) : "memory");
      __syncwarp();
      if (col < p.N) {  // warp-uniform
        const uint32_t mine = stg + lane * 128, x = lane & 7;
#pragma unroll
        for (int h = 0; h < COLS / 32; ++h) {
          uint32_t acc[32];
          tmem_ld_32x32(t_addr + c * COLS + h * 32, acc);
          tmem_ld_wait();
          const float* f = reinterpret_cast<const float*>(acc);
          if constexpr (FP32) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const uint4 o = lds16(mine + ((i ^ x) << 4));
              sts16(mine + ((i ^ x) << 4), __float_as_uint(f[4 * i] + __uint_as_float(o.x)), __float_as_uint(f[4 * i + 1] + __uint_as_float(o.y)),
                    __float_as_uint(f[4 * i + 2] + __uint_as_float(o.z)), __float_as_uint(f[4 * i + 3] + __uint_as_float(o.w)));
            }
          } else {  // added in fp32, rounded once
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t at = mine + (((h * 4 + i) ^ x) << 4);
              const uint4 o = lds16(at);
              const __nv_bfloat162* ob = reinterpret_cast<const __nv_bfloat162*>(&o);
              const float2 o0 = __bfloat1622float2(ob[0]), o1 = __bfloat1622float2(ob[1]), o2 = __bfloat1622float2(ob[2]), o3 = __bfloat1622float2(ob[3]);
              sts16(at, pack_bf16(f[8 * i] + o0.x, f[8 * i + 1] + o0.y), pack_bf16(f[8 * i + 2] + o1.x, f[8 * i + 3] + o1.y),
                    pack_bf16(f[8 * i + 4] + o2.x, f[8 * i + 5] + o2.y), pack_bf16(f[8 * i + 6] + o3.x, f[8 * i + 7] + o3.y));
            }
          }
        }
        __syncwarp();
        const int rows = t.row_end - row0 - lane / 8;
        uint8_t* at = static_cast<uint8_t*>(p.c) + (t.c_base + (row0 + lane / 8) * p.ldc + col) * ESZ + (lane & 7) * 16;
        const long long step = 4 * p.ldc * ESZ;
#pragma unroll
        for (int it = 0; it < 8; ++it, at += step) {
          const int r = it * 4 + lane / 8;
          const uint4 v = lds16(stg + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
          if (it * 4 < rows) *reinterpret_cast<uint4*>(at) = v;
        }
        __syncwarp();
      }
      const bool own = c + AHEAD < PIECES;
      if (own || more) ask(p, own ? t : next, own ? row0 : next_row0, own ? c + AHEAD : c + AHEAD - PIECES, lane, half, stg);
      else asm volatile("cp.async.commit_group;" ::: "memory");
    }
  }
};

// CG = 2: a pair of CTAs (a cluster) multiplies 256 x 256 tiles with `cta_group::2`: each holds its 128 rows of A and half of B's,
// so that a tile's operands are read from shared memory, and from L2, two thirds as often for the same work. That is what bounds the
// one-CTA tile: per 16 of K it reads 12 KB of shared memory and receives another 12 KB in the 128 clocks of its product (at 128 bytes
// a clock), and under the power cap those reads cost clock. The CTA of rank 0 issues; its `full` barrier counts both CTAs' copies, its
// `tempty` both epilogues; `empty` and `tfull` are raised in both by its commits. Sums are those of one CTA bit for bit.
// Measured over seconds, at the power cap, TFLOP/s one CTA -> pair: 8192^3 1181 -> 1283 (cuBLAS 1372), 16384 x 5120 x 2048 1170 ->
// 1233, 9216 x 24576 x 4096 1202 -> 1288, its weight gradient 1116 -> 1209, 2048 x 151936 x 2048 to fp32 1044 -> 1159. Grouped
// contractions gain nothing (131072 rows over 128 experts 872 and 893, 65536 rows 668 and 656) and stay with one CTA.
//
// EPI_GLU: the accumulator of a tile holds 128 gate columns and their 128 up columns, and silu(gate) * up leaves instead of them (or
// beside them, for a backward): rounded to bf16 before the activation, as the separate kernel reads them, so the same bits. What it
// saves is the activation's launch and its pass over gate and up. 131072 rows over 128 experts
// of 768 x 2048: 931 -> 741 us (924 with gate and up kept), 65536 rows 492 -> 386 (429), 8000 rows 162 -> 144.
//
// EPI_SCORES: the log-probabilities of an LM head need three numbers per row of its 150 thousand logits. Every thread of the
// epilogue keeps maximum, sum of exponentials and their first moment about the maximum over 128 columns of its row, and
// logprob.cu merges them: the logits need not be written, or not be read again. Scores of 12288
// rows over 151936 x 2048 (in chunks of 2048 with their logits in fp32 through memory before): a pass of 16384 tokens 30.3 -> 28.8 ms.
template <int BLOCK_N, bool A_MN, bool B_MN, int STAGES, int CG, int EPI>
__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                 const KArgs p) {
  constexpr bool GLU = EPI == EPI_GLU, SCORES = EPI == EPI_SCORES;
  constexpr int ADD_BUFFERS = add_buffers(BLOCK_N, STAGES, CG);
  constexpr int B_ROWS = BLOCK_N / CG;  // of this CTA
  constexpr int B_STAGE_BYTES = B_ROWS * BLOCK_K * 2;
  constexpr uint32_t TMEM_COLS = 2 * BLOCK_N;  // 256 or 512: a power of two >= 32
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t a_smem = smem_base;
  const uint32_t b_smem = a_smem + STAGES * A_STAGE_BYTES;
  const uint32_t bar_base = b_smem + STAGES * B_STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  const uint32_t tmem_slot = bar_base + 8u * (2 * STAGES + 4);
  const uint32_t stage_buf = (bar_base + 8u * (2 * STAGES + 5) + 127u) & ~127u;  // epilogue staging, 4 KB per warp (whole rows of a 128-wide tile: 8 KB of every second one)
  __shared__ int abort_flag_s;
  __shared__ uint32_t tmem_base_s;
  volatile int* abort_flag = &abort_flag_s;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = CG == 2 ? static_cast<int>(cluster_ctarank()) : 0;
  const int first_tile = blockIdx.x / CG, tile_step = gridDim.x / CG;

  if (threadIdx.x == 0) {
    abort_flag_s = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar(a), 1);
      mbar_init(tempty_bar(a), 8 * CG);  // one arrive per epilogue warp
    }
    fence_barrier_init();
    prefetch_tensormap(&tma_a);
    prefetch_tensormap(&tma_b);
  }
  if (warp == 1) {
    if constexpr (CG == 2) {
      tmem_alloc_pair(tmem_slot, TMEM_COLS);
    } else {
      tmem_alloc(tmem_slot, TMEM_COLS);
      tmem_relinquish();
    }
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
  const uint32_t tmem_base = tmem_base_s;
  if constexpr (CG == 2) cluster_sync_all();  // both CTAs' barriers and TMEM are there before either uses the other's
  pdl_enter();

  const int total_tiles = num_tiles_of<BLOCK_N, B_MN, CG, EPI>(p);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      const auto load = [](uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
        if constexpr (CG == 2) tma_load_2d_pair(dst, map, bar, c0, c1);
        else tma_load_2d(dst, map, bar, c0, c1);
      };
      for (int t = first_tile; ok && t < total_tiles; t += tile_step) {
        const Tile tl = decode_tile<BLOCK_N, B_MN, CG, EPI>(p, t, rank);
        const int b_mn0 = tl.b_mn0 + rank * (GLU ? p.N / 2 : B_ROWS);  // (GLU, a pair: gate rows in the first CTA, up rows in the other)
        for (int kb = 0; kb < tl.k_iters; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.status, ERR_WAIT_EMPTY)) {
            ok = false;
            break;
          }
          if (rank == 0) mbar_expect_tx(full_bar(stage), CG * (A_STAGE_BYTES + B_STAGE_BYTES));
          const uint32_t full = CG == 2 ? map_to_rank(full_bar(stage), 0) : full_bar(stage);
          const uint32_t a_dst = a_smem + stage * A_STAGE_BYTES;
          const uint32_t b_dst = b_smem + stage * B_STAGE_BYTES;
          const int ka = tl.a_k0 + kb * BLOCK_K;
          const int kbb = tl.b_k0 + kb * BLOCK_K;
          if (A_MN) {
#pragma unroll
            for (int i = 0; i < BLOCK_M / 64; ++i) load(a_dst + i * (BLOCK_K * 128), &tma_a, full, tl.a_mn0 + 64 * i, ka);
          } else {
            load(a_dst, &tma_a, full, ka, tl.a_mn0);
          }
          if (B_MN) {
#pragma unroll
            for (int i = 0; i < B_ROWS / 64; ++i) load(b_dst + i * (BLOCK_K * 128), &tma_b, full, b_mn0 + 64 * i, kbb);
          } else {
            load(b_dst, &tma_b, full, kbb, b_mn0);
            if (GLU && CG == 1) load(b_dst + BLOCK_N / 2 * (BLOCK_K * 2), &tma_b, full, kbb, b_mn0 + p.N / 2);
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if constexpr (CG == 2) {  // the other CTA's commits have arrived before this one leaves
        for (int s = 0; ok && s < STAGES; ++s) {
          ok = mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.status, ERR_WAIT_EMPTY);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (!ok) {
        // Give copies that are already in flight a bounded chance to land before smem is released.
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 2000000ull) {
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    constexpr uint32_t idesc = make_idesc_bf16(BLOCK_M * CG, BLOCK_N, A_MN, B_MN);
    const auto commit = [](uint32_t bar) {
      if constexpr (CG == 2) umma_commit_pair(bar);
      else umma_commit(bar);
    };
    int stage = 0;
    uint32_t phase = 0;
    int iter = 0;  // counts only tiles that use an accumulator, so both roles stay in phase
    bool ok = true;
    for (int t = first_tile; ok && rank == 0 && t < total_tiles; t += tile_step) {
      const Tile tl = decode_tile<BLOCK_N, B_MN, CG, EPI>(p, t, rank);
      if (tl.k_iters == 0) continue;  // epilogue writes zeros without touching TMEM
      const int acc = iter & 1;
      const uint32_t acc_phase = (iter >> 1) & 1u;
      if (!mbar_wait(tempty_bar(acc), acc_phase ^ 1u, abort_flag, p.status, ERR_WAIT_TMEM_EMPTY)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + acc * BLOCK_N;
      for (int kb = 0; kb < tl.k_iters; ++kb) {
        if (!mbar_wait(full_bar(stage), phase, abort_flag, p.status, ERR_WAIT_FULL)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (lane == 0) {
          const uint32_t a_addr = a_smem + stage * A_STAGE_BYTES;
          const uint32_t b_addr = b_smem + stage * B_STAGE_BYTES;
#pragma unroll
          for (int k = 0; k < BLOCK_K / UMMA_K; ++k) {
            const uint64_t adesc = A_MN ? make_smem_desc(a_addr + k * UMMA_K * 128, BLOCK_K * 128, 1024)
                                        : make_smem_desc(a_addr + k * UMMA_K * 2, 16, 1024);
            const uint64_t bdesc = B_MN ? make_smem_desc(b_addr + k * UMMA_K * 128, BLOCK_K * 128, 1024)
                                        : make_smem_desc(b_addr + k * UMMA_K * 2, 16, 1024);
            if constexpr (CG == 2) umma_f16_pair(d_tmem, adesc, bdesc, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            else umma_f16(d_tmem, adesc, bdesc, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          commit(empty_bar(stage));
        }
        __syncwarp();
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok && lane == 0) commit(tfull_bar(acc));
      __syncwarp();
      ++iter;
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quad = warp & 3;  // TMEM lane quadrant this warp may read
    const int half = (warp - 2) >> 2;
    const bool staged = BLOCK_N >= 64 && p.vec_ok && !p.row_ptrs && p.n_dest == 0;
    int iter = 0;
    bool ok = true;
    const auto release = [&](int acc) {  // this warp's share of the accumulator has been read
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2 && rank != 0) mbar_arrive_remote(map_to_rank(tempty_bar(acc), 0));
        else mbar_arrive(tempty_bar(acc));
      }
    };
    auto add_tiles = [&](auto e) {
      const uint32_t stg = stage_buf + static_cast<uint32_t>(warp - 2) * 4096;
      int ready = -1;  // the tile whose first old values are on their way
      for (int t = first_tile; t < total_tiles; t += tile_step) {
        const Tile tl = decode_tile<BLOCK_N, B_MN, CG, EPI>(p, t, rank);
        if (tl.k_iters == 0) continue;
        const int row0 = tl.c_row0 + quad * 32, acc = iter & 1, tn = t + tile_step;
        if (ready != t) e.begin(p, tl, row0, lane, half);
        const Tile next = decode_tile<BLOCK_N, B_MN, CG, EPI>(p, tn < total_tiles ? tn : t, rank);
        const bool more = tn < total_tiles && next.k_iters > 0;
        if (!__all_sync(0xffffffffu, mbar_wait(tfull_bar(acc), (iter >> 1) & 1u, abort_flag, p.status, ERR_WAIT_TMEM_FULL))) break;
        tc_fence_after();
        const uint32_t t_addr = tmem_base + acc * BLOCK_N + (static_cast<uint32_t>(quad * 32) << 16);
        ready = e.run(p, tl, next, more, row0, next.c_row0 + quad * 32, lane, half, t_addr, stg) ? tn : -1;
        release(acc);
        ++iter;
      }
    };
    if constexpr (EPI == EPI_ADD) {
      const uint32_t stg = stage_buf + static_cast<uint32_t>(warp - 2) * (ADD_BUFFERS * 4096);
      auto add_pieces = [&](auto e) {
        using E = decltype(e);
        bool asked = false;  // the next tile's first pieces
        for (int t = first_tile; t < total_tiles; t += tile_step) {
          const Tile tl = decode_tile<BLOCK_N, B_MN, CG, EPI>(p, t, rank);
          if (tl.k_iters == 0) continue;
          const int row0 = tl.c_row0 + quad * 32, acc = iter & 1, tn = t + tile_step;
          if (!asked)
            for (int c = 0; c < E::AHEAD; ++c) E::ask(p, tl, row0, c, lane, half, stg + c * 4096);
          const Tile next = decode_tile<BLOCK_N, B_MN, CG, EPI>(p, tn < total_tiles ? tn : t, rank);
          asked = tn < total_tiles && next.k_iters > 0;
          if (!__all_sync(0xffffffffu, mbar_wait(tfull_bar(acc), (iter >> 1) & 1u, abort_flag, p.status, ERR_WAIT_TMEM_FULL))) break;
          tc_fence_after();
          E::run(p, tl, next, asked, row0, next.c_row0 + quad * 32, lane, half,
                 tmem_base + acc * BLOCK_N + (static_cast<uint32_t>(quad * 32) << 16), stg);
          release(acc);
          ++iter;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      };
      if (p.out_fp32) add_pieces(AddEpilogue<BLOCK_N, true, ADD_BUFFERS>());
      else add_pieces(AddEpilogue<BLOCK_N, false, ADD_BUFFERS>());
    }
    const bool adds = EPI == EPI_ADD || (EPI == EPI_PLAIN && staged && p.accumulate);
    if constexpr (BLOCK_N >= 64 && EPI == EPI_PLAIN) {
      if (adds && p.out_fp32) add_tiles(StagedEpilogue<BLOCK_N, true, true>());
      else if (adds) add_tiles(StagedEpilogue<BLOCK_N, false, true>());
    }
    for (int t = first_tile; ok && !adds && t < total_tiles; t += tile_step) {
      const Tile tl = decode_tile<BLOCK_N, B_MN, CG, EPI>(p, t, rank);
      const int row = tl.c_row0 + quad * 32 + lane;
      int target = -1;
      if (SCORES && row < tl.row_end) target = p.targets[row];
      uint32_t acc_regs[32];
      if (tl.k_iters == 0) {
        if (!p.accumulate) {
#pragma unroll 1
          for (int c = half; c < BLOCK_N / 32; c += 2)
            if (tl.c_col0 + c * 32 < p.N) store_chunk(p, tl, row, tl.c_col0 + c * 32, acc_regs, true);
        }
        continue;
      }
      const int acc = iter & 1;
      const uint32_t acc_phase = (iter >> 1) & 1u;
      const uint32_t t_addr = tmem_base + acc * BLOCK_N + (static_cast<uint32_t>(quad * 32) << 16);
      if (!mbar_wait(tfull_bar(acc), acc_phase, abort_flag, p.status, ERR_WAIT_TMEM_FULL)) {
        ok = false;
        break;
      }
      tc_fence_after();
      if constexpr (SCORES) {
        const uint32_t stg = stage_buf + static_cast<uint32_t>(warp - 2) * 4096;
        const int row0 = tl.c_row0 + quad * 32, col0 = tl.c_col0 + half * (BLOCK_N / 2);
        float m = -3.402823466e38f, s = 0.f, sy = 0.f;
#pragma unroll 1
        for (int c = 0; c < BLOCK_N / 64; ++c) {
          const int col = col0 + c * 32;
          if (col >= p.N) break;  // warp-uniform
          tmem_ld_32x32(t_addr + half * (BLOCK_N / 2) + c * 32, acc_regs);
          tmem_ld_wait();
          if (p.c) {
            if (p.vec_ok && col + 32 <= p.N) {  // rows of 128 bytes, through shared memory
              const uint32_t mine = stg + lane * 128, x = lane & 7;
#pragma unroll
              for (int i = 0; i < 8; ++i) sts16(mine + ((i ^ x) << 4), acc_regs[4 * i], acc_regs[4 * i + 1], acc_regs[4 * i + 2], acc_regs[4 * i + 3]);
              __syncwarp();
              const int rows = tl.row_end - row0 - lane / 8;
              float* at = static_cast<float*>(p.c) + (row0 + lane / 8) * p.ldc + col + (lane & 7) * 4;
#pragma unroll
              for (int it = 0; it < 8; ++it, at += 4 * p.ldc) {
                const int r = it * 4 + lane / 8;
                const uint4 v = lds16(stg + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
                if (it * 4 < rows) *reinterpret_cast<uint4*>(at) = v;
              }
              __syncwarp();
            } else {
              store_chunk(p, tl, row, col, acc_regs, false);
            }
          }
          float v[32], mx = m;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            v[i] = col + i < p.N ? __uint_as_float(acc_regs[i]) * p.inv_temp : -3.402823466e38f;
            mx = fmaxf(mx, v[i]);
          }
          if (target >= col && target < col + 32) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (target == col + i) p.score_target[row] = v[i];
          }
          const float scale = __expf(m - mx);
          sy = scale * (sy + s * (s > 0.f ? m - mx : 0.f));
          s *= scale;
          m = mx;
          float ps[4] = {0.f, 0.f, 0.f, 0.f}, py[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float y = v[i] - m, e = __expf(y);
            ps[i & 3] += e;
            if (e > 0.f) py[i & 3] += e * y;  // (a masked column's y is -infinity)
          }
          s += (ps[0] + ps[1]) + (ps[2] + ps[3]);
          sy += (py[0] + py[1]) + (py[2] + py[3]);
        }
        if (row < tl.row_end && col0 < p.N) p.score_part[static_cast<long long>(col0 / (BLOCK_N / 2)) * p.M + row] = make_float4(m, s, sy, 0.f);
      } else if constexpr (GLU) {
        const uint32_t stg = stage_buf + static_cast<uint32_t>(warp - 2) * 4096;
        const int row0 = tl.c_row0 + quad * 32, col = tl.c_col0 + half * 64, width = p.N / 2;
        if (row0 >= tl.row_end) {  // (warp-uniform; the tiles of a few rows that decode steps have leave three of four quadrants empty)
          release(acc);
          ++iter;
          continue;
        }
        // Sixteen columns at a time in a rolled loop: unrolled, the activation is thousands of instructions, which a launch of a few
        // tiles per CTA fetches cold (4000 rows of 8 choices over 128 experts 242 -> 232 us).
        const uint32_t mine = stg + lane * 128, x = lane & 7;
        const auto pass = [&](void* c, long long ld, bool gate, bool up) {  // gate columns, up columns, or silu(gate) * up of both
#pragma unroll 1
          for (int i = 0; i < 4; ++i) {
            uint32_t g[16], u[16];
            if (gate) tmem_ld_32x16(t_addr + half * 64 + i * 16, g);
            if (up) tmem_ld_32x16(t_addr + BLOCK_N / 2 + half * 64 + i * 16, u);
            tmem_ld_wait();
            uint32_t w[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint32_t gw = gate ? pack_bf16(__uint_as_float(g[2 * j]), __uint_as_float(g[2 * j + 1])) : 0u;
              const uint32_t uw = up ? pack_bf16(__uint_as_float(u[2 * j]), __uint_as_float(u[2 * j + 1])) : 0u;
              if (gate && up) {
                const float2 gf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&gw));
                const float2 uf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&uw));
                w[j] = pack_bf16(gf.x / (1.f + __expf(-gf.x)) * uf.x, gf.y / (1.f + __expf(-gf.y)) * uf.y);
              } else {
                w[j] = gate ? gw : uw;
              }
            }
            sts16(mine + (((2 * i) ^ x) << 4), w[0], w[1], w[2], w[3]);
            sts16(mine + (((2 * i + 1) ^ x) << 4), w[4], w[5], w[6], w[7]);
          }
          store_rows64(c, ld, row0, tl.row_end, col, width, lane, stg);
        };
        if (p.gu) {
          pass(p.gu, p.gu_ld, true, false);
          pass(static_cast<__nv_bfloat16*>(p.gu) + width, p.gu_ld, false, true);
        }
        pass(p.c, p.ldc, true, true);
      } else if (BLOCK_N == 128 && (p.n_dest > 0 || p.row_ptrs) && half == 1) {
        // (one warp per quadrant stages whole rows below)
      } else if (BLOCK_N == 128 && p.n_dest > 0) {
        // Replicated tile (tensor-parallel partial sums): same staging, every row segment goes to each destination.
        const uint32_t stg = stage_buf + static_cast<uint32_t>(quad) * (32 * 256);
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          tmem_ld_32x32(t_addr + c * 32, acc_regs);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t v0 = pack_bf16(__uint_as_float(acc_regs[8 * i + 0]), __uint_as_float(acc_regs[8 * i + 1]));
            const uint32_t v1 = pack_bf16(__uint_as_float(acc_regs[8 * i + 2]), __uint_as_float(acc_regs[8 * i + 3]));
            const uint32_t v2 = pack_bf16(__uint_as_float(acc_regs[8 * i + 4]), __uint_as_float(acc_regs[8 * i + 5]));
            const uint32_t v3 = pack_bf16(__uint_as_float(acc_regs[8 * i + 6]), __uint_as_float(acc_regs[8 * i + 7]));
            const uint32_t chunk = static_cast<uint32_t>(c * 4 + i) ^ static_cast<uint32_t>(lane & 7);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stg + lane * 256 + chunk * 16), "r"(v0), "r"(v1),
                         "r"(v2), "r"(v3)
                         : "memory");
          }
        }
        __syncwarp();
#pragma unroll 1
        for (int it = 0; it < 16; ++it) {
          const int rl = it * 2 + (lane >> 4);
          const int ch = lane & 15;
          uint4 v;
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                       : "r"(stg + rl * 256 + ((ch ^ (rl & 7)) * 16)));
          const int grow = tl.c_row0 + quad * 32 + rl;
          const int col = tl.c_col0 + ch * 8;
          if (grow < tl.row_end && col + 8 <= p.N) {
            const long long off = static_cast<long long>(grow) * p.ldc + col;
            for (int d = 0; d < p.n_dest; ++d) *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.dest[d]) + off) = v;
          }
        }
        __syncwarp();
      } else if (BLOCK_N == 128 && p.row_ptrs) {
        // Scattered rows (expert-parallel return): pass the warp's 32 x 128 block through shared memory so that
        // every store instruction writes two whole 256-byte row segments instead of thirty-two 64-byte pieces;
        // over NVLink the size of a write decides how much of the link carries payload.
        const uint32_t stg = stage_buf + static_cast<uint32_t>(quad) * (32 * 256);
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          tmem_ld_32x32(t_addr + c * 32, acc_regs);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t v0 = pack_bf16(__uint_as_float(acc_regs[8 * i + 0]), __uint_as_float(acc_regs[8 * i + 1]));
            const uint32_t v1 = pack_bf16(__uint_as_float(acc_regs[8 * i + 2]), __uint_as_float(acc_regs[8 * i + 3]));
            const uint32_t v2 = pack_bf16(__uint_as_float(acc_regs[8 * i + 4]), __uint_as_float(acc_regs[8 * i + 5]));
            const uint32_t v3 = pack_bf16(__uint_as_float(acc_regs[8 * i + 6]), __uint_as_float(acc_regs[8 * i + 7]));
            const uint32_t chunk = static_cast<uint32_t>(c * 4 + i) ^ static_cast<uint32_t>(lane & 7);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stg + lane * 256 + chunk * 16), "r"(v0), "r"(v1),
                         "r"(v2), "r"(v3)
                         : "memory");
          }
        }
        const unsigned long long my_ptr = (row < tl.row_end) ? p.row_ptrs[row] : 0ull;
        __syncwarp();
#pragma unroll 1
        for (int it = 0; it < 16; ++it) {
          const int rl = it * 2 + (lane >> 4);
          const int ch = lane & 15;
          const unsigned long long base = __shfl_sync(0xffffffffu, my_ptr, rl);
          uint4 v;
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                       : "r"(stg + rl * 256 + ((ch ^ (rl & 7)) * 16)));
          const int col = tl.c_col0 + ch * 8;
          if (base != 0ull && col + 8 <= p.N) *reinterpret_cast<uint4*>(base + static_cast<unsigned long long>(col) * 2) = v;
        }
        __syncwarp();
      } else if (!staged) {
#pragma unroll 1
        for (int c = half; c < BLOCK_N / 32; c += 2) {
          if (tl.c_col0 + c * 32 >= p.N) break;  // warp-uniform
          tmem_ld_32x32(t_addr + c * 32, acc_regs);
          tmem_ld_wait();
          store_chunk(p, tl, row, tl.c_col0 + c * 32, acc_regs, false);
        }
      } else if constexpr (BLOCK_N >= 64) {
        const uint32_t stg = stage_buf + static_cast<uint32_t>(warp - 2) * 4096;
        const int row0 = tl.c_row0 + quad * 32;
        if (p.out_fp32) {
          StagedEpilogue<BLOCK_N, true, false> e;
          e.run(p, tl, tl, false, row0, row0, lane, half, t_addr, stg);
        } else {
          StagedEpilogue<BLOCK_N, false, false> e;
          e.run(p, tl, tl, false, row0, row0, lane, half, t_addr, stg);
        }
      }
      release(acc);
      ++iter;
    }
    if (p.row_ptrs || p.n_dest > 0) __threadfence_system();  // peer stores are visible before the CTA reports in
  }

  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) cluster_sync_all();  // neither CTA leaves while the other's products, copies or arrivals may reach it
  if (warp == 1) {
    tc_fence_after();
    if constexpr (CG == 2) tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (p.sig_ctrl && threadIdx.x == 0) {
    __threadfence_system();
    const unsigned long long done = atomicAdd(&p.sig_ctrl[5], 1ull);
    if (done == gridDim.x - 1) {  // every CTA has stored and fenced: raise the return flags of this epoch
      __threadfence_system();
      const unsigned long long epoch = p.sig_ctrl[2] + 1;
      for (int d = 0; d < p.sig_nranks; ++d)
        asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p.sig_flags[d] + p.sig_me), "l"(epoch) : "memory");
      p.sig_ctrl[5] = 0;
      p.sig_ctrl[2] = epoch;
    }
  }
}

// ---------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

std::string g_err;
EncodeTiledFn g_encode = nullptr;
std::once_flag g_once;

EncodeTiledFn get_encode() {
  std::call_once(g_once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  });
  return g_encode;
}

int fail(const std::string& m) {
  g_err = m;
  return -1;
}

}  // namespace

int gemm_fail(const std::string& m) { return fail(m); }

// 2-D bf16 tensor map over a row-major [rows, cols] matrix with a [box_rows, 64] box.
int gemm_make_map(CUtensorMap* map, const GemmOperand& op, int box_rows) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return fail("cuTensorMapEncodeTiled is not available");
  if ((reinterpret_cast<uintptr_t>(op.ptr) & 15) != 0) return fail("operand base must be 16-byte aligned");
  if ((op.ld * 2) % 16 != 0) return fail("operand row pitch must be a multiple of 16 bytes");
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(op.cols), static_cast<cuuint64_t>(op.rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(op.ld) * 2};
  cuuint32_t box[2] = {64u, static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1u, 1u};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(op.ptr), dims, strides, box,
                   estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail("cuTensorMapEncodeTiled failed with code " + std::to_string(int(r)));
  return 0;
}

namespace {

template <int BLOCK_N, bool A_MN, bool B_MN, int CG = 1, int EPI = EPI_PLAIN, int FEWER = 0>
int launch(const GemmProblem& p, const KArgs& ka, cudaStream_t stream) {
  // (the 32 KB staging buffer takes a pipeline stage from the 128-wide variant; FEWER more go to the adding epilogue's buffers)
  constexpr int STAGES = (CG == 2 ? 6 : (BLOCK_N == 256 ? 4 : (BLOCK_N == 128 ? 5 : 8))) - FEWER;
  constexpr int B_STAGE_BYTES = BLOCK_N / CG * BLOCK_K * 2;
  constexpr int SMEM = STAGES * (A_STAGE_BYTES + B_STAGE_BYTES) + 8 * (2 * STAGES + 5) + 1024 +
                       8 * 4096 * (EPI == EPI_ADD ? add_buffers(BLOCK_N, STAGES, CG) : 1) + 128;
  CUtensorMap ma, mb_;
  if (gemm_make_map(&ma, p.a, A_MN ? BLOCK_K : BLOCK_M)) return -1;
  if (gemm_make_map(&mb_, p.b, B_MN ? BLOCK_K : EPI == EPI_GLU ? BLOCK_N / 2 : BLOCK_N / CG)) return -1;
  auto kern = gemm_bf16_kernel<BLOCK_N, A_MN, B_MN, STAGES, CG, EPI>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess)  // per (function, device)
    return fail("cudaFuncSetAttribute(MaxDynamicSharedMemorySize) failed");
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long m_tiles = (p.M + CG * BLOCK_M - 1) / (CG * BLOCK_M);
  const long long n_tiles = (p.N + BLOCK_N - 1) / BLOCK_N;
  long long tiles = (p.mode == GEMM_GROUPED_ROWS ? static_cast<long long>(p.max_tiles) : m_tiles) * n_tiles *
                    (p.mode == GEMM_GROUPED_CONTR ? p.num_groups : 1);
  int grid = static_cast<int>(tiles < sms / CG ? tiles : sms / CG);
  if (p.max_ctas > 0 && grid > p.max_ctas / CG) grid = p.max_ctas / CG;
  if (grid <= 0) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid * CG;
  cfg.blockDim = kThreads;
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CG;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CG == 2 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ma, mb_, ka);
  if (e != cudaSuccess) {
    cudaGetLastError();  // (reported here)
    return fail(std::string("gemm launch failed: ") + cudaGetErrorString(e));
  }
  return 0;
}

}  // namespace

const char* gemm_last_error() { return g_err.c_str(); }

int gemm_bf16_launch(const GemmProblem& p, cudaStream_t stream) {
  if (p.M <= 0 || p.N <= 0) return 0;
  if (p.mode != GEMM_GROUPED_CONTR && p.K <= 0) return fail("K must be positive");
  if (p.mode == GEMM_GROUPED_ROWS && (!p.tile_group || !p.num_m_tiles)) return fail("grouped-rows GEMM needs tile_group and num_m_tiles");
  if (p.mode == GEMM_GROUPED_ROWS && p.b.mn_major && p.K % BLOCK_K != 0) return fail("grouped-rows GEMM with an MN-major B needs K % 64 == 0");
  if (p.mode == GEMM_GROUPED_CONTR && (!p.group_offsets || !p.a.mn_major || !p.b.mn_major)) return fail("grouped-contraction GEMM needs MN-major operands and group_offsets");
  KArgs ka;
  memset(&ka, 0, sizeof(ka));
  ka.mode = p.mode;
  ka.M = p.M;
  ka.N = p.N;
  ka.K = p.K;
  ka.num_groups = p.num_groups;
  ka.max_tiles = p.max_tiles;
  ka.tile_group = p.tile_group;
  ka.num_m_tiles = p.num_m_tiles;
  ka.group_offsets = p.group_offsets;
  ka.c = p.c;
  ka.ldc = p.ldc;
  ka.c_group_stride = p.c_group_stride;
  ka.accumulate = p.accumulate ? 1 : 0;
  ka.out_fp32 = p.out_fp32 ? 1 : 0;
  ka.status = p.status;
  ka.row_ptrs = p.row_ptrs;
  ka.sig_ctrl = (p.row_ptrs || p.n_dest > 0) ? p.sig_ctrl : nullptr;
  ka.n_dest = p.n_dest;
  for (int i = 0; i < 8; ++i) ka.dest[i] = p.dest[i];
  if (p.n_dest > 0 && (p.out_fp32 || p.accumulate || p.N % 8 != 0 || p.mode != GEMM_DENSE || p.n_dest > 8 || p.ldc % 8 != 0))
    return fail("replicated output needs a dense bf16 problem without accumulation, N % 8 == 0 and ldc % 8 == 0");
  for (int i = 0; i < 8; ++i) ka.sig_flags[i] = p.sig_flags[i];
  ka.sig_nranks = p.sig_nranks;
  ka.sig_me = p.sig_me;
  if (p.row_ptrs && (p.out_fp32 || p.accumulate || p.N % 8 != 0 || p.mode == GEMM_GROUPED_CONTR))
    return fail("scattered output needs bf16, no accumulation, N % 8 == 0 and a row-major problem");
  const int esz = p.out_fp32 ? 4 : 2;
  const int vec = 16 / esz;
  ka.vec_ok = ((reinterpret_cast<uintptr_t>(p.c) & 15) == 0 && p.ldc % vec == 0 && p.c_group_stride % vec == 0) ? 1 : 0;

  if (p.glu) {
    const auto rows16 = [](const void* c, long long ld) { return (reinterpret_cast<uintptr_t>(c) & 15) == 0 && ld % 8 == 0; };
    if (p.mode == GEMM_GROUPED_CONTR || p.a.mn_major || p.b.mn_major || p.out_fp32 || p.accumulate || p.row_ptrs || p.n_dest > 0 || p.N % 16 != 0 ||
        !rows16(p.c, p.ldc) || (p.gu && !rows16(p.gu, p.gu_ld)))
      return fail("a gated product needs K-major operands, N % 16 == 0 and aligned bf16 outputs that are not added to");
    ka.gu = p.gu;
    ka.gu_ld = p.gu_ld;
  }

  if (p.score_part) {
    if (p.mode != GEMM_DENSE || p.a.mn_major || p.b.mn_major || (p.c && !p.out_fp32) || p.accumulate || p.row_ptrs || p.n_dest > 0 || p.glu ||
        !p.targets || !p.score_target)
      return fail("vocabulary scores need a dense K-major product, targets, and fp32 logits or none");
    ka.score_part = reinterpret_cast<float4*>(p.score_part);
    ka.targets = p.targets;
    ka.score_target = p.score_target;
    ka.inv_temp = p.inv_temp;
  }

  int bn = p.glu || p.score_part ? 256 : p.block_n;
  const bool amn = p.a.mn_major, bmn = p.b.mn_major;
  if (bn == 0 && gemm_is_skinny(p)) return gemm_skinny_launch(p, nullptr, stream);
  if (bn == 0) {
    const int sms = 148;
    const long long m_tiles = p.mode == GEMM_GROUPED_ROWS ? p.max_tiles : (p.M + BLOCK_M - 1) / BLOCK_M;
    const long long groups = p.mode == GEMM_GROUPED_CONTR ? p.num_groups : 1;
    auto tiles = [&](int b) { return m_tiles * ((p.N + b - 1) / b) * groups; };
    if (p.mode == GEMM_GROUPED_ROWS) {
      // (how many row tiles are live is known on the device only: prefer the 128x256 tile unless even the capacity leaves most
      // SMs idle or it wastes a large share of the tile)
      const bool waste256 = (p.N % 256) != 0 && (p.N % 256) <= 128;
      bn = (tiles(256) >= sms && !waste256) || (p.N >= 256 && tiles(256) >= 2 * sms) ? 256 : 128;
    } else {
      // A wave of 128x256 tiles takes as long as one of 128x128 tiles, which are bound by what they read from shared memory
      // (777 x 2048, K = 9728, one wave of either: 59 and 62 us), so the wider tile whenever it needs fewer waves (2048 x 2048,
      // K = 151936, 128 or 256 tiles: 905 us against 1402).
      const auto waves = [&](int b) { return (tiles(b) + sms - 1) / sms; };
      bn = waves(256) < waves(128) ? 256 : 128;
    }
    if (p.N <= 128) bn = 128;
    // Skinny problems (decode projections): narrower tiles spread the weight stream over more SMs.
    if (!amn && !bmn && tiles(bn) < sms) {
      if (bn == 128 && tiles(128) < sms / 2 && p.N >= 64) bn = 64;
      if (bn == 64 && tiles(64) < sms / 2 && p.N >= 32) bn = 32;
    }
  }
  // Tiles of two CTAs where they need no more waves than the one-CTA tiles (rows that a pair pads cost as much as others: 777 x 5120,
  // K = 2048, two waves instead of one, 906 -> 575 TFLOP/s) and a wave is long enough to carry the pair's start: K of 1024 at least
  // (5120 x 2048, two tiles per CTA, K = 2000 817 -> 843, K = 777 582 -> 573), or many waves (151936 x 2048, K = 583: 544 -> 557).
  // More than one wave, because a single one gains nothing (2000 x 2048, K = 4096: 1114 and 1088).
  bool pair = bn == 256 && p.mode == GEMM_DENSE && !p.row_ptrs && p.n_dest == 0 && (p.max_ctas == 0 || p.max_ctas >= 2) && p.pair != 1;
  if (pair && p.pair == 0) {
    const long long n_tiles = (p.N + 255) / 256, sms = 148;
    const long long single = ((p.M + 127) / 128 * n_tiles + sms - 1) / sms, paired = ((p.M + 255) / 256 * n_tiles + sms / 2 - 1) / (sms / 2);
    pair = p.block_n == 0 && paired <= single && single > 1 && (p.K >= 1024 || single >= 16);
  }
  if (p.row_ptrs || p.n_dest > 0) bn = 128;  // the staged scatter epilogue lives in the 128-wide variant
  if (bn != 32 && bn != 64 && bn != 128 && bn != 256) return fail("block_n must be 32, 64, 128 or 256");
  if ((bn == 32 || bn == 64) && (amn || bmn)) return fail("narrow tiles support K-major operands only");
  if (bn == 32) return launch<32, false, false>(p, ka, stream);
  if (bn == 64) return launch<64, false, false>(p, ka, stream);
  if (p.glu) return pair ? launch<256, false, false, 2, EPI_GLU>(p, ka, stream) : launch<256, false, false, 1, EPI_GLU>(p, ka, stream);
  if (p.score_part) return pair ? launch<256, false, false, 2, EPI_SCORES>(p, ka, stream) : launch<256, false, false, 1, EPI_SCORES>(p, ka, stream);
  // Weight gradients add to whole pieces of 128 bytes (what ends within one stays with the staged epilogue, whose ragged columns find
  // their lines in L1: 1000 x 1048, K = 333, 9.5 and 12.4 us). One CTA's 256-wide tiles take the adding epilogue's second buffer from
  // their stages, which long contractions miss. us staged / two buffers and three stages / one and four, by rows per group:
  //   128 of 1536 x 2048   128 455 / 293 / 387, 384 455 / 387 / 418, 448 486 / 450 / 445, 704 636 / 648 / 597, 1024 808 / 871 / 816
  //   64 of 2048 x 1408    256 310 / 179 / 222, 448 282 / 218 / 226, 576 280 / 253 / 245, 832 323 / 339 / 317, 1536 665 / 706 / 675
  //   16 of 8192 x 4096    256 605 / 433 / 551, 448 677 / 601 / 615, 704 951 / 945 / 878, 1024 1136 / 1222 / 1121, 1536 1508 / 1662 / 1555
  // so the lines lie within 4 % of the best everywhere. Dense in fp32, by K:
  //   8192 x 2048          64 41 / 33 / 41, 333 43 / 35 / 43, 777 47 / 45 / 47, 960 47 / 49 / 49, 2048 70 / 78 / 72
  //   4096 x 12288         64 111 / 76 / 96, 333 113 / 80 / 102, 777 115 / 115 / 111, 960 117 / 127 / 113, 1536 150 / 170 / 150
  //   2560 x 2560          64 25 / 20 / 25, 777 29 / 27 / 29, 1088 31 / 31 / 31, 2048 41 / 43 / 41
  if (p.accumulate && amn && bmn && ka.vec_ok && p.N % (p.out_fp32 ? 32 : 64) == 0) {
    if (pair) return launch<256, true, true, 2, EPI_ADD, 1>(p, ka, stream);
    if (bn == 128) return launch<128, true, true, 1, EPI_ADD>(p, ka, stream);
    const bool grouped = p.mode == GEMM_GROUPED_CONTR;
    const long long k = grouped ? p.a.rows / (p.num_groups > 0 ? p.num_groups : 1) : p.K;
    if (k < (grouped ? 448 : 800)) return launch<256, true, true, 1, EPI_ADD, 1>(p, ka, stream);
    if (grouped && k < 800) return launch<256, true, true, 1, EPI_ADD>(p, ka, stream);
  }
  if (pair) {
    if (!amn && !bmn) return launch<256, false, false, 2>(p, ka, stream);
    if (!amn && bmn) return launch<256, false, true, 2>(p, ka, stream);
    if (amn && !bmn) return launch<256, true, false, 2>(p, ka, stream);
    return launch<256, true, true, 2>(p, ka, stream);
  }
#define MB_DISPATCH(BN)                                                     \
  if (!amn && !bmn) return launch<BN, false, false>(p, ka, stream);         \
  if (!amn && bmn) return launch<BN, false, true>(p, ka, stream);           \
  if (amn && !bmn) return launch<BN, true, false>(p, ka, stream);           \
  return launch<BN, true, true>(p, ka, stream);
  if (bn == 256) {
    MB_DISPATCH(256)
  } else {
    MB_DISPATCH(128)
  }
#undef MB_DISPATCH
}

}  // namespace mb
