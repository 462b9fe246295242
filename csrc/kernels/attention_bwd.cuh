// What the attention backward kernels for head_dim 64 and 128 share: which part of the work a CTA takes.
#pragma once
#include "common.cuh"

namespace cpb {

// A CTA owns a K/V tile and sweeps the (query head, query tile) pairs that see it: `it_chunk` of them at most when that is not 0, and
// then several CTAs share a tile and each writes a part of dK / dV in fp32 (dkv_mode 3).
struct BwdWork {
  int kt, hkv, b;
  int it0;                 // first pair of the sweep
};
// K/V tiles that have a part number c: under a causal mask over positions 0 .. Tq - 1 (`local`) those with more than c chunk visible pairs.
__host__ __device__ __forceinline__ int bwd_tiles(int c, int it_chunk, int n_kt, int nq, int G, int k_off, int local) {
  if (!local) return n_kt;
  const int last = nq - 1 - (int)((long)c * it_chunk / G);             // last first-visible query tile
  const long end = 128L * last + 127 - k_off;
  return last < 0 || end < 0 ? 0 : (int)(end / 128 + 1 < n_kt ? end / 128 + 1 : n_kt);
}
// `local` here: causal and local
template <bool PARTS>
__device__ __forceinline__ BwdWork bwd_work(int it_chunk, int n_kt, int nq, int G, int Hkv, int B, int k_off, int local) {
  if (!PARTS) return BwdWork{(int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z, 0};
  // part 0 of every tile, the longest first over all heads and batches, then part 1 of those that have one, ...: longest first within a part
  // number, not over all of them (a second part may be longer than the first of a later tile)
  int i = (int)blockIdx.x, c = 0;
  const int hb = Hkv * B;
  for (int n; i >= (n = bwd_tiles(c, it_chunk, n_kt, nq, G, k_off, local) * hb); ++c) i -= n;
  return BwdWork{i / hb, i % Hkv, (i / Hkv) % B, c * it_chunk};
}

}  // namespace cpb
