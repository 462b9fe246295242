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
__device__ __forceinline__ BwdWork bwd_work(int it_chunk, int n_kt, int Hkv, int B) {
  if (it_chunk == 0) return BwdWork{(int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z, 0};
  // longest first over all heads and batches: the parts of a tile are numbered last
  const int i = (int)blockIdx.x, hb = Hkv * B, kc = i / hb;
  return BwdWork{kc % n_kt, i % Hkv, (i / Hkv) % B, kc / n_kt * it_chunk};
}

}  // namespace cpb
