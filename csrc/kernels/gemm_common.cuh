// Epilogues of the bf16 GEMM (gemm.cu): parameters, epilogue kinds, and the way a finished accumulator tile leaves the SM.
//
// A thread of an epilogue warp owns one row of the tile (its tensor-memory lane).  Storing its columns straight to global
// memory puts the 32 lanes of every instruction on 32 different rows: 32 partial sectors per instruction, 4096 load/store
// cycles per 128 x 256 bf16 tile and 8192 for fp32 or for two bf16 outputs, while the main loop of the tile needs only
// 512 cycles per 64 of K.  So a warp writes 32 rows x 128 bytes into its own 128-byte-swizzled staging buffer in shared
// memory (conflict-free 16-byte stores) and one lane hands the buffer to TMA, which writes whole lines, clips the edges of
// the matrix and, for the accumulating epilogue, adds in L2 without the SM reading C first.  Two buffers per warp: one is
// drained while the other is filled.
#pragma once
#include "common.cuh"

namespace cpb {

constexpr int GEMM_BM = 128;           // rows of A per CTA; a CTA pair computes 256 rows
constexpr int GEMM_BK = 64;
constexpr int GEMM_THREADS = 192;

enum : int {
  EPI_BF16 = 0,        // C(bf16) = acc (+bias)
  EPI_F32 = 1,         // C(f32)  = acc (+bias)
  EPI_F32_ACC = 2,     // C(f32) += acc (+bias)
  EPI_BF16_GELU = 3,   // C(bf16) = gelu_tanh(acc + bias); aux(bf16) = acc + bias (pre-activation) when aux != null
  EPI_BF16_SWIGLU = 4, // B tile = [gate rows | up rows]; C(bf16)[:, n] = silu(g)*u ; aux gets [g | u] when aux != null
  EPI_HEAD_STATS = 5,  // language-model head: (max, sum of exponentials) of the tile's columns per row, no C
  EPI_HEAD_STORE = 6,  // both: EPI_HEAD_STATS, and C(f32) = acc
  EPI_HEAD_GRAD = 7,   // C(bf16) = (softmax - onehot(target)) * grad_scale from the rows' (max, grad_scale / sum)
};

// Cross entropy in the epilogue of the head's GEMM (xent.cu has the kernel between the two passes).
struct HeadParams {
  const int64_t* targets;    // [M]; a row whose target is outside [0, n_valid) has neither loss nor gradient
  float2* stats;             // [tiles along N][M] (max, sum of exp(x - max))
  float* target_logit;       // [M], written where the target is in range
  const float2* row_coef;    // [M] (max, grad_scale / sum), (max, 0) for ignored rows
  int n_valid;               // columns from here on are padding
  float grad_scale;
};

struct GemmParams {
  int M, N, K;
  int epi;
  int num_m_tiles, num_n_blocks, num_k_blocks;
  int splits, k_per_split;   // split-K: 64-wide K blocks per work item.  EPI_F32_ACC: the first split adds to C, the others go to a
                             // workspace [splits - 1][M][N] for gemm_add_partials_kernel.  EPI_F32 (a bf16 result): all splits go to
                             // a workspace [splits][M][N] for gemm_sum_partials_kernel
  int swiglu_half;     // number of output features F when epi == SWIGLU (B has 2F rows)
  int band;            // pair-rows per band of the tile order (1 = rows of tiles, columns fastest)
  int has_aux;
  const float* bias;
  HeadParams head;
  int* status;
};

// gelu = 0.5 x (1 + tanh(u)), tanh(u) = 1 - 2 / (exp(2u) + 1).  One exponential and one division per value: two values that share
// an approximate reciprocal of the product of their denominators, with the exponent clamped, save 11 to 25 % of the time of a
// GEMM of shallow K, but below about -40 SwiGLU came out as x * 2^-57 and not as x * exp(x).
__device__ __forceinline__ float gelu_tanh_f(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float u = k0 * (x + k1 * x * x * x);
  const float e = __expf(2.f * u);
  const float t = 1.f - 2.f / (e + 1.f);
  return 0.5f * x * (1.f + t);
}
__device__ __forceinline__ float silu_f(float x) { return x / (1.f + __expf(-x)); }

// One warp's way out: two staging buffers of 32 rows x 128 bytes, used in turn.
struct WarpStore {
  uint8_t* buf;        // 2 x 4096 bytes, 1024-byte aligned
  uint32_t use;        // stores issued so far
  bool issuer;         // lane 0: issues and waits

  // Claim the next buffer: it is free once at most the newest bulk group is still being read.
  __device__ __forceinline__ uint8_t* row_ptr(int lane) {
    if (issuer) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
    __syncwarp();
    return buf + (use & 1) * 4096 + lane * 128;
  }
  // v: this lane's 128 bytes, sixteen bytes to chunk position (chunk ^ row % 8)
  __device__ __forceinline__ void fill(uint8_t* row, int lane, const uint32_t (&v)[32]) {
#pragma unroll
    for (int c = 0; c < 8; ++c)
      *(uint4*)(row + ((c ^ (lane & 7)) << 4)) = make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    fence_proxy_async_smem();
    __syncwarp();
  }
  __device__ __forceinline__ void store(const CUtensorMap* m, int x, int y) {
    if (issuer) {
      asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];"
                   ::"l"((uint64_t)m), "r"(smem_u32(buf + (use & 1) * 4096)), "r"(x), "r"(y) : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    ++use;
  }
  __device__ __forceinline__ void store3(const CUtensorMap* m, int x, int y, int z) {
    if (issuer) {
      asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
                   ::"l"((uint64_t)m), "r"(smem_u32(buf + (use & 1) * 4096)), "r"(x), "r"(y), "r"(z) : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    ++use;
  }
  __device__ __forceinline__ void add(const CUtensorMap* m, int x, int y) {
    if (issuer) {
      asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
                   ::"l"((uint64_t)m), "r"(smem_u32(buf + (use & 1) * 4096)), "r"(x), "r"(y) : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    ++use;
  }
  __device__ __forceinline__ void drain() {
    if (issuer) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
};

__device__ __forceinline__ void pack_row(const float (&f)[64], uint32_t (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = pack_bf16(f[2 * j], f[2 * j + 1]);
}

__device__ __forceinline__ float head_exp(float x, float m) { return ex2f((x - m) * 1.4426950408889634f); }

// f[at] without dynamic register indexing (at in [0, 64))
__device__ __forceinline__ float pick64(const float (&f)[64], int at) {
  float r = 0.f;
#pragma unroll
  for (int j = 0; j < 64; ++j) r = j == at ? f[j] : r;
  return r;
}

// What a thread needs of its row, read before the accumulator is waited for.
struct HeadRow {
  int target;                // column, or negative
  float2 coef;
};
__device__ __forceinline__ HeadRow head_row(const GemmParams& p, int row) {
  HeadRow h{-1, {0.f, 0.f}};
  if (p.epi >= EPI_HEAD_STATS && row < p.M) {
    const int64_t t = __ldg(p.head.targets + row);
    h.target = t >= 0 && t < p.head.n_valid ? (int)t : -1;
    if (p.epi == EPI_HEAD_GRAD) h.coef = __ldg(p.head.row_coef + row);
  }
  return h;
}

// Bound by the main loop from a K of about 300 on: a tile's 256 exponentials per thread take the special-function unit 2048 cycles,
// 64 of K take 370 ns.
template <int BN, class Release>
__device__ __forceinline__ void head_epilogue(const GemmParams& p, const CUtensorMap* tmC, WarpStore& ws, uint32_t t_row, int row0, int nb,
                                              int lane, const HeadRow& h, Release release) {
  const int row = row0 + lane;
  const bool live = row0 < p.M;
  float m = -INFINITY, s = 0.f;
#pragma unroll 1
  for (int c = 0; c < BN; c += 64) {
    const int col = nb * BN + c;
    float f[64];
    tmem_ld32(t_row + c, *(uint32_t(*)[32])&f[0]);
    tmem_ld32(t_row + c + 32, *(uint32_t(*)[32])&f[32]);
    tmem_wait_ld();
    if (c + 64 == BN) release();
    if (!live || col >= p.N) continue;
    const int at = h.target - col;
    const bool hit = at >= 0 && at < 64;
    if (p.epi != EPI_HEAD_GRAD) {
      if (p.epi == EPI_HEAD_STORE) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (col + 32 * h >= p.N) break;
          ws.fill(ws.row_ptr(lane), lane, *(uint32_t(*)[32])&f[32 * h]);
          ws.store(tmC, col + 32 * h, row0);
        }
      }
      if (col >= p.head.n_valid) continue;
      if (hit) p.head.target_logit[row] = pick64(f, at);
      if (col + 64 > p.head.n_valid) {
#pragma unroll
        for (int j = 0; j < 64; ++j) if (col + j >= p.head.n_valid) f[j] = -INFINITY;
      }
      float mx[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        mx[q] = fmaxf(f[q], f[q + 4]);
#pragma unroll
        for (int j = 8; j < 64; j += 8) mx[q] = fmax3(mx[q], f[j + q], f[j + q + 4]);
      }
      const float mt = fmax3(fmaxf(mx[0], mx[1]), mx[2], mx[3]);
      if (mt > m) { s = m == -INFINITY ? s : s * head_exp(m, mt); m = mt; }
      // a row of nothing but -inf so far adds nothing; NaN gets into the sum, whatever the maximum says
      const float ref = m == -INFINITY ? 0.f : m;
      const uint64_t nm = pack_f32x2(-ref, -ref), l2e = pack_f32x2(1.4426950408889634f, 1.4426950408889634f);
      uint64_t acc[2] = {pack_f32x2(0.f, 0.f), pack_f32x2(0.f, 0.f)};
#pragma unroll
      for (int j = 0; j < 64; j += 2) {
        float x0, x1;
        unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(f[j], f[j + 1]), nm), l2e), x0, x1);
        acc[(j >> 1) & 1] = add_f32x2(acc[(j >> 1) & 1], pack_f32x2(ex2f(x0), ex2f(x1)));
      }
      float a, b;
      unpack_f32x2(add_f32x2(acc[0], acc[1]), a, b);
      s += a + b;
    } else {
      const uint64_t nm = pack_f32x2(-h.coef.x, -h.coef.x), l2e = pack_f32x2(1.4426950408889634f, 1.4426950408889634f);
      const uint64_t inv = pack_f32x2(h.coef.y, h.coef.y);
#pragma unroll
      for (int j = 0; j < 64; j += 2) {
        float x0, x1;
        unpack_f32x2(mul_f32x2(add_f32x2(pack_f32x2(f[j], f[j + 1]), nm), l2e), x0, x1);
        unpack_f32x2(mul_f32x2(pack_f32x2(ex2f(x0), ex2f(x1)), inv), f[j], f[j + 1]);
      }
      if (col + 64 > p.head.n_valid) {
#pragma unroll
        for (int j = 0; j < 64; ++j) if (col + j >= p.head.n_valid) f[j] = 0.f;
      }
      if (hit) {
#pragma unroll
        for (int j = 0; j < 64; ++j) f[j] = j == at ? f[j] - p.head.grad_scale : f[j];
      }
      uint32_t v[32];
      pack_row(f, v);
      ws.fill(ws.row_ptr(lane), lane, v);
      ws.store(tmC, col, row0);
    }
  }
  if (p.epi != EPI_HEAD_GRAD && row < p.M) p.head.stats[(size_t)nb * p.M + row] = make_float2(m, s);
}

// Epilogue of one 32-row slice of a 128 x BN accumulator tile: `t_row` is the tensor-memory address of this warp's lanes at
// the accumulator's first column, `row0` the slice's first output row, `nb` the tile's index along N, `split` its range of K (the
// first one brings the bias).  `release` runs as soon as the accumulator has been read.
template <int BN, class Release>
__device__ __forceinline__ void gemm_epilogue(const GemmParams& p, const CUtensorMap* tmC, const CUtensorMap* tmX, WarpStore& ws,
                                              uint32_t t_row, int row0, int nb, int lane, int split, Release release) {
  const bool live = row0 < p.M;
  const float* bias = split == 0 ? p.bias : nullptr;
  if (p.epi == EPI_BF16_SWIGLU) {
    // accumulator columns [0, BN/2) = gate, [BN/2, BN) = up, for features f0 .. f0 + BN/2
#pragma unroll 1
    for (int c = 0; c < BN / 2; c += 64) {
      const int f = nb * (BN / 2) + c;
      float g[64], u[64];
      tmem_ld32(t_row + c, *(uint32_t(*)[32])&g[0]);
      tmem_ld32(t_row + c + 32, *(uint32_t(*)[32])&g[32]);
      tmem_ld32(t_row + BN / 2 + c, *(uint32_t(*)[32])&u[0]);
      tmem_ld32(t_row + BN / 2 + c + 32, *(uint32_t(*)[32])&u[32]);
      tmem_wait_ld();
      if (c + 64 == BN / 2) release();
      if (!live || f >= p.swiglu_half) continue;
      uint32_t v[32];
      if (p.has_aux) {
        pack_row(g, v);
        ws.fill(ws.row_ptr(lane), lane, v);
        ws.store3(tmX, f, 0, row0);
        pack_row(u, v);
        ws.fill(ws.row_ptr(lane), lane, v);
        ws.store3(tmX, f, 1, row0);
      }
#pragma unroll
      for (int j = 0; j < 64; j += 2) v[j >> 1] = pack_bf16(silu_f(g[j]) * u[j], silu_f(g[j + 1]) * u[j + 1]);
      ws.fill(ws.row_ptr(lane), lane, v);
      ws.store(tmC, f, row0);
    }
  } else if (p.epi == EPI_F32 || p.epi == EPI_F32_ACC) {
#pragma unroll 1
    for (int c = 0; c < BN; c += 32) {
      const int col = nb * BN + c;
      uint32_t v[32];
      tmem_ld32(t_row + c, v);
      tmem_wait_ld();
      if (c + 32 == BN) release();
      if (!live || col >= p.N) continue;
      if (bias != nullptr) {
#pragma unroll
        for (int j = 0; j < 32; j += 8)
          if (col + j < p.N) {                 // N is a multiple of 8
#pragma unroll
            for (int q = 0; q < 8; q += 4) {
              const float4 b = __ldg((const float4*)(bias + col + j + q));
              v[j + q] = __float_as_uint(__uint_as_float(v[j + q]) + b.x);
              v[j + q + 1] = __float_as_uint(__uint_as_float(v[j + q + 1]) + b.y);
              v[j + q + 2] = __float_as_uint(__uint_as_float(v[j + q + 2]) + b.z);
              v[j + q + 3] = __float_as_uint(__uint_as_float(v[j + q + 3]) + b.w);
            }
          }
      }
      ws.fill(ws.row_ptr(lane), lane, v);
      if (p.splits > 1 && p.epi == EPI_F32) ws.store3(tmX, col, row0, split);
      else if (split > 0) ws.store3(tmX, col, row0, split - 1);
      else if (p.epi == EPI_F32_ACC) ws.add(tmC, col, row0);
      else ws.store(tmC, col, row0);
    }
  } else {
#pragma unroll 1
    for (int c = 0; c < BN; c += 64) {
      const int col = nb * BN + c;
      float f[64];
      tmem_ld32(t_row + c, *(uint32_t(*)[32])&f[0]);
      tmem_ld32(t_row + c + 32, *(uint32_t(*)[32])&f[32]);
      tmem_wait_ld();
      if (c + 64 == BN) release();
      if (!live || col >= p.N) continue;
      if (bias != nullptr) {
#pragma unroll
        for (int j = 0; j < 64; j += 8)
          if (col + j < p.N) {
#pragma unroll
            for (int q = 0; q < 8; q += 4) {
              const float4 b = __ldg((const float4*)(bias + col + j + q));
              f[j + q] += b.x; f[j + q + 1] += b.y; f[j + q + 2] += b.z; f[j + q + 3] += b.w;
            }
          }
      }
      uint32_t v[32];
      if (p.epi == EPI_BF16_GELU) {
        if (p.has_aux) {
          pack_row(f, v);
          ws.fill(ws.row_ptr(lane), lane, v);
          ws.store(tmX, col, row0);
        }
#pragma unroll
        for (int j = 0; j < 64; ++j) f[j] = gelu_tanh_f(f[j]);
      }
      pack_row(f, v);
      ws.fill(ws.row_ptr(lane), lane, v);
      ws.store(tmC, col, row0);
    }
  }
}

}  // namespace cpb
