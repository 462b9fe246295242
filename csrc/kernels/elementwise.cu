// Memory-bound kernels: RMSNorm / LayerNorm (with fused residual add), SwiGLU / GELU backward,
// bias gradient, embedding, QK-norm + RoPE on a packed QKV buffer, RoPE cache builders
// (YaRN / LongRoPE), HeadTail gather, K/V pack, LSE merge, gradient-norm + AdamW.
//
// They replace the reference's external tensor-library kernels (rms_norm, layer_norm, gelu,
// swiglu, embedding, rope_forward_cuda, AdamW, clip_grad_norm_) and its own headtail / kv-pack
// kernels (context_parallel/headtail_kernel.cu:26-105, context_parallel/KVPackKernel.cu:13-37),
// and fold the SDPA merge (context_parallel/SDPAMerger.h:108-121) into one launch.
// Everything is bf16 in / bf16 out with fp32 statistics, 16-byte vector accesses, one warp per row
// for the row reductions.
#include "common.cuh"
#include "host_utils.h"

namespace cpb {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  f[0] = bf16_lo(u.x); f[1] = bf16_hi(u.x); f[2] = bf16_lo(u.y); f[3] = bf16_hi(u.y);
  f[4] = bf16_lo(u.z); f[5] = bf16_hi(u.z); f[6] = bf16_lo(u.w); f[7] = bf16_hi(u.w);
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}

// eight consecutive fp32 parameters (vector c of a row) as two 16-byte loads; `fill` when the parameter is absent
__device__ __forceinline__ void load8f(const float* __restrict__ p, int c, float fill, float (&f)[8]) {
  if (p == nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = fill;
    return;
  }
  const float4 a = __ldg((const float4*)p + 2 * c), b = __ldg((const float4*)p + 2 * c + 1);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// ============================================================================ norm forward
// One warp per row; d % 8 == 0; MAXV = max 16-byte vectors per lane (d <= 256*MAXV).
// If `res` != null: x_new = x + res is written to `xout` and normalised.
// LAYER = true -> LayerNorm (mean/var, optional bias); false -> RMSNorm.
template <bool LAYER, int MAXV>
__global__ void norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                                const float* __restrict__ w, const float* __restrict__ b,
                                __nv_bfloat16* __restrict__ xout, __nv_bfloat16* __restrict__ y,
                                float* __restrict__ stats, int rows, int d, float eps) {
  pdl_release();
  pdl_wait();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const int nvec = d >> 3;
  const uint4* xr = (const uint4*)(x + (size_t)row * d);
  const uint4* rr = res ? (const uint4*)(res + (size_t)row * d) : nullptr;
  // every load of the row is issued before the first use; the row then stays in registers as bf16 (the rounded x + res,
  // exactly what later kernels re-read)
  uint4 px[MAXV], pr[MAXV];
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int c = lane + i * 32;
    if (c < nvec) {
      px[i] = xr[c];
      if (rr) pr[i] = rr[c];
    }
  }
  float s = 0.f, ss = 0.f;
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int c = lane + i * 32;
    if (c < nvec) {
      float v[8];
      unpack8(px[i], v);
      if (rr) {
        float r8[8];
        unpack8(pr[i], r8);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] += r8[j];
        px[i] = pack8(v);
        ((uint4*)(xout + (size_t)row * d))[c] = px[i];
        unpack8(px[i], v);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) { s += v[j]; ss += v[j] * v[j]; }
    }
  }
  s = warp_sum(s); ss = warp_sum(ss);
  float mean = 0.f, rstd;
  if (LAYER) {
    mean = s / d;
    float var = fmaxf(ss / d - mean * mean, 0.f);
    rstd = rsqrtf(var + eps);
  } else {
    rstd = rsqrtf(ss / d + eps);
  }
  if (stats && lane == 0) { stats[2 * (size_t)row] = mean; stats[2 * (size_t)row + 1] = rstd; }
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int c = lane + i * 32;
    if (c < nvec) {
      float v[8], o[8], g[8], bb[8];
      unpack8(px[i], v);
      load8f(w, c, 1.f, g);
      if (LAYER) load8f(b, c, 0.f, bb);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = (v[j] - mean) * rstd * g[j] + (LAYER ? bb[j] : 0.f);
      ((uint4*)(y + (size_t)row * d))[c] = pack8(o);
    }
  }
}

// ============================================================================ norm backward
// dx = rstd * (g*dy - xhat * mean(g*dy*xhat) [- mean(g*dy)])  (+ dres_in) ; dw += sum dy*xhat ; db += sum dy
// Bound by memory (x, dy, dres in, dx out).  A group of G threads owns the d columns, eight each, and takes four rows at a time:
// all loads are issued before the first use, the rows share one reduction, and dw / db stay in registers until the end.
// One warp per row, with dw / db added to shared memory, spent its time in those additions (compare-and-swap loops).
// Cold L2, one warp per row -> this, us: 32768 x 4096 757 -> 206 (5.2 TB/s); 131072 x 2048 732 -> 367 (5.9); 8192 x 2048
// 71 -> 36; 8192 x 384 20.5 -> 16.4; layer norm 4096 x 768 20.5 -> 16.3, 4096 x 384 16.4 -> 12.3.
template <bool LAYER, int G>
__global__ void __launch_bounds__(G > 256 ? 512 : 256, G > 256 ? 1 : 2)
norm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                const __nv_bfloat16* __restrict__ dres, const float* __restrict__ w,
                const float* __restrict__ stats, __nv_bfloat16* __restrict__ dx,
                float* __restrict__ dw, float* __restrict__ db, int rows, int d) {
  pdl_release();
  pdl_wait();
  constexpr int TB = G > 256 ? 512 : 256, NG = TB / G, W = G / 32, R = 4;
  __shared__ float4 red[2][NG][W][LAYER ? 2 : 1];            // per warp: four rows' sums; two buffers, one barrier per turn
  __shared__ float part[NG > 1 ? TB * 8 : 1];                // used only when a block holds several groups
  const int g = threadIdx.x / G, c = threadIdx.x % G, lane = threadIdx.x & 31, warp = c >> 5;
  const bool on = c < (d >> 3);
  float wv[8], aw[8], ab[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) { wv[j] = 0.f; aw[j] = 0.f; ab[j] = 0.f; }
  if (on) load8f(w, c, 1.f, wv);
  int buf = 0;
  for (long base = (long)blockIdx.x * NG * R; base < rows; base += (long)gridDim.x * NG * R, buf ^= 1) {
    const long row0 = base + g * R;
    uint4 px[R], pd[R], pr[R];
    float mean[R], rstd[R], s1[R], s2[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      px[r] = pd[r] = pr[r] = make_uint4(0, 0, 0, 0);
      mean[r] = rstd[r] = 0.f;
      if (row0 + r < rows) {
        const size_t off = (size_t)(row0 + r) * d;
        if (on) {
          px[r] = ((const uint4*)(x + off))[c];
          pd[r] = ((const uint4*)(dy + off))[c];
          if (dres) pr[r] = ((const uint4*)(dres + off))[c];
        }
        if (LAYER) mean[r] = stats[2 * (row0 + r)];
        rstd[r] = stats[2 * (row0 + r) + 1];
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float xv[8], dv[8];
      unpack8(px[r], xv); unpack8(pd[r], dv);
      s1[r] = s2[r] = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = (xv[j] - mean[r]) * rstd[r], gg = dv[j] * wv[j];
        s1[r] += gg * xh;
        if (LAYER) { s2[r] += gg; ab[j] += dv[j]; }
        aw[j] += dv[j] * xh;
      }
      s1[r] = warp_sum(s1[r]);
      if (LAYER) s2[r] = warp_sum(s2[r]);
    }
    if (W > 1) {
      if (lane == 0) {
        red[buf][g][warp][0] = make_float4(s1[0], s1[1], s1[2], s1[3]);
        if (LAYER) red[buf][g][warp][LAYER ? 1 : 0] = make_float4(s2[0], s2[1], s2[2], s2[3]);
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < R; ++r) s1[r] = s2[r] = 0.f;
#pragma unroll
      for (int i = 0; i < W; ++i) {
        const float4 v = red[buf][g][i][0];
        s1[0] += v.x; s1[1] += v.y; s1[2] += v.z; s1[3] += v.w;
        if (LAYER) {
          const float4 u = red[buf][g][i][LAYER ? 1 : 0];
          s2[0] += u.x; s2[1] += u.y; s2[2] += u.z; s2[3] += u.w;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (!on || row0 + r >= rows) continue;
      float xv[8], dv[8], r8[8], o[8];
      unpack8(px[r], xv); unpack8(pd[r], dv); unpack8(pr[r], r8);
      const float m1 = s1[r] / d, m2 = LAYER ? s2[r] / d : 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = (xv[j] - mean[r]) * rstd[r], gg = dv[j] * wv[j];
        o[j] = rstd[r] * (gg - xh * m1 - m2);
        if (dres) o[j] += r8[j];
      }
      ((uint4*)(dx + (size_t)(row0 + r) * d))[c] = pack8(o);
    }
  }
  // the groups of a block are added in shared memory, the blocks in global memory.  One group: four columns per addition (one
  // column at a time, 32 bytes from lane to lane, takes 33 us at 2048 x 1032, where 256 blocks meet on every column).
  for (int pass = 0; pass < (LAYER ? 2 : 1); ++pass) {
    float* dst = pass ? db : dw;
    if (dst == nullptr) continue;
    if (NG == 1) {
      if (on) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = pass ? ab[j] : aw[j];
        if (((uintptr_t)dst & 15) == 0) {
          red_add_v4(dst + c * 8, v[0], v[1], v[2], v[3]);
          red_add_v4(dst + c * 8 + 4, v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) atomicAdd(&dst[c * 8 + j], v[j]);
        }
      }
    } else {
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 8; ++j) part[threadIdx.x * 8 + j] = pass ? ab[j] : aw[j];
      __syncthreads();
      for (int i = threadIdx.x; i < d; i += TB) {
        float v = 0.f;
        for (int k = 0; k < NG; ++k) v += part[k * G * 8 + i];
        atomicAdd(&dst[i], v);
      }
    }
  }
}

// ============================================================================ activations (backward)
// gu: [rows, 2F] = [gate | up]; dact: [rows, F]; dgu: [rows, 2F]
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ dact,
                                  __nv_bfloat16* __restrict__ dgu, size_t rows, int F) {
  pdl_release();
  pdl_wait();
  const size_t nvec = rows * (size_t)(F >> 3);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nvec; i += (size_t)gridDim.x * blockDim.x) {
    const size_t row = i / (F >> 3);
    const int c = (int)(i % (F >> 3)) * 8;
    float g[8], u[8], da[8], dg[8], du[8];
    uint4 ug = *(const uint4*)(gu + row * 2 * F + c);
    uint4 uu = *(const uint4*)(gu + row * 2 * F + F + c);
    uint4 ud = *(const uint4*)(dact + row * F + c);
    unpack8(ug, g); unpack8(uu, u); unpack8(ud, da);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float s = 1.f / (1.f + __expf(-g[j]));
      float silu = g[j] * s;
      dg[j] = da[j] * u[j] * (s + silu * (1.f - s));
      du[j] = da[j] * silu;
    }
    *(uint4*)(dgu + row * 2 * F + c) = pack8(dg);
    *(uint4*)(dgu + row * 2 * F + F + c) = pack8(du);
  }
}

// forward (standalone, used when the GEMM epilogue fusion is not): act = silu(g)*u
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ act, size_t rows, int F) {
  pdl_release();
  pdl_wait();
  const size_t nvec = rows * (size_t)(F >> 3);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nvec; i += (size_t)gridDim.x * blockDim.x) {
    const size_t row = i / (F >> 3);
    const int c = (int)(i % (F >> 3)) * 8;
    float g[8], u[8], o[8];
    uint4 ug = *(const uint4*)(gu + row * 2 * F + c);
    uint4 uu = *(const uint4*)(gu + row * 2 * F + F + c);
    unpack8(ug, g); unpack8(uu, u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    *(uint4*)(act + row * F + c) = pack8(o);
  }
}

__device__ __forceinline__ float gelu_tanh_grad(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * (x + k1 * x * x * x);
  float e = __expf(2.f * u);
  float t = 1.f - 2.f / (e + 1.f);
  float du = k0 * (1.f + 3.f * k1 * x * x);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * du;
}
__device__ __forceinline__ float gelu_tanh_val(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  float u = k0 * (x + k1 * x * x * x);
  float e = __expf(2.f * u);
  float t = 1.f - 2.f / (e + 1.f);
  return 0.5f * x * (1.f + t);
}
// mode 0: y = gelu(x) ; mode 1: y = dy * gelu'(x)
__global__ void gelu_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                            __nv_bfloat16* __restrict__ y, size_t n8, int mode) {
  pdl_release();
  pdl_wait();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n8; i += (size_t)gridDim.x * blockDim.x) {
    float xv[8], o[8];
    uint4 ux = ((const uint4*)x)[i];
    unpack8(ux, xv);
    if (mode == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = gelu_tanh_val(xv[j]);
    } else {
      float dv[8];
      uint4 ud = ((const uint4*)dy)[i];
      unpack8(ud, dv);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = dv[j] * gelu_tanh_grad(xv[j]);
    }
    ((uint4*)y)[i] = pack8(o);
  }
}

// y = a + b (bf16), 8 elements per thread
__global__ void add_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                           __nv_bfloat16* __restrict__ y, size_t n8) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n8; i += (size_t)gridDim.x * blockDim.x) {
    float av[8], bv[8];
    uint4 ua = ((const uint4*)a)[i], ub = ((const uint4*)b)[i];
    unpack8(ua, av); unpack8(ub, bv);
#pragma unroll
    for (int j = 0; j < 8; ++j) av[j] += bv[j];
    ((uint4*)y)[i] = pack8(av);
  }
}

// db[n] += sum_rows dy[row, n]; grid (ceil(N/64), row_blocks); block 256 = 8 row-lanes x 32 col-pairs
__global__ void bias_grad_kernel(const __nv_bfloat16* __restrict__ dy, float* __restrict__ db, int rows, int N, int rows_per_block) {
  pdl_release();
  pdl_wait();
  __shared__ float red[8][64];
  const int cp = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int col = blockIdx.x * 64 + cp * 2;
  const int r0 = blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  float a0 = 0.f, a1 = 0.f;
  if (col < N) {
    for (int r = r0 + rl; r < r1; r += 8) {
      uint32_t u = *(const uint32_t*)(dy + (size_t)r * N + col);
      a0 += bf16_lo(u); a1 += bf16_hi(u);
    }
  }
  red[rl][cp * 2] = a0; red[rl][cp * 2 + 1] = a1;
  __syncthreads();
  if (threadIdx.x < 64) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += red[i][threadIdx.x];
    const int c = blockIdx.x * 64 + threadIdx.x;
    if (c < N) atomicAdd(&db[c], s);
  }
}

// ============================================================================ embedding
// out[row, :] = wte[idx[row], :] (+ wpe[pos[row], :])
__global__ void embedding_fwd_kernel(const int64_t* __restrict__ idx, const int64_t* __restrict__ pos,
                                     const __nv_bfloat16* __restrict__ wte, const __nv_bfloat16* __restrict__ wpe,
                                     __nv_bfloat16* __restrict__ out, size_t rows, int d, int pos_period) {
  pdl_release();
  pdl_wait();
  const int nvec = d >> 3;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < rows * nvec; i += (size_t)gridDim.x * blockDim.x) {
    const size_t row = i / nvec;
    const int c = (int)(i % nvec);
    uint4 u = ((const uint4*)(wte + (size_t)idx[row] * d))[c];
    if (wpe) {
      float a[8], b[8];
      uint4 up = ((const uint4*)(wpe + (size_t)pos[row % pos_period] * d))[c];
      unpack8(u, a); unpack8(up, b);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += b[j];
      u = pack8(a);
    }
    ((uint4*)(out + row * d))[c] = u;
  }
}
// dwte[idx[row], :] += dout[row, :] ; dwpe[pos[row], :] += dout[row, :]   (fp32 atomics)
__global__ void embedding_bwd_kernel(const int64_t* __restrict__ idx, const int64_t* __restrict__ pos,
                                     const __nv_bfloat16* __restrict__ dout, float* __restrict__ dwte,
                                     float* __restrict__ dwpe, size_t rows, int d, int pos_period) {
  pdl_release();
  pdl_wait();
  const bool wide = (((uintptr_t)dwte | (uintptr_t)dwpe) & 15) == 0;       // d is a multiple of eight
  const int nvec = d >> 3;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < rows * nvec; i += (size_t)gridDim.x * blockDim.x) {
    const size_t row = i / nvec;
    const int c = (int)(i % nvec) * 8;
    float g[8];
    uint4 u = *(const uint4*)(dout + row * d + c);
    unpack8(u, g);
    const auto add = [&](float* dst) {
      if (wide) {
        red_add_v4(dst, g[0], g[1], g[2], g[3]);
        red_add_v4(dst + 4, g[4], g[5], g[6], g[7]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) atomicAdd(dst + j, g[j]);
      }
    };
    add(dwte + (size_t)idx[row] * d + c);
    if (dwpe) add(dwpe + (size_t)pos[row % pos_period] * d + c);
  }
}

// ============================================================================ QK-norm + RoPE
// Packed QKV [rows = B*T, (Hq + 2*Hkv) * D] bf16.  For every q and k head vector: optional RMS-norm with gain
// gamma_q / gamma_k, then NeoX rotation by cache row pos[t] (element e pairs with e + D/2); v is copied.
// A head vector is handled by D/8 adjacent lanes, each holding 8 consecutive elements (one 16-byte access), so a warp
// covers 4 (D = 64) or 2 (D = 128) vectors at a time; the lanes of the first half of the vector exchange values with
// the lanes of the second half by shuffle, and the sum of squares is reduced inside the lane group.
// Output: out (same packed shape, may alias in).  rstd (optional) [rows, Hq+Hkv] fp32.
template <int D>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = D / 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void load8_f32(const float* p, float (&v)[8]) {
  const float4 a = *(const float4*)p, b = *(const float4*)(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// One warp per token row: the row's cos / sin values (this lane's 8 positions inside a half) and its position are
// loaded once and reused for every q and k head of the row; without that reuse each head re-reads its 2 * D floats of the
// cache row, as many bytes as the packed QKV itself.  The heads of the row are swept 32 * 8 / D at a time, U sweeps' loads
// issued before the first use.
template <int D>
__global__ void __launch_bounds__(256, 3) qk_norm_rope_fwd_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out,
                                        const float* __restrict__ gq, const float* __restrict__ gk,
                                        const float* __restrict__ cache, const int64_t* __restrict__ pos,
                                        float* __restrict__ rstd, size_t rows, int T, int Hq, int Hkv, float eps,
                                        int cache_len, int* status) {
  pdl_release();
  pdl_wait();
  constexpr int GL = D / 8, VPW = 32 / GL, half = D / 2, U = 4;
  const int H = Hq + 2 * Hkv;
  const int lane = threadIdx.x & 31;
  const int gl = lane % GL;                         // lane inside its vector's group
  const int hv = lane / GL;                         // which of the VPW heads of a sweep this lane works on
  const bool second = gl >= GL / 2;                 // this lane holds elements of the second half
  const int e0 = gl * 8;                            // first element this lane holds
  const int eh = (gl % (GL / 2)) * 8;               // the same position inside a half (index into cos / sin)
  const size_t warps = (size_t)gridDim.x * (blockDim.x >> 5);
  float gqv[8], gkv[8];
  if (gq) load8_f32(gq + e0, gqv);
  if (gk) load8_f32(gk + e0, gkv);
  for (size_t row = blockIdx.x * (size_t)(blockDim.x >> 5) + (threadIdx.x >> 5); row < rows; row += warps) {
    float c[8], sn[8];
    bool have_cs = false;
    if (cache) {
      const int64_t p = pos[row % T];
      if (p >= 0 && p < cache_len) {
        const float* cr = cache + (size_t)p * D;
        load8_f32(cr + eh, c); load8_f32(cr + half + eh, sn);
        have_cs = true;
      } else {
        report(status, ST_BAD_INDEX, 400, (int)p);
      }
    }
    const __nv_bfloat16* irow = in + row * (size_t)H * D;
    __nv_bfloat16* orow = out + row * (size_t)H * D;
    for (int h0 = 0; h0 < H; h0 += VPW * U) {
      uint4 raw[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int h = h0 + u * VPW + hv;
        raw[u] = h < H ? *(const uint4*)(irow + (size_t)h * D + e0) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int h = h0 + u * VPW + hv;
        const bool live = h < H;
        const bool rot = live && h < Hq + Hkv;          // uniform inside a lane group
        const bool isq = h < Hq;
        float x[8];
        unpack8(raw[u], x);
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += x[i] * x[i];
        ss = group_sum<D>(ss);
        if (rot && (isq ? gq != nullptr : gk != nullptr)) {
          const float r = rsqrtf(ss / D + eps);
          if (rstd && gl == 0) rstd[row * (size_t)(Hq + Hkv) + h] = r;
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] = x[i] * r * (isq ? gqv[i] : gkv[i]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float other = __shfl_xor_sync(0xffffffffu, x[i], GL / 2);      // the paired element of the other half
          if (rot && have_cs) x[i] = second ? other * sn[i] + x[i] * c[i] : x[i] * c[i] - other * sn[i];
        }
        if (live) *(uint4*)(orow + (size_t)h * D + e0) = pack8(x);
      }
    }
  }
}

// Backward of the above on the packed gradient: din = d(in); dgq / dgk (fp32, +=) accumulate the gain gradients.
// `in` is the ORIGINAL (pre-norm, pre-rotation) packed QKV.  Same row-per-warp sweep as the forward kernel.
template <int D>
// Bound by memory (in, dout read, din written) and, with few rows, by latency.  The gamma gradients are added by shuffles and plain
// stores before they meet in memory: additions to shared memory are compare-and-swap loops, 32 lanes to an address here.  Cold L2,
// with those and two heads per lane and turn -> this, us: 8192 x (6 + 4) x 64 33.8 -> 21.5, 8192 x (32 + 16) x 64 66.5 -> 54.2,
// 131072 rows 657 -> 593, 32768 x 48 x 128 345 -> 308.
__global__ void __launch_bounds__(256, 2) qk_norm_rope_bwd_kernel(const __nv_bfloat16* __restrict__ in, const __nv_bfloat16* __restrict__ dout,
                                        __nv_bfloat16* __restrict__ din, const float* __restrict__ gq,
                                        const float* __restrict__ gk, const float* __restrict__ cache,
                                        const int64_t* __restrict__ pos, float* __restrict__ dgq, float* __restrict__ dgk,
                                        size_t rows, int T, int Hq, int Hkv, float eps, int cache_len) {
  pdl_release();
  pdl_wait();
  constexpr int GL = D / 8, VPW = 32 / GL, half = D / 2, U = 4;
  __shared__ float sg[8][2 * D];                   // per warp: dgq, dgk
  const int H = Hq + 2 * Hkv;
  const int lane = threadIdx.x & 31;
  const int gl = lane % GL, hv = lane / GL;
  const bool second = gl >= GL / 2;
  const int e0 = gl * 8, eh = (gl % (GL / 2)) * 8;
  const size_t warps = (size_t)gridDim.x * (blockDim.x >> 5);
  float accq[8], acck[8], gqv[8], gkv[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) accq[i] = acck[i] = 0.f;
  if (gq) load8_f32(gq + e0, gqv);
  if (gk) load8_f32(gk + e0, gkv);
  for (size_t row = blockIdx.x * (size_t)(blockDim.x >> 5) + (threadIdx.x >> 5); row < rows; row += warps) {
    float c[8], sn[8];
    bool have_cs = false;
    if (cache) {
      const int64_t p = pos[row % T];
      if (p >= 0 && p < cache_len) {
        const float* cr = cache + (size_t)p * D;
        load8_f32(cr + eh, c); load8_f32(cr + half + eh, sn);
        have_cs = true;
      }
    }
    const size_t rbase = row * (size_t)H * D;
    for (int h0 = 0; h0 < H; h0 += VPW * U) {
      uint4 rawd[U], rawx[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int h = h0 + u * VPW + hv;
        const bool live = h < H;
        const bool normed = live && h < Hq + Hkv && (h < Hq ? gq != nullptr : gk != nullptr);
        rawd[u] = live ? *(const uint4*)(dout + rbase + (size_t)h * D + e0) : make_uint4(0, 0, 0, 0);
        rawx[u] = normed ? *(const uint4*)(in + rbase + (size_t)h * D + e0) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int h = h0 + u * VPW + hv;
        const bool live = h < H;
        const bool rot = live && h < Hq + Hkv;
        const bool isq = h < Hq;
        const bool normed = rot && (isq ? gq != nullptr : gk != nullptr);
        float d[8], xh[8];
        unpack8(rawd[u], d);
        unpack8(rawx[u], xh);
        // every shuffle below is executed by the whole warp: lane groups of one warp may hold different kinds of heads
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float other = __shfl_xor_sync(0xffffffffu, d[i], GL / 2);
          if (rot && have_cs) d[i] = second ? d[i] * c[i] - other * sn[i] : d[i] * c[i] + other * sn[i];   // transpose of the rotation
        }
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += xh[i] * xh[i];
        ss = group_sum<D>(ss);
        const float r = rsqrtf(ss / D + eps);
        float dot = 0.f;
        if (normed) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            xh[i] *= r;
            if (isq) accq[i] += d[i] * xh[i]; else acck[i] += d[i] * xh[i];
            d[i] *= isq ? gqv[i] : gkv[i];
            dot += d[i] * xh[i];
          }
        }
        dot = group_sum<D>(dot) / D;
        if (normed) {
#pragma unroll
          for (int i = 0; i < 8; ++i) d[i] = r * (d[i] - xh[i] * dot);
        }
        if (live) *(uint4*)(din + rbase + (size_t)h * D + e0) = pack8(d);
      }
    }
  }
  // the lane groups of a warp by shuffles, the warps through shared memory, the blocks in global memory
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int o = GL; o < 32; o <<= 1) {
      accq[i] += __shfl_xor_sync(0xffffffffu, accq[i], o);
      acck[i] += __shfl_xor_sync(0xffffffffu, acck[i], o);
    }
  if (hv == 0) {
    float* g = sg[threadIdx.x >> 5];
#pragma unroll
    for (int i = 0; i < 8; ++i) { g[e0 + i] = accq[i]; g[D + e0 + i] = acck[i]; }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += sg[w][i];
    float* dst = i < D ? dgq : dgk;
    if (dst) atomicAdd(&dst[i < D ? i : i - D], v);
  }
}

// ============================================================================ RoPE caches
// cache[p, i] = cos(p * f_i) * m ; cache[p, i + half] = sin(p * f_i) * m, with f_i from `inv_freq` (YaRN:
// ramp-blended on the host; LongRoPE: base_freq, divided by lambda_i when p >= n_hat).
__global__ void rope_cache_kernel(float* __restrict__ cache, const float* __restrict__ inv_freq,
                                  const float* __restrict__ lambda, const int64_t* __restrict__ positions,
                                  int64_t seq_len, int half, int64_t n_hat, float mscale) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)seq_len * half; i += (size_t)gridDim.x * blockDim.x) {
    const int64_t r = (int64_t)(i / half);
    const int d = (int)(i % half);
    const int64_t p = positions ? positions[r] : r;
    float f = inv_freq[d];
    float ang = (float)p * f;
    if (lambda && p >= n_hat) ang = (float)p * f / lambda[d];
    float s, c;
    sincosf(ang, &s, &c);
    cache[(size_t)r * 2 * half + d] = c * mscale;
    cache[(size_t)r * 2 * half + d + half] = s * mscale;
  }
}
// out[r, :] = cache[labels[r], :]   (CREAM / PoSE / RandPos relabelling)
__global__ void gather_rows_f32_kernel(const float* __restrict__ src, const int64_t* __restrict__ index,
                                       float* __restrict__ out, int64_t rows, int width, int64_t src_rows, int* status) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < (size_t)rows * width; i += (size_t)gridDim.x * blockDim.x) {
    const int64_t r = (int64_t)(i / width);
    const int64_t s = index[r];
    if (s < 0 || s >= src_rows) { report(status, ST_BAD_INDEX, 410, (int)s); continue; }
    out[i] = src[(size_t)s * width + (i % width)];
  }
}

// ============================================================================ sequence permutations
// Generic gather along the sequence axis of a [outer, T_src, inner_bytes] tensor:
//   out[o, j, :] = in[o, index[j], :]       (16-byte vectors when inner_bytes % 16 == 0)
// index = HeadTail permutation -> loadbalance; inverse -> unloadbalance; local positions -> shard.
template <typename V>
__global__ void gather_seq_kernel(const V* __restrict__ in, V* __restrict__ out, const int64_t* __restrict__ index,
                                  int64_t outer, int64_t t_src, int64_t t_dst, int64_t inner, int* status) {
  const size_t total = (size_t)outer * t_dst * inner;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int64_t c = (int64_t)(i % inner);
    const int64_t j = (int64_t)((i / inner) % t_dst);
    const int64_t o = (int64_t)(i / (inner * t_dst));
    const int64_t s = index[j];
    if (s < 0 || s >= t_src) { report(status, ST_BAD_INDEX, 420, (int)s); continue; }
    out[i] = in[((size_t)o * t_src + s) * inner + c];
  }
}

// K,V (strided [B,T,H,D] views) -> contiguous [2][B,T,H,D] buffer
__global__ void kv_pack_kernel(const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
                               __nv_bfloat16* __restrict__ out, size_t rows, int hd, size_t k_row_stride, size_t v_row_stride) {
  const int nvec = hd >> 3;
  const size_t total = rows * nvec;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < 2 * total; i += (size_t)gridDim.x * blockDim.x) {
    const int which = i >= total;
    const size_t j = which ? i - total : i;
    const size_t row = j / nvec;
    const int c = (int)(j % nvec);
    const __nv_bfloat16* src = which ? v + row * v_row_stride : k + row * k_row_stride;
    ((uint4*)(out + (size_t)which * rows * hd + row * hd))[c] = ((const uint4*)src)[c];
  }
}

// ============================================================================ LSE merge
// out, blk: [B,T,H,D] bf16 ; lse, blk_lse: [B,H,T] fp32.  Rows t in [t_begin, T) are merged (t_begin = T/2
// reproduces the reference's `partial` second-half update).  One warp per (b,t,h) row.
__global__ void lse_merge_kernel(__nv_bfloat16* __restrict__ out, float* __restrict__ lse,
                                 const __nv_bfloat16* __restrict__ blk, const float* __restrict__ blk_lse,
                                 int B, int T, int H, int D, int t_begin, int blk_T, int blk_t_offset) {
  const int lane = threadIdx.x & 31;
  const size_t nrow = (size_t)B * (T - t_begin) * H;
  for (size_t w = blockIdx.x * (size_t)(blockDim.x >> 5) + (threadIdx.x >> 5); w < nrow; w += (size_t)gridDim.x * (blockDim.x >> 5)) {
    const int h = (int)(w % H);
    const int t = (int)((w / H) % (T - t_begin)) + t_begin;
    const int b = (int)(w / ((size_t)H * (T - t_begin)));
    const int tb = t - blk_t_offset;          // row inside the block result
    const float l0 = lse[((size_t)b * H + h) * T + t];
    const float l1 = blk_lse[((size_t)b * H + h) * blk_T + tb];
    float wgt, lnew;
    if (l1 == -INFINITY) { wgt = 0.f; lnew = l0; }
    else if (l0 == -INFINITY) { wgt = 1.f; lnew = l1; }
    else {
      const float dlt = l1 - l0;
      wgt = 1.f / (1.f + __expf(-dlt));
      const float mx = fmaxf(l0, l1);
      lnew = mx + log1pf(__expf(-fabsf(dlt)));
    }
    __nv_bfloat16* o = out + (((size_t)b * T + t) * H + h) * D;
    const __nv_bfloat16* s = blk + (((size_t)b * blk_T + tb) * H + h) * D;
    for (int e = lane; e < D; e += 32) {
      const float ov = __bfloat162float(o[e]), sv = __bfloat162float(s[e]);
      o[e] = __float2bfloat16(ov - wgt * (ov - sv));
    }
    if (lane == 0) lse[((size_t)b * H + h) * T + t] = lnew;
  }
}

// ============================================================================ optimiser
// partial[blockIdx.x] = sum g^2 over the block's grid-stride range ; the last block (ticket) folds the
// partials into out[0] = total sum of squares (not sqrt) so the next kernel can consume it.
__global__ void sumsq_kernel(const float* __restrict__ g, size_t n, float* __restrict__ partial,
                             unsigned int* __restrict__ ticket, float* __restrict__ out) {
  __shared__ float red[32];
  __shared__ bool last;
  float s = 0.f;
  const size_t n4 = n >> 2;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
    float4 v = ((const float4*)g)[i];
    s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  if (blockIdx.x == 0)
    for (size_t i = (n4 << 2) + threadIdx.x; i < n; i += blockDim.x) s += g[i] * g[i];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    t = warp_sum(t);
    if (threadIdx.x == 0) {
      partial[blockIdx.x] = t;
      __threadfence();
      last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
    }
  }
  __syncthreads();
  if (last) {
    float t = 0.f;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) t += ((volatile float*)partial)[i];
    t = warp_sum(t);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x < 32) {
      float u = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
      u = warp_sum(u);
      if (threadIdx.x == 0) { out[0] = u; *ticket = 0; }
    }
  }
}

// AdamW on flat fp32 master / moment buffers, writing the bf16 compute copy in the same pass.
//   gscale = grad_prescale * min(1, clip / (sqrt(sumsq)*grad_prescale + 1e-6))   (sumsq read on device, no host sync)
// If sumsq is not finite the step is skipped (NaN/Inf guard) and flag[0] is set.
// Bound by memory: 30 bytes per parameter, four parameters per thread and turn.
__global__ void adamw_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                             float* __restrict__ v, __nv_bfloat16* __restrict__ p16, size_t n, float lr, float b1,
                             float b2, float eps, float wd, float bc1, float bc2, float grad_prescale, float clip,
                             const float* __restrict__ sumsq, int* __restrict__ flag) {
  float gs = grad_prescale;
  if (sumsq) {
    const float ssq = sumsq[0];
    if (!isfinite(ssq)) { if (flag && blockIdx.x == 0 && threadIdx.x == 0) flag[0] = 1; return; }
    const float norm = sqrtf(ssq) * grad_prescale;
    if (clip > 0.f) gs *= fminf(1.f, clip / (norm + 1e-6f));
  }
  const float inv_bc2_sqrt = rsqrtf(bc2);
  const auto step = [&](float gr, float& pi, float& mi, float& vi) {
    const float gi = gr * gs;
    pi *= 1.f - lr * wd;
    mi = b1 * mi + (1.f - b1) * gi;
    vi = b2 * vi + (1.f - b2) * gi * gi;
    pi -= (lr / bc1) * mi / (sqrtf(vi) * inv_bc2_sqrt + eps);
  };
  const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x, nt = (size_t)gridDim.x * blockDim.x;
  const bool wide = ((((uintptr_t)p | (uintptr_t)g | (uintptr_t)m | (uintptr_t)v) & 15) | ((uintptr_t)p16 & 7)) == 0;
  const size_t n4 = wide ? n >> 2 : 0;
  for (size_t i = tid; i < n4; i += nt) {
    const float4 gr = ((const float4*)g)[i];
    float4 a = ((const float4*)p)[i], b = ((const float4*)m)[i], c = ((const float4*)v)[i];
    step(gr.x, a.x, b.x, c.x); step(gr.y, a.y, b.y, c.y); step(gr.z, a.z, b.z, c.z); step(gr.w, a.w, b.w, c.w);
    ((float4*)p)[i] = a; ((float4*)m)[i] = b; ((float4*)v)[i] = c;
    if (p16) ((uint2*)p16)[i] = make_uint2(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w));
  }
  for (size_t i = 4 * n4 + tid; i < n; i += nt) {
    float a = p[i], b = m[i], c = v[i];
    step(g[i], a, b, c);
    p[i] = a; m[i] = b; v[i] = c;
    if (p16) p16[i] = __float2bfloat16(a);
  }
}

// AdamW over this rank's shard of a sharded optimiser state.  master/m/v/g are shard-contiguous; every segment
// (blockIdx.y) maps a run of shard elements to the flat parameter index it updates, so the refreshed compute copy is
// written at its flat position: bf16 for matrices (decay != 0, flat index < n_decay) and fp32 for vectors.
struct AdamSeg {
  long shard_begin;     // first element inside the shard buffers
  long flat_begin;      // flat parameter index of that element
  long n;
  long decay;           // 1: weight decay applies and the compute copy is bf16; 0: no decay, fp32 copy
};
__global__ void adamw_sharded_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                                     float* __restrict__ v, __nv_bfloat16* __restrict__ p16, float* __restrict__ p32,
                                     long n_decay, const AdamSeg* __restrict__ segs, float lr, float b1, float b2,
                                     float eps, float wd, float bc1, float bc2, float grad_prescale, float clip,
                                     const float* __restrict__ sumsq, int* __restrict__ flag) {
  float gs = grad_prescale;
  if (sumsq) {
    const float ssq = sumsq[0];
    if (!isfinite(ssq)) { if (flag && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) flag[0] = 1; return; }
    const float norm = sqrtf(ssq) * grad_prescale;
    if (clip > 0.f) gs *= fminf(1.f, clip / (norm + 1e-6f));
  }
  const AdamSeg sg = segs[blockIdx.y];
  const float decay = sg.decay ? (1.f - lr * wd) : 1.f;
  const float inv_bc2_sqrt = rsqrtf(bc2);
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < sg.n; i += (long)gridDim.x * blockDim.x) {
    const long s = sg.shard_begin + i, f = sg.flat_begin + i;
    const float gi = g[s] * gs;
    float pi = p[s] * decay;
    const float mi = b1 * m[s] + (1.f - b1) * gi;
    const float vi = b2 * v[s] + (1.f - b2) * gi * gi;
    pi -= (lr / bc1) * mi / (sqrtf(vi) * inv_bc2_sqrt + eps);
    p[s] = pi; m[s] = mi; v[s] = vi;
    if (sg.decay) p16[f] = __float2bfloat16(pi);
    else p32[f - n_decay] = pi;
  }
}

__global__ void cast_f32_bf16_kernel(const float* __restrict__ in, __nv_bfloat16* __restrict__ out, size_t n, float scale) {
  pdl_release();
  pdl_wait();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16(in[i] * scale);
}
// fp32 -> bf16 rows `stride` elements apart; eight elements per thread (32 bytes in, 16 out).
struct CastPiece {
  __nv_bfloat16* out;
  size_t n8;               // sixteen-byte groups of the result
  int c8;                  // of one row
  long stride;             // elements from row to row
};
// The parts of dK and dV that several CTAs of the attention backward wrote for one K/V tile of 128 rows (see cpb_flash_attn_bwd): part j
// of a matrix starts j * n8 groups after it.
struct CastParts {
  int count;               // parts of every tile; with `local` a tile has ceil(G (nq - first visible query tile) / chunk) of them
  int local, Tk, k_off, nq, G, chunk;
};
__device__ __forceinline__ int tile_parts(const CastParts& q, size_t row) {
  if (!q.local) return q.count;
  const int seen = q.nq - max(0, q.k_off + (int)(row % q.Tk) / 128 * 128) / 128;
  return seen <= 0 ? 0 : (q.G * seen + q.chunk - 1) / q.chunk;
}
// in: the rows of `a`, then the parts of `b`, then those of `c`, added in their order.
__global__ void cast_f32_bf16_rows_kernel(const float* __restrict__ in, CastPiece a, CastPiece b, CastPiece c, CastParts q, float scale) {
  pdl_release();
  pdl_wait();
  const size_t total = a.n8 + b.n8 + c.n8;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const bool in_a = i < a.n8, in_b = !in_a && i < a.n8 + b.n8;
    __nv_bfloat16* out = in_a ? a.out : in_b ? b.out : c.out;
    const int c8 = in_a ? a.c8 : in_b ? b.c8 : c.c8;
    const long stride = in_a ? a.stride : in_b ? b.stride : c.stride;
    const size_t k = in_a ? i : in_b ? i - a.n8 : i - a.n8 - b.n8, r = k / c8;
    const float4* src = (const float4*)in + 2 * (in_a ? i : a.n8 + (in_b ? 0 : b.n8 * q.count) + k);
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
    const int parts = in_a ? 1 : tile_parts(q, r);
    if (parts > 0) { x = src[0]; y = src[1]; }
    for (int j = 1; j < parts; ++j) {
      const float4 u = src[2 * j * b.n8], v = src[2 * j * b.n8 + 1];
      x.x += u.x; x.y += u.y; x.z += u.z; x.w += u.w;
      y.x += v.x; y.y += v.y; y.z += v.z; y.w += v.w;
    }
    *(uint4*)(out + r * stride + (k - r * c8) * 8) = make_uint4(pack_bf16(x.x * scale, x.y * scale), pack_bf16(x.z * scale, x.w * scale),
                                                                pack_bf16(y.x * scale, y.y * scale), pack_bf16(y.z * scale, y.w * scale));
  }
}
__global__ void cast_bf16_f32_kernel(const __nv_bfloat16* __restrict__ in, float* __restrict__ out, size_t n, float scale, int accumulate) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float v = __bfloat162float(in[i]) * scale;
    out[i] = accumulate ? out[i] + v : v;
  }
}

static inline int grid_for(size_t work, int block, int per_sm = 8) {
  size_t g = (work + block - 1) / block;
  size_t cap = (size_t)sm_count() * per_sm;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace cpb

using namespace cpb;

#define NORM_DISPATCH(KERN, LAYER)                                                   \
  do {                                                                               \
    const int nv = (d / 8 + 31) / 32;                                                \
    if (nv <= 1) kern = KERN<LAYER, 1>;                                              \
    else if (nv <= 2) kern = KERN<LAYER, 2>;                                         \
    else if (nv <= 4) kern = KERN<LAYER, 4>;                                         \
    else if (nv <= 8) kern = KERN<LAYER, 8>;                                         \
    else if (nv <= 16) kern = KERN<LAYER, 16>;                                       \
    else return set_error(CPB_ERR_LIMIT, "norm: d=%d exceeds 4096", d);              \
  } while (0)

// x (+res) -> xout (only when res != null), y ; stats [rows,2] (mean, rstd) optional
extern "C" int cpb_norm_fwd(const void* x, const void* res, const float* w, const float* b, void* xout, void* y,
                            float* stats, int rows, int d, float eps, int layer, cudaStream_t stream) {
  if (d % 8) return set_error(CPB_ERR_ARG, "norm: d=%d must be a multiple of 8", d);
  if (rows <= 0) return CPB_OK;
  const int wpb = 8;
  decltype(&norm_fwd_kernel<true, 1>) kern;
  if (layer) NORM_DISPATCH(norm_fwd_kernel, true);
  else NORM_DISPATCH(norm_fwd_kernel, false);
  CPB_CUDA_OK(launch_pdl(kern, (rows + wpb - 1) / wpb, wpb * 32, 0, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)res, w, b, (__nv_bfloat16*)xout, (__nv_bfloat16*)y, stats, rows, d, eps));
  return check_launch("norm_fwd");
}

// dw / db are fp32 and accumulated into (+=).
extern "C" int cpb_norm_bwd(const void* x, const void* dy, const void* dres, const float* w, const float* stats,
                            void* dx, float* dw, float* db, int rows, int d, int layer, cudaStream_t stream) {
  if (d % 8) return set_error(CPB_ERR_ARG, "norm: d=%d must be a multiple of 8", d);
  if (rows <= 0) return CPB_OK;
  const int nvec = d / 8;
  if (nvec > 512) return set_error(CPB_ERR_LIMIT, "norm: d=%d exceeds 4096", d);
#define NORM_BWD(G)                                                                                                             \
  do {                                                                                                                          \
    const int tb = G > 256 ? 512 : 256, per_block = 4 * (tb / G);                                                               \
    const int cap = sm_count() * (G > 256 ? 1 : 2), need = (rows + per_block - 1) / per_block, blocks = need < cap ? need : cap; \
    auto kern = layer ? norm_bwd_kernel<true, G> : norm_bwd_kernel<false, G>;                                                   \
    CPB_CUDA_OK(launch_pdl(kern, blocks, tb, 0, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)dres, w, stats,    \
                                    (__nv_bfloat16*)dx, dw, db, rows, d));                                                       \
  } while (0)
  if (nvec <= 32) NORM_BWD(32);
  else if (nvec <= 64) NORM_BWD(64);
  else if (nvec <= 128) NORM_BWD(128);
  else if (nvec <= 256) NORM_BWD(256);
  else NORM_BWD(512);
#undef NORM_BWD
  return check_launch("norm_bwd");
}

extern "C" int cpb_swiglu_fwd(const void* gu, void* act, long rows, int F, cudaStream_t stream) {
  if (F % 8) return set_error(CPB_ERR_ARG, "swiglu: F must be a multiple of 8");
  if (rows <= 0) return CPB_OK;
  CPB_CUDA_OK(launch_pdl(swiglu_fwd_kernel, grid_for((size_t)rows * (F / 8), 256), 256, 0, stream, (const __nv_bfloat16*)gu, (__nv_bfloat16*)act, (size_t)rows, F));
  return check_launch("swiglu_fwd");
}
extern "C" int cpb_swiglu_bwd(const void* gu, const void* dact, void* dgu, long rows, int F, cudaStream_t stream) {
  if (F % 8) return set_error(CPB_ERR_ARG, "swiglu: F must be a multiple of 8");
  if (rows <= 0) return CPB_OK;
  CPB_CUDA_OK(launch_pdl(swiglu_bwd_kernel, grid_for((size_t)rows * (F / 8), 256), 256, 0, stream, (const __nv_bfloat16*)gu, (const __nv_bfloat16*)dact, (__nv_bfloat16*)dgu, (size_t)rows, F));
  return check_launch("swiglu_bwd");
}
extern "C" int cpb_gelu(const void* x, const void* dy, void* y, long n, int mode, cudaStream_t stream) {
  if (n % 8) return set_error(CPB_ERR_ARG, "gelu: n must be a multiple of 8");
  if (n <= 0) return CPB_OK;
  CPB_CUDA_OK(launch_pdl(gelu_kernel, grid_for((size_t)n / 8, 256), 256, 0, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)dy, (__nv_bfloat16*)y, (size_t)n / 8, mode));
  return check_launch("gelu");
}
extern "C" int cpb_add_bf16(const void* a, const void* b, void* y, long n, cudaStream_t stream) {
  if (n % 8) return set_error(CPB_ERR_ARG, "add: n must be a multiple of 8");
  if (n <= 0) return CPB_OK;
  add_kernel<<<grid_for((size_t)n / 8, 256), 256, 0, stream>>>((const __nv_bfloat16*)a, (const __nv_bfloat16*)b, (__nv_bfloat16*)y, (size_t)n / 8);
  return check_launch("add");
}
extern "C" int cpb_bias_grad(const void* dy, float* db, int rows, int N, cudaStream_t stream) {
  if (N % 2) return set_error(CPB_ERR_ARG, "bias_grad: N must be even");
  if (rows <= 0) return CPB_OK;
  int rb = sm_count() * 4 / ((N + 63) / 64);
  if (rb < 1) rb = 1;
  int rpb = (rows + rb - 1) / rb;
  if (rpb < 64) rpb = 64;
  rb = (rows + rpb - 1) / rpb;
  CPB_CUDA_OK(launch_pdl(bias_grad_kernel, dim3((N + 63) / 64, rb), 256, 0, stream, (const __nv_bfloat16*)dy, db, rows, N, rpb));
  return check_launch("bias_grad");
}
extern "C" int cpb_embedding_fwd(const int64_t* idx, const int64_t* pos, const void* wte, const void* wpe, void* out,
                                 long rows, int d, int pos_period, cudaStream_t stream) {
  if (d % 8) return set_error(CPB_ERR_ARG, "embedding: d must be a multiple of 8");
  if (rows <= 0) return CPB_OK;
  CPB_CUDA_OK(launch_pdl(embedding_fwd_kernel, grid_for((size_t)rows * (d / 8), 256), 256, 0, stream, idx, pos, (const __nv_bfloat16*)wte, (const __nv_bfloat16*)wpe, (__nv_bfloat16*)out, (size_t)rows, d, pos_period));
  return check_launch("embedding_fwd");
}
extern "C" int cpb_embedding_bwd(const int64_t* idx, const int64_t* pos, const void* dout, float* dwte, float* dwpe,
                                 long rows, int d, int pos_period, cudaStream_t stream) {
  if (d % 8) return set_error(CPB_ERR_ARG, "embedding: d must be a multiple of 8");
  if (rows <= 0) return CPB_OK;
  CPB_CUDA_OK(launch_pdl(embedding_bwd_kernel, grid_for((size_t)rows * (d / 8), 256), 256, 0, stream, idx, pos, (const __nv_bfloat16*)dout, dwte, dwpe, (size_t)rows, d, pos_period));
  return check_launch("embedding_bwd");
}

extern "C" int cpb_qk_norm_rope_fwd(const void* in, void* out, const float* gq, const float* gk, const float* cache,
                                    const int64_t* pos, float* rstd, long rows, int T, int Hq, int Hkv, int D,
                                    float eps, int cache_len, int* status, cudaStream_t stream) {
  if (rows <= 0) return CPB_OK;
  const int grid = grid_for((size_t)rows, 8, 3);      // one warp per token row, eight warps per block
  if (D == 64) CPB_CUDA_OK(launch_pdl(qk_norm_rope_fwd_kernel<64>, grid, 256, 0, stream, (const __nv_bfloat16*)in, (__nv_bfloat16*)out, gq, gk, cache, pos, rstd, (size_t)rows, T, Hq, Hkv, eps, cache_len, status));
  else if (D == 128) CPB_CUDA_OK(launch_pdl(qk_norm_rope_fwd_kernel<128>, grid, 256, 0, stream, (const __nv_bfloat16*)in, (__nv_bfloat16*)out, gq, gk, cache, pos, rstd, (size_t)rows, T, Hq, Hkv, eps, cache_len, status));
  else return set_error(CPB_ERR_ARG, "qk_norm_rope: head_dim %d not in {64,128}", D);
  return check_launch("qk_norm_rope_fwd");
}
extern "C" int cpb_qk_norm_rope_bwd(const void* in, const void* dout, void* din, const float* gq, const float* gk,
                                    const float* cache, const int64_t* pos, float* dgq, float* dgk, long rows, int T,
                                    int Hq, int Hkv, int D, float eps, int cache_len, cudaStream_t stream) {
  if (rows <= 0) return CPB_OK;
  const int grid = grid_for((size_t)rows, 8, 2);         // as many blocks as fit: each ends with additions to the same 2 D values
  if (D == 64) CPB_CUDA_OK(launch_pdl(qk_norm_rope_bwd_kernel<64>, grid, 256, 0, stream, (const __nv_bfloat16*)in, (const __nv_bfloat16*)dout, (__nv_bfloat16*)din, gq, gk, cache, pos, dgq, dgk, (size_t)rows, T, Hq, Hkv, eps, cache_len));
  else if (D == 128) CPB_CUDA_OK(launch_pdl(qk_norm_rope_bwd_kernel<128>, grid, 256, 0, stream, (const __nv_bfloat16*)in, (const __nv_bfloat16*)dout, (__nv_bfloat16*)din, gq, gk, cache, pos, dgq, dgk, (size_t)rows, T, Hq, Hkv, eps, cache_len));
  else return set_error(CPB_ERR_ARG, "qk_norm_rope: head_dim %d not in {64,128}", D);
  return check_launch("qk_norm_rope_bwd");
}

extern "C" int cpb_rope_cache(float* cache, const float* inv_freq, const float* lambda, const int64_t* positions,
                              long seq_len, int half, long n_hat, float mscale, cudaStream_t stream) {
  if (seq_len <= 0) return CPB_OK;
  rope_cache_kernel<<<grid_for((size_t)seq_len * half, 256), 256, 0, stream>>>(cache, inv_freq, lambda, positions, seq_len, half, n_hat, mscale);
  return check_launch("rope_cache");
}
extern "C" int cpb_gather_rows_f32(const float* src, const int64_t* index, float* out, long rows, int width,
                                   long src_rows, int* status, cudaStream_t stream) {
  if (rows <= 0) return CPB_OK;
  gather_rows_f32_kernel<<<grid_for((size_t)rows * width, 256), 256, 0, stream>>>(src, index, out, rows, width, src_rows, status);
  return check_launch("gather_rows_f32");
}
// in/out: [outer, T, inner_bytes] raw bytes
extern "C" int cpb_gather_seq(const void* in, void* out, const int64_t* index, long outer, long t_src, long t_dst,
                              long inner_bytes, int* status, cudaStream_t stream) {
  if (outer * t_dst * inner_bytes <= 0) return CPB_OK;
  const bool vec16 = (inner_bytes % 16 == 0) && (((uintptr_t)in | (uintptr_t)out) % 16 == 0);
  if (vec16) {
    const long inner = inner_bytes / 16;
    gather_seq_kernel<uint4><<<grid_for((size_t)outer * t_dst * inner, 256), 256, 0, stream>>>((const uint4*)in, (uint4*)out, index, outer, t_src, t_dst, inner, status);
  } else if (inner_bytes % 8 == 0 && (((uintptr_t)in | (uintptr_t)out) % 8 == 0)) {
    const long inner = inner_bytes / 8;
    gather_seq_kernel<uint2><<<grid_for((size_t)outer * t_dst * inner, 256), 256, 0, stream>>>((const uint2*)in, (uint2*)out, index, outer, t_src, t_dst, inner, status);
  } else {
    gather_seq_kernel<uint8_t><<<grid_for((size_t)outer * t_dst * inner_bytes, 256), 256, 0, stream>>>((const uint8_t*)in, (uint8_t*)out, index, outer, t_src, t_dst, inner_bytes, status);
  }
  return check_launch("gather_seq");
}
extern "C" int cpb_kv_pack(const void* k, const void* v, void* out, long rows, int hd, long k_row_stride,
                           long v_row_stride, cudaStream_t stream) {
  if (hd % 8 || k_row_stride % 8 || v_row_stride % 8) return set_error(CPB_ERR_ARG, "kv_pack: sizes must be multiples of 8 elements");
  if (rows <= 0) return CPB_OK;
  kv_pack_kernel<<<grid_for((size_t)2 * rows * (hd / 8), 256), 256, 0, stream>>>((const __nv_bfloat16*)k, (const __nv_bfloat16*)v, (__nv_bfloat16*)out, (size_t)rows, hd, (size_t)k_row_stride, (size_t)v_row_stride);
  return check_launch("kv_pack");
}
extern "C" int cpb_lse_merge(void* out, float* lse, const void* blk, const float* blk_lse, int B, int T, int H, int D,
                             int t_begin, int blk_T, int blk_t_offset, cudaStream_t stream) {
  const size_t nrow = (size_t)B * (T - t_begin) * H;
  if (nrow == 0) return CPB_OK;
  lse_merge_kernel<<<grid_for(nrow, 8), 256, 0, stream>>>((__nv_bfloat16*)out, lse, (const __nv_bfloat16*)blk, blk_lse, B, T, H, D, t_begin, blk_T, blk_t_offset);
  return check_launch("lse_merge");
}

// scratch: >= (1024 + 2) floats: [0..1023] partials, [1024] ticket (zero-initialised once), out separate
extern "C" int cpb_sumsq(const float* g, long n, float* partial, unsigned int* ticket, float* out, cudaStream_t stream) {
  int grid = grid_for((size_t)(n / 4 + 1), 256, 4);
  if (grid > 1024) grid = 1024;
  sumsq_kernel<<<grid, 256, 0, stream>>>(g, (size_t)n, partial, ticket, out);
  return check_launch("sumsq");
}
// segs: device array of {shard_begin, flat_begin, n, decay} (four longs each).
extern "C" int cpb_adamw_sharded(float* p, const float* g, float* m, float* v, void* p16, float* p32, long n_decay,
                                 const void* segs, int n_segs, int ctas_per_seg, float lr, float b1, float b2, float eps,
                                 float wd, int step, float grad_prescale, float clip, const float* sumsq, int* flag,
                                 cudaStream_t stream) {
  if (n_segs <= 0) return CPB_OK;
  if (n_segs > 65535) return set_error(CPB_ERR_LIMIT, "adamw_sharded: at most 65535 segments");
  const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  dim3 grid(ctas_per_seg < 1 ? 1 : ctas_per_seg, n_segs);
  adamw_sharded_kernel<<<grid, 256, 0, stream>>>(p, g, m, v, (__nv_bfloat16*)p16, p32, n_decay, (const AdamSeg*)segs, lr, b1, b2,
                                                 eps, wd, bc1, bc2, grad_prescale, clip, sumsq, flag);
  return check_launch("adamw_sharded");
}

extern "C" int cpb_adamw(float* p, const float* g, float* m, float* v, void* p16, long n, float lr, float b1, float b2,
                         float eps, float wd, int step, float grad_prescale, float clip, const float* sumsq, int* flag,
                         cudaStream_t stream) {
  if (n <= 0) return CPB_OK;
  const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  adamw_kernel<<<grid_for((size_t)n, 256), 256, 0, stream>>>(p, g, m, v, (__nv_bfloat16*)p16, (size_t)n, lr, b1, b2, eps, wd, bc1, bc2, grad_prescale, clip, sumsq, flag);
  return check_launch("adamw");
}
// in: fp32, rows_q x cols_q values and then twice `parts` matrices of rows_k x cols_k (parts 0: none), the parts to be added; each result goes
// to bf16 rows q_stride / kv_stride elements apart.  Tk, k_off, nq, G, chunk, local: see CastParts.
extern "C" int cpb_cast_f32_bf16_rows(const float* in, void* out_q, long rows_q, int cols_q, long q_stride, void* out_k, void* out_v, long rows_k,
                                      int cols_k, long kv_stride, int parts, int Tk, int k_off, int nq, int G, int chunk, int local, float scale,
                                      cudaStream_t stream) {
  if ((cols_q % 8) || (q_stride % 8) || ((uintptr_t)in & 15) || ((uintptr_t)out_q & 15)) return set_error(CPB_ERR_ARG, "cast_rows: columns, stride and pointers must be multiples of 16 bytes");
  if (parts > 0 && ((cols_k % 8) || (kv_stride % 8) || (((uintptr_t)out_k | (uintptr_t)out_v) & 15) || Tk <= 0 || chunk <= 0))
    return set_error(CPB_ERR_ARG, "cast_rows: columns, stride and pointers must be multiples of 16 bytes");
  const CastPiece q{(__nv_bfloat16*)out_q, (size_t)(rows_q > 0 ? rows_q : 0) * (cols_q / 8), cols_q > 0 ? cols_q / 8 : 1, q_stride};
  const size_t nk = parts > 0 ? (size_t)rows_k * (cols_k / 8) : 0;
  const CastPiece k{(__nv_bfloat16*)out_k, nk, cols_k > 0 ? cols_k / 8 : 1, kv_stride}, v{(__nv_bfloat16*)out_v, nk, k.c8, kv_stride};
  const size_t total = q.n8 + 2 * nk;
  if (total == 0) return CPB_OK;
  CPB_CUDA_OK(launch_pdl(cast_f32_bf16_rows_kernel, grid_for(total, 256, 32), 256, 0, stream, in, q, k, v, CastParts{parts, local, Tk, k_off, nq, G, chunk}, scale));
  return check_launch("cast_rows");
}
extern "C" int cpb_cast_f32_bf16(const float* in, void* out, long n, float scale, cudaStream_t stream) {
  if (n <= 0) return CPB_OK;
  if (n % 8 == 0 && (((uintptr_t)in | (uintptr_t)out) & 15) == 0)
    return cpb_cast_f32_bf16_rows(in, out, n / 8, 8, 8, nullptr, nullptr, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, scale, stream);
  CPB_CUDA_OK(launch_pdl(cast_f32_bf16_kernel, grid_for((size_t)n, 256), 256, 0, stream, in, (__nv_bfloat16*)out, (size_t)n, scale));
  return check_launch("cast_f32_bf16");
}
extern "C" int cpb_cast_bf16_f32(const void* in, float* out, long n, float scale, int accumulate, cudaStream_t stream) {
  if (n <= 0) return CPB_OK;
  cast_bf16_f32_kernel<<<grid_for((size_t)n, 256), 256, 0, stream>>>((const __nv_bfloat16*)in, out, (size_t)n, scale, accumulate);
  return check_launch("cast_bf16_f32");
}
