// Softmax cross-entropy.  The language-model head never materialises [tokens, vocab] for the whole sequence: the host loops over row
// chunks, the head's GEMM leaves statistics per column tile (gemm_common.cuh), xent_rows_kernel makes losses and gradient coefficients of
// them and xent_dlogits_kernel dlogits = (softmax - onehot) * grad_scale of logits that were stored; two more GEMMs then produce dX
// and accumulate dW.  Replaces the reference's materialised logits + sparse_cross_entropy_loss (Scripts/Blutrain/bluscriptCP.cpp:452-459,1712).
//
// cpb_xent is for fp32 logits that a caller has: loss and dlogits in one launch.  With gradients the row is read from memory once: a
// cluster of CTAs keeps it in shared memory between the two passes (xent_smem_kernel).  Without gradients, or when a row does not fit, one
// CTA per row computes max and sum(exp) online and, if asked to, re-reads the row for dlogits (xent_kernel).  Rows whose target is
// negative are ignored everywhere (zero gradient, no loss).
#include "common.cuh"
#include "host_utils.h"

namespace cpb {

__global__ void __launch_bounds__(512)
xent_kernel(const float* __restrict__ logits, const int64_t* __restrict__ targets, __nv_bfloat16* __restrict__ dlogits,
            float* __restrict__ loss_sum, float* __restrict__ row_loss, int rows, int V, int Vcols, long ld_logits, long ld_dlogits,
            float grad_scale, int* status) {
  pdl_release();
  pdl_wait();
  __shared__ float red_m[16], red_s[16];
  __shared__ float s_max, s_sum;
  const int row = blockIdx.x;
  if (row >= rows) return;
  const float* x = logits + (size_t)row * ld_logits;
  const int64_t tgt = targets[row];
  if (tgt >= V) report(status, ST_BAD_INDEX, 1200, (int)tgt);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float m = -INFINITY, s = 0.f;
  const int V4 = V >> 2;
  for (int i = threadIdx.x; i < V4; i += blockDim.x) {
    const float4 v = ((const float4*)x)[i];
    const float mx = fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w));
    if (mx > m) { s *= __expf(m - mx); m = mx; }
    s += __expf(v.x - m) + __expf(v.y - m) + __expf(v.z - m) + __expf(v.w - m);
  }
  for (int i = (V4 << 2) + threadIdx.x; i < V; i += blockDim.x) {
    const float v = x[i];
    if (v > m) { s *= __expf(m - v); m = v; }
    s += __expf(v - m);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
    const float mn = fmaxf(m, m2);
    s = (m == -INFINITY ? 0.f : s * __expf(m - mn)) + (m2 == -INFINITY ? 0.f : s2 * __expf(m2 - mn));
    m = mn;
  }
  if (lane == 0) { red_m[warp] = m; red_s[warp] = s; }
  __syncthreads();
  if (warp == 0) {
    m = lane < nw ? red_m[lane] : -INFINITY;
    s = lane < nw ? red_s[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
      const float mn = fmaxf(m, m2);
      s = (m == -INFINITY ? 0.f : s * __expf(m - mn)) + (m2 == -INFINITY ? 0.f : s2 * __expf(m2 - mn));
      m = mn;
    }
    if (lane == 0) { s_max = m; s_sum = s; }
  }
  __syncthreads();
  m = s_max; s = s_sum;
  const bool ignore = tgt < 0 || tgt >= V;
  if (threadIdx.x == 0) {
    const float l = ignore ? 0.f : (m + __logf(s) - x[tgt]);
    if (row_loss) row_loss[row] = l;
    if (loss_sum && !ignore) atomicAdd(loss_sum, l);
  }
  if (dlogits == nullptr) return;
  __nv_bfloat16* d = dlogits + (size_t)row * ld_dlogits;
  const float inv = ignore ? 0.f : grad_scale / s;
  const int VC4 = Vcols >> 2;       // Vcols (>= V, multiple of 4): padded width; padding columns get zero gradient
  for (int i = threadIdx.x; i < VC4; i += blockDim.x) {
    const float4 v = ((const float4*)x)[i];
    const int c = i << 2;
    float p0 = c < V ? __expf(v.x - m) * inv : 0.f, p1 = c + 1 < V ? __expf(v.y - m) * inv : 0.f;
    float p2 = c + 2 < V ? __expf(v.z - m) * inv : 0.f, p3 = c + 3 < V ? __expf(v.w - m) * inv : 0.f;
    if (!ignore && tgt >= c && tgt < c + 4) {
      if (tgt == c) p0 -= grad_scale; else if (tgt == c + 1) p1 -= grad_scale; else if (tgt == c + 2) p2 -= grad_scale; else p3 -= grad_scale;
    }
    *(uint2*)(d + c) = make_uint2(pack_bf16(p0, p1), pack_bf16(p2, p3));
  }
}

// Bytes of a row that one CTA of a cluster keeps: two such CTAs fit an SM, so one computes while the other's row arrives (four
// CTAs of half the size and clusters of twice as many: 300 and 805 us at the sizes below).
constexpr int XE_SEG_BYTES = 104 * 1024;
constexpr int XE_PARTS = 4;            // bulk copies per segment: the first pass starts when a quarter has arrived
constexpr int XE_THREADS = 512;

// x, m, s: online softmax over four values at once
__device__ __forceinline__ void xe_online4(const float4 v, float& m, float& s) {
  const float mx = fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w));
  if (mx > m) { s *= __expf(m - mx); m = mx; }
  s += __expf(v.x - m) + __expf(v.y - m) + __expf(v.z - m) + __expf(v.w - m);
}
__device__ __forceinline__ void xe_merge(float& m, float& s, float m2, float s2) {
  const float mn = fmaxf(m, m2);
  s = (m == -INFINITY ? 0.f : s * __expf(m - mn)) + (m2 == -INFINITY ? 0.f : s2 * __expf(m2 - mn));
  m = mn;
}

// Bound by memory: 4 bytes in and 2 out per logit.  One CTA per row that re-reads the row for the second pass moved 10 bytes
// instead of 6, because the rows in flight (four per SM, 119 MB at 50304 columns) do not stay in L2.  Here cluster rank r
// loads columns [r seg, (r+1) seg) with bulk copies, the ranks exchange (max, sum) through distributed shared memory, and
// the second pass reads shared memory.  Measured, cold L2, one CTA per
// row -> cluster: 4096 x 50304 323 -> 274 us, 4096 x 128256 808 -> 746, 1000 x 50304 94 -> 78.
__global__ void __launch_bounds__(XE_THREADS)
xent_smem_kernel(const float* __restrict__ logits, const int64_t* __restrict__ targets, __nv_bfloat16* __restrict__ dlogits,
                 float* __restrict__ loss_sum, float* __restrict__ row_loss, int V, int Vcols, int seg, int ranks,
                 long ld_logits, long ld_dlogits, float grad_scale, int* status) {
  pdl_release();
  pdl_wait();
  extern __shared__ __align__(16) float xs[];
  __shared__ __align__(8) uint64_t bars[XE_PARTS];
  __shared__ float red_m[XE_THREADS / 32], red_s[XE_THREADS / 32];
  __shared__ float2 mine;                                          // this rank's (max, sum)
  __shared__ int abort_flag;
  const int rank = (int)(blockIdx.x % ranks), row = (int)(blockIdx.x / ranks);
  const int c0 = rank * seg, n = min(seg, Vcols - c0);             // columns of this rank (a multiple of four)
  const int part = (n / 4 + XE_PARTS - 1) / XE_PARTS * 4;
  const float* x = logits + (size_t)row * ld_logits;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    for (int i = 0; i < XE_PARTS; ++i) mbar_init(&bars[i], 1);
    abort_flag = 0;
    fence_mbar_init();
    for (int i = 0; i < XE_PARTS; ++i) {
      const int len = min(part, n - i * part);
      if (len <= 0) break;
      mbar_expect_tx(&bars[i], len * 4);
      bulk_load_1d(xs + i * part, x + c0 + i * part, len * 4, &bars[i]);
    }
  }
  const int64_t tgt = targets[row];
  __syncthreads();
  float m = -INFINITY, s = 0.f;
  bool ok = true;
  for (int i = 0; i < XE_PARTS && i * part < n; ++i) {
    ok = ok && mbar_wait(&bars[i], 0, &abort_flag, status, 1210);
    if (!ok) break;
    const int end = min((i + 1) * part, n);
    for (int c = i * part + 4 * (int)threadIdx.x; c < end; c += 4 * XE_THREADS) {
      const float4 v = *(const float4*)(xs + c);
      if (c0 + c + 3 < V) {
        xe_online4(v, m, s);
      } else {
        const float e[4] = {v.x, v.y, v.z, v.w};
        for (int k = 0; k < 4; ++k)
          if (c0 + c + k < V) {
            if (e[k] > m) { s *= __expf(m - e[k]); m = e[k]; }
            s += __expf(e[k] - m);
          }
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) xe_merge(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
  if (lane == 0) { red_m[warp] = m; red_s[warp] = s; }
  __syncthreads();
  if (warp == 0) {
    m = lane < XE_THREADS / 32 ? red_m[lane] : -INFINITY;
    s = lane < XE_THREADS / 32 ? red_s[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) xe_merge(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
    if (lane == 0) mine = make_float2(m, s);
  }
  __syncwarp();                                                    // the aligned forms want the whole warp at the same instruction
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  m = -INFINITY; s = 0.f;
  for (int r = 0; r < ranks; ++r) {
    uint32_t addr;
    float m2, s2;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(&mine)), "r"(r));
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(m2), "=f"(s2) : "r"(addr) : "memory");
    xe_merge(m, s, m2, s2);
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");    // this thread has read every rank's pair
  const bool ignore = tgt < 0 || tgt >= V;
  if (rank == 0 && threadIdx.x == 0) {
    if (tgt >= V) report(status, ST_BAD_INDEX, 1200, (int)tgt);
    const float l = ignore ? 0.f : (m + __logf(s) - x[tgt]);
    if (row_loss) row_loss[row] = l;
    if (loss_sum && !ignore) atomicAdd(loss_sum, l);
  }
  if (ok) {
    __nv_bfloat16* d = dlogits + (size_t)row * ld_dlogits + c0;
    const float inv = ignore ? 0.f : grad_scale / s;
    const int t = ignore || tgt < c0 || tgt >= c0 + n ? -1 : (int)(tgt - c0);
    for (int c = 4 * (int)threadIdx.x; c < n; c += 4 * XE_THREADS) {
      const float4 v = *(const float4*)(xs + c);
      float p0 = c0 + c < V ? __expf(v.x - m) * inv : 0.f, p1 = c0 + c + 1 < V ? __expf(v.y - m) * inv : 0.f;
      float p2 = c0 + c + 2 < V ? __expf(v.z - m) * inv : 0.f, p3 = c0 + c + 3 < V ? __expf(v.w - m) * inv : 0.f;
      if ((t & ~3) == c) {
        if (t == c) p0 -= grad_scale; else if (t == c + 1) p1 -= grad_scale; else if (t == c + 2) p2 -= grad_scale; else p3 -= grad_scale;
      }
      *(uint2*)(d + c) = make_uint2(pack_bf16(p0, p1), pack_bf16(p2, p3));
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");      // no rank leaves while another may still read its pair
}

// Between the two passes of the head's GEMM (cpb_gemm_head): per row the maximum and the sum of exponentials over all column tiles,
// the loss, and the coefficients of the gradient.  A block takes 32 rows, a warp every eighth tile of them (the lanes' pairs are
// adjacent in memory), and warp 0 adds the eight parts, always in the same order.
constexpr int XR_WARPS = 8;
__global__ void __launch_bounds__(XR_WARPS * 32)
xent_rows_kernel(const float2* __restrict__ stats, const float* __restrict__ target_logit, const int64_t* __restrict__ targets,
                 float2* __restrict__ row_coef, float* __restrict__ row_loss, float* __restrict__ loss_sum, int rows, int tiles, int V,
                 float grad_scale, int* status) {
  pdl_release();
  pdl_wait();
  __shared__ float2 part[XR_WARPS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = blockIdx.x * 32 + lane;
  float m = -INFINITY, s = 0.f;
  // a part without a finite maximum contributes its sum as it is: zero, or NaN
  const auto add = [&](float2 v) {
    const float mn = fmaxf(m, v.x);
    s = (m == -INFINITY ? s : s * __expf(m - mn)) + (v.x == -INFINITY ? v.y : v.y * __expf(v.x - mn));
    m = mn;
  };
  if (row < rows) {
    int t = warp;
    for (; t + 3 * XR_WARPS < tiles; t += 4 * XR_WARPS) {
      float2 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = stats[(size_t)(t + k * XR_WARPS) * rows + row];
#pragma unroll
      for (int k = 0; k < 4; ++k) add(v[k]);
    }
    for (; t < tiles; t += XR_WARPS) add(stats[(size_t)t * rows + row]);
  }
  part[warp][lane] = make_float2(m, s);
  __syncthreads();
  if (warp != 0) return;
  for (int k = 1; k < XR_WARPS; ++k) add(part[k][lane]);
  float l = 0.f;
  if (row < rows) {
    const int64_t tgt = targets[row];
    if (tgt >= V) report(status, ST_BAD_INDEX, 1200, (int)tgt);
    const bool ignore = tgt < 0 || tgt >= V;
    if (!ignore) l = m + __logf(s) - target_logit[row];
    if (row_loss) row_loss[row] = l;
    if (row_coef) row_coef[row] = make_float2(m, ignore ? 0.f : grad_scale / s);
  }
  if (loss_sum) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (lane == 0) atomicAdd(loss_sum, l);
  }
}

// dlogits = (softmax - onehot) * grad_scale from stored logits and the rows' (max, grad_scale / sum).  Bound by memory: 4 bytes in and 2
// out per logit; four 16-byte loads per thread before the first use.
constexpr int XD_COLS = 256 * 16;
__global__ void __launch_bounds__(256)
xent_dlogits_kernel(const float* __restrict__ logits, const int64_t* __restrict__ targets, const float2* __restrict__ row_coef,
                    __nv_bfloat16* __restrict__ dlogits, int V, int Vcols, long ld_logits, long ld_dlogits, float grad_scale) {
  pdl_release();
  pdl_wait();
  const int row = blockIdx.y, c0 = blockIdx.x * XD_COLS + 4 * threadIdx.x;
  const float4* x = (const float4*)(logits + (size_t)row * ld_logits);
  const float2 coef = row_coef[row];
  const int64_t tgt = targets[row];
  float4 v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) if (c0 + 1024 * k < Vcols) v[k] = x[(c0 + 1024 * k) >> 2];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = c0 + 1024 * k;
    if (c >= Vcols) break;
    float p[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      p[e] = c + e < V ? __expf(p[e] - coef.x) * coef.y : 0.f;
      if (tgt == c + e && c + e < V) p[e] -= grad_scale;
    }
    *(uint2*)(dlogits + (size_t)row * ld_dlogits + c) = make_uint2(pack_bf16(p[0], p[1]), pack_bf16(p[2], p[3]));
  }
}

}  // namespace cpb

using namespace cpb;

// logits fp32 [rows, Vcols] and row_coef as written by cpb_gemm_head and cpb_xent_rows; dlogits bf16 [rows, Vcols], zero from column V on.
extern "C" int cpb_xent_dlogits(const float* logits, const int64_t* targets, const float* row_coef, void* dlogits, int rows, int V, int Vcols,
                                long ld_logits, long ld_dlogits, float grad_scale, cudaStream_t stream) {
  if (rows <= 0) return CPB_OK;
  if (Vcols < V || (Vcols % 4) || (ld_logits % 4) || (ld_dlogits % 4) || ((uintptr_t)logits & 15) || ((uintptr_t)dlogits & 7) || rows > 65535)
    return set_error(CPB_ERR_ARG, "xent_dlogits: columns and strides must be multiples of 4, rows at most 65535");
  CPB_CUDA_OK(launch_pdl(xent_dlogits_kernel, dim3((Vcols + XD_COLS - 1) / XD_COLS, rows), 256, 0, stream, logits, targets, (const float2*)row_coef,
                         (__nv_bfloat16*)dlogits, V, Vcols, ld_logits, ld_dlogits, grad_scale));
  return check_launch("xent_dlogits");
}

// stats [tiles][rows] (max, sum) pairs and target_logit [rows] of cpb_gemm_head; row_coef [rows] pairs, row_loss [rows] and
// loss_sum (fp32 scalar, +=) are optional.  V: columns that are real vocabulary.
extern "C" int cpb_xent_rows(const float* stats, const float* target_logit, const int64_t* targets, float* row_coef, float* row_loss,
                             float* loss_sum, int rows, int tiles, int V, float grad_scale, int* status, cudaStream_t stream) {
  if (rows <= 0) return CPB_OK;
  CPB_CUDA_OK(launch_pdl(xent_rows_kernel, (rows + 31) / 32, XR_WARPS * 32, 0, stream, (const float2*)stats, target_logit, targets, (float2*)row_coef, row_loss,
                                                                    loss_sum, rows, tiles, V, grad_scale, status));
  return check_launch("xent_rows");
}

// logits fp32 [rows, Vcols] (row stride ld_logits, multiple of 4) of which the first V columns are real vocabulary;
// dlogits bf16 [rows, Vcols] (row stride multiple of 4) or null; loss_sum (fp32 scalar, +=) and row_loss [rows] optional.
extern "C" int cpb_xent(const float* logits, const int64_t* targets, void* dlogits, float* loss_sum, float* row_loss,
                        int rows, int V, int Vcols, long ld_logits, long ld_dlogits, float grad_scale, int* status, cudaStream_t stream) {
  if (rows <= 0) return CPB_OK;
  if (Vcols < V || (Vcols % 4)) return set_error(CPB_ERR_ARG, "xent: Vcols must be >= V and a multiple of 4");
  if ((ld_logits % 4) || (dlogits && (ld_dlogits % 4))) return set_error(CPB_ERR_ARG, "xent: row strides must be multiples of 4");
  // A cluster of up to eight CTAs (the portable limit) holds rows of up to 213000 columns.  Rows that fit one CTA stay with the
  // kernel below: they are in L2 when it re-reads them (4096 x 8192: 55 us there, 63 us here).  So do rows in great number of
  // which four per SM, those in flight there, come to 80 MB at most (us there and here: 4096 x 26752 130 and 144, 2400 x 32000 101
  // and 106; but 4096 x 36096 194 and 183, and with few rows, 64 x 32000, 7.8 and 6.4, 600 x 26752 30 and 27).
  const int ranks = (int)(((long)Vcols * 4 + XE_SEG_BYTES - 1) / XE_SEG_BYTES);
  const bool resident = rows > 8 * sm_count() && (long)Vcols * 4 * 4 * sm_count() <= 80000000L;
  if (dlogits != nullptr && !resident && ranks > 1 && ranks <= 8 && ((uintptr_t)logits & 15) == 0 && ((uintptr_t)dlogits & 7) == 0) {
    const int seg = (Vcols / 4 + ranks - 1) / ranks * 4;
    if (seg * (ranks - 1) < Vcols && (long)rows * ranks <= 0x7fffffffL) {
      static bool cfg = false;
      if (!cfg) { CPB_CUDA_OK(cudaFuncSetAttribute(xent_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, XE_SEG_BYTES + 64)); cfg = true; }
      cudaLaunchConfig_t lc = {};
      lc.gridDim = dim3((unsigned)(rows * ranks)); lc.blockDim = dim3(XE_THREADS); lc.dynamicSmemBytes = (size_t)seg * 4; lc.stream = stream;
      cudaLaunchAttribute at[2];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = ranks; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
      at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[1].val.programmaticStreamSerializationAllowed = 1;
      lc.attrs = at; lc.numAttrs = 2;
      CPB_CUDA_OK(cudaLaunchKernelEx(&lc, xent_smem_kernel, logits, targets, (__nv_bfloat16*)dlogits, loss_sum, row_loss, V, Vcols, seg, ranks,
                                     ld_logits, ld_dlogits, grad_scale, status));
      return check_launch("xent");
    }
  }
  CPB_CUDA_OK(launch_pdl(xent_kernel, rows, 512, 0, stream, logits, targets, (__nv_bfloat16*)dlogits, loss_sum, row_loss, rows, V, Vcols, ld_logits, ld_dlogits, grad_scale, status));
  return check_launch("xent");
}
