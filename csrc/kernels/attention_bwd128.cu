// Flash-attention backward specialised for head_dim 128.
//
// One CTA owns one 128-row K/V tile of one KV head and sweeps the query tiles (of every query head of the GQA group) that
// see it, with the K/V rows in tensor-memory lanes:
//
//     S^T  = K Q^T            (smem x smem)      P^T  = exp2(S^T c - LSE)        (registers -> tensor memory, bf16)
//     dP^T = V dO^T           (smem x smem)      dS^T = P^T o (dP^T - Delta)     (registers -> tensor memory and smem, bf16)
//     dV  += P^T dO           (tmem x smem)      dK  += dS^T Q                   (tmem x smem)
//     dQ   = dS K             (smem x smem, dS^T read M-major) -> staged in shared memory -> TMA reduce-add (fp32)
//
// What bounds it: shared-memory bandwidth.  Per 128 x 128 tile the five products take 2560 tensor-core cycles, but the
// operands they read from shared memory (64 KB for each smem x smem product, 32 KB for the two whose A operand is in tensor
// memory), the dS^T tile, the TMA fills and the fp32 dQ staging (64 KB in, 64 KB out) are about 490 KB, 3840 cycles at
// 128 bytes per cycle.  Hence P^T and dS^T stay in tensor memory for dV and dK, and everything else is arranged so that the
// tensor core never waits for the warps for long:
//
// Tensor memory (512 columns): S^T / P^T 128 | dP^T / dS^T / dQ 128 | dV 128 | dK 128.  P^T overwrites the part of S^T its
// thread has read, dS^T that of dP^T, and dQ all of dP^T once dK has read dS^T.  Issue order of the MMA warp:
//     dV(i), S(i+1)      when the warps have stored P(i): both run while the warps form dS(i)
//     dK(i), dQ(i)       when dS(i) is stored: both run while the warps take the exponentials of tile i+1
//     dP(i+1)            when dQ(i) has been read out of tensor memory
// The drain warps load a whole dQ row (128 columns) into registers and release tensor memory at once, then pass it through the
// staging buffer in two rounds of 64 columns.  Shared memory: K 32 KB, V 32, Q two stages 64, dO one stage 32 (dO(i) is done with dV(i), long
// before dP(i+1) wants the next one), dS^T 32, dQ staging 32, LSE and Delta of two stages 2: all of it.
//
// Measured (T 32768, 32/8 heads, causal, the kernel alone): 33.8 ms = 650 TFLOP/s for the kernel this one replaces (query rows in
// lanes, P and dS through shared memory, dQ over S: fully serialised), 23.0 ms = 956 with the drain warps storing dQ before they
// release tensor memory, 20.3 ms = 1084 now.  With the clock beside it, on another GPU: back to back for two seconds 20.7 ms at 1.47
// GHz and 1002 W, which is 4280 cycles per tile, of which shared memory needs 3840; one launch at a time 18.1 ms.  So on long runs
// the power cap sets the clock and shared memory nine tenths of the cycles.  The second tile half of dP^T is loaded after
// the first is used: loading both at once spills in the 72 registers of these warps (24.4 ms).
//
// Masking is on global positions, dK/dV output modes and bounded waits are those of the head_dim-64 kernel.  Replaces
// mem_efficient_bwd_unified_kernel_exp11 (context_parallel/AttentionBackward.cu:300-541) and gqa_fused_rope_bwd_dQ / _dKdV
// (context_parallel/GQA_fused_bwd_sm103_cp.cu:135-565).
//
// Warp roles (768 threads): 0 = TMA loader, 1 = MMA issuer, 2, 3 idle, 4..19 = softmax-gradient warps (thread = key row, 32
// queries), 20..23 = dQ drain warps (thread = query row).
#include "attention_bwd.cuh"
#include "common.cuh"
#include "host_utils.h"

#include <stdlib.h>

namespace cpb {

constexpr int B128_T = 128;
constexpr int B128_D = 128;
constexpr int B128_CW = 32;                              // query columns per softmax-gradient thread
constexpr int B128_THREADS = 6 * 128;                     // six warpgroups
// Registers per thread and warpgroup: the launch gives every thread 80 (768 x 80); the loader / issuer warpgroup hands back
// what the drain warps need to hold a whole dQ row.  48 + 4 x 72 + 144 = 6 x 80.
constexpr int B128_REGS_ISSUE = 48, B128_REGS_GRAD = 72, B128_REGS_DRAIN = 144;

struct Bwd128Params {
  int B, Tq, Tk, Hq, Hkv, Tq_pad;
  int causal, k_off;
  float scale, scale_log2;
  const float* lse2;            // [B,Hq,Tq_pad] LSE * log2(e), +inf in the padding
  const float* delta;           // [B,Hq,Tq_pad] rowsum(dO o O), 0 in the padding
  const int* q_pos;             // [Tq_pad] global positions, INT_MAX in the padding
  void* dk; void* dv;           // [B,Tk,Hkv,D] bf16 (store) or fp32 (accumulate)
  long dkv_st;                  // elements from one token of dk / dv to the next (heads adjacent, batches dense)
  int dkv_mode;                 // 0 bf16 store, 1 fp32 accumulate, 2 routed red.add (fused ring), 3 fp32 store to the part of this CTA (several per tile)
  int it_chunk;                 // pairs of (query head, query tile) per CTA, 0: all (see BwdWork)
  long part_st;                 // mode 3: floats from one part of dk / dv to the next
  int local;                    // q_pos is 0 .. Tq - 1: the first visible query tile needs no search
  const uint64_t* route_k;      // mode 2: per chunk of route_rows K/V rows the address of its owner's fp32 accumulator
  const uint64_t* route_v;
  int route_rows, route_tl;
  int debug_skip_dq;            // diagnostic: do not add dQ tiles to global memory (timing experiments only)
  int* status;
};

struct Bwd128Smem {
  static constexpr int TILE = B128_T * B128_D * 2;       // 32 KB: two 64-wide halves of 128 rows x 128 bytes
  static constexpr int HALF = B128_T * 128;
  static constexpr int K_OFF = 0;
  static constexpr int V_OFF = TILE;
  static constexpr int Q_OFF = 2 * TILE;                 // two stages
  static constexpr int DO_OFF = 4 * TILE;                // one stage
  static constexpr int DS_OFF = 5 * TILE;                // dS^T: two 64-query halves of 128 key rows x 128 bytes
  static constexpr int DQS_OFF = 6 * TILE;               // per drain warp two boxes of 32 rows x 32 fp32
  static constexpr int VEC_OFF = 7 * TILE;               // two stages of lse2[128], delta[128]
  static constexpr int BAR_OFF = VEC_OFF + 2048;
  static constexpr int TOTAL = BAR_OFF + 256;            // 231,680 bytes; the base must be 1024-byte aligned as it is
};


// PARTS (several CTAs per tile) is an instance of its own: its state in the whole sweep's softmax warps raised the spilled loads from 24
// to 144 bytes, and 32749 tokens of 4/1 heads took 2590 us instead of 2455.
template <bool PARTS>
__global__ void __launch_bounds__(B128_THREADS, 1)
flash_bwd128_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                    const __grid_constant__ CUtensorMap tmDQ, Bwd128Params p) {
  using L = Bwd128Smem;
  constexpr int D = B128_D, CW = B128_CW;
  constexpr uint32_t ST_COL = 0, DPT_COL = 128, DV_COL = 256, DK_COL = 384;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) { pdl_wait(); report(p.status, ST_BAD_INDEX, 870, (int)smem_u32(smem)); return; }
  uint64_t* bars = (uint64_t*)(smem + L::BAR_OFF);
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;        // [2]
  uint64_t* q_empty = bars + 3;       // [2]
  uint64_t* do_full = bars + 5;
  uint64_t* do_empty = bars + 6;
  uint64_t* s_ready = bars + 7;
  uint64_t* p_ready = bars + 8;
  uint64_t* dp_ready = bars + 9;
  uint64_t* ds_ready = bars + 10;
  uint64_t* dq_full = bars + 11;
  uint64_t* dq_empty = bars + 12;
  uint64_t* acc_done = bars + 13;
  uint32_t* tmem_slot = (uint32_t*)(bars + 14);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  int* qt_start_s = (int*)(tmem_slot + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.Hq / p.Hkv, num_q_tiles = p.Tq_pad / B128_T;
  const BwdWork work = bwd_work<PARTS>(p.it_chunk, (p.Tk + B128_T - 1) / B128_T, num_q_tiles, G, p.Hkv, p.B, p.k_off, p.causal && p.local);
  const int kt = work.kt, hkv = work.hkv, b = work.b;
  const int k0 = kt * B128_T;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < 2; ++s) { mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 1); }
    mbar_init(do_full, 1); mbar_init(do_empty, 1);
    mbar_init(s_ready, 1); mbar_init(p_ready, 16); mbar_init(dp_ready, 1); mbar_init(ds_ready, 16);
    mbar_init(dq_full, 1); mbar_init(dq_empty, 4); mbar_init(acc_done, 1);
    *abort_flag = 0;
    *qt_start_s = num_q_tiles;
    if (PARTS) qt_start_s[1] = work.it0 / p.it_chunk;
    fence_mbar_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();                               // and no pdl_release(), see common.cuh
  const uint32_t tmem_base = *tmem_slot;

  // first query tile that can see this K/V tile (q_pos is non-decreasing)
  if (p.causal && p.local) {
    if (threadIdx.x == 0 && p.k_off + k0 < p.Tq) *qt_start_s = max(0, p.k_off + k0) / B128_T;
  } else if (p.causal) {
    const int kpos_min = p.k_off + k0;
    for (int t = threadIdx.x; t < num_q_tiles; t += blockDim.x) {
      const int last = min(t * B128_T + B128_T, p.Tq) - 1;
      if (p.q_pos[last] >= kpos_min) { atomicMin(qt_start_s, t); break; }
    }
  } else if (threadIdx.x == 0) {
    *qt_start_s = 0;
  }
  __syncthreads();
  const int qt_start = *qt_start_s;
  const int n_qt = num_q_tiles - qt_start;
  const int n_it = PARTS ? max(0, min(p.it_chunk, n_qt * G - work.it0)) : n_qt * G;          // this CTA's pairs
  const int hq0 = hkv * G + (PARTS && n_it ? work.it0 / n_qt : 0), t0 = PARTS && n_it ? work.it0 % n_qt : 0;       // the first of them

  if (warp < 4) {
  regs_give<B128_REGS_ISSUE>();
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA loader
    if (lane == 0 && n_it > 0) {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmDO);
      mbar_expect_tx(kv_full, 2 * L::TILE);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        tma_load_4d(smem + L::K_OFF + h * L::HALF, &tmK, kv_full, h * 64, hkv, k0, b);
        tma_load_4d(smem + L::V_OFF + h * L::HALF, &tmV, kv_full, h * 64, hkv, k0, b);
      }
      int hq = hq0, t = t0;
      for (int i = 0; i < n_it; ++i) {
        const int st = i & 1;
        const int q0 = (qt_start + t) * B128_T;
        if (!mbar_wait_lean(&q_empty[st], ((i >> 1) & 1) ^ 1, abort_flag, 800)) break;
        mbar_expect_tx(&q_full[st], L::TILE + 1024);
#pragma unroll
        for (int h = 0; h < 2; ++h) tma_load_4d(smem + L::Q_OFF + st * L::TILE + h * L::HALF, &tmQ, &q_full[st], h * 64, hq, q0, b);
        const size_t row_off = ((size_t)b * p.Hq + hq) * p.Tq_pad + q0;
        bulk_load_1d(smem + L::VEC_OFF + st * 1024, p.lse2 + row_off, 512, &q_full[st]);
        bulk_load_1d(smem + L::VEC_OFF + st * 1024 + 512, p.delta + row_off, 512, &q_full[st]);
        if (!mbar_wait_lean(do_empty, (i & 1) ^ 1, abort_flag, 801)) break;
        mbar_expect_tx(do_full, L::TILE);
#pragma unroll
        for (int h = 0; h < 2; ++h) tma_load_4d(smem + L::DO_OFF + h * L::HALF, &tmDO, do_full, h * 64, hq, q0, b);
        if (++t == n_qt) { t = 0; ++hq; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp runs this code convergently; only the elected lane issues the MMAs and commits.
    if (n_it > 0) {
      const uint32_t leader = elect_one() ? 1u : 0u;
      constexpr uint32_t idesc_s = make_idesc_bf16(B128_T, B128_T, false, false);     // S^T, dP^T
      constexpr uint32_t idesc_acc = make_idesc_bf16(B128_T, D, false, true);         // dV, dK: A in tensor memory, B N-major
      constexpr uint32_t idesc_dq = make_idesc_bf16(B128_T, D, true, true);           // dQ: A M-major smem, B N-major
      const SDesc dK_k = sdesc_split(sdesc_kmajor(smem_u32(smem + L::K_OFF))), dV_k = sdesc_split(sdesc_kmajor(smem_u32(smem + L::V_OFF)));
      const SDesc dQ_k = sdesc_split(sdesc_kmajor(smem_u32(smem + L::Q_OFF))), dDO_k = sdesc_split(sdesc_kmajor(smem_u32(smem + L::DO_OFF)));
      const SDesc dQ_n = sdesc_split(make_sdesc(smem_u32(smem + L::Q_OFF), L::HALF, 1024));
      const SDesc dDO_n = sdesc_split(make_sdesc(smem_u32(smem + L::DO_OFF), L::HALF, 1024));
      const SDesc dK_n = sdesc_split(make_sdesc(smem_u32(smem + L::K_OFF), L::HALF, 1024));
      const SDesc dDS_m = sdesc_split(make_sdesc(smem_u32(smem + L::DS_OFF), L::HALF, 1024));
      const uint32_t t_s = tmem_base + ST_COL, t_dp = tmem_base + DPT_COL, t_dv = tmem_base + DV_COL, t_dk = tmem_base + DK_COL;
      auto issue_s = [&](int st) {          // S^T = K Q^T
        const SDesc q = SDesc{dQ_k.lo + (uint32_t)st * (L::TILE >> 4), dQ_k.hi};
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = (k / 4) * L::HALF + (k % 4) * 32;
          if (k == 0) umma_ss_cp<false>(leader, t_s, sdesc_at(dK_k, off), sdesc_at(q, off), idesc_s);
          else umma_ss_cp<true>(leader, t_s, sdesc_at(dK_k, off), sdesc_at(q, off), idesc_s);
        }
        umma_commit_p(leader, s_ready);
      };
      auto issue_dp = [&]() {               // dP^T = V dO^T
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = (k / 4) * L::HALF + (k % 4) * 32;
          if (k == 0) umma_ss_cp<false>(leader, t_dp, sdesc_at(dV_k, off), sdesc_at(dDO_k, off), idesc_s);
          else umma_ss_cp<true>(leader, t_dp, sdesc_at(dV_k, off), sdesc_at(dDO_k, off), idesc_s);
        }
        umma_commit_p(leader, dp_ready);
      };
      // the bf16 A operand of queries 16k .. 16k+15 sits in the front half of its writer's 32-column span
      auto a_col = [](int k) { return (uint32_t)(((16 * k) / CW) * CW + (((16 * k) % CW) / 16) * 8); };
      bool ok = __all_sync(0xffffffffu, mbar_wait_lean(kv_full, 0, abort_flag, 900) && mbar_wait_lean(&q_full[0], 0, abort_flag, 901) &&
                                            mbar_wait_lean(do_full, 0, abort_flag, 902));
      if (ok) {
        tc_fence_after();
        issue_s(0);
        issue_dp();
      }
      for (int i = 0; ok && i < n_it; ++i) {
        const int st = i & 1, sn = st ^ 1;
        const bool more = i + 1 < n_it;
        if (!__all_sync(0xffffffffu, mbar_wait_lean(p_ready, i & 1, abort_flag, 903))) break;
        tc_fence_after();
        umma_ts_p(leader, t_dv, t_s, sdesc_at(dDO_n, 0), idesc_acc, i != 0);              // dV += P^T dO
#pragma unroll
        for (int k = 1; k < B128_T / 16; ++k) umma_ts_cp<true>(leader, t_dv, t_s + a_col(k), sdesc_at(dDO_n, k * 2048), idesc_acc);
        umma_commit_p(leader, do_empty);
        if (more) {
          if (!__all_sync(0xffffffffu, mbar_wait_lean(&q_full[sn], ((i + 1) >> 1) & 1, abort_flag, 904))) break;
          tc_fence_after();
          issue_s(sn);                                                                     // over P(i), which dV(i) has read
        }
        if (!__all_sync(0xffffffffu, mbar_wait_lean(ds_ready, i & 1, abort_flag, 905))) break;
        tc_fence_after();
        const SDesc qn = SDesc{dQ_n.lo + (uint32_t)st * (L::TILE >> 4), dQ_n.hi};
        umma_ts_p(leader, t_dk, t_dp, sdesc_at(qn, 0), idesc_acc, i != 0);                // dK += dS^T Q
#pragma unroll
        for (int k = 1; k < B128_T / 16; ++k) umma_ts_cp<true>(leader, t_dk, t_dp + a_col(k), sdesc_at(qn, k * 2048), idesc_acc);
        umma_commit_p(leader, &q_empty[st]);
        umma_ss_cp<false>(leader, t_dp, sdesc_at(dDS_m, 0), sdesc_at(dK_n, 0), idesc_dq); // dQ = dS K, over dS^T, which dK(i) has read
#pragma unroll
        for (int k = 1; k < B128_T / 16; ++k) umma_ss_cp<true>(leader, t_dp, sdesc_at(dDS_m, k * 2048), sdesc_at(dK_n, k * 2048), idesc_dq);
        umma_commit_p(leader, dq_full);
        if (more) {
          if (!__all_sync(0xffffffffu, mbar_wait_lean(do_full, (i + 1) & 1, abort_flag, 906))) break;
          if (!__all_sync(0xffffffffu, mbar_wait_lean(dq_empty, i & 1, abort_flag, 907))) break;
          tc_fence_after();
          issue_dp();
        }
      }
      umma_commit_p(leader, acc_done);
    }
  }
  } else if (warp < 20) {
    // ------------------------------------------------------------------ softmax-gradient warps (thread = key row, 32 queries)
    regs_give<B128_REGS_GRAD>();
    const int quarter = warp & 3;
    const int grp = (warp - 4) >> 2;                    // which 32 query columns of the tile this thread owns
    const int cbase = grp * CW;
    const int r = quarter * 32 + lane;                  // key row inside the tile
    const int kidx = k0 + r;
    const bool k_valid = kidx < p.Tk;
    const int kpos = p.k_off + kidx;
    const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
    uint8_t* ds_row = smem + L::DS_OFF + (cbase / 64) * L::HALF + r * 128;
    const int chunk0 = (cbase % 64) / 8;
    bool alive = true;
    // first query position of a tile decides whether it needs masking; read one tile ahead, straight from global memory
    int qmin_next = n_it > 0 ? ld_ahead_s32(p.q_pos + (qt_start + t0) * B128_T) : 0;
    for (int i = 0; i < n_it && alive; ++i) {
      const int st = i & 1;
      const int qmin = qmin_next;
      if (i + 1 < n_it) qmin_next = ld_ahead_s32(p.q_pos + (qt_start + (t0 + i + 1) % n_qt) * B128_T);
      // slow path only for tiles that touch the causal diagonal or the end of the key sequence
      const bool need_mask = (k0 + B128_T > p.Tk) || (p.causal && (p.k_off + k0 + B128_T - 1 > qmin));
      const float* vec = (const float*)(smem + L::VEC_OFF + st * 1024) + cbase;
      bool ok = mbar_wait_lean(&q_full[st], (i >> 1) & 1, abort_flag, 1000) && mbar_wait_lean(s_ready, i & 1, abort_flag, 1001);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) { alive = false; break; }
      tc_fence_after();
      uint32_t sv[CW];
      tmem_ld32(t_lane + ST_COL + cbase, sv);
      tmem_wait_ld();
      if (!need_mask) {
        const uint64_t c2 = pack_f32x2(p.scale_log2, p.scale_log2);
#pragma unroll
        for (int j = 0; j < CW; j += 4) {
          const float4 l = *(const float4*)(vec + j);
          float x0, x1, x2, x3;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[j]), __uint_as_float(sv[j + 1])), c2, pack_f32x2(-l.x, -l.y)), x0, x1);
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[j + 2]), __uint_as_float(sv[j + 3])), c2, pack_f32x2(-l.z, -l.w)), x2, x3);
          sv[j] = __float_as_uint(ex2f(x0)); sv[j + 1] = __float_as_uint(ex2f(x1));
          sv[j + 2] = __float_as_uint(ex2f(x2)); sv[j + 3] = __float_as_uint(ex2f(x3));
        }
      } else {
        const int lim = (p.causal ? kpos : -0x7fffffff - 1);               // visible: lim <= q position
        const int4* qp = (const int4*)(p.q_pos + (qt_start + (t0 + i) % n_qt) * B128_T + cbase);
#pragma unroll
        for (int j = 0; j < CW; j += 4) {
          const float4 l = *(const float4*)(vec + j);
          const int4 q = __ldg(qp + (j >> 2));
          sv[j] = (k_valid && lim <= q.x) ? __float_as_uint(ex2f(fmaf(__uint_as_float(sv[j]), p.scale_log2, -l.x))) : 0u;
          sv[j + 1] = (k_valid && lim <= q.y) ? __float_as_uint(ex2f(fmaf(__uint_as_float(sv[j + 1]), p.scale_log2, -l.y))) : 0u;
          sv[j + 2] = (k_valid && lim <= q.z) ? __float_as_uint(ex2f(fmaf(__uint_as_float(sv[j + 2]), p.scale_log2, -l.z))) : 0u;
          sv[j + 3] = (k_valid && lim <= q.w) ? __float_as_uint(ex2f(fmaf(__uint_as_float(sv[j + 3]), p.scale_log2, -l.w))) : 0u;
        }
      }
      {
        uint32_t pk[CW / 2];                            // P^T of this thread's queries as bf16 pairs, over its own scores
#pragma unroll
        for (int j = 0; j < CW; j += 2) pk[j >> 1] = pack_bf16(__uint_as_float(sv[j]), __uint_as_float(sv[j + 1]));
        tmem_st16(t_lane + ST_COL + cbase, pk);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(p_ready);
      // dp_ready(i): dP(i) is complete, and so is dQ(i-1), which read the previous dS^T in shared memory
      ok = mbar_wait_lean(dp_ready, i & 1, abort_flag, 1002);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) { alive = false; break; }
      tc_fence_after();
      uint32_t dsk[CW / 2];                             // dS^T = P^T o (dP^T - Delta) with P in fp32
#pragma unroll
      for (int ch = 0; ch < CW; ch += 16) {
        uint32_t dpv[16];
        tmem_ld16(t_lane + DPT_COL + cbase + ch, dpv);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const float4 dl = *(const float4*)(vec + 128 + ch + j);
          float e0, e1, e2, e3;
          unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(sv[ch + j]), __uint_as_float(sv[ch + j + 1])),
                                 add_f32x2(pack_f32x2(__uint_as_float(dpv[j]), __uint_as_float(dpv[j + 1])), pack_f32x2(-dl.x, -dl.y))), e0, e1);
          unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(sv[ch + j + 2]), __uint_as_float(sv[ch + j + 3])),
                                 add_f32x2(pack_f32x2(__uint_as_float(dpv[j + 2]), __uint_as_float(dpv[j + 3])), pack_f32x2(-dl.z, -dl.w))), e2, e3);
          dsk[(ch + j) >> 1] = pack_bf16(e0, e1);
          dsk[((ch + j) >> 1) + 1] = pack_bf16(e2, e3);
        }
      }
      tmem_st16(t_lane + DPT_COL + cbase, dsk);
#pragma unroll
      for (int c8 = 0; c8 < CW / 8; ++c8)
        *(uint4*)(ds_row + (((chunk0 + c8) ^ (r & 7)) << 4)) = make_uint4(dsk[4 * c8], dsk[4 * c8 + 1], dsk[4 * c8 + 2], dsk[4 * c8 + 3]);
      tmem_wait_st();
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive_warp(ds_ready);
    }
    // final: dK, dV -> global
    if (n_it == 0) {
      if (PARTS && k_valid && grp == 0) {
        const size_t at = qt_start_s[1] * p.part_st + ((size_t)b * p.Tk + kidx) * p.dkv_st + hkv * D;
        for (int c = 0; c < D; c += 4) {
          *(float4*)((float*)p.dk + at + c) = make_float4(0.f, 0.f, 0.f, 0.f);
          *(float4*)((float*)p.dv + at + c) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      if (!PARTS && p.dkv_mode == 0 && k_valid && grp == 0) {
        __nv_bfloat16* dkr = (__nv_bfloat16*)p.dk + ((size_t)b * p.Tk + kidx) * p.dkv_st + hkv * D;
        __nv_bfloat16* dvr = (__nv_bfloat16*)p.dv + ((size_t)b * p.Tk + kidx) * p.dkv_st + hkv * D;
#pragma unroll
        for (int c = 0; c < D; c += 8) { *(uint4*)(dkr + c) = make_uint4(0, 0, 0, 0); *(uint4*)(dvr + c) = make_uint4(0, 0, 0, 0); }
      }
    } else if (alive) {
      bool ok = mbar_wait_lean(acc_done, 0, abort_flag, 1003);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        tc_fence_after();
        const size_t off = ((size_t)b * p.Tk + (k_valid ? kidx : 0)) * p.dkv_st + hkv * D;
        const int which = grp >> 1;                      // groups 0, 1 drain dK, groups 2, 3 dV: 64 columns each
        const int c_lo = (grp & 1) * 64;
        void* base = which ? p.dv : p.dk;
        const float osc = which ? 1.f : p.scale;         // dS^T was accumulated without the softmax scale
#pragma unroll 1
        for (int c = c_lo; c < c_lo + 64; c += 32) {
          uint32_t v[32];
          tmem_ld32(t_lane + (which ? DV_COL : DK_COL) + c, v);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * osc);
          if (k_valid) {
            if (!PARTS && p.dkv_mode == 2) {
              const int ch = kidx / p.route_rows, lrow = kidx % p.route_rows;
              float* dst = (float*)(which ? p.route_v[ch] : p.route_k[ch]) + (((size_t)b * p.route_tl + lrow) * p.Hkv + hkv) * D + c;
#pragma unroll
              for (int j = 0; j < 32; j += 4)
                red_add_v4(dst + j, __uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
            } else if (PARTS) {
              uint4* dst = (uint4*)((float*)base + qt_start_s[1] * p.part_st + off + c);
#pragma unroll
              for (int j = 0; j < 32; j += 4) dst[j >> 2] = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            } else if (p.dkv_mode == 1) {
              float* dst = (float*)base + off + c;
#pragma unroll
              for (int j = 0; j < 32; j += 4) {
                float4 o = *(float4*)(dst + j);
                o.x += __uint_as_float(v[j]); o.y += __uint_as_float(v[j + 1]);
                o.z += __uint_as_float(v[j + 2]); o.w += __uint_as_float(v[j + 3]);
                *(float4*)(dst + j) = o;
              }
            } else {
              __nv_bfloat16* dst = (__nv_bfloat16*)base + off + c;
#pragma unroll
              for (int j = 0; j < 32; j += 8) {
                uint4 o;
                o.x = pack_bf16(__uint_as_float(v[j]), __uint_as_float(v[j + 1]));
                o.y = pack_bf16(__uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                o.z = pack_bf16(__uint_as_float(v[j + 4]), __uint_as_float(v[j + 5]));
                o.w = pack_bf16(__uint_as_float(v[j + 6]), __uint_as_float(v[j + 7]));
                *(uint4*)(dst + j) = o;
              }
            }
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ dQ drain warps (20..23)
    regs_take<B128_REGS_DRAIN>();
    // tensor memory -> registers -> 128B-swizzled fp32 staging -> TMA reduce-add into the global fp32 dQ (rows past the end
    // of the sequence are clipped by the tensor map).  Every warp drains its own 32 query rows through its own two boxes
    // with its own bulk groups.  The whole row is loaded first and tensor memory released at once: dP(i+1) waits for that.
    const int quarter = warp & 3;
    const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16) + DPT_COL;
    uint8_t* stage = smem + L::DQS_OFF + quarter * 8192;      // [2 boxes][32 rows][128 B]
    const bool issuer = (lane == 0);
    if (issuer) tma_prefetch_desc(&tmDQ);
    for (int i = 0; i < n_it; ++i) {
      bool ok = mbar_wait_lean(dq_full, i & 1, abort_flag, 1100);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int hq = hq0 + (t0 + i) / n_qt;
      const int q0 = (qt_start + (t0 + i) % n_qt) * B128_T;
      uint32_t v[4][32];
#pragma unroll
      for (int h = 0; h < 4; ++h) tmem_ld32(t_lane + 32 * h, v[h]);
      tmem_wait_ld();
      tc_fence_before();
      mbar_arrive_warp(dq_empty);
#pragma unroll
      for (int rnd = 0; rnd < 2; ++rnd) {
        if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the boxes have been read out
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint8_t* rowp = stage + h * 4096 + lane * 128;
          const uint32_t (&w)[32] = v[2 * rnd + h];
#pragma unroll
          for (int c4 = 0; c4 < 8; ++c4)                  // dS was formed without the softmax scale: apply it here
            *(float4*)(rowp + ((c4 ^ (lane & 7)) << 4)) = make_float4(__uint_as_float(w[4 * c4]) * p.scale, __uint_as_float(w[4 * c4 + 1]) * p.scale,
                                                                      __uint_as_float(w[4 * c4 + 2]) * p.scale, __uint_as_float(w[4 * c4 + 3]) * p.scale);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (issuer && !p.debug_skip_dq) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
            asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                         ::"l"((uint64_t)&tmDQ), "r"(smem_u32(stage + h * 4096)), "r"(rnd * 64 + h * 32), "r"(hq), "r"(q0 + quarter * 32), "r"(b)
                         : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
    }
    if (issuer) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
  if (threadIdx.x == 0 && *abort_flag) report(p.status, ST_TIMEOUT_MBAR, *abort_flag, 0);
}

static int make_tmap4_128(CUtensorMap* m, const void* ptr, int H, int T, int B, long s_head, long s_tok, long s_batch) {
  uint64_t dims[4] = {(uint64_t)B128_D, (uint64_t)H, (uint64_t)T, (uint64_t)B};
  uint64_t strides[4] = {0, (uint64_t)s_head * 2, (uint64_t)s_tok * 2, (uint64_t)s_batch * 2};
  uint32_t box[4] = {64, 1, (uint32_t)B128_T, 1};
  return encode_tmap(m, ptr, 2, 4, dims, strides, box, 1);
}

}  // namespace cpb

using namespace cpb;

// q, k, v: strided views (element strides: head, token, batch); dout contiguous [B,Tq,Hq,D].
// dq: fp32 [B,Tq,Hq,D] (accumulated; caller zeroes).  dk/dv: [B,Tk,Hkv,D] bf16 (written) or fp32 (+=), tokens dkv_st elements apart.
// lse2 / delta: fp32 [B,Hq,Tq_pad] as produced by cpb_flash_bwd_prep; q_pos: int32 [Tq_pad] (INT_MAX padding), required.
extern "C" int cpb_flash_bwd128(const void* q, const void* k, const void* v, const void* dout, const float* lse2,
                                const float* delta, float* dq, void* dk, void* dv,
                                int B, int Tq, int Tk, int Hq, int Hkv, int Tq_pad,
                                long q_sh, long q_st, long q_sb, long k_sh, long k_st, long k_sb,
                                float scale, int causal, int k_off, const int* q_pos, int dkv_mode, long dkv_st,
                                const uint64_t* route_k, const uint64_t* route_v, int route_rows, int route_tl, int it_chunk, int local,
                                int* status, cudaStream_t stream) {
  if (Hq % Hkv) return set_error(CPB_ERR_ARG, "flash_bwd128: Hq %% Hkv != 0");
  if (Tq_pad % B128_T || Tq_pad < Tq) return set_error(CPB_ERR_ARG, "flash_bwd128: bad Tq_pad");
  if (q_pos == nullptr) return set_error(CPB_ERR_ARG, "flash_bwd128: q_pos is required");
  if (((uintptr_t)lse2 | (uintptr_t)delta | (uintptr_t)q_pos) & 15) return set_error(CPB_ERR_ARG, "flash_bwd128: vectors must be 16-byte aligned");
  if (dkv_mode != 2 && (dkv_st < (long)Hkv * B128_D || (dkv_st & 7) || (((uintptr_t)dk | (uintptr_t)dv) & 15)))
    return set_error(CPB_ERR_ARG, "flash_bwd128: dK/dV rows must be 16-byte aligned");
  if (dkv_mode == 2 && (route_k == nullptr || route_v == nullptr || route_rows <= 0))
    return set_error(CPB_ERR_ARG, "flash_bwd128: routed dK/dV needs route tables");
  CUtensorMap tq, tk, tv, tdo, tdq;
  int rc;
  if ((rc = make_tmap4_128(&tq, q, Hq, Tq, B, q_sh, q_st, q_sb)) != CPB_OK) return rc;
  if ((rc = make_tmap4_128(&tk, k, Hkv, Tk, B, k_sh, k_st, k_sb)) != CPB_OK) return rc;
  if ((rc = make_tmap4_128(&tv, v, Hkv, Tk, B, k_sh, k_st, k_sb)) != CPB_OK) return rc;
  if ((rc = make_tmap4_128(&tdo, dout, Hq, Tq, B, B128_D, (long)Hq * B128_D, (long)Tq * Hq * B128_D)) != CPB_OK) return rc;
  {
    uint64_t dims[4] = {(uint64_t)B128_D, (uint64_t)Hq, (uint64_t)Tq, (uint64_t)B};
    uint64_t strides[4] = {0, (uint64_t)B128_D * 4, (uint64_t)Hq * B128_D * 4, (uint64_t)Tq * Hq * B128_D * 4};
    uint32_t box[4] = {32, 1, 32, 1};      // one drain warp: 32 query rows x 32 columns
    if ((rc = encode_tmap(&tdq, dq, 4, 4, dims, strides, box, 1)) != CPB_OK) return rc;
  }
  Bwd128Params p;
  p.B = B; p.Tq = Tq; p.Tk = Tk; p.Hq = Hq; p.Hkv = Hkv; p.Tq_pad = Tq_pad; p.causal = causal; p.k_off = k_off;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.lse2 = lse2; p.delta = delta; p.q_pos = q_pos; p.dk = dk; p.dv = dv; p.dkv_mode = dkv_mode; p.dkv_st = dkv_st; p.status = status;
  p.route_k = route_k; p.route_v = route_v; p.route_rows = route_rows; p.route_tl = route_tl;
  if (it_chunk < 0 || (it_chunk > 0) != (dkv_mode == 3)) return set_error(CPB_ERR_ARG, "flash_bwd128: several CTAs per K/V tile write parts of dK/dV (dkv_mode 3)");
  p.it_chunk = it_chunk; p.local = local; p.part_st = (long)B * Tk * dkv_st;
  static const bool skip_dq = [] {
    const char* e = getenv("CPB_BWD_SKIP_DQ");
    const bool on = e != nullptr && e[0] == '1';
    if (on) fprintf(stderr, "CPB_BWD_SKIP_DQ=1: the attention backward does NOT produce dQ (timing experiment only)\n");
    return on;
  }();
  p.debug_skip_dq = skip_dq;
  const int n_kt = (Tk + B128_T - 1) / B128_T, G = Hq / Hkv, nq = Tq_pad / B128_T;
  dim3 grid(n_kt, Hkv, B);
  if (it_chunk) {
    long ctas = 0;
    for (int c = 0; (long)c * it_chunk < (long)G * nq; ++c) ctas += (long)bwd_tiles(c, it_chunk, n_kt, nq, G, k_off, causal && local) * Hkv * B;
    if (ctas == 0) return CPB_OK;                        // no query sees a key: the cast reads no part
    grid = dim3((unsigned)ctas);
  }
  const auto kernel = it_chunk ? flash_bwd128_kernel<true> : flash_bwd128_kernel<false>;
  static bool cfg[2] = {false, false};
  if (!cfg[it_chunk > 0]) { CPB_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Bwd128Smem::TOTAL)); cfg[it_chunk > 0] = true; }
  CPB_CUDA_OK(launch_pdl(kernel, grid, B128_THREADS, Bwd128Smem::TOTAL, stream, tq, tk, tv, tdo, tdq, p));
  return check_launch("flash_bwd128");
}
