// Flash-attention backward specialised for head_dim 64.
//
// One CTA owns one 128-row K/V tile of one KV head and sweeps the query tiles (of every query head of the GQA group) that
// see it, with the K/V rows in tensor-memory lanes.  A 128 x 128 tile is worked on as two halves of 64 queries, each by
// eight warps of its own and with barriers of its own:
//
//     S^T  = K Q^T            (tmem x smem)      P^T  = exp2(S^T c - LSE)        (registers -> tensor memory, bf16)
//     dP^T = V dO^T           (tmem x smem)      dS^T = P^T o (dP^T - Delta)     (registers -> tensor memory and smem, bf16)
//     dV  += P^T dO           (tmem x smem)      dK  += dS^T Q                   (tmem x smem)
//     dQ   = dS K             (smem x smem, dS^T read M-major, both halves at once) -> staging -> TMA reduce-add (fp32)
//
// What bounds it: the exponentials (16 per clock: 1024 cycles for 16384) if they never pause, then shared memory.  With all
// sixteen warps on one tile the exponential unit idles while they form dS and wait for each other (3150 cycles per tile);
// here one half can take its exponentials while the other forms dS.  N = 64 score products would read
// 192 bytes of operands per tensor-core cycle from shared memory, so K and V are copied into tensor memory once and only Q
// and dO are streamed.  Shared memory then moves about 270 KB per tile (64 KB for four products, 48 KB for dQ, 32 KB of dS^T,
// 64 KB of dQ staging, 33 KB of TMA fills and the LSE / Delta vectors): 2100 cycles at 128 bytes per cycle.
//
// Tensor memory (512 columns): S^T / P^T 128 | dP^T / dS^T 128 | dV 64 | dK 64 | dQ 64 | K 32 | V 32.  P^T overwrites the
// part of S^T its thread has read and dS^T that of dP^T.  Issue order of the MMA warp for tile i (halves A and B):
//     dK_B(i-1), dP_B(i), dQ(i-1)    when dS_B(i-1) is stored        dV_A(i), S_A(i+1)     when P_A(i) is stored
//     dK_A(i), dP_A(i+1)             when dS_A(i) is stored          dV_B(i), S_B(i+1)     when P_B(i) is stored
// so every product a half needs next is issued a whole phase before it is wanted.  dS^T has two buffers in shared memory:
// the commit behind dP of either half for tile i covers dQ(i-2), so no barrier of its own guards them.
//
// Measured against the kernel this one replaces (all sixteen warps on one tile, K and V read from shared memory, LSE and Delta
// as extra K = 16 products; same GPU, cold L2, us): T 32768, 32/8 heads 12886 -> 12244 (898 TFLOP/s); T 16384 2997 -> 2948;
// 2 x 4096, 6/2 heads 194 -> 181; 2 x 1000, 6/2 heads 64.5 -> 56.3 (the vectors' own launch is gone); 4 x 1024, 6/6 50.2 -> 48.2.
// Of the whole gradient (preparation and cast included) 1 to 18 %: 8192, 32/8 heads 1019 -> 924; 4096 queries, 32768 keys, 8/8, not
// causal 786 -> 771.  With the clock beside it: T 32768, 32/8 heads, back to back for two seconds, 12.8 ms at 1.59 GHz and 1004 W,
// 2860 cycles per tile; one launch at a time 11.2 ms (980 TFLOP/s).
//
// Masking is on global positions, dK/dV output modes and bounded waits are those of the head_dim-128 kernel.  Replaces
// mem_efficient_bwd_unified_kernel_exp11 (context_parallel/AttentionBackward.cu:300-541) and gqa_fused_rope_bwd_dQ / _dKdV
// (context_parallel/GQA_fused_bwd_sm103_cp.cu:135-565).
//
// Warp roles (768 threads): 0 = TMA loader, 1 = MMA issuer, 2, 3 idle, 4..11 = softmax-gradient warps of half A, 12..19 of
// half B (thread = key row, 32 queries), 20..23 = dQ drain warps (thread = query row).
#include "attention_bwd.cuh"
#include "common.cuh"
#include "host_utils.h"

#include <stdlib.h>

namespace cpb {

constexpr int B64_T = 128;
constexpr int B64_D = 64;
constexpr int B64_CW = 32;                              // query columns per softmax-gradient thread
constexpr int B64_THREADS = 6 * 128;                     // six warpgroups
// Registers per thread and warpgroup: the launch gives every thread 80 (768 x 80); the loader / issuer warpgroup hands back
// what the drain warps need to hold a whole dQ row.  48 + 4 x 80 + 112 = 6 x 80.
constexpr int B64_REGS_ISSUE = 48, B64_REGS_DRAIN = 112;

struct Bwd64Params {
  int B, Tq, Tk, Hq, Hkv, Tq_pad;
  const __nv_bfloat16* k;       // K and V rows are also read with plain loads, once, into tensor memory
  const __nv_bfloat16* v;
  long k_sh, k_st, k_sb;
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

struct Bwd64Smem {
  static constexpr int TILE = B64_T * B64_D * 2;         // 16 KB: 128 rows x 128 bytes
  static constexpr int NST = 3;                          // Q and dO ring depth
  static constexpr int K_OFF = 0;                        // K once more, as the B operand of dQ
  static constexpr int Q_OFF = TILE;
  static constexpr int DO_OFF = Q_OFF + NST * TILE;
  static constexpr int DS_BYTES = B64_T * B64_T * 2;     // dS^T: two 64-query halves of 128 key rows x 128 bytes
  static constexpr int DS_OFF = DO_OFF + NST * TILE;     // two buffers
  static constexpr int DQS_OFF = DS_OFF + 2 * DS_BYTES;  // per drain warp two boxes of 32 rows x 32 fp32
  static constexpr int VEC_OFF = DQS_OFF + 32768;        // NST x (lse2[128], delta[128])
  static constexpr int BAR_OFF = VEC_OFF + NST * 1024;
  static constexpr int TOTAL = BAR_OFF + 256;            // 216,320 bytes; the base must be 1024-byte aligned as it is
};


// PARTS (several CTAs per tile) is an instance of its own: its state raised the spilled loads of whole sweeps from 80 to 108 bytes, and
// 8192 queries of 65536 keys, 32/8 heads, took 5690 us instead of 5570.
template <bool PARTS>
__global__ void __launch_bounds__(B64_THREADS, 1)
flash_bwd64_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmDO, const __grid_constant__ CUtensorMap tmDQ, Bwd64Params p) {
  using L = Bwd64Smem;
  constexpr int D = B64_D, CW = B64_CW, NST = L::NST;
  constexpr uint32_t ST_COL = 0, DPT_COL = 128, DV_COL = 256, DK_COL = 320, DQ_COL = 384, K_COL = 448, V_COL = 480;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) { pdl_wait(); report(p.status, ST_BAD_INDEX, 870, (int)smem_u32(smem)); return; }
  uint64_t* bars = (uint64_t*)(smem + L::BAR_OFF);
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;        // [NST]
  uint64_t* q_empty = bars + 4;       // [NST]
  uint64_t* do_full = bars + 7;       // [NST]
  uint64_t* do_empty = bars + 10;     // [NST]
  uint64_t* s_ready = bars + 13;      // [2 halves], like the three below
  uint64_t* p_ready = bars + 15;
  uint64_t* dp_ready = bars + 17;
  uint64_t* ds_ready = bars + 19;
  uint64_t* dq_full = bars + 21;
  uint64_t* dq_empty = bars + 22;
  uint64_t* acc_done = bars + 23;
  uint32_t* tmem_slot = (uint32_t*)(bars + 24);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  int* qt_start_s = (int*)(tmem_slot + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.Hq / p.Hkv, num_q_tiles = p.Tq_pad / B64_T;
  const BwdWork work = bwd_work<PARTS>(p.it_chunk, (p.Tk + B64_T - 1) / B64_T, num_q_tiles, G, p.Hkv, p.B, p.k_off, p.causal && p.local);
  const int kt = work.kt, hkv = work.hkv, b = work.b;
  const int k0 = kt * B64_T;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < NST; ++s) { mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 1); mbar_init(&do_full[s], 1); mbar_init(&do_empty[s], 1); }
    for (int h = 0; h < 2; ++h) { mbar_init(&s_ready[h], 1); mbar_init(&p_ready[h], 8); mbar_init(&dp_ready[h], 1); mbar_init(&ds_ready[h], 8); }
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
    if (threadIdx.x == 0 && p.k_off + k0 < p.Tq) *qt_start_s = max(0, p.k_off + k0) / B64_T;
  } else if (p.causal) {
    const int kpos_min = p.k_off + k0;
    for (int t = threadIdx.x; t < num_q_tiles; t += blockDim.x) {
      const int last = min(t * B64_T + B64_T, p.Tq) - 1;
      if (p.q_pos[last] >= kpos_min) { atomicMin(qt_start_s, t); break; }
    }
  } else if (threadIdx.x == 0) {
    *qt_start_s = 0;
  }
  // K and V rows into tensor memory as bf16 A operands (warps 4..7 K, 8..11 V; rows past the end are zero)
  if (warp >= 4 && warp < 12) {
    const int row = k0 + (warp & 3) * 32 + lane;
    const __nv_bfloat16* src = (warp < 8 ? p.k : p.v) + (size_t)b * p.k_sb + (size_t)hkv * p.k_sh + (size_t)(row < p.Tk ? row : 0) * p.k_st;
    uint32_t w[32];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint4 x = row < p.Tk ? *(const uint4*)(src + 8 * c) : make_uint4(0, 0, 0, 0);
      w[4 * c] = x.x; w[4 * c + 1] = x.y; w[4 * c + 2] = x.z; w[4 * c + 3] = x.w;
    }
    tmem_st32(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (warp < 8 ? K_COL : V_COL), w);
    tmem_wait_st();
    tc_fence_before();
  }
  __syncthreads();
  const int qt_start = *qt_start_s;
  const int n_qt = num_q_tiles - qt_start;
  const int n_it = PARTS ? max(0, min(p.it_chunk, n_qt * G - work.it0)) : n_qt * G;          // this CTA's pairs
  const int hq0 = hkv * G + (PARTS && n_it ? work.it0 / n_qt : 0), t0 = PARTS && n_it ? work.it0 % n_qt : 0;       // the first of them

  if (warp < 4) {
  regs_give<B64_REGS_ISSUE>();
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA loader
    if (lane == 0 && n_it > 0) {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmDO);
      mbar_expect_tx(kv_full, L::TILE);
      tma_load_4d(smem + L::K_OFF, &tmK, kv_full, 0, hkv, k0, b);
      int st = 0, ph = 1, hq = hq0, t = t0;
      for (int i = 0; i < n_it; ++i) {
        const int q0 = (qt_start + t) * B64_T;
        if (!mbar_wait_lean(&q_empty[st], ph, abort_flag, 800)) break;
        mbar_expect_tx(&q_full[st], L::TILE + 1024);
        tma_load_4d(smem + L::Q_OFF + st * L::TILE, &tmQ, &q_full[st], 0, hq, q0, b);
        const size_t row_off = ((size_t)b * p.Hq + hq) * p.Tq_pad + q0;
        bulk_load_1d(smem + L::VEC_OFF + st * 1024, p.lse2 + row_off, 512, &q_full[st]);
        bulk_load_1d(smem + L::VEC_OFF + st * 1024 + 512, p.delta + row_off, 512, &q_full[st]);
        if (!mbar_wait_lean(&do_empty[st], ph, abort_flag, 801)) break;
        mbar_expect_tx(&do_full[st], L::TILE);
        tma_load_4d(smem + L::DO_OFF + st * L::TILE, &tmDO, &do_full[st], 0, hq, q0, b);
        if (++st == NST) { st = 0; ph ^= 1; }
        if (++t == n_qt) { t = 0; ++hq; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp runs this code convergently; only the elected lane issues the MMAs and commits.
    if (n_it > 0) {
      const uint32_t leader = elect_one() ? 1u : 0u;
      constexpr uint32_t idesc_s = make_idesc_bf16(B64_T, 64, false, false);        // one half of S^T, dP^T
      constexpr uint32_t idesc_acc = make_idesc_bf16(B64_T, D, false, true);        // dV, dK: A in tensor memory, B N-major
      constexpr uint32_t idesc_dq = make_idesc_bf16(B64_T, D, true, true);          // dQ: A M-major smem, B N-major
      const SDesc dQ_k = sdesc_split(sdesc_kmajor(smem_u32(smem + L::Q_OFF))), dDO_k = sdesc_split(sdesc_kmajor(smem_u32(smem + L::DO_OFF)));
      const SDesc dQ_n = sdesc_split(make_sdesc(smem_u32(smem + L::Q_OFF), B64_T * 128, 1024));
      const SDesc dDO_n = sdesc_split(make_sdesc(smem_u32(smem + L::DO_OFF), B64_T * 128, 1024));
      const SDesc dK_n = sdesc_split(make_sdesc(smem_u32(smem + L::K_OFF), B64_T * 128, 1024));
      const SDesc dDS_m = sdesc_split(make_sdesc(smem_u32(smem + L::DS_OFF), B64_T * 128, 1024));
      const uint32_t t_s = tmem_base + ST_COL, t_dp = tmem_base + DPT_COL, t_dv = tmem_base + DV_COL, t_dk = tmem_base + DK_COL,
                     t_dq = tmem_base + DQ_COL, t_k = tmem_base + K_COL, t_v = tmem_base + V_COL;
      auto stage = [](const SDesc& d, int st) { return SDesc{d.lo + (uint32_t)st * (L::TILE >> 4), d.hi}; };
      // one half of S^T = K Q^T (resp. dP^T = V dO^T): 64 query rows of the stage are 8 KB
      auto issue_half = [&](uint32_t t_out, uint32_t t_a, const SDesc& d, int h, uint64_t* ready) {
        umma_ts_cp<false>(leader, t_out + 64 * h, t_a, sdesc_at(d, 8192 * h), idesc_s);
#pragma unroll
        for (int k = 1; k < D / 16; ++k) umma_ts_cp<true>(leader, t_out + 64 * h, t_a + 8 * k, sdesc_at(d, 8192 * h + 32 * k), idesc_s);
        umma_commit_p(leader, &ready[h]);
      };
      // dV += P^T dO (resp. dK += dS^T Q) over the 64 queries of one half; the bf16 operand of 16 queries is 8 columns and
      // sits in the front half of its writer's 32-column span
      auto issue_acc = [&](uint32_t t_out, uint32_t t_a, const SDesc& d, int h, uint32_t acc) {
        umma_ts_p(leader, t_out, t_a + 64 * h, sdesc_at(d, 8192 * h), idesc_acc, acc);
        umma_ts_cp<true>(leader, t_out, t_a + 64 * h + 8, sdesc_at(d, 8192 * h + 2048), idesc_acc);
        umma_ts_cp<true>(leader, t_out, t_a + 64 * h + 32, sdesc_at(d, 8192 * h + 4096), idesc_acc);
        umma_ts_cp<true>(leader, t_out, t_a + 64 * h + 40, sdesc_at(d, 8192 * h + 6144), idesc_acc);
      };
      bool ok = __all_sync(0xffffffffu, mbar_wait_lean(kv_full, 0, abort_flag, 900) && mbar_wait_lean(&q_full[0], 0, abort_flag, 901) &&
                                            mbar_wait_lean(&do_full[0], 0, abort_flag, 902));
      if (ok) {
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) issue_half(t_s, t_k, dQ_k, h, s_ready);
#pragma unroll
        for (int h = 0; h < 2; ++h) issue_half(t_dp, t_v, dDO_k, h, dp_ready);
      }
      int st = 0, ph = 0;                      // stage of tile i and the parity of its fill
      int sp = 0;                              // stage of tile i - 1
      for (int i = 0; ok && i <= n_it; ++i) {
        int sn = st + 1, pn = ph;              // stage and parity of tile i + 1
        if (sn == NST) { sn = 0; pn ^= 1; }
        const bool more = i + 1 < n_it;
        if (i > 0) {
          if (!__all_sync(0xffffffffu, mbar_wait_lean(&ds_ready[1], (i - 1) & 1, abort_flag, 903))) break;
          tc_fence_after();
          issue_acc(t_dk, t_dp, stage(dQ_n, sp), 1, 1);
          umma_commit_p(leader, &q_empty[sp]);
          if (i < n_it) issue_half(t_dp, t_v, stage(dDO_k, st), 1, dp_ready);       // dO(i) has arrived: dP_A(i) waited for it
          if (i > 1 && !__all_sync(0xffffffffu, mbar_wait_lean(dq_empty, i & 1, abort_flag, 904))) break;
          tc_fence_after();
          const SDesc ds = SDesc{dDS_m.lo + (uint32_t)((i - 1) & 1) * (L::DS_BYTES >> 4), dDS_m.hi};
          umma_ss_cp<false>(leader, t_dq, sdesc_at(ds, 0), sdesc_at(dK_n, 0), idesc_dq);
#pragma unroll
          for (int k = 1; k < B64_T / 16; ++k) umma_ss_cp<true>(leader, t_dq, sdesc_at(ds, k * 2048), sdesc_at(dK_n, k * 2048), idesc_dq);
          umma_commit_p(leader, dq_full);
          if (i == n_it) break;
        }
        if (!__all_sync(0xffffffffu, mbar_wait_lean(&p_ready[0], i & 1, abort_flag, 905))) break;
        tc_fence_after();
        issue_acc(t_dv, t_s, stage(dDO_n, st), 0, i != 0);
        if (more) {
          if (!__all_sync(0xffffffffu, mbar_wait_lean(&q_full[sn], pn, abort_flag, 906))) break;
          tc_fence_after();
          issue_half(t_s, t_k, stage(dQ_k, sn), 0, s_ready);                        // over P_A(i), which dV has read
        }
        if (!__all_sync(0xffffffffu, mbar_wait_lean(&ds_ready[0], i & 1, abort_flag, 907))) break;
        tc_fence_after();
        issue_acc(t_dk, t_dp, stage(dQ_n, st), 0, i != 0);
        if (more) {
          if (!__all_sync(0xffffffffu, mbar_wait_lean(&do_full[sn], pn, abort_flag, 908))) break;
          tc_fence_after();
          issue_half(t_dp, t_v, stage(dDO_k, sn), 0, dp_ready);                     // over dS_A(i), which dK has read
        }
        if (!__all_sync(0xffffffffu, mbar_wait_lean(&p_ready[1], i & 1, abort_flag, 909))) break;
        tc_fence_after();
        issue_acc(t_dv, t_s, stage(dDO_n, st), 1, 1);
        umma_commit_p(leader, &do_empty[st]);
        if (more) issue_half(t_s, t_k, stage(dQ_k, sn), 1, s_ready);
        sp = st; st = sn; ph = pn;
      }
      umma_commit_p(leader, acc_done);
    }
  }
  } else if (warp < 20) {
    // ------------------------------------------------------------------ softmax-gradient warps (thread = key row, 32 queries)
    const int quarter = warp & 3;
    const int grp = (warp - 4) >> 2;                    // which 32 query columns of the tile this thread owns
    const int half = grp >> 1;
    const int cbase = grp * CW;
    const int r = quarter * 32 + lane;                  // key row inside the tile
    const int kidx = k0 + r;
    const bool k_valid = kidx < p.Tk;
    const int kpos = p.k_off + kidx;
    const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
    uint8_t* ds_row = smem + L::DS_OFF + half * (B64_T * 128) + r * 128;
    const int chunk0 = (cbase % 64) / 8;
    bool alive = true;
    // first query position of a half tile decides whether it needs masking; read one tile ahead, straight from global memory
    const int* qp0 = p.q_pos + qt_start * B64_T + 64 * half;
    int qmin_next = n_it > 0 ? ld_ahead_s32(qp0 + t0 * B64_T) : 0;
    int st = 0, ph = 0, t = t0;
    for (int i = 0; i < n_it && alive; ++i) {
      const int qmin = qmin_next;
      const int t_cur = t;
      if (++t == n_qt) t = 0;
      if (i + 1 < n_it) qmin_next = ld_ahead_s32(qp0 + t * B64_T);
      // slow path only for tiles that touch the causal diagonal or the end of the key sequence
      const bool need_mask = (k0 + B64_T > p.Tk) || (p.causal && (p.k_off + k0 + B64_T - 1 > qmin));
      const float* vec = (const float*)(smem + L::VEC_OFF + st * 1024) + cbase;
      bool ok = mbar_wait_lean(&q_full[st], ph, abort_flag, 1000) && mbar_wait_lean(&s_ready[half], i & 1, abort_flag, 1001);
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
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const uint64_t x = fma_f32x2(pack_f32x2(__uint_as_float(sv[j + e]), __uint_as_float(sv[j + e + 1])), c2, e ? pack_f32x2(-l.z, -l.w) : pack_f32x2(-l.x, -l.y));
            float x0, x1;
            unpack_f32x2(x, x0, x1);
            sv[j + e] = __float_as_uint(ex2f(x0)); sv[j + e + 1] = __float_as_uint(ex2f(x1));
          }
        }
      } else {
        const int lim = (p.causal ? kpos : -0x7fffffff - 1);               // visible: lim <= q position
        const int4* qp = (const int4*)(p.q_pos + (qt_start + t_cur) * B64_T + cbase);
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
      mbar_arrive_warp(&p_ready[half]);
      // dp_ready(i): dP(i) of this half is complete, and so is dQ(i-2), which read the dS^T buffer written below
      ok = mbar_wait_lean(&dp_ready[half], i & 1, abort_flag, 1002);
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
      uint8_t* dsb = ds_row + (i & 1) * L::DS_BYTES;
#pragma unroll
      for (int c8 = 0; c8 < CW / 8; ++c8)
        *(uint4*)(dsb + (((chunk0 + c8) ^ (r & 7)) << 4)) = make_uint4(dsk[4 * c8], dsk[4 * c8 + 1], dsk[4 * c8 + 2], dsk[4 * c8 + 3]);
      tmem_wait_st();
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive_warp(&ds_ready[half]);
      if (++st == NST) { st = 0; ph ^= 1; }
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
        const int which = grp >> 1;                      // groups 0, 1 drain dK, groups 2, 3 dV: 32 columns each
        const int c = (grp & 1) * 32;
        void* base = which ? p.dv : p.dk;
        const float osc = which ? 1.f : p.scale;         // dS^T was accumulated without the softmax scale
        {
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
    regs_take<B64_REGS_DRAIN>();
    // tensor memory -> registers -> 128B-swizzled fp32 staging -> TMA reduce-add into the global fp32 dQ (rows past the end
    // of the sequence are clipped by the tensor map).  Every warp drains its own 32 query rows through its own two boxes
    // with its own bulk group, so the four warps never wait for one another.
    const int quarter = warp & 3;
    const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16) + DQ_COL;
    uint8_t* stage = smem + L::DQS_OFF + quarter * 8192;      // [2 boxes][32 rows][128 B]
    const bool issuer = (lane == 0);
    if (issuer) tma_prefetch_desc(&tmDQ);
    int hq = hq0, t = t0;
    for (int i = 0; i < n_it; ++i) {
      bool ok = mbar_wait_lean(dq_full, i & 1, abort_flag, 1100);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int q0 = (qt_start + t) * B64_T;
      uint32_t v[2][32];
      tmem_ld32(t_lane, v[0]);
      tmem_ld32(t_lane + 32, v[1]);
      tmem_wait_ld();
      tc_fence_before();
      mbar_arrive_warp(dq_empty);                           // tensor-memory dQ is free again
      if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the boxes have been read out
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint8_t* rowp = stage + h * 4096 + lane * 128;
#pragma unroll
        for (int c4 = 0; c4 < 8; ++c4)                      // dS was formed without the softmax scale: apply it here
          *(float4*)(rowp + ((c4 ^ (lane & 7)) << 4)) = make_float4(__uint_as_float(v[h][4 * c4]) * p.scale, __uint_as_float(v[h][4 * c4 + 1]) * p.scale,
                                                                    __uint_as_float(v[h][4 * c4 + 2]) * p.scale, __uint_as_float(v[h][4 * c4 + 3]) * p.scale);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (issuer && !p.debug_skip_dq) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
          asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                       ::"l"((uint64_t)&tmDQ), "r"(smem_u32(stage + h * 4096)), "r"(h * 32), "r"(hq), "r"(q0 + quarter * 32), "r"(b)
                       : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
      if (++t == n_qt) { t = 0; ++hq; }
    }
    if (issuer) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
  if (threadIdx.x == 0 && *abort_flag) report(p.status, ST_TIMEOUT_MBAR, *abort_flag, 0);
}

static int make_tmap4_64(CUtensorMap* m, const void* ptr, int H, int T, int B, long s_head, long s_tok, long s_batch) {
  uint64_t dims[4] = {(uint64_t)B64_D, (uint64_t)H, (uint64_t)T, (uint64_t)B};
  uint64_t strides[4] = {0, (uint64_t)s_head * 2, (uint64_t)s_tok * 2, (uint64_t)s_batch * 2};
  uint32_t box[4] = {64, 1, (uint32_t)B64_T, 1};
  return encode_tmap(m, ptr, 2, 4, dims, strides, box, 1);
}

}  // namespace cpb

using namespace cpb;

// q, k, v: strided views (element strides: head, token, batch); dout contiguous [B,Tq,Hq,D].
// dq: fp32 [B,Tq,Hq,D] (accumulated; caller zeroes).  dk/dv: [B,Tk,Hkv,D] bf16 (written) or fp32 (+=), tokens dkv_st elements apart.
// lse2 / delta: fp32 [B,Hq,Tq_pad] as produced by cpb_flash_bwd_prep; q_pos: int32 [Tq_pad] (INT_MAX padding), required.
extern "C" int cpb_flash_bwd64(const void* q, const void* k, const void* v, const void* dout, const float* lse2,
                                const float* delta, float* dq, void* dk, void* dv,
                                int B, int Tq, int Tk, int Hq, int Hkv, int Tq_pad,
                                long q_sh, long q_st, long q_sb, long k_sh, long k_st, long k_sb,
                                float scale, int causal, int k_off, const int* q_pos, int dkv_mode, long dkv_st,
                                const uint64_t* route_k, const uint64_t* route_v, int route_rows, int route_tl, int it_chunk, int local,
                                int* status, cudaStream_t stream) {
  if (Hq % Hkv) return set_error(CPB_ERR_ARG, "flash_bwd64: Hq %% Hkv != 0");
  if (Tq_pad % B64_T || Tq_pad < Tq) return set_error(CPB_ERR_ARG, "flash_bwd64: bad Tq_pad");
  if (q_pos == nullptr) return set_error(CPB_ERR_ARG, "flash_bwd64: q_pos is required");
  if (((uintptr_t)k | (uintptr_t)v) & 15 || (k_sh | k_st | k_sb) & 7) return set_error(CPB_ERR_ARG, "flash_bwd64: K/V rows must be 16-byte aligned");
  if (((uintptr_t)lse2 | (uintptr_t)delta | (uintptr_t)q_pos) & 15) return set_error(CPB_ERR_ARG, "flash_bwd64: vectors must be 16-byte aligned");
  if (dkv_mode != 2 && (dkv_st < (long)Hkv * B64_D || (dkv_st & 7) || (((uintptr_t)dk | (uintptr_t)dv) & 15)))
    return set_error(CPB_ERR_ARG, "flash_bwd64: dK/dV rows must be 16-byte aligned");
  if (dkv_mode == 2 && (route_k == nullptr || route_v == nullptr || route_rows <= 0))
    return set_error(CPB_ERR_ARG, "flash_bwd64: routed dK/dV needs route tables");
  CUtensorMap tq, tk, tdo, tdq;
  int rc;
  if ((rc = make_tmap4_64(&tq, q, Hq, Tq, B, q_sh, q_st, q_sb)) != CPB_OK) return rc;
  if ((rc = make_tmap4_64(&tk, k, Hkv, Tk, B, k_sh, k_st, k_sb)) != CPB_OK) return rc;
  if ((rc = make_tmap4_64(&tdo, dout, Hq, Tq, B, B64_D, (long)Hq * B64_D, (long)Tq * Hq * B64_D)) != CPB_OK) return rc;
  {
    uint64_t dims[4] = {(uint64_t)B64_D, (uint64_t)Hq, (uint64_t)Tq, (uint64_t)B};
    uint64_t strides[4] = {0, (uint64_t)B64_D * 4, (uint64_t)Hq * B64_D * 4, (uint64_t)Tq * Hq * B64_D * 4};
    uint32_t box[4] = {32, 1, 32, 1};      // one drain warp: 32 query rows x 32 columns
    if ((rc = encode_tmap(&tdq, dq, 4, 4, dims, strides, box, 1)) != CPB_OK) return rc;
  }
  Bwd64Params p;
  p.B = B; p.Tq = Tq; p.Tk = Tk; p.Hq = Hq; p.Hkv = Hkv; p.Tq_pad = Tq_pad; p.causal = causal; p.k_off = k_off;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.k = (const __nv_bfloat16*)k; p.v = (const __nv_bfloat16*)v; p.k_sh = k_sh; p.k_st = k_st; p.k_sb = k_sb;
  p.lse2 = lse2; p.delta = delta; p.q_pos = q_pos; p.dk = dk; p.dv = dv; p.dkv_mode = dkv_mode; p.dkv_st = dkv_st; p.status = status;
  p.route_k = route_k; p.route_v = route_v; p.route_rows = route_rows; p.route_tl = route_tl;
  if (it_chunk < 0 || (it_chunk > 0) != (dkv_mode == 3)) return set_error(CPB_ERR_ARG, "flash_bwd64: several CTAs per K/V tile write parts of dK/dV (dkv_mode 3)");
  p.it_chunk = it_chunk; p.local = local; p.part_st = (long)B * Tk * dkv_st;
  static const bool skip_dq = [] {
    const char* e = getenv("CPB_BWD_SKIP_DQ");
    const bool on = e != nullptr && e[0] == '1';
    if (on) fprintf(stderr, "CPB_BWD_SKIP_DQ=1: the attention backward does NOT produce dQ (timing experiment only)\n");
    return on;
  }();
  p.debug_skip_dq = skip_dq;
  const int n_kt = (Tk + B64_T - 1) / B64_T, G = Hq / Hkv, nq = Tq_pad / B64_T;
  dim3 grid(n_kt, Hkv, B);
  if (it_chunk) {
    long ctas = 0;
    for (int c = 0; (long)c * it_chunk < (long)G * nq; ++c) ctas += (long)bwd_tiles(c, it_chunk, n_kt, nq, G, k_off, causal && local) * Hkv * B;
    if (ctas == 0) return CPB_OK;                        // no query sees a key: the cast reads no part
    grid = dim3((unsigned)ctas);
  }
  const auto kernel = it_chunk ? flash_bwd64_kernel<true> : flash_bwd64_kernel<false>;
  static bool cfg[2] = {false, false};
  if (!cfg[it_chunk > 0]) { CPB_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Bwd64Smem::TOTAL)); cfg[it_chunk > 0] = true; }
  CPB_CUDA_OK(launch_pdl(kernel, grid, B64_THREADS, Bwd64Smem::TOTAL, stream, tq, tk, tdo, tdq, p));
  return check_launch("flash_bwd64");
}
