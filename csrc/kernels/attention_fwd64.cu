// Flash-attention forward for head_dim 64: four CTAs per SM, each with one query tile and steps of 64 keys.  Same contract as
// flash_fwd_kernel (attention_fwd.cu), readiness flags, copy CTAs and scatter epilogue included.
//
// What bounds it: the exponentials, 16 per clock and SM, as long as some warp of every scheduler is always in its exponential phase.
// A softmax warp spends longer on waits, tensor-memory round trips and the row maximum than a tile's products take, so it needs
// others beside it that are independent of it: here a scheduler has one softmax warp of each of four CTAs (thread = query row, 64
// key columns: no exchange of row maxima).  P overwrites the scores it was made from, so 128 tensor-memory columns do (S / P 64,
// O 64); P V(j) and S(j+1) are issued together, and S(j+1) ready implies that P V(j) has finished.
//
// Measured against two CTAs per SM with steps of 128 keys (attention_fwd.cu), cold L2, us: 32768 keys, 32/8 heads 5712 -> 5272 (834
// TFLOP/s), 65536 keys 23345 -> 22326, 40 sequences of 1024 449 -> 331; few long sequences are slower (see fwd_kernel).  At 16384 keys the special-function unit is
// 74 % busy, half of the issue slots are used, and the softmax warps wait for tensor memory most of the time (counters).
// Polynomial exponentials for one column in eight take 5046 us, but leave an LSE error of 1e-5 where this has 1e-6.
#include <stdlib.h>
#include "attention_fwd.cuh"

namespace cpb {

constexpr int F64_THREADS = 192;      // warp 0: loader, 1: MMA issuer, 2..5: softmax
constexpr int F64_BK = 64;            // keys per step

struct F64Smem {
  static constexpr int ST = 2;                             // K and V ring depth
  static constexpr int Q_BYTES = FA_BQ * 128;
  static constexpr int KV_BYTES = F64_BK * 128;
  static constexpr int K_OFF = Q_BYTES;
  static constexpr int V_OFF = K_OFF + ST * KV_BYTES;
  static constexpr int BAR_OFF = V_OFF + ST * KV_BYTES;
  static constexpr int TOTAL = BAR_OFF + 128;              // 49,280 bytes; the base must be 1024-byte aligned as it is
};

template <int POLY>
__global__ void __launch_bounds__(F64_THREADS, 4)
flash_fwd64_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                   FwdParams p) {
  using L = F64Smem;
  if (p.n_copy > 0 && blockIdx.x < (unsigned)p.n_copy) {
    pdl_wait();
    if (blockIdx.y == 0 && blockIdx.z == 0) ring_copy_cta(p.segs, p.n_segs, p.n_copy, blockIdx.x, p.ready);
    return;
  }
  constexpr int D = 64, ST = L::ST;
  constexpr uint32_t O_COL = 64;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023) { pdl_wait(); report(p.status, ST_BAD_INDEX, 570, (int)smem_u32(smem)); return; }
  uint64_t* bars = (uint64_t*)(smem + L::BAR_OFF);
  uint64_t* q_full = bars + 0;
  uint64_t* k_full = bars + 1;              // [ST]
  uint64_t* k_empty = k_full + ST;
  uint64_t* v_full = k_empty + ST;
  uint64_t* v_empty = v_full + ST;
  uint64_t* s_full = v_empty + ST;
  uint64_t* p_full = s_full + 1;
  uint64_t* o_done = s_full + 2;
  uint32_t* tmem_slot = (uint32_t*)(s_full + 3);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bx = (int)blockIdx.x - p.n_copy;
  const int G = p.Hq / p.Hkv;
  const int qt = (p.Tq + FA_BQ - 1) / FA_BQ - 1 - bx / G;     // heaviest tiles first
  const int hkv = blockIdx.y;
  const int hq = hkv * G + bx % G;
  const int b = blockIdx.z;
  const int q0 = qt * FA_BQ;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < ST; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    mbar_init(s_full, 1);
    mbar_init(p_full, 4);
    mbar_init(o_done, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 128); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();                               // and no pdl_release(), see common.cuh

  // Range of K/V steps this query tile attends to.
  const int q_last = min(q0 + FA_BQ, p.Tq) - 1;
  const int qpos_min = p.q_pos ? p.q_pos[q0] : q0;
  const int qpos_max = p.q_pos ? p.q_pos[q_last] : q_last;
  int n_kv = (p.Tk + F64_BK - 1) / F64_BK;
  if (p.causal) {
    const int last_idx = qpos_max - p.k_off;                  // last visible K index
    n_kv = last_idx < 0 ? 0 : min(n_kv, last_idx / F64_BK + 1);
  }
  // Order of the K/V sweep: step (j + j_start) % n_kv.  With readiness flags the sweep starts at the chunk
  // that contains this tile's own positions (resident locally), so remote chunks have time to arrive.
  int j_start = 0;
  if (p.ready != nullptr && n_kv > 0 && (p.block_rows % F64_BK) == 0) {
    const int c = max(qpos_min - p.k_off, 0) / p.block_rows;
    j_start = min(c * (p.block_rows / F64_BK), n_kv - 1);
  }
  auto key0 = [&](int j) { const int jj = j + j_start; return (jj >= n_kv ? jj - n_kv : jj) * F64_BK; };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA loader
    if (lane == 0 && n_kv > 0) {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
      mbar_expect_tx(q_full, L::Q_BYTES);
      tma_load_4d(smem, &tmQ, q_full, 0, hq, q0, b);
      int ready_block = -1;
      for (int j = 0; j < n_kv; ++j) {
        const int st = j % ST;
        const uint32_t free_phase = ((j / ST) & 1) ^ 1;
        if (!mbar_wait_lean(&k_empty[st], free_phase, abort_flag, 500)) break;
        const int k0 = key0(j);
        if (p.ready != nullptr) {
          // a step may straddle two blocks when block_rows is not a multiple of it
          const int blk_hi = min(k0 + F64_BK, p.Tk) - 1;
          for (int c = k0 / p.block_rows; c <= blk_hi / p.block_rows; ++c) {
            if (c == ready_block) continue;
            if (!wait_flag_ge(p.ready + c, p.ready_epoch, abort_flag, p.status, 501)) break;
            ready_block = c;
          }
          if (*abort_flag) break;
          // The copy CTAs wrote these rows with ordinary (generic-proxy) stores; the loads below go through the
          // async proxy (TMA): the acquire above orders generic accesses only.
          asm volatile("fence.proxy.async.global;" ::: "memory");
        }
        mbar_expect_tx(&k_full[st], L::KV_BYTES);
        tma_load_4d(smem + L::K_OFF + st * L::KV_BYTES, &tmK, &k_full[st], 0, hkv, k0, b);
        if (!mbar_wait_lean(&v_empty[st], free_phase, abort_flag, 502)) break;
        mbar_expect_tx(&v_full[st], L::KV_BYTES);
        tma_load_4d(smem + L::V_OFF + st * L::KV_BYTES, &tmV, &v_full[st], 0, hkv, k0, b);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (convergent warp, elected lane issues)
    if (n_kv > 0) {
      const uint32_t leader = elect_one() ? 1u : 0u;
      constexpr uint32_t idesc_qk = make_idesc_bf16(FA_BQ, F64_BK, false, false);
      constexpr uint32_t idesc_pv = make_idesc_bf16(FA_BQ, D, false, true);
      const SDesc dq = sdesc_split(sdesc_kmajor(smem_u32(smem)));
      const SDesc dk0 = sdesc_split(sdesc_kmajor(smem_u32(smem + L::K_OFF)));
      const SDesc dv0 = sdesc_split(make_sdesc(smem_u32(smem + L::V_OFF), F64_BK * 128, 1024));           // V, N-major
      const uint32_t s_tmem = tmem_base, o_tmem = tmem_base + O_COL;
      auto issue_qk = [&](int j) {
        const SDesc dk = SDesc{dk0.lo + (uint32_t)(j % ST) * (L::KV_BYTES >> 4), dk0.hi};
        umma_ss_cp<false>(leader, s_tmem, sdesc_at(dq, 0), sdesc_at(dk, 0), idesc_qk);
#pragma unroll
        for (int k = 1; k < D / 16; ++k) umma_ss_cp<true>(leader, s_tmem, sdesc_at(dq, k * 32), sdesc_at(dk, k * 32), idesc_qk);
        umma_commit_p(leader, s_full);
        umma_commit_p(leader, &k_empty[j % ST]);
      };
      bool ok = mbar_wait_lean(q_full, 0, abort_flag, 600) && mbar_wait_lean(&k_full[0], 0, abort_flag, 601);
      if (__all_sync(0xffffffffu, ok)) {
        tc_fence_after();
        issue_qk(0);
        for (int j = 0; j < n_kv; ++j) {
          const int st = j % ST;
          const bool more = j + 1 < n_kv;
          bool w = mbar_wait_lean(&v_full[st], (j / ST) & 1, abort_flag, 603);
          if (more) w = w && mbar_wait_lean(&k_full[(j + 1) % ST], ((j + 1) / ST) & 1, abort_flag, 604);
          w = w && mbar_wait_lean(p_full, j & 1, abort_flag, 602);
          if (!__all_sync(0xffffffffu, w)) break;
          tc_fence_after();
          const SDesc dv = SDesc{dv0.lo + (uint32_t)st * (L::KV_BYTES >> 4), dv0.hi};
          // A = P (bf16, 8 tensor-memory columns per 16 keys, 32 keys over the columns of their scores); B = V, 16 key rows = 2 KB
          umma_ts_p(leader, o_tmem, s_tmem, sdesc_at(dv, 0), idesc_pv, j != 0);
#pragma unroll
          for (int k = 1; k < F64_BK / 16; ++k)
            umma_ts_cp<true>(leader, o_tmem, s_tmem + (k >> 1) * 32 + (k & 1) * 8, sdesc_at(dv, k * 2048), idesc_pv);
          if (more) issue_qk(j + 1);                        // over P(j), which P V(j) has read by then
          else umma_commit_p(leader, o_done);
          umma_commit_p(leader, &v_empty[st]);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue (warps 2..5, thread = query row)
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const int qi = q0 + row;
    const bool row_valid = qi < p.Tq;
    // last visible key index of this row; rows past the end see everything (their results are dropped)
    const int k_last = min(p.causal ? (row_valid ? (p.q_pos ? p.q_pos[qi] : qi) : 0x7fffffff) - p.k_off : 0x7fffffff, p.Tk - 1);
    const int k_clear = p.causal ? min(qpos_min - p.k_off, p.Tk - 1) : p.Tk - 1;      // every row of the tile sees the keys up to here
    const uint32_t t_s = tmem_base + ((uint32_t)(quarter * 32) << 16), t_o = t_s + O_COL;
    float m_used = -INFINITY;    // running max (scaled, log2 domain) the accumulators are relative to
    float l = 0.f;
    bool alive = true;
    for (int j = 0; j < n_kv; ++j) {
      const int k0 = key0(j);
      bool ok = mbar_wait_lean(s_full, j & 1, abort_flag, 700);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) { alive = false; break; }
      tc_fence_after();
      const bool need_mask = k0 + F64_BK - 1 > k_clear;
      const int kmax = k_last - k0;                         // last visible column
      // the first 32 scores are read again after the second 32 are done with: 64 of them do not fit into 80 registers
      uint32_t sv[32];
      float mx = -INFINITY;
      {
        uint32_t lo[32];
        tmem_ld32(t_s, lo);
        tmem_ld32(t_s + 32, sv);
        tmem_wait_ld();
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (i <= kmax) mx = fmaxf(mx, __uint_as_float(lo[i]));
            if (32 + i <= kmax) mx = fmaxf(mx, __uint_as_float(sv[i]));
          }
        } else {
          float m4[4];                                      // four independent chains of three-input maxima
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            m4[c] = fmaxf(__uint_as_float(lo[8 * c]), __uint_as_float(sv[8 * c]));
#pragma unroll
            for (int i = 1; i < 8; ++i) m4[c] = fmax3(m4[c], __uint_as_float(lo[8 * c + i]), __uint_as_float(sv[8 * c + i]));
          }
          mx = fmaxf(fmax3(m4[0], m4[1], m4[2]), m4[3]);
        }
      }
      const float m_new = fmaxf(m_used, mx * p.scale_log2);
      // lazy rescale: keep the old reference maximum unless it fell behind by more than 2^8
      const bool need = (m_new > m_used + 8.f);
      if (__any_sync(0xffffffffu, need)) {
        float alpha = 1.f;
        if (need) {
          alpha = (m_used == -INFINITY) ? 0.f : ex2f(m_used - m_new);
          m_used = m_new;
          l *= alpha;
        }
        if (j > 0) {                                        // P V(j-1) has finished: S(j) came after it
#pragma unroll 1
          for (int c = 0; c < D; c += 16) {
            uint32_t v[16];
            tmem_ld16(t_o + c, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
            tmem_st16(t_o + c, v);
          }
        }
      }
      const float m_sub = (m_used == -INFINITY) ? 0.f : m_used;
      // p = exp2(s*scale - m) as bf16 pairs over the scores; two copies of the loop: the common one carries no compare per element
#pragma unroll
      for (int h = 1; h >= 0; --h) {
        if (h == 0) {
          tmem_ld32(t_s, sv);
          tmem_wait_ld();
        }
        uint32_t pk[16];
        if (!need_mask) {
          const uint64_t c2 = pack_f32x2(p.scale_log2, p.scale_log2), m2 = pack_f32x2(-m_sub, -m_sub);
          uint64_t l2 = pack_f32x2(0.f, 0.f);
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float p0, p1;
            const uint64_t x2 = fma_f32x2(pack_f32x2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), c2, m2);
            if (((i >> 1) & 7) >= 8 - POLY) {                  // resolved at compile time (the loop is unrolled)
              const uint64_t p2 = exp2_poly_f32x2(x2);
              l2 = add_f32x2(l2, p2);
              unpack_f32x2(p2, p0, p1);
            } else {
              float x0, x1;
              unpack_f32x2(x2, x0, x1);
              p0 = ex2f(x0); p1 = ex2f(x1);
              l2 = add_f32x2(l2, pack_f32x2(p0, p1));
            }
            pk[i >> 1] = pack_bf16(p0, p1);
          }
          float l0, l1;
          unpack_f32x2(l2, l0, l1);
          l += l0 + l1;
        } else {
          float l0 = 0.f, l1 = 0.f;
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float p0 = (h * 32 + i > kmax) ? 0.f : ex2f(fmaf(__uint_as_float(sv[i]), p.scale_log2, -m_sub));
            const float p1 = (h * 32 + i + 1 > kmax) ? 0.f : ex2f(fmaf(__uint_as_float(sv[i + 1]), p.scale_log2, -m_sub));
            l0 += p0; l1 += p1;
            pk[i >> 1] = pack_bf16(p0, p1);
          }
          l += l0 + l1;
        }
        tmem_st16(t_s + 32 * h, pk);                        // over the scores it came from
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(p_full);
    }
    // epilogue: O / l -> bf16, LSE
    __nv_bfloat16* orow = p.O + (((size_t)b * p.Tq + (row_valid ? qi : 0)) * p.Hq + hq) * D;
    if (p.o_peers != nullptr && row_valid) {
      const int peer = qi / p.o_rows_per_peer, lrow = qi % p.o_rows_per_peer;
      orow = (__nv_bfloat16*)(p.o_peers[peer] + p.o_off) + (((size_t)b * p.o_rows_per_peer + lrow) * p.o_heads_total + p.o_head_off + hq) * D;
    }
    if (n_kv == 0) {
      // no visible key at all: zero output, LSE = -inf
      if (row_valid) {
#pragma unroll
        for (int c = 0; c < D; c += 8) *(uint4*)(orow + c) = make_uint4(0, 0, 0, 0);
        p.lse[((size_t)b * p.Hq + hq) * p.Tq + qi] = -INFINITY;
      }
    } else if (alive) {
      bool ok = mbar_wait_lean(o_done, 0, abort_flag, 701);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        tc_fence_after();
        const float inv_l = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
        for (int c = 0; c < D; c += 32) {
          uint32_t v[32];
          tmem_ld32(t_o + c, v);
          tmem_wait_ld();
          if (row_valid) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 o;
              o.x = pack_bf16(__uint_as_float(v[i]) * inv_l, __uint_as_float(v[i + 1]) * inv_l);
              o.y = pack_bf16(__uint_as_float(v[i + 2]) * inv_l, __uint_as_float(v[i + 3]) * inv_l);
              o.z = pack_bf16(__uint_as_float(v[i + 4]) * inv_l, __uint_as_float(v[i + 5]) * inv_l);
              o.w = pack_bf16(__uint_as_float(v[i + 6]) * inv_l, __uint_as_float(v[i + 7]) * inv_l);
              *(uint4*)(orow + c + i) = o;
            }
          }
        }
        if (row_valid) p.lse[((size_t)b * p.Hq + hq) * p.Tq + qi] = l > 0.f ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 128); }
  if (threadIdx.x == 0 && *abort_flag) report(p.status, ST_TIMEOUT_MBAR, *abort_flag, 0);
}

template <int POLY>
static int launch_poly(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p, cudaStream_t stream) {
  static bool cfg = false;
  if (!cfg) { CPB_CUDA_OK(cudaFuncSetAttribute(flash_fwd64_kernel<POLY>, cudaFuncAttributeMaxDynamicSharedMemorySize, F64Smem::TOTAL)); cfg = true; }
  const dim3 grid(p.n_copy + (p.Tq + FA_BQ - 1) / FA_BQ * (p.Hq / p.Hkv), p.Hkv, p.B);
  CPB_CUDA_OK(launch_pdl(flash_fwd64_kernel<POLY>, grid, F64_THREADS, F64Smem::TOTAL, stream, tq, tk, tv, p));
  return check_launch("flash_fwd");
}

// tk, tv: boxes of 64 keys
int launch_flash_fwd64(int poly, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p, cudaStream_t stream) {
  switch (poly) {
    case 0: return launch_poly<0>(tq, tk, tv, p, stream);
    case 1: return launch_poly<1>(tq, tk, tv, p, stream);
    case 2: return launch_poly<2>(tq, tk, tv, p, stream);
    case 4: return launch_poly<4>(tq, tk, tv, p, stream);
    case 5: return launch_poly<5>(tq, tk, tv, p, stream);
    default: return launch_poly<3>(tq, tk, tv, p, stream);
  }
}

}  // namespace cpb
