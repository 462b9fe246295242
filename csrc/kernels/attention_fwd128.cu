// Flash-attention forward for head_dim 128 and long key sequences: two query tiles of one head per CTA.  Same contract as
// flash_fwd_kernel (attention_fwd.cu), readiness flags, copy CTAs and scatter epilogue included.
//
// One softmax warpgroup per query tile (thread = query row, 128 key columns): the tensor core works on one tile while the
// other tile's warps take exponentials, where one tile per CTA leaves it idle between its score products.  P overwrites the
// front half of the scores it was made from (the two S / P and the two O fill the 512 tensor-memory columns), so P V(j) and
// S(j+1) of a tile are issued together, and S(j+1) ready implies that P V(j) has finished: the warps wait for one barrier per
// tile, need no exchange of row maxima, and can rescale O (rarely) without another.
//
// What bounds it: the chain of one tile (clock counters in the kernel: about 3450 cycles for two tiles of 2 x 1024 tensor-core
// cycles, 1650 of them from the store of P until the next scores are in registers), and on long runs the power cap: T 32768, 32/8
// heads, back to back for two seconds, 8.0 ms at an SM clock of 1.64 GHz (1104 TFLOP/s, 3680 cycles per pair of tiles, 1005 W); one
// launch at a time 7.1 ms.
// Measured against one tile per CTA (attention_fwd.cu), same GPU, cold L2, us: 32768 keys, 32/8 heads 8740 -> 7760; 4/1 heads
// 1110 -> 1026; 16384, 16/4 heads 1131 -> 1017; 8192, 32/8 heads 615 -> 552.  Share of polynomial exponentials 0, 1, 3 of 8: 992,
// 925, 906 us at 16384 keys (another GPU); two, as in the other kernel, because three gave up accuracy.  Making the two tiles'
// warps take turns on the exponentials: 966.
#include "attention_fwd.cuh"

namespace cpb {

constexpr int FP_THREADS = 384;    // warpgroup 0: loader, MMA issuer, two idle warps; 1 and 2: softmax of one query tile each
constexpr int FP_REGS_ISSUE = 56, FP_REGS_SOFTMAX = 224;      // 56 + 2 x 224 = 3 x 168

struct FpSmem {
  static constexpr int D = 128, KST = 3, VST = 2;
  static constexpr int Q_BYTES = FA_BQ * D * 2;
  static constexpr int KV_BYTES = FA_BK * D * 2;
  static constexpr int K_OFF = 2 * Q_BYTES;
  static constexpr int V_OFF = K_OFF + KST * KV_BYTES;
  static constexpr int BAR_OFF = V_OFF + VST * KV_BYTES;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

// POLY: of the 8 column pairs of every 16-column group, the last POLY take exp2_poly_f32x2 and the others ex2.approx.
template <int POLY>
__global__ void __launch_bounds__(FP_THREADS, 1)
flash_fwd128_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, FwdParams p) {
  using L = FpSmem;
  constexpr int D = L::D;
  if (p.n_copy > 0 && blockIdx.x < (unsigned)p.n_copy) {
    pdl_wait();
    if (blockIdx.y == 0 && blockIdx.z == 0) ring_copy_cta(p.segs, p.n_segs, p.n_copy, blockIdx.x, p.ready);
    return;
  }
  const int bx = (int)blockIdx.x - p.n_copy;
  constexpr int DH = D / 64;                // 64-wide halves of the head dimension
  constexpr uint32_t S_COL = 0, O_COL = 256;     // S / P of tile t at 128 t, O at 256 + 128 t
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + L::BAR_OFF);
  uint64_t* q_full = bars + 0;              // [2 tiles]
  uint64_t* s_full = bars + 2;              // [2]
  uint64_t* p_full = bars + 4;              // [2]
  uint64_t* o_done = bars + 6;
  uint64_t* k_full = bars + 7;              // [KST]
  uint64_t* k_empty = k_full + L::KST;
  uint64_t* v_full = k_empty + L::KST;      // [VST]
  uint64_t* v_empty = v_full + L::VST;
  uint32_t* tmem_slot = (uint32_t*)(v_empty + L::VST);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.Hq / p.Hkv;
  const int num_pairs = (p.Tq + 2 * FA_BQ - 1) / (2 * FA_BQ);
  const int qt = num_pairs - 1 - bx / G;                     // heaviest tiles first
  const int hkv = blockIdx.y;
  const int hq = hkv * G + bx % G;
  const int b = blockIdx.z;
  const int q0 = qt * 2 * FA_BQ;

  if (threadIdx.x == 0) {
    for (int t = 0; t < 2; ++t) { mbar_init(&q_full[t], 1); mbar_init(&s_full[t], 1); mbar_init(&p_full[t], 4); }
    for (int s = 0; s < L::KST; ++s) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
    for (int s = 0; s < L::VST; ++s) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    mbar_init(o_done, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();                               // and no pdl_release(), see common.cuh

  // K/V tiles that each of the two query tiles attends to: 0 .. n_t - 1
  const int qpos_min0 = p.q_pos ? p.q_pos[q0] : q0;
  int n0 = (p.Tk + FA_BK - 1) / FA_BK, n1 = n0;
  if (p.causal) {
    const int l0 = min(q0 + FA_BQ, p.Tq) - 1, l1 = min(q0 + 2 * FA_BQ, p.Tq) - 1;
    const int v0 = (p.q_pos ? p.q_pos[l0] : l0) - p.k_off, v1 = (p.q_pos ? p.q_pos[l1] : l1) - p.k_off;   // last visible key
    n0 = v0 < 0 ? 0 : min(n0, v0 / FA_BK + 1);
    n1 = v1 < 0 ? 0 : min(n1, v1 / FA_BK + 1);
  }
  if (q0 + FA_BQ >= p.Tq) n1 = 0;
  const int n_kv = max(n0, n1);
  // Order of the K/V sweep: tile (j + j_start) % n_kv.  With readiness flags the sweep starts at the chunk
  // that contains this tile's own positions (resident locally), so remote chunks have time to arrive.
  int j_start = 0;
  if (p.ready != nullptr && n_kv > 0 && (p.block_rows % FA_BK) == 0) {
    const int c = max(qpos_min0 - p.k_off, 0) / p.block_rows;
    j_start = min(c * (p.block_rows / FA_BK), n_kv - 1);
  }
  // a wrapped sweep visits every tile for both query tiles (what a tile cannot see is masked)
  const int cnt0 = n0 == 0 || j_start == 0 ? n0 : n_kv, cnt1 = n1 == 0 || j_start == 0 ? n1 : n_kv;
  auto kv_tile = [&](int j) { const int jj = j + j_start; return jj >= n_kv ? jj - n_kv : jj; };

  if (warp < 4) {
    regs_give<FP_REGS_ISSUE>();
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA loader
      if (lane == 0 && n_kv > 0) {
        tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if ((t ? n1 : n0) == 0) continue;
          mbar_expect_tx(&q_full[t], L::Q_BYTES);
#pragma unroll
          for (int h = 0; h < DH; ++h)
            tma_load_4d(smem + t * L::Q_BYTES + h * (FA_BQ * 128), &tmQ, &q_full[t], h * 64, hq, q0 + t * FA_BQ, b);
        }
        int ready_block = -1;
        int ks = 0, kp = 1, vs = 0, vp = 1;
        for (int j = 0; j < n_kv; ++j) {
          if (!mbar_wait_lean(&k_empty[ks], kp, abort_flag, 500)) break;
          const int k0 = kv_tile(j) * FA_BK;
          if (p.ready != nullptr) {
            // a tile may straddle two blocks when block_rows is not a multiple of the tile
            const int blk_hi = min(k0 + FA_BK, p.Tk) - 1;
            for (int c = k0 / p.block_rows; c <= blk_hi / p.block_rows; ++c) {
              if (c == ready_block) continue;
              if (!wait_flag_ge(p.ready + c, p.ready_epoch, abort_flag, p.status, 501)) break;
              ready_block = c;
            }
            if (*abort_flag) break;
            // The copy CTAs wrote these rows with ordinary (generic-proxy) stores; the loads below go through the
            // async proxy (TMA).  The acquire above orders generic accesses only, so a cross-proxy fence is needed
            // before the first bulk-tensor read of a freshly arrived block.
            asm volatile("fence.proxy.async.global;" ::: "memory");
          }
          mbar_expect_tx(&k_full[ks], L::KV_BYTES);
#pragma unroll
          for (int h = 0; h < DH; ++h) tma_load_4d(smem + L::K_OFF + ks * L::KV_BYTES + h * (FA_BK * 128), &tmK, &k_full[ks], h * 64, hkv, k0, b);
          if (!mbar_wait_lean(&v_empty[vs], vp, abort_flag, 502)) break;
          mbar_expect_tx(&v_full[vs], L::KV_BYTES);
#pragma unroll
          for (int h = 0; h < DH; ++h) tma_load_4d(smem + L::V_OFF + vs * L::KV_BYTES + h * (FA_BK * 128), &tmV, &v_full[vs], h * 64, hkv, k0, b);
          if (++ks == L::KST) { ks = 0; kp ^= 1; }
          if (++vs == L::VST) { vs = 0; vp ^= 1; }
        }
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer
      // The whole warp runs this code convergently and only the elected lane issues: the descriptors then stay
      // warp-uniform, and stepping one is a single add (see sdesc_at).
      if (n_kv > 0) {
        const uint32_t leader = elect_one() ? 1u : 0u;
        constexpr uint32_t idesc_qk = make_idesc_bf16(FA_BQ, FA_BK, false, false);
        constexpr uint32_t idesc_pv = make_idesc_bf16(FA_BQ, D, false, true);
        const SDesc dq = sdesc_split(sdesc_kmajor(smem_u32(smem)));
        const SDesc dk0 = sdesc_split(sdesc_kmajor(smem_u32(smem + L::K_OFF)));                            // stage 0
        const SDesc dv0 = sdesc_split(make_sdesc(smem_u32(smem + L::V_OFF), FA_BK * 128, 1024));           // V tile, N-major
        const uint32_t s_tmem = tmem_base + S_COL, o_tmem = tmem_base + O_COL;
        auto issue_qk = [&](int t, int ks) {
          const SDesc q = SDesc{dq.lo + (uint32_t)t * (L::Q_BYTES >> 4), dq.hi};
          const SDesc k_ = SDesc{dk0.lo + (uint32_t)ks * (L::KV_BYTES >> 4), dk0.hi};
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint32_t off = (k / 4) * (FA_BQ * 128) + (k % 4) * 32;
            if (k == 0) umma_ss_cp<false>(leader, s_tmem + 128 * t, sdesc_at(q, off), sdesc_at(k_, off), idesc_qk);
            else umma_ss_cp<true>(leader, s_tmem + 128 * t, sdesc_at(q, off), sdesc_at(k_, off), idesc_qk);
          }
          umma_commit_p(leader, &s_full[t]);
        };
        bool ok = true;
        int ks = 0, kp = 0, vs = 0, vp = 0;              // stages of the next K tile and of V(j)
        // S(jn) of tile t, over P(jn - 1), which the P V issued before it has read
        auto scores = [&](int t, int jn, bool& k_in) {
          bool w = jn > 0 || mbar_wait_lean(&q_full[t], 0, abort_flag, 600);
          if (!k_in) w = w && mbar_wait_lean(&k_full[ks], kp, abort_flag, 604);
          k_in = true;
          if (!__all_sync(0xffffffffu, w)) return false;
          tc_fence_after();
          issue_qk(t, ks);
          return true;
        };
        auto next_k = [&] {
          umma_commit_p(leader, &k_empty[ks]);
          if (++ks == L::KST) { ks = 0; kp ^= 1; }
        };
        {
          bool k_in = false;
#pragma unroll
          for (int t = 0; t < 2; ++t) if (ok && (t ? cnt1 : cnt0) > 0) ok = scores(t, 0, k_in);
          next_k();
        }
        for (int j = 0; ok && j < n_kv; ++j) {
          const int jn = j + 1;
          bool k_in = false, v_in = false;
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int cnt = t ? cnt1 : cnt0;
            if (ok && j < cnt) {
              bool w = mbar_wait_lean(&p_full[t], j & 1, abort_flag, 602);
              if (!v_in) w = w && mbar_wait_lean(&v_full[vs], vp, abort_flag, 603);
              v_in = true;
              if (!__all_sync(0xffffffffu, w)) { ok = false; break; }
              tc_fence_after();
              const SDesc dv = SDesc{dv0.lo + (uint32_t)vs * (L::KV_BYTES >> 4), dv0.hi};
              // A = P (bf16, 8 tensor-memory columns per 16 keys); B = V tile, N-major: 16 key rows = 2 KB
              umma_ts_p(leader, o_tmem + D * t, s_tmem + 128 * t, sdesc_at(dv, 0), idesc_pv, j != 0);
#pragma unroll
              for (int k = 1; k < FA_BK / 16; ++k)
                umma_ts_cp<true>(leader, o_tmem + D * t, s_tmem + 128 * t + k * 8, sdesc_at(dv, k * 2048), idesc_pv);
            }
            if (t == 1) umma_commit_p(leader, &v_empty[vs]);
            if (ok && jn < cnt) ok = scores(t, jn, k_in);
          }
          if (!ok) break;
          if (jn < n_kv) next_k();
          if (++vs == L::VST) { vs = 0; vp ^= 1; }
        }
        umma_commit_p(leader, o_done);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue (warps 4..7: tile 0, 8..11: tile 1)
    regs_take<FP_REGS_SOFTMAX>();
    const int quarter = warp & 3;
    const int t = (warp - 4) >> 2;
    const int row = quarter * 32 + lane;
    const int qt0 = q0 + t * FA_BQ;                    // first query row of this tile
    const int qi = qt0 + row;
    const bool row_valid = qi < p.Tq;
    const int nt = t ? n1 : n0;
    const int qpos_min = qt0 < p.Tq ? (p.q_pos ? p.q_pos[qt0] : qt0) : 0;
    const int my_qpos = row_valid ? (p.q_pos ? p.q_pos[qi] : qi) : 0x7fffffff;
    const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t t_s = t_lane + S_COL + 128 * t, t_o = t_lane + O_COL + D * t;
    const int cnt = t ? cnt1 : cnt0;
    float m_used = -INFINITY;    // running max (scaled, log2 domain) the accumulators are relative to
    float l = 0.f;
    bool alive = true;
    for (int j = 0; j < cnt; ++j) {
      const int k0 = kv_tile(j) * FA_BK;
      bool ok = mbar_wait_lean(&s_full[t], j & 1, abort_flag, 700);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) { alive = false; break; }
      tc_fence_after();
      const bool need_mask = (k0 + FA_BK > p.Tk) || (p.causal && (k0 + FA_BK - 1 + p.k_off > qpos_min));
      uint32_t sv[4][32];
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) tmem_ld32(t_s + 32 * ch, sv[ch]);
      tmem_wait_ld();
      const int kmax = min(p.causal ? (my_qpos - p.k_off) : 0x7fffffff, p.Tk - 1) - k0;        // last visible column
      float mx = -INFINITY;
      if (need_mask) {
#pragma unroll
        for (int ch = 0; ch < 4; ++ch)
#pragma unroll
          for (int i = 0; i < 32; ++i) if (ch * 32 + i <= kmax) mx = fmaxf(mx, __uint_as_float(sv[ch][i]));
      } else {
        // eight independent chains of three-input maxima
        float m8[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          m8[c] = fmaxf(__uint_as_float(sv[c >> 1][(c & 1) * 16]), __uint_as_float(sv[c >> 1][(c & 1) * 16 + 1]));
#pragma unroll
          for (int i = 2; i < 16; i += 2) m8[c] = fmax3(m8[c], __uint_as_float(sv[c >> 1][(c & 1) * 16 + i]), __uint_as_float(sv[c >> 1][(c & 1) * 16 + i + 1]));
        }
        mx = fmax3(fmax3(m8[0], m8[1], m8[2]), fmax3(m8[3], m8[4], m8[5]), fmaxf(m8[6], m8[7]));
      }
      const float m_new = fmaxf(m_used, mx * p.scale_log2);
      // lazy rescale: keep the old reference maximum unless it fell behind by more than 2^8
      const bool need = (m_new > m_used + 8.f);
      float alpha = 1.f;
      if (need) {
        alpha = (m_used == -INFINITY) ? 0.f : ex2f(m_used - m_new);
        m_used = m_new;
        l *= alpha;
      }
      const float m_sub = (m_used == -INFINITY) ? 0.f : m_used;
      // p = exp2(s*scale - m) as bf16 pairs into the front half of the score columns, 32 columns at a time
      const uint64_t c2 = pack_f32x2(p.scale_log2, p.scale_log2), m2 = pack_f32x2(-m_sub, -m_sub);
      uint64_t la = pack_f32x2(0.f, 0.f), lb = la;
      // two copies of the loop: the common one (no tile edge, not on the diagonal) carries no compare/select per element
      if (!need_mask) {
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float p0, p1;
            uint64_t p2;
            const uint64_t x2 = fma_f32x2(pack_f32x2(__uint_as_float(sv[ch][i]), __uint_as_float(sv[ch][i + 1])), c2, m2);
            if (((i % 16) >> 1) >= 8 - POLY) {               // resolved at compile time (the loop is unrolled)
              p2 = exp2_poly_f32x2(x2);
              unpack_f32x2(p2, p0, p1);
            } else {
              float x0, x1;
              unpack_f32x2(x2, x0, x1);
              p0 = ex2f(x0); p1 = ex2f(x1);
              p2 = pack_f32x2(p0, p1);
            }
            if (i & 2) lb = add_f32x2(lb, p2); else la = add_f32x2(la, p2);
            pk[i >> 1] = pack_bf16(p0, p1);
          }
          tmem_st16(t_s + 16 * ch, pk);
        }
      } else {
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float p0 = (ch * 32 + i > kmax) ? 0.f : ex2f(fmaf(__uint_as_float(sv[ch][i]), p.scale_log2, -m_sub));
            const float p1 = (ch * 32 + i + 1 > kmax) ? 0.f : ex2f(fmaf(__uint_as_float(sv[ch][i + 1]), p.scale_log2, -m_sub));
            la = add_f32x2(la, pack_f32x2(p0, p1));
            pk[i >> 1] = pack_bf16(p0, p1);
          }
          tmem_st16(t_s + 16 * ch, pk);
        }
      }
      if (j > 0 && __any_sync(0xffffffffu, need)) {       // P V of the previous tile finished before S was written
#pragma unroll 1
        for (int c = 0; c < D; c += 32) {
          uint32_t v[32];
          tmem_ld32(t_o + c, v);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
          tmem_st32(t_o + c, v);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(&p_full[t]);
      float l0, l1;
      unpack_f32x2(add_f32x2(la, lb), l0, l1);
      l += l0 + l1;
    }
    // epilogue: O / l -> bf16, LSE
    __nv_bfloat16* orow = p.O + (((size_t)b * p.Tq + (row_valid ? qi : 0)) * p.Hq + hq) * D;
    if (p.o_peers != nullptr && row_valid) {
      const int peer = qi / p.o_rows_per_peer, lrow = qi % p.o_rows_per_peer;
      orow = (__nv_bfloat16*)(p.o_peers[peer] + p.o_off) +
             (((size_t)b * p.o_rows_per_peer + lrow) * p.o_heads_total + p.o_head_off + hq) * D;
    }
    if (nt > 0 && alive) {
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
        if (row_valid)
          p.lse[((size_t)b * p.Hq + hq) * p.Tq + qi] = l > 0.f ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
      }
    } else if (nt == 0 && row_valid) {
      // no visible key at all: zero output, LSE = -inf
#pragma unroll
      for (int c = 0; c < D; c += 8) *(uint4*)(orow + c) = make_uint4(0, 0, 0, 0);
      p.lse[((size_t)b * p.Hq + hq) * p.Tq + qi] = -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
  if (threadIdx.x == 0 && *abort_flag) report(p.status, ST_TIMEOUT_MBAR, *abort_flag, 0);
}

template <int POLY>
static int launch_pair(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p, cudaStream_t stream) {
  static bool cfg = false;
  if (!cfg) { CPB_CUDA_OK(cudaFuncSetAttribute(flash_fwd128_pair_kernel<POLY>, cudaFuncAttributeMaxDynamicSharedMemorySize, FpSmem::TOTAL)); cfg = true; }
  const dim3 grid(p.n_copy + (p.Tq + 2 * FA_BQ - 1) / (2 * FA_BQ) * (p.Hq / p.Hkv), p.Hkv, p.B);
  CPB_CUDA_OK(launch_pdl(flash_fwd128_pair_kernel<POLY>, grid, FP_THREADS, FpSmem::TOTAL, stream, tq, tk, tv, p));
  return check_launch("flash_fwd");
}

int launch_flash_fwd128_pair(int poly, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p, cudaStream_t stream) {
  switch (poly) {
    case 0: return launch_pair<0>(tq, tk, tv, p, stream);
    case 1: return launch_pair<1>(tq, tk, tv, p, stream);
    case 3: return launch_pair<3>(tq, tk, tv, p, stream);
    case 4: return launch_pair<4>(tq, tk, tv, p, stream);
    default: return launch_pair<2>(tq, tk, tv, p, stream);
  }
}

}  // namespace cpb
