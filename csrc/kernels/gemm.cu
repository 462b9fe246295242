// Persistent bf16 GEMM for sm_100a on CTA pairs (tcgen05 cta_group::2): two CTAs of a cluster compute one 256 x BN output
// tile together, TMA -> shared memory -> tcgen05.mma -> tensor memory -> registers -> shared memory -> TMA, warp-specialised,
// with a double-buffered accumulator so that the epilogue of one tile overlaps the main loop of the next.
//
//   C[M,N] (op)= A * B        A is M x K, B is N x K ("NT": both K-major) by default.
//   a_mn = 1 : A is stored as [K, M] (M contiguous)   -> weight-gradient GEMM  dW = dY^T X
//   b_mn = 1 : B is stored as [K, N] (N contiguous)   -> data-gradient GEMM    dX = dY W
// Both majors are native UMMA operand layouts, so no transposed copies are ever made.
//
// Replaces the cuBLAS GEMMs behind nn::Linear in the reference trainers
// (Scripts/Blutrain/bluscriptCP.cpp:212-330, Makefile:129).
//
// Why pairs: with one CTA per tile (128 x 256) every K=16 step of the tensor core reads (128 + 256) x 16 x 2 = 12 KB of
// operands from shared memory while TMA writes the same 12 KB, i.e. 192 bytes per tensor-core cycle against the 128 bytes
// per cycle a shared memory delivers.  In a pair each CTA stages its own 128 rows of A and only HALF of the B tile; one MMA
// instruction issued by the even CTA drives both tensor cores and each of them reads the other CTA's B half through the
// pair link, so a CTA moves (128 + 128) x 16 x 2 = 8 KB in and 8 KB out per step: 128 bytes per cycle.
//
// Protocol (per CTA: warp 0 = TMA producer, warp 1 = tensor-memory owner and, in the even CTA, MMA issuer, warps 2..5 =
// epilogue).  Every TMA load of either CTA (cta_group::2 form, no multicast) signals the EVEN CTA's `full` barrier, which
// expects the bytes of both CTAs.  After the MMAs of a stage the issuer commits twice, once to its own `empty` barrier and
// once to the odd CTA's (a cluster address), and likewise for the accumulator-ready barriers; the odd CTA's epilogue
// warps release an accumulator by a remote arrival on the even CTA's barrier.  Tensor memory is allocated with the
// cta_group::2 form by the same warp of both CTAs, so an accumulator has the same address in both; each CTA's epilogue
// drains its own 128 rows.  All waits are bounded like everywhere else in this library.
#include "common.cuh"
#include "gemm_common.cuh"
#include "host_utils.h"
#include <stdlib.h>

namespace cpb {

template <int BN>
struct GemmSmem {
  static constexpr int STAGES = BN == 384 ? 4 : BN > 128 ? 6 : 8;       // 160 to 192 KB of operands in flight
  static constexpr int A_BYTES = GEMM_BM * GEMM_BK * 2;          // 128 rows of A
  static constexpr int B_GROUPS = (BN / 2 + 63) / 64;            // this CTA's half of B's columns, in groups of 64 (N-major: 96 columns
  static constexpr int B_BYTES = B_GROUPS * 64 * GEMM_BK * 2;    // take two groups, the last 32 columns are loaded and not used)
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int ACCS = BN == 384 ? 1 : 2;                 // accumulators
  static constexpr int ACC_COLS = BN == 384 ? 512 : BN > 128 ? 256 : 128;      // tensor-memory columns of one (a power of two)
  static constexpr int STORE_OFFSET = STAGES * STAGE_BYTES;      // 4 epilogue warps x 2 buffers x 4 KB
  static constexpr int BAR_OFFSET = STORE_OFFSET + 32768;
  static constexpr int TOTAL = BAR_OFFSET + 256 + 1024;
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();                                 // the aligned forms want the whole warp at the same instruction
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load of a CTA pair: the data lands in THIS CTA's shared memory, the bytes are counted on the barrier at `bar_addr`
// (a cluster address: the even CTA's barrier).  No multicast.
__device__ __forceinline__ void tma_load_2d_pair(void* smem, const CUtensorMap* m, uint32_t bar_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem)), "l"((uint64_t)m), "r"(bar_addr), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {      // same warp of both CTAs
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
template <bool ACC>
__device__ __forceinline__ void umma_pair_ss_cp(uint32_t leader, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "n"(ACC ? 1 : 0), "r"(leader) : "memory");
}
__device__ __forceinline__ void umma_pair_ss_p(uint32_t leader, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
// Arrive on the barrier at `cluster_addr` (any CTA of the cluster) once every MMA issued so far has completed.
__device__ __forceinline__ void umma_pair_commit_p(uint32_t leader, uint32_t cluster_addr) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(cluster_addr), "r"(leader) : "memory");
}

// Tile order: bands of `band` pair-rows swept along N, rows fastest.  With band = 8 the 74 pairs running at one time
// share 8 row tiles of A and about 9 column tiles of B, and successive waves keep the band's A rows in L2, so a GEMM
// whose B operand does not fit in L2 beside A's band (8192^3: 134 MB against 126 MB) streams B once per band instead of
// once per 2.3 rows of tiles.  band = 1 is the plain order (columns fastest), kept while B stays resident anyway.
__device__ __forceinline__ void pair_tile_coords(int tile, int num_m_tiles, int num_n_blocks, int band_rows, int& mt, int& nb) {
  const int per_band = band_rows * num_n_blocks;
  const int band = tile / per_band, idx = tile - band * per_band;
  const int rows = min(band_rows, num_m_tiles - band * band_rows);
  nb = idx / rows;
  mt = band * band_rows + (idx - nb * rows);
}

template <int BN, bool A_MN, bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
gemm_pair_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmX, GemmParams p) {
  using L = GemmSmem<BN>;
  constexpr int STAGES = L::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = (uint64_t*)(smem + L::BAR_OFFSET);      // used in the even CTA only
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;     // [2]
  uint64_t* tempty_bar = tfull_bar + 2;         // [2], used in the even CTA only
  uint32_t* tmem_slot = (uint32_t*)(tempty_bar + 2);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();      // 0: even CTA (issues the MMAs), 1: odd CTA
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int num_tiles = p.num_m_tiles * p.num_n_blocks;
  const int num_items = num_tiles * p.splits;   // item = split * num_tiles + tile: items of one K range run together

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&tfull_bar[s], 1); mbar_init(&tempty_bar[s], 8); }      // 4 epilogue warps of each CTA
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, L::ACCS * L::ACC_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                           // both CTAs' barriers exist before anything arrives on them remotely
  tc_fence_after();
  // not before a launch that adds the splits' parts: its waiting blocks made the pair of launches slower (us with and without:
  // 136 x 768 x 3072 in twelve 14.4 and 9.1, 1152 x 384 x 4096 in seven 17.3 and 15.2, 384 x 384 x 4096 in eleven 10.6 and 9.4)
  if (p.splits == 1) pdl_release();
  pdl_wait();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      int stage = 0; uint32_t phase = 0;
      for (int item = pair; item < num_items; item += num_pairs) {
        const int split = item / num_tiles;
        int mt, nb;
        pair_tile_coords(item - split * num_tiles, p.num_m_tiles, p.num_n_blocks, p.band, mt, nb);
        const int m0 = mt * (2 * GEMM_BM) + (int)rank * GEMM_BM;      // this CTA's rows
        const int kb1 = min(p.num_k_blocks, (split + 1) * p.k_per_split);
        for (int kb = split * p.k_per_split; kb < kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, 110)) break;
          uint8_t* sa = smem + stage * L::STAGE_BYTES;
          uint8_t* sb = sa + L::A_BYTES;
          const uint32_t full_even = map_to_cta(smem_u32(&full_bar[stage]), 0);
          if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * (L::A_BYTES + (B_MN ? L::B_BYTES : BN * GEMM_BK)));    // the bytes of both CTAs
          const int k0 = kb * GEMM_BK;
          if (A_MN) {
#pragma unroll
            for (int g = 0; g < GEMM_BM / 64; ++g) tma_load_2d_pair(sa + g * 8192, &tmA, full_even, m0 + g * 64, k0);
          } else {
            tma_load_2d_pair(sa, &tmA, full_even, k0, m0);
          }
          if (p.epi == EPI_BF16_SWIGLU) {
            // the even CTA stages the gate rows of features nb*BN/2.., the odd CTA the matching up rows
            const int f0 = nb * (BN / 2);
            tma_load_2d_pair(sb, &tmB, full_even, k0, (rank == 0 ? 0 : p.swiglu_half) + f0);
          } else if (BN == 384) {
            // columns of the 256-wide product, 128 per CTA, then those of the 128-wide one, 64 per CTA
            const int n0 = nb * BN + (int)rank * 128, n2 = nb * BN + 256 + (int)rank * 64;
#pragma unroll
            for (int g = 0; g < 3; ++g) {
              const int n = g < 2 ? n0 + g * 64 : n2;
              tma_load_2d_pair(sb + g * 8192, &tmB, full_even, B_MN ? n : k0, B_MN ? k0 : n);
            }
          } else if (B_MN) {
            const int n0 = nb * BN + (int)rank * (BN / 2);
#pragma unroll
            for (int g = 0; g < L::B_GROUPS; ++g) tma_load_2d_pair(sb + g * 8192, &tmB, full_even, n0 + g * 64, k0);
          } else {
            tma_load_2d_pair(sb, &tmB, full_even, k0, nb * BN + (int)rank * (BN / 2));
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (*abort_flag) break;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (even CTA only; convergent warp, elected lane)
    if (rank == 0) {
      const uint32_t leader = elect_one() ? 1u : 0u;
      constexpr uint32_t idesc = make_idesc_bf16(2 * GEMM_BM, BN == 384 ? 256 : BN, A_MN, B_MN);
      constexpr uint32_t idesc2 = make_idesc_bf16(2 * GEMM_BM, 128, A_MN, B_MN);       // the last 128 of 384 columns
      const uint32_t s0 = smem_u32(smem);
      const SDesc da0 = sdesc_split(A_MN ? make_sdesc(s0, 8192, 1024) : sdesc_kmajor(s0));
      const SDesc db0 = sdesc_split(B_MN ? make_sdesc(s0 + L::A_BYTES, 8192, 1024) : sdesc_kmajor(s0 + L::A_BYTES));
      constexpr uint32_t A_STEP = A_MN ? 2048 : 32, B_STEP = B_MN ? 2048 : 32;
      int stage = 0; uint32_t phase = 0;
      int it = 0;
      bool alive = true;
      for (int item = pair; item < num_items && alive; item += num_pairs, ++it) {
        const int acc = L::ACCS == 2 ? it & 1 : 0;
        const uint32_t acc_phase = (L::ACCS == 2 ? it >> 1 : it) & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(&tempty_bar[acc], acc_phase ^ 1, abort_flag, p.status, 210))) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * L::ACC_COLS;
        const int split = item / num_tiles;
        const int kb0 = split * p.k_per_split, kb1 = min(p.num_k_blocks, kb0 + p.k_per_split);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, abort_flag, p.status, 211))) { alive = false; break; }
          tc_fence_after();
          const uint32_t so = (uint32_t)stage * (L::STAGE_BYTES >> 4);
          const SDesc da = SDesc{da0.lo + so, da0.hi}, db = SDesc{db0.lo + so, db0.hi};
          umma_pair_ss_p(leader, d_tmem, sdesc_at(da, 0), sdesc_at(db, 0), idesc, kb != kb0);
          if (BN == 384) umma_pair_ss_p(leader, d_tmem + 256, sdesc_at(da, 0), sdesc_at(db, 16384), idesc2, kb != kb0);
#pragma unroll
          for (int k = 1; k < GEMM_BK / 16; ++k) {
            umma_pair_ss_cp<true>(leader, d_tmem, sdesc_at(da, k * A_STEP), sdesc_at(db, k * B_STEP), idesc);
            if (BN == 384) umma_pair_ss_cp<true>(leader, d_tmem + 256, sdesc_at(da, k * A_STEP), sdesc_at(db, 16384 + k * B_STEP), idesc2);
          }
          // the stage is free in both CTAs once these MMAs have read it
          const uint32_t e_own = smem_u32(&empty_bar[stage]);
          umma_pair_commit_p(leader, e_own);
          umma_pair_commit_p(leader, map_to_cta(e_own, 1));
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        const uint32_t t_own = smem_u32(&tfull_bar[acc]);
        umma_pair_commit_p(leader, t_own);
        umma_pair_commit_p(leader, map_to_cta(t_own, 1));
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5 of both CTAs: own 128 rows)
    const int quarter = warp & 3;
    WarpStore ws{smem + L::STORE_OFFSET + quarter * 8192, 0u, lane == 0};
    int it = 0;
    for (int item = pair; item < num_items; item += num_pairs, ++it) {
      const int acc = L::ACCS == 2 ? it & 1 : 0;
      const uint32_t acc_phase = (L::ACCS == 2 ? it >> 1 : it) & 1;
      int mt, nb;
      pair_tile_coords(item % num_tiles, p.num_m_tiles, p.num_n_blocks, p.band, mt, nb);
      const int row0 = mt * (2 * GEMM_BM) + (int)rank * GEMM_BM + quarter * 32;
      const HeadRow head = head_row(p, row0 + lane);
      bool ok = mbar_wait(&tfull_bar[acc], acc_phase, abort_flag, p.status, 310);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * L::ACC_COLS;
      const auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (rank == 0) mbar_arrive(&tempty_bar[acc]);
          else mbar_arrive_cluster(map_to_cta(smem_u32(&tempty_bar[acc]), 0));
        }
      };
      if (p.epi >= EPI_HEAD_STATS) head_epilogue<BN>(p, &tmC, ws, t_row, row0, nb, lane, head, release);
      else gemm_epilogue<BN>(p, &tmC, &tmX, ws, t_row, row0, nb, lane, item / num_tiles, release);
    }
    ws.drain();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // the even CTA's MMAs have finished reading the odd CTA's operands; no remote arrival is in flight
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, L::ACCS * L::ACC_COLS);
  }
}

template <int BN, bool A_MN, bool B_MN>
static int launch_pair(const CUtensorMap (&tm)[4], const GemmParams& p, cudaStream_t stream) {
  auto kern = gemm_pair_bf16_kernel<BN, A_MN, B_MN>;
  static bool configured = false;
  if (!configured) {
    CPB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmSmem<BN>::TOTAL));
    configured = true;
  }
  const int items = p.num_m_tiles * p.num_n_blocks * p.splits;
  const int max_pairs = sm_count() / 2;
  const int pairs = items < max_pairs ? items : max_pairs;
  CPB_CUDA_OK(launch_pdl(kern, 2 * pairs, GEMM_THREADS, GemmSmem<BN>::TOTAL, stream, tm[0], tm[1], tm[2], tm[3], p));
  return check_launch("gemm_pair_bf16");
}

template <int BN>
static int dispatch_pair(const CUtensorMap (&tm)[4], const GemmParams& p, int a_mn, int b_mn, cudaStream_t stream) {
  if (!a_mn && !b_mn) return launch_pair<BN, false, false>(tm, p, stream);
  if (!a_mn && b_mn) return launch_pair<BN, false, true>(tm, p, stream);
  if (a_mn && !b_mn) return launch_pair<BN, true, false>(tm, p, stream);
  return launch_pair<BN, true, true>(tm, p, stream);
}

// C += partials[0] + partials[1] + ..., always in that order and after the first split has been added, so that a weight gradient
// repeats bit for bit (all splits adding to C in L2 as they finish, in one launch, do not).  
__global__ void __launch_bounds__(256)
gemm_add_partials_kernel(float* __restrict__ C, const float4* __restrict__ partials, unsigned n4, unsigned total4, long ldc, int count) {
  pdl_release();
  pdl_wait();
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total4; i += gridDim.x * blockDim.x) {
    const unsigned r = i / n4;
    float4* dst = (float4*)(C + r * ldc) + (i - r * n4);
    const float4 c = *dst;
    float4 a = partials[i];
#pragma unroll 4
    for (int s = 1; s < count; ++s) {
      const float4 v = partials[(size_t)s * total4 + i];
      a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    }
    *dst = make_float4(c.x + a.x, c.y + a.y, c.z + a.z, c.w + a.w);
  }
}

// C (bf16) = partials[0] + partials[1] + ... (+ bias), in that order.
__global__ void __launch_bounds__(256)
gemm_sum_partials_kernel(__nv_bfloat16* __restrict__ C, const float4* __restrict__ partials, const float* __restrict__ bias, unsigned n8,
                         unsigned total8, long ldc, int count) {
  pdl_release();
  pdl_wait();
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total8; i += gridDim.x * blockDim.x) {
    const unsigned r = i / n8, c = i - r * n8;
    float4 a = partials[2 * (size_t)i], b = partials[2 * (size_t)i + 1];
#pragma unroll 4
    for (int s = 1; s < count; ++s) {
      const float4 u = partials[2 * ((size_t)s * total8 + i)], v = partials[2 * ((size_t)s * total8 + i) + 1];
      a.x += u.x; a.y += u.y; a.z += u.z; a.w += u.w;
      b.x += v.x; b.y += v.y; b.z += v.z; b.w += v.w;
    }
    if (bias != nullptr) {
      const float4 u = __ldg((const float4*)bias + 2 * c), v = __ldg((const float4*)bias + 2 * c + 1);
      a.x += u.x; a.y += u.y; a.z += u.z; a.w += u.w;
      b.x += v.x; b.y += v.y; b.z += v.z; b.w += v.w;
    }
    *(uint4*)(C + r * ldc + 8 * (long)c) = make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
  }
}

// Tile width and K split.  The work items of a launch (tiles x splits) run on 74 pairs, so the time is that of the pair
// with the most items: items / 74 rounded up, each the longer of its main loop and its epilogue, plus one epilogue at the
// end.  Nanoseconds, measured: main loop per 64 of K 370 at 256 columns (8192^3: 694 us), 300 at 192 and 240 at 128 columns (892 us),
// so narrow tiles pay only where they fill a wave (M 4096, N 384, K 50304: 238 us at 256 columns, 182 at 128; M 4096, K 3072, N 768: 19.4
// at 256 and 15.4 at 192; M 8192, N 384, K 1024 10.4 at 128 and 8.3 at 192).
//
// The accumulating and the bf16 epilogue may be split: all splits but the first (bf16: all) go through a workspace of at most 128 MB,
// and a second launch adds them in a fixed order.  On the GPU that costs 1.4 us and, per split, a write and a read of the fp32 matrix in L2 at
// about 16 TB/s (M 3072, N 2048, K 8192: 106 us unsplit, 86 in two; M 384, N 384, K 8192: 36.6 unsplit, 22.6 in two, 11.7 in
// twelve; M 2048, N 2048, K 8192: 50 unsplit, 57 in two); the host pays 4 us for the launch and the workspace.  So a split has to
// save 8 us: with 1.4 us as the bar the small training steps, which wait for the host, were 1 to 3 % slower, and without any
// split 1 to 2 %.  All splits adding to C in L2 from one launch took 9.0 us in twelve and 75.7 in two, but in the order in
// which they finished: weight gradients did not repeat.
// With all pairs on narrow tiles their operands come to 15 TB/s out of L2 and 64 of K takes 290 instead of 240, 400 instead of 300 (M 3072,
// N 768, K 4096: 24 us, against 22 in two splits of wide tiles).  bf16 in splits: M 136, N 768, K 3072 14.6 us unsplit, 9.1 in twelve.
// `want` > 0 asks for the time at that many splits, 0 for the best number of them; -1: no such split.
static long plan_width(int cand, int M, int N, int K, int epi, int has_aux, int want, int& splits) {
  const long nk = (K + GEMM_BK - 1) / GEMM_BK;
  const long m_tiles = (M + 2 * GEMM_BM - 1) / (2 * GEMM_BM), pairs = sm_count() > 1 ? sm_count() / 2 : 1;
  const long pass = (long)M * N * 8 / 16000;
  const bool sums = epi == EPI_F32_ACC || epi == EPI_BF16;
  const int per_tile = epi == EPI_BF16_SWIGLU ? cand / 2 : cand;
  const long tiles = m_tiles * ((N + per_tile - 1) / per_tile);
  long ce = epi == EPI_F32 || epi == EPI_F32_ACC ? 1200 : epi == EPI_BF16_GELU ? (has_aux ? 1600 : 1400) : epi == EPI_BF16_SWIGLU ? (has_aux ? 1300 : 1000) : 650;
  if (cand != 256) ce = ce * cand / 256 + 50;
  const long max_split = want > 0 ? want : sums ? (nk + 3) / 4 : 1;                     // at least four K blocks per item
  long best = -1;
  for (long s = want > 0 ? want : 1; s <= max_split; ++s) {
    const bool sum16 = epi == EPI_BF16 && s > 1;
    if (s > 1 && want == 0 && (sum16 ? s : s - 1) * (long)M * N > (32L << 20)) break;          // the workspace
    const long kps = (nk + s - 1) / s;
    if ((nk + kps - 1) / kps != s) continue;                         // the same items as a smaller split
    const long waves = (tiles * s + pairs - 1) / pairs, busy = tiles * s < pairs ? tiles * s : pairs;
    const long main = kps * (cand == 384 ? 620 : cand == 256 ? 370 : cand == 192 ? (epi == EPI_F32_ACC || sum16 ? 300 + 100 * busy / pairs : 300) : epi == EPI_F32_ACC || sum16 ? 240 + 50 * busy / pairs : 240);
    const long out = !sum16 ? ce : cand == 256 ? 1200 : 1200 * cand / 256 + 50;
    // with one accumulator the epilogue is not hidden behind the next item's main loop
    long t = cand == 384 ? waves * (main + out) : waves * (main > out ? main : out) + (main > out ? out : main);
    if (s > 1) t += 8000 + (sum16 ? 3 * s + 1 : s + 1) * pass;       // 1.4 us and what a split has to save
    if (best < 0 || t < best) { best = t; splits = (int)s; }
  }
  return best;
}

// The best of the usual widths.
static long plan_narrow(int M, int N, int K, int epi, int has_aux, int want, int& bn, int& splits) {
  long best = -1;
  for (const int cand : {256, 192, 128}) {
    if (cand == 192 && epi == EPI_BF16_SWIGLU) continue;
    int s = 1;
    const long t = plan_width(cand, M, N, K, epi, has_aux, want, s);
    if (t >= 0 && (best < 0 || t < best)) { best = t; bn = cand; splits = s; }
  }
  return best;
}

// Tiles of 384 columns where N is one column of them and two of the others, and L2 does not hold A: it is read once, which is worth a
// tenth of the time that the plan expects of the others.  us, the best of the other widths and this one: bf16 4096 x 264 x 50304 157 and 134,
// x 384 157 and 132, 131072 x 384 x 2056 217 and 170, 37888 x 320 x 2056 66 and 59, 55000 x 264 x 3072 100 and 95; accumulating 50304 x 320 x 4096 163
// and 138, 33000 x 264 x 1024 53 and 43.  Left to the others: bf16 24000 x 384 x 3072 (94 tiles for 74 pairs) 60 and 68, 65536 x 384 x 1024 56 and
// 60.  Over 224 such sizes, bf16 and accumulating, the choice is 1 % above the better of the two.
// Splits of it: not where the others do without (8192 x 384 x 4104 in two 39 and 42), but with few tiles whatever the plan expects
// (bf16 4096 x 384 x 8192 in four 43 and 38).  Rows of A that do not all start on a 128-byte line are dear to read twice: bf16 then takes
// half full waves too (20360 x 384 x 4104 97 and 92, 42000 x 320 x 4104 142 and 131, 65536 x 264 x 4104 197 and 164; from a K of 2048 on above 320
// columns: 20360 x 384 x 2056 51 and 53, 42000 78 and 78, 65536 109 and 102).  With two and more columns of tiles it costs more than it
// saves (4096 x 768 x 50304 217 to 234 and 233 to 255, 50304 x 768 x 4096 238 and 267).
static bool one_column(int M, int N, int K, int epi) {
  if ((epi != EPI_F32_ACC && epi != EPI_BF16) || N <= 256 || N > 384 || K < 1024 || (long)M * K * 2 < (64L << 20)) return false;
  const long m_tiles = (M + 2 * GEMM_BM - 1) / (2 * GEMM_BM), pairs = sm_count() > 1 ? sm_count() / 2 : 1;
  int bn, s = 1, narrow_s = 1;
  const long t = plan_width(384, M, N, K, epi, 0, 0, s), narrow_t = plan_narrow(M, N, K, epi, 0, 0, bn, narrow_s);
  if (s > 1 && 10 * m_tiles >= 4 * pairs) return false;
  const long items = m_tiles * s, slots = (items + pairs - 1) / pairs * pairs;
  return 10 * t <= 11 * narrow_t || (s > 1 && 5 * items >= 4 * slots) || (epi == EPI_BF16 && K % 64 != 0 && K >= (N > 320 ? 2048 : 4096) && 2 * items >= slots);
}

// `want` > 0 asks for the best width at that many splits, 0 for the best of both.
static void plan_tiles(int M, int N, int K, int epi, int has_aux, int want, int& bn, int& splits) {
  if (one_column(M, N, K, epi)) plan_width(bn = 384, M, N, K, epi, has_aux, want, splits);
  else plan_narrow(M, N, K, epi, has_aux, want, bn, splits);
}

// banded tile order once B (N x K bf16) reaches 64 MB, half of L2; CPB_GEMM_BAND (read once) overrides
static int tile_band(int N, int K) {
  static const int band_env = [] { const char* e = getenv("CPB_GEMM_BAND"); return e ? atoi(e) : 0; }();
  return band_env > 0 ? band_env : (((size_t)N * K * 2 >= ((size_t)64 << 20)) ? 8 : 1);
}

static int kmajor_tmap(CUtensorMap* m, const void* ptr, int rows, int K, int ld, int box_rows) {
  uint64_t dims[2] = {(uint64_t)K, (uint64_t)rows}, strides[2] = {0, (uint64_t)ld * 2};
  uint32_t box[2] = {GEMM_BK, (uint32_t)box_rows};
  return encode_tmap(m, ptr, 2, 2, dims, strides, box, 1);
}
static int mnmajor_tmap(CUtensorMap* m, const void* ptr, int rows, int K, int ld) {
  uint64_t dims[2] = {(uint64_t)rows, (uint64_t)K}, strides[2] = {0, (uint64_t)ld * 2};
  uint32_t box[2] = {64, GEMM_BK};
  return encode_tmap(m, ptr, 2, 2, dims, strides, box, 1);
}

}  // namespace cpb

using namespace cpb;

// A: bf16, [M,K] row stride lda (a_mn=0) or [K,M] row stride lda (a_mn=1).
// B: bf16, [N,K] row stride ldb (b_mn=0) or [K,N] row stride ldb (b_mn=1).
// epi: see EPI_* above.  For EPI_BF16_SWIGLU B is the fused [2F, K] weight, N = F output features.
// splits > 1 (accumulating and bf16 epilogues, see cpb_gemm_plan): K is split that often; partials is a 16-byte aligned workspace of
// splits - 1 (bf16: splits) matrices of M x N floats, and a second launch adds them to C (bf16: sums them, adds the bias and rounds once).
extern "C" int cpb_gemm_bf16(const void* A, const void* B, void* C, void* aux, const float* bias,
                             int M, int N, int K, int lda, int ldb, int ldc, int ld_aux,
                             int a_mn, int b_mn, int epi, float* partials, int splits, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return set_error(CPB_ERR_ARG, "gemm: empty problem %dx%dx%d", M, N, K);
  // the contiguous dimension of every operand and every row stride must be a multiple of 8 elements (16 bytes)
  if ((N % 8) || (lda % 8) || (ldb % 8)) return set_error(CPB_ERR_ARG, "gemm: N,lda,ldb must be multiples of 8 (got N=%d lda=%d ldb=%d)", N, lda, ldb);
  if ((!a_mn || !b_mn) && (K % 8)) return set_error(CPB_ERR_ARG, "gemm: K=%d must be a multiple of 8 for a K-major operand", K);
  if (a_mn && (M % 8)) return set_error(CPB_ERR_ARG, "gemm: M must be a multiple of 8 when A is M-major");
  if (epi == EPI_BF16_SWIGLU && (a_mn || b_mn)) return set_error(CPB_ERR_ARG, "gemm: swiglu epilogue needs K-major operands");
  if (bias != nullptr && ((uintptr_t)bias & 15)) return set_error(CPB_ERR_ARG, "gemm: bias must be 16-byte aligned");
  if (epi != EPI_BF16_GELU && epi != EPI_BF16_SWIGLU) aux = nullptr;
  if (splits < 1) splits = 1;
  {
    const int nk = (K + GEMM_BK - 1) / GEMM_BK, kps = (nk + splits - 1) / splits;
    if (splits > 1 && ((epi != EPI_F32_ACC && epi != EPI_BF16) || partials == nullptr || ((uintptr_t)partials & 15) || (nk + kps - 1) / kps != splits))
      return set_error(CPB_ERR_ARG, "gemm: %d splits of K=%d need the accumulating or the bf16 epilogue and a 16-byte aligned workspace", splits, K);
    if (splits > 1 && (((uintptr_t)C & 15) || (ldc & (epi == EPI_BF16 ? 7 : 3)) || (long)M * N >= (1L << 32)))
      return set_error(CPB_ERR_ARG, "gemm: a split C must have 16-byte aligned rows and less than 2^32 elements");
  }
  int bn = 256;
  plan_tiles(M, N, K, epi, aux != nullptr, splits, bn, splits);
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.epi = epi;
  p.num_m_tiles = (M + 2 * GEMM_BM - 1) / (2 * GEMM_BM);
  p.num_k_blocks = (K + GEMM_BK - 1) / GEMM_BK;
  p.k_per_split = (p.num_k_blocks + splits - 1) / splits;
  p.splits = splits;
  p.swiglu_half = (epi == EPI_BF16_SWIGLU) ? N : 0;
  p.band = tile_band(N, K);
  const int per_tile = epi == EPI_BF16_SWIGLU ? bn / 2 : bn;
  p.num_n_blocks = (N + per_tile - 1) / per_tile;
  p.has_aux = aux != nullptr; p.bias = bias; p.status = status;
  const bool sum16 = splits > 1 && epi == EPI_BF16;      // every split goes to the workspace, the sum kernel writes C
  if (sum16) { p.epi = EPI_F32; p.bias = nullptr; }

  CUtensorMap tm[4];
  int rc;
  const int b_rows = epi == EPI_BF16_SWIGLU ? 2 * N : N;
  if ((rc = a_mn ? mnmajor_tmap(&tm[0], A, M, K, lda) : kmajor_tmap(&tm[0], A, M, K, lda, GEMM_BM)) != CPB_OK) return rc;
  if ((rc = b_mn ? mnmajor_tmap(&tm[1], B, b_rows, K, ldb) : kmajor_tmap(&tm[1], B, b_rows, K, ldb, bn == 384 ? 64 : bn / 2)) != CPB_OK) return rc;
  {
    // one store box = 32 rows x 128 bytes; the map's extents clip the edges of C
    const int eb = (epi == EPI_F32 || epi == EPI_F32_ACC) ? 4 : 2;
    uint64_t dims[2] = {(uint64_t)N, (uint64_t)M}, strides[2] = {0, (uint64_t)ldc * eb};
    uint32_t box[2] = {(uint32_t)(128 / eb), 32};
    if ((rc = encode_tmap(&tm[2], C, eb, 2, dims, strides, box, 1)) != CPB_OK) return rc;
  }
  tm[3] = tm[2];
  if (aux != nullptr && epi == EPI_BF16_SWIGLU) {      // [g | u] as [M][2][F]: a box never crosses from gate into up
    uint64_t dims[3] = {(uint64_t)N, 2, (uint64_t)M}, strides[3] = {0, (uint64_t)N * 2, (uint64_t)ld_aux * 2};
    uint32_t box[3] = {64, 1, 32};
    if ((rc = encode_tmap(&tm[3], aux, 2, 3, dims, strides, box, 1)) != CPB_OK) return rc;
  } else if (aux != nullptr) {
    uint64_t dims[2] = {(uint64_t)N, (uint64_t)M}, strides[2] = {0, (uint64_t)ld_aux * 2};
    uint32_t box[2] = {64, 32};
    if ((rc = encode_tmap(&tm[3], aux, 2, 2, dims, strides, box, 1)) != CPB_OK) return rc;
  }
  if (splits > 1) {
    uint64_t dims[3] = {(uint64_t)N, (uint64_t)M, (uint64_t)(sum16 ? splits : splits - 1)}, strides[3] = {0, (uint64_t)N * 4, (uint64_t)M * N * 4};
    uint32_t box[3] = {32, 32, 1};
    if ((rc = encode_tmap(&tm[3], partials, 4, 3, dims, strides, box, 1)) != CPB_OK) return rc;
  }
  rc = bn == 384 ? dispatch_pair<384>(tm, p, a_mn, b_mn, stream) : bn == 256 ? dispatch_pair<256>(tm, p, a_mn, b_mn, stream) : bn == 192 ? dispatch_pair<192>(tm, p, a_mn, b_mn, stream) : dispatch_pair<128>(tm, p, a_mn, b_mn, stream);
  if (rc != CPB_OK || splits == 1) return rc;
  const unsigned total = (unsigned)((long)M * N / (sum16 ? 8 : 4)), blocks = (total + 255) / 256, cap = (unsigned)sm_count() * 8;
  const unsigned grid = blocks < cap ? blocks : cap;
  if (sum16) CPB_CUDA_OK(launch_pdl(gemm_sum_partials_kernel, grid, 256, 0, stream, (__nv_bfloat16*)C, (const float4*)partials, bias, (unsigned)N / 8, total, (long)ldc, splits));
  else CPB_CUDA_OK(launch_pdl(gemm_add_partials_kernel, grid, 256, 0, stream, (float*)C, (const float4*)partials, (unsigned)N / 4, total, (long)ldc, splits - 1));
  return check_launch("gemm_add_partials");
}

// Cross entropy of the language-model head, logits = x w^T (x [M,K], w [N,K], both K-major).  out == null or fp32 (grad == 0): per row and
// 256-wide tile (max, sum of exponentials) to stats [ceil(N / 256)][M] and the target's logit; out, if given, gets the logits as well.
// grad == 1: out (bf16) = (softmax - onehot) * grad_scale from row_coef (cpb_xent_rows).  out: [M,N], row stride ldc.
//
// The gradient pass computes the logits again, 2 K operations for each, where storing them in fp32 moves 4 bytes for the GEMM and 4
// more for the kernel that turns them into dlogits; beyond a K of about a thousand storing them is cheaper (cpb_xent_dlogits).
extern "C" int cpb_gemm_head(const void* x, const void* w, void* out, const int64_t* targets, float* stats, float* target_logit,
                             const float* row_coef, int M, int N, int K, int ldx, int ldw, int ldc, int n_valid, int grad, float grad_scale,
                             int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return set_error(CPB_ERR_ARG, "gemm_head: empty problem %dx%dx%d", M, N, K);
  if ((N % 8) || (K % 8) || (ldx % 8) || (ldw % 8) || (out && (ldc % 8)))
    return set_error(CPB_ERR_ARG, "gemm_head: N,K,ldx,ldw,ldc must be multiples of 8 (got N=%d K=%d ldx=%d ldw=%d ldc=%d)", N, K, ldx, ldw, ldc);
  if (n_valid <= 0 || n_valid > N) return set_error(CPB_ERR_ARG, "gemm_head: n_valid=%d outside 1..%d", n_valid, N);
  if (grad ? (out == nullptr || row_coef == nullptr) : (stats == nullptr || target_logit == nullptr)) return set_error(CPB_ERR_ARG, "gemm_head: missing buffers");
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.epi = grad ? EPI_HEAD_GRAD : out ? EPI_HEAD_STORE : EPI_HEAD_STATS;
  p.num_m_tiles = (M + 2 * GEMM_BM - 1) / (2 * GEMM_BM);
  p.num_n_blocks = (N + 255) / 256;
  p.num_k_blocks = p.k_per_split = (K + GEMM_BK - 1) / GEMM_BK;
  p.splits = 1;
  p.band = tile_band(N, K);
  p.head = HeadParams{targets, (float2*)stats, target_logit, (const float2*)row_coef, n_valid, grad_scale};
  p.status = status;
  CUtensorMap tm[4];
  int rc;
  if ((rc = kmajor_tmap(&tm[0], x, M, K, ldx, GEMM_BM)) != CPB_OK) return rc;
  if ((rc = kmajor_tmap(&tm[1], w, N, K, ldw, 128)) != CPB_OK) return rc;
  tm[2] = tm[0];
  if (out) {
    const int eb = grad ? 2 : 4;
    uint64_t dims[2] = {(uint64_t)N, (uint64_t)M}, strides[2] = {0, (uint64_t)ldc * eb};
    uint32_t box[2] = {(uint32_t)(128 / eb), 32};
    if ((rc = encode_tmap(&tm[2], out, eb, 2, dims, strides, box, 1)) != CPB_OK) return rc;
  }
  tm[3] = tm[2];
  return launch_pair<256, false, false>(tm, p, stream);
}

// The plan of a GEMM of this shape and epilogue: tile width << 16 | how often K is split (at least 1).  For a split the caller brings the
// workspace, splits - 1 matrices of M x N floats for the accumulating epilogue, splits for the bf16 one.
extern "C" int cpb_gemm_plan(int M, int N, int K, int epi, int has_aux) {
  int bn = 256, splits = 1;
  if (M > 0 && N > 0 && K > 0) plan_tiles(M, N, K, epi, has_aux, 0, bn, splits);
  return bn << 16 | splits;
}
