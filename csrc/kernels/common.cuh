// Device-side building blocks shared by every sm_100a kernel in this library:
// mbarrier / TMA / tcgen05 (UMMA + tensor memory) PTX wrappers, shared-memory and
// instruction descriptors, bounded waits and the status word they report into.
//
// Rules every kernel here follows:
//   * every spin (mbarrier, peer flag) is bounded; on expiry the waiter writes a code to the
//     kernel's status word, raises a CTA-wide abort flag and the kernel drains and returns
//     normally, freeing any tensor memory it holds;
//   * TMA loads never use cluster multicast;
//   * a tiled TMA copy always starts at an inner coordinate that is a multiple of 16 bytes.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cpb {

// ------------------------------------------------------------------ status codes
enum : int {
  ST_OK = 0,
  ST_TIMEOUT_MBAR = 1,     // an mbarrier wait ran out
  ST_TIMEOUT_FLAG = 2,     // a peer-flag wait ran out
  ST_BAD_INDEX = 3,        // debug bounds check tripped
};

// status word layout: [0]=code, [1]=site id, [2]=blockIdx.x, [3]=aux
struct Status { int code, site, block, aux; };

__device__ __forceinline__ void report(int* status, int code, int site, int aux) {
  if (status != nullptr && atomicCAS(status, 0, code) == 0) {
    status[1] = site; status[2] = (int)blockIdx.x; status[3] = aux;
  }
}

// ------------------------------------------------------------------ misc
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

// ------------------------------------------------------------------ programmatic dependent launch
// A kernel started with launch_pdl (host_utils.h) may begin while the one before it on the stream still runs: its blocks set up
// barriers, tensor memory and descriptors, and pdl_wait() returns once every earlier kernel has finished and its writes are
// visible.  So pdl_wait() comes before the first access to global memory, weights included (the optimiser may be what runs before),
// and every block gets there: a grid that ended without it could end before its predecessor.
// pdl_release() lets the next kernel's blocks in as soon as every block of this one has got that far: after the block has its
// tensor memory, or a waiting block on the same SM could hold the columns that a running one still wants, and never in a kernel
// that waits for other GPUs, whose SMs the blocks let in would keep from the kernels of other streams.
// Nor in the attention kernels: their CTAs are long and uneven, and the blocks that wait on the SMs already done slow down the ones still
// running (32749 tokens, 4/1 heads of 128, us per pass, one after the other: all releasing 3900, without the backward's 3896, without
// the forward's either 3742, before dependent launches 3766; the backward kernel 2552 to 2680 and 2494 to 2507; the whole
// gradient in a chain, with and without: 2 x 1000, 6/2 heads of 64 25.0 and 23.5, 1024, 32/8 of 128 55.6 and 53.4, 4000, 8/2 105.4 and 98.5; with
// the forward before it 2 x 1000 39.6 and 41.7, 2 x 300 28.5 and 25.3, 1024, 32/8 of 128 78.8 and 77.3).  Up to 1024 keys the
// forward does all the same, its CTAs are short there (one window of GPT-2 124M, us without and with: 136 tokens 633 and 624, 4 x 1024
// tokens 1499 and 1486; of the 48M model, 1024 tokens 381 and 370; 2048 and 4096 tokens the same).
// us per GEMM in a chain, without and with: 136 x 768 x 64 4.6 and 3.7, 136 x 2304 x 768 7.2 and 6.1, 4096 x 1536 x 384 8.7 and 8.0.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// One arrival for a whole warp: per-thread arrivals on one barrier word serialise (32 per warp instruction), which at
// 256 arrivals per tile costs hundreds of cycles on the critical path.  Every lane must have completed its own work
// (tcgen05.wait, proxy fence, tcgen05.fence::before_thread_sync) before the call; __syncwarp orders the lanes' writes
// before the elected arrival.
__device__ __forceinline__ void mbar_arrive_warp(uint64_t* bar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}

// try_wait with a suspend-time hint: the hardware parks the thread until the phase completes or the hint
// (nanoseconds) runs out, so a waiting warp does not burn issue slots and shared-memory bandwidth that the
// working warps of the same SM partition need.
__device__ __forceinline__ bool mbar_try_wait_hint(uint64_t* bar, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(ns) : "memory");
  return ok != 0;
}

// Bounded wait.  `abort_flag` lives in shared memory; once any waiter of the CTA has timed out
// every later wait returns at once so the kernel drains in bounded time.  Worst case: CPB_WAIT_SPINS
// suspensions of CPB_WAIT_HINT_NS each (about 2 s).
#ifndef CPB_WAIT_SPINS
#define CPB_WAIT_SPINS (100000u)
#endif
#ifndef CPB_WAIT_FAST_SPINS
#define CPB_WAIT_FAST_SPINS 256
#endif
#ifndef CPB_WAIT_HINT_NS
#define CPB_WAIT_HINT_NS (20000u)
#endif
// Out of line on purpose: the warp-specialised kernels wait in dozens of places, and their hot loops must stay small
// enough for the instruction cache.  Reached only when the first probe of the barrier fails.
static __device__ __noinline__ bool mbar_wait_slow(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                   int* status, int site) {
  // short waits (the common case inside a pipelined kernel) spin; long waits are parked by the hardware
#pragma unroll 1
  for (int it = 0; it < CPB_WAIT_FAST_SPINS; ++it)
    if (mbar_try_wait(bar, parity)) return true;
#pragma unroll 1
  for (uint32_t it = 0; it < CPB_WAIT_SPINS; ++it) {
    if (mbar_try_wait_hint(bar, parity, CPB_WAIT_HINT_NS)) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  report(status, ST_TIMEOUT_MBAR, site, (int)parity);
  return false;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          int* status, int site) {
  if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_slow(bar, parity, abort_flag, status, site);
}

// The same wait without a call and without the report: for kernels that move registers between warpgroups (setmaxnreg does
// not go together with calls).  A few instructions in line; an expired wait leaves its site in `abort_site`, which the
// kernel reports once all its roles are done.
__device__ __forceinline__ bool mbar_wait_lean(uint64_t* bar, uint32_t parity, volatile int* abort_site, int site) {
  if (mbar_try_wait(bar, parity)) return true;
#pragma unroll 1
  for (uint32_t it = 0; it < CPB_WAIT_SPINS; ++it) {
    if (mbar_try_wait_hint(bar, parity, CPB_WAIT_HINT_NS)) return true;
    if (*abort_site) return false;
  }
  *abort_site = site;
  return false;
}

// Registers moved between warpgroups (setmaxnreg, all four warps of the warpgroup).
template <int R> __device__ __forceinline__ void regs_give() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R> __device__ __forceinline__ void regs_take() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }

// ------------------------------------------------------------------ proxies / fences
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ------------------------------------------------------------------ TMA (no multicast anywhere)
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)m) : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* smem, const CUtensorMap* m, uint64_t* bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem)), "l"((uint64_t)m), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// Untiled bulk copy: both addresses and the size are multiples of 16 bytes.
__device__ __forceinline__ void bulk_load_1d(void* smem, const void* gmem, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem)), "l"((uint64_t)gmem), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// A global load that stays where it is written (the compiler would otherwise sink it to its first use, one tile later).
__device__ __forceinline__ int ld_ahead_s32(const int* ptr) {
  int v;
  asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(ptr));
  return v;
}
__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {      // addr 16-byte aligned
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// ------------------------------------------------------------------ tensor memory
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {   // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
               ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {      // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 32 lanes x 32 columns of 32-bit: thread t of the warp gets lane (base_lane + t), 32 consecutive columns.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ------------------------------------------------------------------ UMMA descriptors
// Shared-memory matrix descriptor, 128-byte swizzle, descriptor version 1 (Blackwell).
//   K-major  : rows of 128 B (64 bf16 along K); groups of 8 rows are `sbo` bytes apart (1024 when
//              dense); the leading-offset field is unused and holds 1.
//   MN-major : rows of 128 B (64 bf16 along M/N), one row per K index; groups of 8 K-rows are `sbo`
//              bytes apart, successive 64-element M/N groups are `lbo` bytes apart.
__device__ __forceinline__ uint64_t make_sdesc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;       // version
  d |= (uint64_t)2 << 61;       // SWIZZLE_128B
  return d;
}
__device__ __forceinline__ uint64_t sdesc_kmajor(uint32_t smem_addr) { return make_sdesc(smem_addr, 16, 1024); }

// Instruction descriptor for kind::f16 with bf16 operands and fp32 accumulation.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N, bool a_mn_major, bool b_mn_major) {
  return (1u << 4)                       // D format: f32
       | (1u << 7)                       // A format: bf16
       | (1u << 10)                      // B format: bf16
       | ((a_mn_major ? 1u : 0u) << 15)
       | ((b_mn_major ? 1u : 0u) << 16)
       | ((uint32_t)(N >> 3) << 17)
       | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A * B with A in shared memory (umma_ss...) or tensor memory (umma_ts...) and B in shared memory.
// Lean issue path.  One thread issues every MMA of a CTA, and at N <= 128 an MMA lasts only 45-64 cycles, so the
// scalar instructions between two MMAs decide the tensor-core rate.  A descriptor is kept as two 32-bit halves: the
// start-address field is lo[13:0] in 16-byte units, so stepping it by a byte offset (address stays below 256 KB) is
// one 32-bit add with an immediate; the accumulate flag is a template constant unless it depends on the iteration.
struct SDesc { uint32_t lo, hi; };
__device__ __forceinline__ SDesc sdesc_split(uint64_t d) { return SDesc{(uint32_t)d, (uint32_t)(d >> 32)}; }
__device__ __forceinline__ uint64_t sdesc_at(SDesc d, uint32_t byte_off) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(d.lo + (byte_off >> 4)), "r"(d.hi));
  return r;
}
// Issued by the elected lane of a warp that runs the surrounding code convergently: operands that are
// warp-uniform can then stay in uniform registers instead of being moved there before every MMA.
template <bool ACC>
__device__ __forceinline__ void umma_ss_cp(uint32_t leader, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "n"(ACC ? 1 : 0), "r"(leader) : "memory");
}
template <bool ACC>
__device__ __forceinline__ void umma_ts_cp(uint32_t leader, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "n"(ACC ? 1 : 0), "r"(leader) : "memory");
}
__device__ __forceinline__ void umma_ss_p(uint32_t leader, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
__device__ __forceinline__ void umma_ts_p(uint32_t leader, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
// Arrive on `bar` once every MMA issued so far by the elected lane has completed.
__device__ __forceinline__ void umma_commit_p(uint32_t leader, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(smem_u32(bar)), "r"(leader) : "memory");
}

// ------------------------------------------------------------------ small math helpers
#ifdef CPB_PROF_ORDER      // diagnostic builds: keep the math between the clock reads that bracket it
#define CPB_MATH_ASM asm volatile
#else
#define CPB_MATH_ASM asm
#endif
// Packed pairs of fp32 (sm_100): one instruction for two fused multiply-adds / adds / multiplies.  The softmax warps are
// bound by issue slots, so halving their FFMA and FADD counts is worth more than anything done to the exponential unit.
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  CPB_MATH_ASM("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  CPB_MATH_ASM("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  CPB_MATH_ASM("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {     // one instruction on sm_100
  float r;
  CPB_MATH_ASM("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float ex2f(float x) {
  float y;
  CPB_MATH_ASM("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t r;
  CPB_MATH_ASM("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// exp2 of two floats on the FMA and integer pipes instead of the special-function unit: x = n + f with n = round(x),
// f in [-0.5, 0.5]; 2^f from a cubic (maximum relative error 7.6e-5, far below the bf16 rounding the result gets);
// the result's exponent field is then advanced by n with an integer add.  The special-function unit delivers 16
// exponentials per clock per SM and a 128x128 attention tile needs 16384 of them; sending a share of the columns
// through this routine shortens the exponential phase of the attention kernels.
// Valid for x <= 100; arguments below -126 are clamped (the result is then 2^-126 instead of a denormal or zero).
__device__ __forceinline__ uint64_t exp2_poly_f32x2(uint64_t x2) {
  float x0, x1;
  unpack_f32x2(x2, x0, x1);
  x0 = fmaxf(x0, -126.f); x1 = fmaxf(x1, -126.f);
  x2 = pack_f32x2(x0, x1);
  const uint64_t magic = pack_f32x2(12582912.f, 12582912.f);          // 1.5 * 2^23: adding it rounds to an integer
  const uint64_t t = add_f32x2(x2, magic);
  const uint64_t r = add_f32x2(t, pack_f32x2(-12582912.f, -12582912.f));
  const uint64_t f = fma_f32x2(r, pack_f32x2(-1.f, -1.f), x2);
  uint64_t p = fma_f32x2(f, pack_f32x2(0.05520550534129143f, 0.05520550534129143f), pack_f32x2(0.24261397123336792f, 0.24261397123336792f));
  p = fma_f32x2(p, f, pack_f32x2(0.6932547688484192f, 0.6932547688484192f));
  p = fma_f32x2(p, f, pack_f32x2(0.9999276995658875f, 0.9999276995658875f));
  float t0, t1, p0, p1;
  unpack_f32x2(t, t0, t1);
  unpack_f32x2(p, p0, p1);
  // the low mantissa bits of t hold n in two's complement; shifted into the exponent field they add n to p's exponent
  p0 = __uint_as_float(__float_as_uint(p0) + (__float_as_uint(t0) << 23));
  p1 = __uint_as_float(__float_as_uint(p1) + (__float_as_uint(t1) << 23));
  return pack_f32x2(p0, p1);
}
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }

}  // namespace cpb
