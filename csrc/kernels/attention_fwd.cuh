// What the two attention forward kernels share: parameters, the wait for a block of K/V, the launcher of the pair kernel.
#pragma once
#include "common.cuh"
#include "host_utils.h"
#include "ring_copy.cuh"

namespace cpb {

constexpr int FA_BQ = 128;
constexpr int FA_BK = 128;

struct FwdParams {
  int B, Tq, Tk, Hq, Hkv;
  int causal;
  int k_off;                 // global position of K row 0
  float scale_log2;          // softmax scale * log2(e)
  const int* q_pos;          // [Tq] global position of each query row, or null (= row index)
  __nv_bfloat16* O;          // [B,Tq,Hq,D]
  float* lse;                // [B,Hq,Tq]
  // fused-ring readiness flags: K/V rows [c*block_rows, (c+1)*block_rows) may be read once
  // ready[c] >= ready_epoch.  null -> everything is ready.
  int* ready;
  int ready_epoch;
  int block_rows;
  // fused ring: the first n_copy CTAs (blockIdx.x < n_copy, y = z = 0) pull the K/V blocks listed in segs into
  // the local position-ordered buffer and bump ready[]; the compute CTAs start on the chunk that holds
  // their own diagonal (local data) and wrap around while remote chunks land.
  const CopySeg* segs;
  int n_segs;
  int n_copy;
  // Ulysses: when o_peers != null the epilogue stores each output row straight into the arena of the rank
  // that owns the token: row qi -> peer qi / o_rows_per_peer, local row qi % o_rows_per_peer, layout
  // [B, o_rows_per_peer, o_heads_total, D] at byte offset o_off, head slot o_head_off + hq.
  const uint64_t* o_peers;
  long o_off;
  int o_rows_per_peer, o_head_off, o_heads_total;
  int* status;
};

// Bounded acquire-spin on a readiness flag in global memory (written by a copy kernel or a peer).
__device__ __forceinline__ bool wait_flag_ge(const int* flag, int value, volatile int* abort_flag, int* status, int site) {
  for (uint32_t it = 0; it < (1u << 22); ++it) {
    int v;
    asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (v >= value) return true;
    if (*abort_flag) return false;
    __nanosleep(200);
  }
  *abort_flag = 1;
  report(status, ST_TIMEOUT_FLAG, site, value);
  return false;
}

// attention_fwd128.cu: head_dim 128, two query tiles per CTA; poly = share (of 8) of polynomial exponentials, 0 to 4
int launch_flash_fwd128_pair(int poly, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p, cudaStream_t stream);

// attention_fwd64.cu: head_dim 64, tk and tv with boxes of 64 keys; poly as above, 0 to 5
int launch_flash_fwd64(int poly, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p, cudaStream_t stream);

}  // namespace cpb
