// Arguments of a decode step, shared by the general kernel and the one with caller-supplied window logits.
#pragma once

#include "nha_common.cuh"

namespace nha {

struct DecodeArgs {
  const bf16* q; const bf16* sq; const bf16* k; const bf16* v; const bf16* g; const bf16* s;
  const bf16* sw_k; const bf16* sw_v; const bf16* cosp; const bf16* sinp; const bf16* win_logits;
  float* hk; float* hv; bf16* o; float* win_prob;
  float* part_o;      // [B*H, SPLITS, NG, V] unnormalised partial outputs
  float* part_ml;     // [B*H, SPLITS, NG, 2] running max and sum of each split
  int* tickets;       // [B*H] arrival counters, zero between calls
  int64_t cs_batch, cs_row;
  int B, HQ, H, K, V, M, W, NG, SPLITS, KS, KSp, MQ, zero_state;
  float scale;
  // shared-memory byte offsets
  int off_qraw, off_sqA, off_oks, off_eg, off_sv, off_kpop, off_vpop, off_ml, off_P, off_hk, off_hv, off_kst, off_vst,
      off_S;
};

}  // namespace nha
