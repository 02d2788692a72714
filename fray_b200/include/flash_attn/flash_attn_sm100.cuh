#pragma once
// Entry points the JIT-generated `launch` bodies call for the attention forward path.
// Replaces fray::flash_attn_cute<R,C,D> (fray/include/flash_attn/flashattn_cute.cuh:166-239):
// same fp16 [B,H,S,D] operands and in-place output, plus explicit strides, an optional
// causal mask and an explicit softmax scale.

#include "fwd_simple_sm100.cuh"
#include "host_sm100.cuh"
#include "fwd_ws_sm100.cuh"
#include "fwd_alt_sm100.cuh"
#include "fwd_one_sm100.cuh"
#include "fwd_duo_sm100.cuh"
#include "fwd_split_sm100.cuh"

namespace fray {

// Kernel families selectable from the tuning space.
enum AttnKernelKind : int {
  kAttnSimple = 0,           // one 128-row tile per CTA, single role, no overlap; two CTAs per SM
  kAttnWarpSpecialized = 1,  // two 128-row tiles per CTA, producer / MMA / softmax / correction roles
  kAttnAlternating = 2,        // one 128-row tile per CTA, scores and probabilities in separate tensor-memory buffers,
                             // two softmax groups on alternate KV steps
  kAttnPaired = 3,           // the same on a pair of CTAs (cta_group::2): 256 rows per pair, half of K and V per CTA
  kAttnOneTile = 4,          // one 128-row tile per CTA, producer / MMA / softmax roles, 256 tensor-memory columns:
                             // two CTAs per SM cover each other's start, end and softmax phases
  kAttnFewQueries = 6,       // all rows of a K/V head's group in one tile, keys split over a cluster of CTAs; what does
                             // not have that form runs as kind 1
  kAttnDuo = 7,              // two 128-row tiles, two softmax threads per row, one CTA per SM that walks through the work
                             // items
  kAttnPersistent = 5,       // kind 1 in that form, until kind 7 was faster in all of it: the number now means kind 7
};

// KIND, D, BLOCK_N, STAGES are compile-time tuning keys (BLOCK_N: KV tile of the single-role kernel, 128
// elsewhere; STAGES: K/V ring depth of kind 1, K ring depth of kinds 2 and 3); everything else is a
// run-time argument.  K and V have num_kv_heads heads
// (a divisor of num_heads; query head h uses K/V head h / (num_heads / num_kv_heads)) and seq_len_kv rows
// (seq_len is the number of queries); lse is null or an
// fp32 [B, H, S] array that receives the log-sum-exp of every query row.  `rc` receives an
// AttnReturnCode; a non-zero value means nothing was launched.
template <int KIND, int D, int BLOCK_N, int STAGES>
inline void flash_attn_sm100(const operand_t* q, const operand_t* k, const operand_t* v, operand_t* o, int batch_size,
                             int num_heads, int seq_len, int q_sb, int q_sh, int q_ss, int k_sb, int k_sh, int k_ss,
                             int v_sb, int v_sh, int v_ss, int o_sb, int o_sh, int o_ss, int num_kv_heads,
                             int seq_len_kv, float* lse, bool causal, float scale, cudaStream_t stream, int& rc) {
  const AttnShape shp{batch_size, num_heads, seq_len, D};
  const bool bad_shape = num_kv_heads <= 0 || num_heads % num_kv_heads != 0 || seq_len_kv <= 0 ||
                         !(scale > 0.f) || !(scale <= 3.0e38f);  // also false for NaN
  if (bad_shape || (reinterpret_cast<uintptr_t>(lse) & 3u) != 0) {
    rc = bad_shape ? kAttnBadShape : kAttnBadPointer;
    return;
  }
  const AttnExtras ex{num_heads / num_kv_heads, lse, seq_len_kv};
  const AttnStrides st[4] = {{q_sb, q_sh, q_ss}, {k_sb, k_sh, k_ss}, {v_sb, v_sh, v_ss}, {o_sb, o_sh, o_ss}};
  const AttnShape shp_kv{batch_size, num_kv_heads, seq_len_kv, D};
  rc = validate_attn_args(q, k, v, o, shp, shp_kv, st);
  if (rc != kAttnOk) return;
  if constexpr (KIND == kAttnSimple) {
    rc = sm100::launch_attn_fwd_simple<D, BLOCK_N>(q, k, v, o, shp, st, ex, causal, scale, stream);
  } else if constexpr (KIND == kAttnWarpSpecialized) {
    rc = sm100::launch_attn_fwd_ws<D, BLOCK_N, STAGES>(q, k, v, o, shp, st, ex, causal, scale, stream);
  } else if constexpr (KIND == kAttnAlternating) {
    rc = sm100::launch_attn_fwd_alt<D, STAGES, 1>(q, k, v, o, shp, st, ex, causal, scale, stream);
  } else if constexpr (KIND == kAttnOneTile) {
    rc = sm100::launch_attn_fwd_one<D, BLOCK_N, STAGES>(q, k, v, o, shp, st, ex, causal, scale, stream);
  } else if constexpr (KIND == kAttnDuo || KIND == kAttnPersistent) {
    static_assert(BLOCK_N == 128, "written for 128-key tiles");
    rc = sm100::launch_attn_fwd_duo<D, STAGES>(q, k, v, o, shp, st, ex, causal, scale, stream);
  } else if constexpr (KIND == kAttnFewQueries) {
    if (sm100::split_applies(shp, ex, causal)) {
      rc = sm100::launch_attn_fwd_split<D>(q, k, v, o, shp, st, ex, scale, stream);
    } else {
      rc = sm100::launch_attn_fwd_ws<D, BLOCK_N, STAGES>(q, k, v, o, shp, st, ex, causal, scale, stream);
    }
  } else {
    static_assert(KIND == kAttnPaired, "unknown kernel kind");
    static_assert(D == 128, "the paired kernel is built for head dim 128");
    rc = sm100::launch_attn_fwd_alt<D, STAGES, 2>(q, k, v, o, shp, st, ex, causal, scale, stream);
  }
}

// The arguments of flash_attn_sm100 that stay the same from call to call of one tensor layout.
struct AttnLayout {
  int batch_size, num_heads, seq_len;
  int q_sb, q_sh, q_ss, k_sb, k_sh, k_ss, v_sb, v_sh, v_ss, o_sb, o_sh, o_ss;
  int num_kv_heads, seq_len_kv, causal;
  float scale;
};

template <int KIND, int D, int BLOCK_N, int STAGES>
inline void flash_attn_layout(void* q, void* k, void* v, void* o, void* lse, void* stream, const AttnLayout& l, int& rc) {
  flash_attn_sm100<KIND, D, BLOCK_N, STAGES>(
      static_cast<const operand_t*>(q), static_cast<const operand_t*>(k), static_cast<const operand_t*>(v),
      static_cast<operand_t*>(o), l.batch_size, l.num_heads, l.seq_len, l.q_sb, l.q_sh, l.q_ss, l.k_sb, l.k_sh, l.k_ss,
      l.v_sb, l.v_sh, l.v_ss, l.o_sb, l.o_sh, l.o_ss, l.num_kv_heads, l.seq_len_kv, static_cast<float*>(lse), l.causal != 0,
      l.scale, static_cast<cudaStream_t>(stream), rc);
}

// How a launch of this layout on the current device deals its work, for tests and tools: mode (DuoMode; 0 for every other kind) and
// CTAs per work item.  Returns an AttnReturnCode.
template <int KIND, int D, int STAGES>
inline int flash_attn_form(const AttnLayout& l, int* mode, int* parts) {
  *mode = 0;
  *parts = 1;
  if constexpr (KIND == kAttnDuo || KIND == kAttnPersistent) {
    sm100::DuoPlan plan;
    const int rc = sm100::duo_plan<D, STAGES>(AttnShape{l.batch_size, l.num_heads, l.seq_len, D},
                                              AttnShape{l.batch_size, l.num_kv_heads, l.seq_len_kv, D}, l.causal != 0, nullptr, plan);
    if (rc != kAttnOk) return rc;
    *mode = plan.mode;
    *parts = plan.parts;
  }
  return kAttnOk;
}

// Whether a launch of this layout on the current device puts a pair of CTAs to every work item (DuoPair), or a negative AttnReturnCode.
template <int KIND, int D, int STAGES>
inline int flash_attn_pair(const AttnLayout& l) {
  if constexpr (KIND == kAttnDuo || KIND == kAttnPersistent) {
    sm100::DuoPlan plan;
    const int rc = sm100::duo_plan<D, STAGES>(AttnShape{l.batch_size, l.num_heads, l.seq_len, D},
                                              AttnShape{l.batch_size, l.num_kv_heads, l.seq_len_kv, D}, l.causal != 0, nullptr, plan);
    return rc == kAttnOk ? plan.pair : -rc;
  }
  return 0;
}

// Whether a launch of this layout on the current device runs four independent streams per CTA (1), or a negative AttnReturnCode.
template <int KIND, int D, int STAGES>
inline int flash_attn_four_streams(const AttnLayout& l) {
  if constexpr (KIND == kAttnDuo || KIND == kAttnPersistent) {
    sm100::DuoPlan plan;
    const int rc = sm100::duo_plan<D, STAGES>(AttnShape{l.batch_size, l.num_heads, l.seq_len, D},
                                              AttnShape{l.batch_size, l.num_kv_heads, l.seq_len_kv, D}, l.causal != 0, nullptr, plan);
    return rc == kAttnOk ? plan.quad : -rc;
  }
  return 0;
}

}  // namespace fray
