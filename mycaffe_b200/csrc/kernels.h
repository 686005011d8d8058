// Internal alias: the kernels implement exactly the raw entry points of the public header.
#pragma once
#include "mycaffe_attn.h"

// Internal: turn the public (bits, bits_t, mask_mode) triple into the kernels' view; *view stays null for no mask.
struct McaMaskBits;
int mca_mask_bits_view(const uint32_t* bits, const uint32_t* bits_t, int mask_mode, int T, int need_transpose, McaMaskBits* out,
                       const McaMaskBits** view);

// Internal: mca_classify_causal_mask in one launch.
struct McaClassifyJob;
struct McaPackJob;
int mca_classify_causal_mask_ws(const McaClassifyJob* job, void* stream);

// Internal: mca_sdpa_backward_f32_layout with room for dS between its two kernels (ds_floats floats, 16-byte aligned; fewer than
// mca_sdpa_backward_f32_ws_bytes asks for, which is 0 where it would not be used: dS is formed twice).
int64_t mca_sdpa_backward_f32_ws_bytes(int B, int H, int T);
int mca_sdpa_backward_f32_ws(const float* q, const float* k, const float* v, const float* dy, const float* y_saved, const float* mask,
                             int mask_mode, const int* causal_flag, const float* row_max, const float* row_sum, float* delta_scratch,
                             int B, int H, int T, int D, float* dq, float* dk, float* dv, float* ds, int64_t ds_floats, int layout,
                             void* stream);

// Internal: mca_sdpa_backward_tc_masked and mca_sdpa_backward_f32_tc_masked with room for dS between their two kernels (16-byte
// aligned; null, or less than ds_rules::plan asks for: dS is formed twice).
int mca_sdpa_backward_tc_ws(const void* q, const void* k, const void* v, const void* y, const void* dy, const float* lse,
                            float* delta_scratch, int dtype, int causal, int B, int H, int T, int D, void* dq, void* dk, void* dv,
                            int* status, int layout, const uint32_t* mask_bits, const uint32_t* mask_bits_t, int mask_mode, void* ds,
                            int64_t ds_bytes, void* stream);
int mca_sdpa_backward_f32_tc_ws(const float* dy, const float* y_copy, const float* lse, float* delta_scratch, int causal, int B, int H,
                                int T, int D, float* dq, float* dk, float* dv, void* workspace, int64_t workspace_bytes, int* status,
                                int layout, const uint32_t* mask_bits, const uint32_t* mask_bits_t, int mask_mode, void* ds,
                                int64_t ds_bytes, void* stream);

// Internal: the fp32 forward of a short call that nothing is kept of, in one launch (attn_small.cu); small_rules::takes says which.
int mca_sdpa_forward_small(const float* q, const float* k, const float* v, const float* mask, int mode, int B, int H, int T, int D, float* y,
                           int layout, void* stream);

// Internal: the two halves of mca_sdpa_forward_f32_tc_masked -- the pre-pass that splits q, k, v (and classifies the caller's
// (T,T) mask, or packs the key mask's bits, in the same launch when `cls` or `pack` is given), and the kernel, which may then be chosen on the class.
int mca_split_forward_prepass(const float* q, const float* k, const float* v, int B, int H, int T, int D, void* workspace,
                              int64_t workspace_bytes, int layout, const McaClassifyJob* cls, const McaPackJob* pack, void* stream);
int mca_split_forward_main(int causal, int B, int H, int T, int D, float* y, float* row_max, float* row_sum, float* y_copy, float* lse,
                           void* workspace, int* status, int layout, const uint32_t* mask_bits, int mask_mode, void* stream);

// Internal: mca_mask_pack whose forward may be let go at its top.
int mca_mask_pack_ahead(const float* mask, int mask_mode, int B, int T, uint32_t* bits, uint32_t* bits_t, int let_go, void* stream);

// Internal: hand the current device's kernels the address of their row of failure words (McaFailWord).
int mca_set_fail_words_fwd(int* words);
int mca_set_fail_words_bwd(int* words);
int mca_set_fail_words_probe(int* words);
int mca_set_fail_words_decode(int* words);
int mca_set_fail_words_proj(int* words);

// Internal: the decode attention inside a step of up to eight sequences.  Where step_rules says so its combine pass is left to
// mca_decode_out_proj_partials (one sequence), which combines the partial results while it stages its activations: *partials
// then says where they are; with nsplit 1 the output is in `out` as mca_decode_attention leaves it.
struct McaDecodePartials {
  const float *acc, *ml;
  const int* pos;
  int n_heads, hs, nsplit, split_len, pos_limit;
};
int mca_decode_attention_partials(const float* q, const float* k_new, const float* v_new, void* k_cache, void* v_cache,
                                  int cache_is_bf16, int64_t cache_batch_stride, const int* pos, int B, int n_heads, int n_kv_heads,
                                  int head_size, int seq_len, int max_len, const float* freq_real, const float* freq_imag,
                                  float* scratch, int64_t scratch_floats, float* out, McaDecodePartials* partials, void* stream);
int mca_decode_out_proj_partials(const McaDecodePartials* partials, const void* wo, int weights_bf16, int dim, float* x_inout, void* stream);
