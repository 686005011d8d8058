// Internal alias: the kernels implement exactly the raw entry points of the public header.
#pragma once
#include "mycaffe_attn.h"

// Internal: turn the public (bits, bits_t, mask_mode) triple into the kernels' view; *view stays null for no mask.
struct McaMaskBits;
int mca_mask_bits_view(const uint32_t* bits, const uint32_t* bits_t, int mask_mode, int T, int need_transpose, McaMaskBits* out,
                       const McaMaskBits** view);

// Internal: mca_classify_causal_mask in one launch.  scratch: two device ints that are zero before the call and zero
// again after it (a mismatch count and a ticket; the last block to finish writes *flag, and host_base + flag to
// *host_flag in pinned host memory unless that is null).
int mca_classify_causal_mask_ws(const float* mask, int T, int* flag, int* host_flag, int host_base, int* scratch, void* stream);

// Internal: hand the current device's kernels the address of the process's failure words (McaFailWord).
int mca_set_fail_words_fwd(int* words);
int mca_set_fail_words_bwd(int* words);
int mca_set_fail_words_probe(int* words);
int mca_set_fail_words_decode(int* words);
int mca_set_fail_words_proj(int* words);
