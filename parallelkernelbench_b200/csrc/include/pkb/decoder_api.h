// C API of the native decoder layer (csrc/kernels/decoder.cu): one call issues all launches of a layer's forward or backward.
#pragma once
#include <stdint.h>

extern "C" {

typedef struct pkb_layer_desc {
  int32_t tokens, hidden, ffn, hq, hkv, head_dim;   // one sequence of `tokens` rows; head_dim 64 or 128
  float eps, scale;                                 // of the norms; of the attention scores
} pkb_layer_desc;

// Bytes of the buffers below.
int pkb_decoder_layer_sizes(const pkb_layer_desc* L, long long* saved, long long* fwd_scratch, long long* bwd_scratch);

// x, out: bf16 [tokens, hidden]; params: the flat bf16 parameters; cos_t / sin_t: bf16 [tokens, head_dim]; saved is written for
// the backward, scratch is free again when the call's launches have run.
int pkb_decoder_layer_fwd(const pkb_layer_desc* L, const void* x, const void* params, const void* cos_t, const void* sin_t, void* out,
                          void* saved, void* scratch, void* stream);

// dout -> dx (bf16 [tokens, hidden]) and dparams (bf16, laid out like params; nothing behind the last parameter is written).
int pkb_decoder_layer_bwd(const pkb_layer_desc* L, const void* x, const void* params, const void* cos_t, const void* sin_t,
                          const void* saved, const void* dout, void* dx, void* dparams, void* scratch, void* stream);
}
