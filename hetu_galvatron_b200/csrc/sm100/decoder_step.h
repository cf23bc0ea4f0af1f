// Arguments of hg_decoder_step (decoder_step.cu), mirrored by ``DecoderStep`` in ops/_lib.py.  x and out are [S * B, H]
// contiguous (S tokens of B sequences, S * B <= 128); the caches point at the first of the B sequences, position 0, and `past`
// positions of them are filled.
#pragma once

struct HgDecoderStep {
  int S, B, H, nh, ng, hd, F, past;
  int rms, act, rot_dim, interleaved;      // act: kind of hg_glu_fwd; rot_dim 0: no rotation
  float eps, scale;
  const void *w_norm1, *b_norm1, *w_qkv, *b_qkv, *w_proj, *b_proj;
  const void *w_norm2, *b_norm2, *w_fc1, *b_fc1, *w_fc2, *b_fc2;
  const void *cos_t, *sin_t;
  void *k_cache, *v_cache;
  long long k_ss, k_sb, v_ss, v_sb;
  const void* x;
  void* out;
  void* ws;
  long long ws_bytes;
  int launches;                            // set by hg_decoder_step: kernels that it has launched
};
