// C entry points that other translation units call.  The files that define them include this header too, so that a
// changed parameter list does not compile where it would link.
#pragma once

#include "attn_tensor.h"

extern "C" {

int hg_norm_fwd(const void* x, const void* residual, const void* w, const void* b, void* y, void* h_out, void* rstd,
                void* mean, int rows, int H, float eps, int rms, void* stream);
int hg_gemm_skinny_bf16(const void* x, const void* W, void* C, const void* bias, int M, int N, int K, int ldx, int ldw,
                        int ldc, int w_mn, int out_mode, int splits, void* stream);
int hg_rope_append(void* qkv, int tokens, int batch, int ng, int qpg, int hd, int pos_offset, const void* cos_t,
                   const void* sin_t, int rot_dim, int interleaved, void* kc, void* vc, long long k_ss, long long k_sb,
                   long long v_ss, long long v_sb, void* stream);
long long hg_flash_decode_scratch(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, int Sq, int Skv, int B,
                                  int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0);
int hg_flash_decode_pays(int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0);
int hg_flash_decode(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, const HgAttnTensor* o, void* lse,
                    void* ws, int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0,
                    float scale, void* stream);
int hg_flash_stream_takes(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, int Sq, int Skv, int B,
                          int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0);
int hg_flash_stream(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, const HgAttnTensor* o, void* lse,
                    int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0, float scale,
                    int settled, void* stream);
int hg_flash_fwd(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, const HgAttnTensor* o, void* lse,
                 int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0, float scale,
                 void* stream);
int hg_glu_fwd(const void* y, void* out, long long rows, int F, int kind, void* stream);
int hg_add_bf16(const void* a, const void* b, void* out, long long n, void* stream);

}  // extern "C"
