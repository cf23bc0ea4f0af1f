// One dense decoder layer of a cached forward (a decode step, or a short prompt), launched by a single native call:
//
//   n = norm(x);  qkv = n Wqkv^T;  rotate, append to the cache, attend;  a = ctx Wproj^T
//   h = x + a;  out = h + act(norm(h) W1^T) W2^T
//
// The kernels are the ones the layer's modules launch one by one: ten, or eleven where the keys of cached attention are
// spread over several ranges (flash_decode.cu).  A decode step of a 7B-sized layer keeps the GPU busy for about 110 us;
// launched through the tensor library and the autograd wrappers it takes the host several times that.  Four 4096-wide
// layers, 4 sequences at 1000 cached positions, embedding and head included: 1400 us a step when each is waited for, 770 us
// from here; one after another 590 us, of which 517 us were kernels.  They are launched as a chain (sm100_common.cuh): each
// may start while the one before it ends, and the products read their first weights meanwhile; the same step as a CUDA graph
// 519 us without and 477 with, 466 with the keys streamed (flash_decode.cu) and their first copies made before the wait, 498
// one after another.  Host code only.
#include "decoder_step.h"
#include "entry_points.h"
#include "sm100_common.cuh"

namespace {

struct Buffers {
  char *norm, *qkv, *ctx, *attn, *h, *fc1, *act, *mlp, *rstd, *mean, *lse, *part;
  long long bytes, part_floats;
};

HgAttnTensor packed(const HgDecoderStep& d, void* base, int qpg, bool query) {
  const long long P = (long long)(d.nh + 2 * d.ng) * d.hd;
  return {base, d.B * P, P, d.nh + 2 * d.ng, qpg + 2, query ? 1 : 0, query ? 0 : qpg};
}

// Carves the scratch; every buffer starts on a 256-byte boundary.
Buffers carve(const HgDecoderStep& d, char* base) {
  Buffers b{};
  long long at = 0;
  auto take = [&](long long bytes) {
    char* p = base + at;
    at += (bytes + 255) / 256 * 256;
    return p;
  };
  const long long T = (long long)d.S * d.B, lp = sizeof(hg_lp_t);
  const int qpg = d.nh / d.ng;
  b.norm = take(T * d.H * lp);
  b.qkv = take(T * (d.nh + 2 * d.ng) * d.hd * lp);
  b.ctx = take(T * d.nh * d.hd * lp);
  b.attn = take(T * d.H * lp);
  b.h = take(T * d.H * lp);
  b.fc1 = take(T * d.F * (d.act == 2 ? 1 : 2) * lp);
  b.act = take(T * d.F * lp);
  b.mlp = take(T * d.H * lp);
  b.rstd = take(T * 4);
  b.mean = take(T * 4);
  b.lse = take(T * d.nh * 4);
  const HgAttnTensor q = packed(d, b.qkv, qpg, true), k{d.k_cache, d.k_ss, d.k_sb, d.ng, 1, 0, 0},
                     v{d.v_cache, d.v_ss, d.v_sb, d.ng, 1, 0, 0};
  b.part_floats = hg_flash_decode_pays(d.S, d.past + d.S, d.B, d.nh, d.ng, d.hd, 1, d.past, 0)
                      ? hg_flash_decode_scratch(&q, &k, &v, d.S, d.past + d.S, d.B, d.nh, d.ng, d.hd, 1, d.past, 0) : -1;
  b.part = take(b.part_floats > 0 ? b.part_floats * 4 : 0);
  b.bytes = at;
  return b;
}

bool valid(const HgDecoderStep& d) {
  return d.S > 0 && d.B > 0 && (long long)d.S * d.B <= 128 && d.H > 0 && d.ng > 0 && d.nh > 0 && d.nh % d.ng == 0 &&
         d.F > 0 && d.past >= 0 && d.act >= 0 && d.act <= 2 && (d.hd == 64 || d.hd == 128);
}

}  // namespace

extern "C" {

// Bytes of scratch (256-byte aligned) that hg_decoder_step needs, or -1 for a layer it does not take.
long long hg_decoder_step_scratch(const HgDecoderStep* d) {
  if (!valid(*d)) return -1;
  char dummy alignas(256)[1];
  return carve(*d, dummy).bytes;
}

int hg_decoder_step(HgDecoderStep* dp, void* stream) {
  const HgDecoderStep& d = *dp;
  if (!valid(d)) return -1;
  const Buffers b = carve(d, static_cast<char*>(d.ws));
  if (b.bytes > d.ws_bytes) return -1;
  const int T = d.S * d.B, qpg = d.nh / d.ng, P = (d.nh + 2 * d.ng) * d.hd, C = d.nh * d.hd;
  const int F1 = d.F * (d.act == 2 ? 1 : 2);
  void* mean = d.rms ? nullptr : b.mean;
  int rc;
  hg_host::Chain chain;
  if ((rc = hg_norm_fwd(d.x, nullptr, d.w_norm1, d.b_norm1, b.norm, nullptr, b.rstd, mean, T, d.H, d.eps, d.rms, stream))) return rc;
  if ((rc = hg_gemm_skinny_bf16(b.norm, d.w_qkv, b.qkv, d.b_qkv, T, P, d.H, d.H, d.H, P, 0, 0, 0, stream))) return rc;
  const size_t lp = sizeof(hg_lp_t);
  if ((rc = hg_rope_append(b.qkv, T, d.B, d.ng, qpg, d.hd, d.past, d.cos_t, d.sin_t, d.rot_dim, d.interleaved,
                           static_cast<char*>(d.k_cache) + size_t(d.past) * d.k_ss * lp,
                           static_cast<char*>(d.v_cache) + size_t(d.past) * d.v_ss * lp, d.k_ss, d.k_sb, d.v_ss, d.v_sb,
                           stream))) return rc;
  const HgAttnTensor q = packed(d, b.qkv, qpg, true), k{d.k_cache, d.k_ss, d.k_sb, d.ng, 1, 0, 0},
                     v{d.v_cache, d.v_ss, d.v_sb, d.ng, 1, 0, 0}, o{b.ctx, (long long)d.B * C, C, d.nh, qpg, 1, 0};
  if (b.part_floats >= 0)
    rc = hg_flash_decode(&q, &k, &v, &o, b.lse, b.part, d.S, d.past + d.S, d.B, d.nh, d.ng, d.hd, 1, d.past, 0, d.scale, stream);
  else if (hg_flash_stream_takes(&q, &k, &v, d.S, d.past + d.S, d.B, d.nh, d.ng, d.hd, 1, d.past, 0))
    rc = hg_flash_stream(&q, &k, &v, &o, b.lse, d.S, d.past + d.S, d.B, d.nh, d.ng, d.hd, 1, d.past, 0, d.scale, d.past, stream);
  else
    rc = hg_flash_fwd(&q, &k, &v, &o, b.lse, d.S, d.past + d.S, d.B, d.nh, d.ng, d.hd, 1, d.past, 0, d.scale, stream);
  if (rc) return rc;
  if ((rc = hg_gemm_skinny_bf16(b.ctx, d.w_proj, b.attn, d.b_proj, T, d.H, C, C, C, d.H, 0, 0, 0, stream))) return rc;
  if ((rc = hg_norm_fwd(b.attn, d.x, d.w_norm2, d.b_norm2, b.norm, b.h, b.rstd, mean, T, d.H, d.eps, d.rms, stream))) return rc;
  if ((rc = hg_gemm_skinny_bf16(b.norm, d.w_fc1, b.fc1, d.b_fc1, T, F1, d.H, d.H, d.H, F1, 0, 0, 0, stream))) return rc;
  if ((rc = hg_glu_fwd(b.fc1, b.act, T, d.F, d.act, stream))) return rc;
  if ((rc = hg_gemm_skinny_bf16(b.act, d.w_fc2, b.mlp, d.b_fc2, T, d.H, d.F, d.F, d.F, d.H, 0, 0, 0, stream))) return rc;
  dp->launches = b.part_floats > 0 ? 11 : 10;   // two for attention whose keys are spread over several ranges, else one
  return hg_add_bf16(b.h, b.mlp, d.out, (long long)T * d.H, stream);
}

}  // extern "C"
