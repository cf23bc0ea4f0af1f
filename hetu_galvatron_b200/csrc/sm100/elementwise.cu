// Memory-bound element-wise kernels: RoPE (in place on the packed QKV projection), SwiGLU / GeGLU /
// GELU forward and backward, embedding gather and its scatter-add gradient, bf16<->fp32 casts.
// Oracles: galvatron/core/runtime/transformer/rope_utils.py:86-120 (rotate-half form),
// galvatron/core/runtime/transformer/fused_kernels.py:19-48,142-168 (activations),
// galvatron/core/runtime/tensor_parallel/layers.py:120-147 (masked vocab-parallel lookup).
#include "entry_points.h"
#include "sm100_common.cuh"

namespace {

__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const hg_lp2_t* p = reinterpret_cast<const hg_lp2_t*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = hg_lp22ff(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 u;
  u.x = hg::pack_bf16(f[0], f[1]);
  u.y = hg::pack_bf16(f[2], f[3]);
  u.z = hg::pack_bf16(f[4], f[5]);
  u.w = hg::pack_bf16(f[6], f[7]);
  return u;
}

// A grid-stride walk over (row, col) pairs of a [rows, width] index space without a division per step: the
// stride is split into whole rows and a remainder once per thread, then every step is an add and a carry.
// (A 64-bit divide per 16-byte access costs more issue slots than the access leaves room for at HBM speed.)
struct RowColWalk {
  int64_t row;
  int col;
  int64_t d_row;
  int d_col;
  int width;
  __device__ __forceinline__ RowColWalk(int width_) : width(width_) {
    const int64_t first = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    row = first / width;
    col = int(first - row * width);
    d_row = stride / width;
    d_col = int(stride - d_row * width);
  }
  __device__ __forceinline__ void next() {
    row += d_row;
    col += d_col;
    if (col >= width) {
      col -= width;
      ++row;
    }
  }
};

// ---------------------------------------------------------------------------------------------
// RoPE, rotate-half (non-interleaved) form, applied in place to `nheads` heads that sit at
// column offsets slot[h] * slot_width (elements) of every token row of a [tokens, row_pitch] buffer.
//   out[i]        = x[i]*cos[i] - x[i+half]*sin[i]
//   out[i+half]   = x[i+half]*cos[i] + x[i]*sin[i]       (sign of sin flipped for the backward)
// Token t has position pos[t] when `pos` is given, else (t / batch) + pos_offset ([S,B] order).
// cos/sin tables are fp32 [max_pos, half].
// ---------------------------------------------------------------------------------------------
__global__ void rope_kernel(hg_lp_t* __restrict__ buf, const int* __restrict__ slot, int slot_width, int nheads,
                            int row_pitch, int tokens, int batch, const int* __restrict__ pos, int pos_offset,
                            const float* __restrict__ cos_t, const float* __restrict__ sin_t, int half, float sign) {
  hg::chain_release();
  const int zero = hg::chain_wait();
  buf += zero;
  slot += zero;
  cos_t += zero;
  sin_t += zero;
  if (pos != nullptr) pos += zero;
  const int vec_per_head = half >> 3;  // uint4 chunks in one half
  const int per_token = nheads * vec_per_head;
  for (RowColWalk w(per_token); w.row < tokens; w.next()) {
    const int t = int(w.row);
    const int h = w.col / vec_per_head, c = w.col - h * vec_per_head;
    const int p = pos ? pos[t] : (t / batch + pos_offset);
    hg_lp_t* base = buf + size_t(t) * row_pitch + slot[h] * slot_width + c * 8;
    float a[8], b[8], cs[8], sn[8];
    unpack8(*reinterpret_cast<const uint4*>(base), a);
    unpack8(*reinterpret_cast<const uint4*>(base + half), b);
    const float4* cp = reinterpret_cast<const float4*>(cos_t + size_t(p) * half + c * 8);
    const float4* sp = reinterpret_cast<const float4*>(sin_t + size_t(p) * half + c * 8);
    *reinterpret_cast<float4*>(cs) = cp[0];
    *reinterpret_cast<float4*>(cs + 4) = cp[1];
    *reinterpret_cast<float4*>(sn) = sp[0];
    *reinterpret_cast<float4*>(sn + 4) = sp[1];
    float oa[8], ob[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = sn[j] * sign;
      oa[j] = a[j] * cs[j] - b[j] * s;
      ob[j] = b[j] * cs[j] + a[j] * s;
    }
    *reinterpret_cast<uint4*>(base) = pack8(oa);
    *reinterpret_cast<uint4*>(base + half) = pack8(ob);
  }
}

// RoPE, interleaved form: channel pairs (2i, 2i+1) rotate by angle i.
//   out[2i]   = x[2i]*cos[i] - x[2i+1]*sin[i]
//   out[2i+1] = x[2i+1]*cos[i] + x[2i]*sin[i]
// One thread takes 8 consecutive channels (4 pairs) of one head of one token.
__global__ void rope_interleaved_kernel(hg_lp_t* __restrict__ buf, const int* __restrict__ slot, int slot_width, int nheads,
                                        int row_pitch, int tokens, int batch, const int* __restrict__ pos,
                                        int pos_offset, const float* __restrict__ cos_t,
                                        const float* __restrict__ sin_t, int half, float sign) {
  hg::chain_release();
  const int zero = hg::chain_wait();
  buf += zero;
  slot += zero;
  cos_t += zero;
  sin_t += zero;
  if (pos != nullptr) pos += zero;
  const int vec_per_head = half >> 2;  // uint4 chunks over the 2*half rotated channels
  const int per_token = nheads * vec_per_head;
  for (RowColWalk w(per_token); w.row < tokens; w.next()) {
    const int t = int(w.row);
    const int h = w.col / vec_per_head, c = w.col - h * vec_per_head;
    const int p = pos ? pos[t] : (t / batch + pos_offset);
    hg_lp_t* base = buf + size_t(t) * row_pitch + slot[h] * slot_width + c * 8;
    float x[8], o[8];
    unpack8(*reinterpret_cast<const uint4*>(base), x);
    const float4 cs = *reinterpret_cast<const float4*>(cos_t + size_t(p) * half + c * 4);
    const float4 sn = *reinterpret_cast<const float4*>(sin_t + size_t(p) * half + c * 4);
    const float cv[4] = {cs.x, cs.y, cs.z, cs.w}, sv[4] = {sn.x * sign, sn.y * sign, sn.z * sign, sn.w * sign};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o[2 * j] = x[2 * j] * cv[j] - x[2 * j + 1] * sv[j];
      o[2 * j + 1] = x[2 * j + 1] * cv[j] + x[2 * j] * sv[j];
    }
    *reinterpret_cast<uint4*>(base) = pack8(o);
  }
}

// ---------------------------------------------------------------------------------------------
// Cached attention: RoPE on the new tokens of a packed projection [tokens, ng * (qpg + 2) * hd] (per kv head: qpg query
// heads, the key head, the value head).  Queries are rotated in place; rotated keys and the values go straight into
// their rows of the cache, so that a decode step makes one launch where rotating, splitting and copying made seven.
// An item is 8 channels of one slot of one token (with the 8 they rotate with in the rotate-half form); half = 0: no
// rotation.  Cache element (s, b, g, d) at base + s * c_ss + b * c_sb + g * hd + d, s and b counted from the new tokens.
// ---------------------------------------------------------------------------------------------
__global__ void rope_append_kernel(hg_lp_t* __restrict__ qkv, int tokens, int batch, int ng, int qpg, int hd,
                                   int pos_offset, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                   int half, int interleaved, hg_lp_t* __restrict__ kc, hg_lp_t* __restrict__ vc,
                                   int64_t k_ss, int64_t k_sb, int64_t v_ss, int64_t v_sb) {
  hg::chain_release();
  const int zero = hg::chain_wait();
  qkv += zero;
  cos_t += zero;
  sin_t += zero;
  kc += zero;
  vc += zero;
  const int vph = hd >> 3, slots = ng * (qpg + 2);
  for (RowColWalk w(slots * vph); w.row < tokens; w.next()) {
    const int t = int(w.row), slot = w.col / vph, c = w.col - slot * vph;
    const int g = slot / (qpg + 2), j = slot - g * (qpg + 2);
    const int s = t / batch, b = t - s * batch;
    hg_lp_t* in = qkv + int64_t(t) * slots * hd + int64_t(slot) * hd + c * 8;
    hg_lp_t* out = j < qpg ? in : j == qpg ? kc + s * k_ss + b * k_sb + g * hd + c * 8
                                           : vc + s * v_ss + b * v_sb + g * hd + c * 8;
    const float* ct = cos_t + int64_t(s + pos_offset) * half;
    const float* st = sin_t + int64_t(s + pos_offset) * half;
    const bool rotates = j <= qpg && c * 8 < 2 * half;
    if (!rotates) {
      if (j >= qpg) *reinterpret_cast<uint4*>(out) = *reinterpret_cast<const uint4*>(in);
    } else if (interleaved) {
      float x[8], o[8];
      unpack8(*reinterpret_cast<const uint4*>(in), x);
      const float4 cs = *reinterpret_cast<const float4*>(ct + c * 4), sn = *reinterpret_cast<const float4*>(st + c * 4);
      const float cv[4] = {cs.x, cs.y, cs.z, cs.w}, sv[4] = {sn.x, sn.y, sn.z, sn.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        o[2 * i] = x[2 * i] * cv[i] - x[2 * i + 1] * sv[i];
        o[2 * i + 1] = x[2 * i + 1] * cv[i] + x[2 * i] * sv[i];
      }
      *reinterpret_cast<uint4*>(out) = pack8(o);
    } else if (c * 8 < half) {                       // the item of channels half + 8c.. is covered here
      float a[8], bb[8], cs[8], sn[8], oa[8], ob[8];
      unpack8(*reinterpret_cast<const uint4*>(in), a);
      unpack8(*reinterpret_cast<const uint4*>(in + half), bb);
      *reinterpret_cast<float4*>(cs) = reinterpret_cast<const float4*>(ct + c * 8)[0];
      *reinterpret_cast<float4*>(cs + 4) = reinterpret_cast<const float4*>(ct + c * 8)[1];
      *reinterpret_cast<float4*>(sn) = reinterpret_cast<const float4*>(st + c * 8)[0];
      *reinterpret_cast<float4*>(sn + 4) = reinterpret_cast<const float4*>(st + c * 8)[1];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        oa[i] = a[i] * cs[i] - bb[i] * sn[i];
        ob[i] = bb[i] * cs[i] + a[i] * sn[i];
      }
      *reinterpret_cast<uint4*>(out) = pack8(oa);
      *reinterpret_cast<uint4*>(out + half) = pack8(ob);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Gated activations on y = [y1 | y2] (each F wide, row pitch 2F):  out = act(y1) * y2
//   kind 0: SwiGLU (silu), kind 1: GeGLU (tanh GELU).  Non-gated kind 2, gelu_kernel: out = gelu_tanh(y) (pitch F).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float silu(float x) { return __fdividef(x, 1.f + __expf(-x)); }
// 0.5 (1 + tanh u) = 1 / (1 + exp(-2u)): one exponential and one reciprocal, and no cancellation where the result is small.
// With tanhf() these kernels were bound by its instructions: 2997 x 6400 forward 26.6 us, backward 32.8; 21.5
// and 27.6 with this alone, 18.4 and 24.6 with four groups a thread (gelu_kernel).
__device__ __forceinline__ float gelu_gate(float x) {
  return __fdividef(1.f, 1.f + __expf(-1.59576912f * x * (1.f + 0.044715f * x * x)));
}
__device__ __forceinline__ float gelu_tanh(float x) { return x * gelu_gate(x); }
__device__ __forceinline__ float gelu_tanh_grad(float x) {
  const float s = gelu_gate(x), s2 = s + s;       // x 2 s (1 - s) (...): the bracket overflows where it did with tanhf(), at 5.6e19
  return x * (s2 - s2 * s) * (0.79788456f + 0.1070322243f * x * x) + s;
}

template <int KIND>
__global__ void glu_fwd_kernel(const hg_lp_t* __restrict__ y, hg_lp_t* __restrict__ out, int64_t rows,
                               int F) {
  hg::chain_release();
  y += hg::chain_wait();
  for (RowColWalk w(F >> 3); w.row < rows; w.next()) {
    const int64_t r = w.row;
    const int c = w.col;
    float a[8], b[8], o[8];
    unpack8(reinterpret_cast<const uint4*>(y + r * 2 * F)[c], a);
    unpack8(reinterpret_cast<const uint4*>(y + r * 2 * F + F)[c], b);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = (KIND == 0 ? silu(a[j]) : gelu_tanh(a[j])) * b[j];
    reinterpret_cast<uint4*>(out + r * F)[c] = pack8(o);
  }
}

template <int KIND>
__global__ void glu_bwd_kernel(const hg_lp_t* __restrict__ g, const hg_lp_t* __restrict__ y,
                               hg_lp_t* __restrict__ dy, int64_t rows, int F) {
  hg::chain_release();
  const int zero = hg::chain_wait();
  g += zero;
  y += zero;
  for (RowColWalk w(F >> 3); w.row < rows; w.next()) {
    const int64_t r = w.row;
    const int c = w.col;
    float gv[8], a[8], b[8], d1[8], d2[8];
    unpack8(reinterpret_cast<const uint4*>(g + r * F)[c], gv);
    unpack8(reinterpret_cast<const uint4*>(y + r * 2 * F)[c], a);
    unpack8(reinterpret_cast<const uint4*>(y + r * 2 * F + F)[c], b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (KIND == 0) {
        const float s = __fdividef(1.f, 1.f + __expf(-a[j]));
        d1[j] = gv[j] * s * (1.f + a[j] * (1.f - s)) * b[j];
        d2[j] = gv[j] * a[j] * s;
      } else {
        d1[j] = gv[j] * gelu_tanh_grad(a[j]) * b[j];
        d2[j] = gv[j] * gelu_tanh(a[j]);
      }
    }
    reinterpret_cast<uint4*>(dy + r * 2 * F)[c] = pack8(d1);
    reinterpret_cast<uint4*>(dy + r * 2 * F + F)[c] = pack8(d2);
  }
}

// out = gelu(y) (BWD: g * gelu'(y)) over n groups of eight.  One stream in and one out: a thread takes U groups, all loads
// before the first use, which a gated kernel's two or three streams have without it.
template <bool BWD, int U>
__global__ void __launch_bounds__(256)
gelu_kernel(const hg_lp_t* __restrict__ y, const hg_lp_t* __restrict__ g, hg_lp_t* __restrict__ out, int64_t n) {
  hg::chain_release();
  const int zero = hg::chain_wait();
  y += zero;
  g += zero;
  const int64_t first = blockIdx.x * int64_t(256 * U) + threadIdx.x;
  uint4 v[U], w[U];
#pragma unroll
  for (int k = 0; k < U; ++k)
    if (first + k * 256 < n) {
      v[k] = reinterpret_cast<const uint4*>(y)[first + k * 256];
      if (BWD) w[k] = reinterpret_cast<const uint4*>(g)[first + k * 256];
    }
#pragma unroll
  for (int k = 0; k < U; ++k)
    if (first + k * 256 < n) {
      float a[8], b[8];
      unpack8(v[k], a);
      if (BWD) unpack8(w[k], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = BWD ? b[j] * gelu_tanh_grad(a[j]) : gelu_tanh(a[j]);
      reinterpret_cast<uint4*>(out)[first + k * 256] = pack8(a);
    }
}

// ---------------------------------------------------------------------------------------------
// Embedding: out[t,:] = (v0 <= id < v1) ? W[id - v0,:] : 0   (+ pos_emb[t / batch,:] optional)
// Gradient: dW[id - v0,:] += dout[t,:] (fp32 atomics)
// ---------------------------------------------------------------------------------------------
__global__ void embedding_fwd_kernel(const int64_t* __restrict__ ids, const hg_lp_t* __restrict__ W,
                                     const hg_lp_t* __restrict__ pos_emb, hg_lp_t* __restrict__ out,
                                     int tokens, int H, int v0, int v1, int batch, int pos_offset) {
  for (RowColWalk w(H >> 3); w.row < tokens; w.next()) {
    const int t = int(w.row), c = w.col;
    const int64_t id = ids[t];
    uint4 v = make_uint4(0, 0, 0, 0);
    if (id >= v0 && id < v1) v = reinterpret_cast<const uint4*>(W + size_t(id - v0) * H)[c];
    if (pos_emb) {
      float a[8], b[8];
      unpack8(v, a);
      unpack8(reinterpret_cast<const uint4*>(pos_emb + size_t(t / batch + pos_offset) * H)[c], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += b[j];
      v = pack8(a);
    }
    reinterpret_cast<uint4*>(out + size_t(t) * H)[c] = v;
  }
}

// Adds eight gradients to eight consecutive fp32 words.  What bounds the scatter is the number of reductions the L2
// executes, not the bytes: two 16-byte reductions do the work of eight 4-byte ones (8192 tokens x 4096, token
// frequencies as in text: 191 us with 4-byte reductions, 59 us).
template <bool VEC>
__device__ __forceinline__ void add8(float* dst, const float (&g)[8]) {
  if (VEC) {
    atomicAdd(reinterpret_cast<float4*>(dst), make_float4(g[0], g[1], g[2], g[3]));
    atomicAdd(reinterpret_cast<float4*>(dst) + 1, make_float4(g[4], g[5], g[6], g[7]));
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) atomicAdd(dst + j, g[j]);
  }
}

// VEC: dW and dpos are 16-byte aligned (their rows then are, too: H is a multiple of 8)
template <bool VEC>
__global__ void embedding_bwd_kernel(const int64_t* __restrict__ ids, const hg_lp_t* __restrict__ dout,
                                     float* __restrict__ dW, float* __restrict__ dpos, int tokens, int H, int v0,
                                     int v1, int batch, int pos_offset) {
  for (RowColWalk w(H >> 3); w.row < tokens; w.next()) {
    const int t = int(w.row), c = w.col;
    const int64_t id = ids[t];
    float g[8];
    unpack8(reinterpret_cast<const uint4*>(dout + size_t(t) * H)[c], g);
    if (id >= v0 && id < v1) add8<VEC>(dW + size_t(id - v0) * H + c * 8, g);
    if (dpos) add8<VEC>(dpos + size_t(t / batch + pos_offset) * H + c * 8, g);
  }
}

// The same gradient with the tokens of a row of dW brought together, for up to kSortTokens tokens: what bounds the scatter above is
// its reductions in L2, and in text more than half of them meet a row that another token of the batch has as well.  One block sorts
// (row, token) in shared memory by a bitonic network (8192 keys 68 us in 91 passes) while the others clear dW.  A block of the
// second kernel then adds the tokens of kRunTokens neighbouring keys in registers and leaves one row of sums per run, as plain stores
// where the run is all of its row's tokens.  8192 tokens x 4096 of 32000 rows, frequencies as in text, us: cleared 72 and scattered 59,
// 114 so; 8200 x 3584 of 152064 354, 322.
constexpr int kSortTokens = 16384, kSortIndexBits = 14, kRunTokens = 8, kClearVecs = 8192;
constexpr unsigned kNoRow = 0xffffffffu;
static_assert(1 << kSortIndexBits == kSortTokens, "an index of a key");

__global__ void __launch_bounds__(1024)
embedding_sort_kernel(const int64_t* __restrict__ ids, unsigned* __restrict__ keys, int tokens, int v0, int v1, float4* __restrict__ dW,
                      int64_t n4) {
  extern __shared__ unsigned k[];
  if (blockIdx.x > 0) {
    const int64_t at = int64_t(blockIdx.x - 1) * kClearVecs + threadIdx.x;
#pragma unroll
    for (int i = 0; i < kClearVecs; i += 1024)
      if (at + i < n4) dW[at + i] = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  int n = 1;
  while (n < tokens) n <<= 1;
  for (int i = threadIdx.x; i < n; i += 1024) {
    const int64_t id = i < tokens ? ids[i] : -1;
    k[i] = id >= v0 && id < v1 && i < tokens ? unsigned(id - v0) << kSortIndexBits | unsigned(i) : kNoRow;
  }
  for (int width = 2; width <= n; width <<= 1)
    for (int d = width >> 1; d > 0; d >>= 1) {
      __syncthreads();
      for (int p = threadIdx.x; p < n >> 1; p += 1024) {
        const int lo = 2 * (p & ~(d - 1)) + (p & (d - 1)), hi = lo + d;
        const unsigned a = k[lo], b = k[hi];
        if ((a > b) == ((lo & width) == 0)) {
          k[lo] = b;
          k[hi] = a;
        }
      }
    }
  __syncthreads();
  for (int i = threadIdx.x; i < tokens; i += 1024) keys[i] = k[i];
}

__global__ void __launch_bounds__(256)
embedding_run_kernel(const unsigned* __restrict__ keys, const hg_lp_t* __restrict__ dout, float* __restrict__ dW, int tokens, int H) {
  const int c = blockIdx.y * 256 + threadIdx.x, first = blockIdx.x * kRunTokens;
  if (c >= H >> 3) return;
  unsigned key[kRunTokens + 2];                     // with a neighbour on either side
#pragma unroll
  for (int i = 0; i < kRunTokens + 2; ++i) {
    const int at = first + i - 1;
    key[i] = at >= 0 && at < tokens ? keys[at] : kNoRow;
  }
  uint4 v[kRunTokens];
#pragma unroll
  for (int i = 0; i < kRunTokens; ++i)
    if (key[i + 1] != kNoRow) v[i] = reinterpret_cast<const uint4*>(dout + size_t(key[i + 1] & (kSortTokens - 1)) * H)[c];
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  bool whole = true;                                // the run starts in this block
#pragma unroll
  for (int i = 1; i <= kRunTokens; ++i) {
    if (key[i] == kNoRow) break;                    // sorted behind all others
    const unsigned row = key[i] >> kSortIndexBits;
    if (i == 1) whole = key[0] == kNoRow || key[0] >> kSortIndexBits != row;
    float g[8];
    unpack8(v[i - 1], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] += g[j];
    const bool goes_on = key[i + 1] != kNoRow && key[i + 1] >> kSortIndexBits == row;
    if (goes_on && i < kRunTokens) continue;
    float* dst = dW + size_t(row) * H + c * 8;
    if (whole && !goes_on) {
      reinterpret_cast<float4*>(dst)[0] = make_float4(s[0], s[1], s[2], s[3]);
      reinterpret_cast<float4*>(dst)[1] = make_float4(s[4], s[5], s[6], s[7]);
    } else {
      add8<true>(dst, s);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = 0.f;
    whole = true;
  }
}

// ---------------------------------------------------------------------------------------------
// Column sums of a 16-bit matrix (bias gradients): out[c] = sum_r x[r, c] in fp32, rounded once, or written or added to fp32.
// A CTA takes 256 columns (32 lanes of eight) and one of `parts` row ranges, its eight warps share the rows.
// x is read once with 16-byte loads and nothing is widened in memory; rows are added in a fixed order.  2997 x 6400 with
// the final sum: 11 us (38 MB; 50 us as a widening copy, a reduction and a cast).
// ---------------------------------------------------------------------------------------------
struct ColsumOut {
  hg_lp_t* lp;                    // 16 bits, or
  float* wide;                    // fp32
  int accumulate;
  __device__ __forceinline__ void put(int c, float t) const {
    if (lp != nullptr) lp[c] = hg_f2lp(t);
    else wide[c] = accumulate ? wide[c] + t : t;
  }
};

__global__ void __launch_bounds__(256)
colsum_kernel(const hg_lp_t* __restrict__ x, int64_t pitch, int rows, int cols, float* __restrict__ partial, const ColsumOut out) {
  hg::chain_release();
  const int zero = hg::chain_wait();
  x += zero;
  __shared__ float red[8][256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c0 = blockIdx.x * 256 + lane * 8;
  const int r0 = int(int64_t(rows) * blockIdx.y / gridDim.y), r1 = int(int64_t(rows) * (blockIdx.y + 1) / gridDim.y);
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (c0 + 8 <= cols) {
    const hg_lp_t* p = x + c0;
    int r = r0 + warp;
    for (; r + 24 < r1; r += 32) {                     // four rows in flight per warp
      uint4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = __ldcs(reinterpret_cast<const uint4*>(p + int64_t(r + 8 * k) * pitch));
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float f[8];
        unpack8(v[k], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] += f[j];
      }
    }
    for (; r < r1; r += 8) {
      float f[8];
      unpack8(*reinterpret_cast<const uint4*>(p + int64_t(r) * pitch), f);
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] += f[j];
    }
  } else {
    for (int r = r0 + warp; r < r1; r += 8)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (c0 + j < cols) s[j] += hg_lp2f(x[int64_t(r) * pitch + c0 + j]);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) red[warp][lane * 8 + j] = s[j];
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < cols) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += red[k][threadIdx.x];
    if (gridDim.y > 1) partial[int64_t(blockIdx.y) * cols + c] = t;
    else out.put(c, t);
  }
}

// 32 columns a CTA, its eight warps share the parts.
__global__ void __launch_bounds__(256)
colsum_final_kernel(const float* __restrict__ partial, int parts, int cols, const ColsumOut out) {
  hg::chain_release();
  const int zero = hg::chain_wait();
  partial += zero;
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float t = 0.f;
  if (c < cols) {
#pragma unroll 8
    for (int p = warp; p < parts; p += 8) t += partial[int64_t(p) * cols + c];
  }
  red[warp][lane] = t;
  __syncthreads();
  if (warp == 0 && c < cols) {
    t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += red[k][lane];
    out.put(c, t);
  }
}

// ---------------------------------------------------------------------------------------------
// Casts and the bf16 residual add
// ---------------------------------------------------------------------------------------------
__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ in, hg_lp_t* __restrict__ out, int64_t n) {
  const int64_t nv = n >> 3;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < nv; i += int64_t(gridDim.x) * blockDim.x) {
    const float4 a = reinterpret_cast<const float4*>(in)[2 * i], b = reinterpret_cast<const float4*>(in)[2 * i + 1];
    const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    reinterpret_cast<uint4*>(out)[i] = pack8(f);
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 7)) out[(nv << 3) + threadIdx.x] = hg_f2lp(in[(nv << 3) + threadIdx.x]);
}

__global__ void add_bf16_kernel(const hg_lp_t* __restrict__ a, const hg_lp_t* __restrict__ b,
                                hg_lp_t* __restrict__ out, int64_t n) {
  hg::chain_release();
  const int zero = hg::chain_wait();
  a += zero;
  b += zero;
  const int64_t nv = n >> 3;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < nv; i += int64_t(gridDim.x) * blockDim.x) {
    float x[8], y[8];
    unpack8(reinterpret_cast<const uint4*>(a)[i], x);
    unpack8(reinterpret_cast<const uint4*>(b)[i], y);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] += y[j];
    reinterpret_cast<uint4*>(out)[i] = pack8(x);
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 7)) {
    const int64_t k = (nv << 3) + threadIdx.x;
    out[k] = hg_f2lp(hg_lp2f(a[k]) + hg_lp2f(b[k]));
  }
}


// Log-sum-exp merge of two partial attention results over disjoint key sets (ring / context-parallel attention):
//   l = log(exp(lse_acc) + exp(lse_new));  out_acc = exp(lse_acc - l) * out_acc + exp(lse_new - l) * out_new;  lse_acc = l
// out_acc fp32 [S, B*h, d] contiguous, out_new bf16 same shape, lse_new fp32 [B*h, S] contiguous, lse_acc fp32 with
// row pitch `lse_pitch` (a slice of a longer sequence).  LPR = d / 8 lanes share a row; they all read the old lse
// before lane 0 replaces it.
template <int LPR>
__global__ void attn_merge_kernel(float* __restrict__ out_acc, float* __restrict__ lse_acc, long long lse_pitch,
                                  const hg_lp_t* __restrict__ out_new, const float* __restrict__ lse_new, int S,
                                  int BH) {
  const int64_t rows = int64_t(S) * BH;
  const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  const int64_t row = t / LPR;
  const int lane = int(t % LPR);
  const bool live = row < rows;
  float wa = 0.f, wb = 0.f, l = 0.f;
  float* lp = nullptr;
  if (live) {
    const int s = int(row / BH), bh = int(row % BH);
    lp = lse_acc + int64_t(bh) * lse_pitch + s;
    const float la = *lp, ln = lse_new[int64_t(bh) * S + s];
    const float m = fmaxf(la, ln);
    if (m == -INFINITY) {   // neither side has seen a key yet
      l = -INFINITY;
    } else {
      l = m + __logf(__expf(la - m) + __expf(ln - m));
      wa = __expf(la - l);
      wb = __expf(ln - l);
    }
    float4* acc = reinterpret_cast<float4*>(out_acc + (row * LPR + lane) * 8);
    float x[8];
    unpack8(reinterpret_cast<const uint4*>(out_new)[row * LPR + lane], x);
    float4 a0 = acc[0], a1 = acc[1];
    a0.x = wa * a0.x + wb * x[0]; a0.y = wa * a0.y + wb * x[1]; a0.z = wa * a0.z + wb * x[2]; a0.w = wa * a0.w + wb * x[3];
    a1.x = wa * a1.x + wb * x[4]; a1.y = wa * a1.y + wb * x[5]; a1.z = wa * a1.z + wb * x[6]; a1.w = wa * a1.w + wb * x[7];
    acc[0] = a0;
    acc[1] = a1;
  }
  __syncwarp();
  if (live && lane == 0) *lp = l;
}

inline int grid_for(int64_t work, int threads) {
  int64_t g = (work + threads - 1) / threads;
  const int64_t cap = 148 * 16;
  return int(g < 1 ? 1 : (g > cap ? cap : g));
}

// Four groups a thread once that still makes eight CTAs for each of 148 SMs.
template <bool BWD>
int launch_gelu(const void* y, const void* g, void* out, int64_t n, cudaStream_t st) {
  const bool four = n >= 148 * 8 * 1024;
  const int64_t per = four ? 1024 : 256, grid = (n + per - 1) / per;
  if (grid > 0x7fffffff) return -1;
  return hg_host::launch_over(four ? gelu_kernel<BWD, 4> : gelu_kernel<BWD, 1>, int(grid), 256, 0, st, (const hg_lp_t*)y,
                         (const hg_lp_t*)g, (hg_lp_t*)out, n);
}

}  // namespace

extern "C" {

int hg_rope(void* buf, const void* slots, int slot_width, int nheads, int row_pitch, int tokens, int batch, const void* pos,
            int pos_offset, const void* cos_t, const void* sin_t, int rot_dim, int flags, void* stream) {
  // flags: bit 0 = backward (rotate by the negative angle), bit 1 = interleaved channel pairs
  if (tokens <= 0 || nheads <= 0) return 0;
  const int half = rot_dim / 2;
  if ((half & 7) || (row_pitch & 7)) return -1;
  const float sign = (flags & 1) ? -1.f : 1.f;
  if (flags & 2) {
    const int64_t work = int64_t(tokens) * nheads * (half >> 2);
    return hg_host::launch_over(rope_interleaved_kernel, grid_for(work, 256), 256, 0, (cudaStream_t)stream, (hg_lp_t*)buf,
                           (const int*)slots, slot_width, nheads, row_pitch, tokens, batch, (const int*)pos, pos_offset,
                           (const float*)cos_t, (const float*)sin_t, half, sign);
  }
  const int64_t work = int64_t(tokens) * nheads * (half >> 3);
  return hg_host::launch_over(rope_kernel, grid_for(work, 256), 256, 0, (cudaStream_t)stream, (hg_lp_t*)buf, (const int*)slots,
                         slot_width, nheads, row_pitch, tokens, batch, (const int*)pos, pos_offset, (const float*)cos_t,
                         (const float*)sin_t, half, sign);
}

// See rope_append_kernel.  rot_dim = 0: no rotation (cos_t / sin_t unused).  Strides in elements, multiples of 8; all
// pointers 16-byte aligned.
int hg_rope_append(void* qkv, int tokens, int batch, int ng, int qpg, int hd, int pos_offset, const void* cos_t,
                   const void* sin_t, int rot_dim, int interleaved, void* kc, void* vc, long long k_ss, long long k_sb,
                   long long v_ss, long long v_sb, void* stream) {
  if (tokens <= 0) return 0;
  const int half = rot_dim / 2;
  if ((hd & 7) || (half & 7) || batch < 1 || ng < 1 || qpg < 1 || ((k_ss | k_sb | v_ss | v_sb) & 7)) return -1;
  if ((uintptr_t(qkv) | uintptr_t(kc) | uintptr_t(vc)) & 15) return -1;
  const int64_t work = int64_t(tokens) * ng * (qpg + 2) * (hd >> 3);
  return hg_host::launch_over(rope_append_kernel, grid_for(work, 256), 256, 0, (cudaStream_t)stream, (hg_lp_t*)qkv, tokens, batch,
                         ng, qpg, hd, pos_offset, (const float*)cos_t, (const float*)sin_t, half, interleaved, (hg_lp_t*)kc,
                         (hg_lp_t*)vc, k_ss, k_sb, v_ss, v_sb);
}

int hg_glu_fwd(const void* y, void* out, long long rows, int F, int kind, void* stream) {
  if (rows <= 0) return 0;
  if (F & 7) return -1;
  const int g = grid_for(rows * (F >> 3), 256);
  cudaStream_t st = (cudaStream_t)stream;
  if (kind == 2) return launch_gelu<false>(y, nullptr, out, rows * (F >> 3), st);
  return hg_host::launch_over(kind == 0 ? glu_fwd_kernel<0> : glu_fwd_kernel<1>, g, 256, 0, st, (const hg_lp_t*)y, (hg_lp_t*)out, rows, F);
}

int hg_glu_bwd(const void* g_, const void* y, void* dy, long long rows, int F, int kind, void* stream) {
  if (rows <= 0) return 0;
  if (F & 7) return -1;
  const int g = grid_for(rows * (F >> 3), 256);
  cudaStream_t st = (cudaStream_t)stream;
  auto G = (const hg_lp_t*)g_;
  if (kind == 2) return launch_gelu<true>(y, g_, dy, rows * (F >> 3), st);
  return hg_host::launch_over(kind == 0 ? glu_bwd_kernel<0> : glu_bwd_kernel<1>, g, 256, 0, st, G, (const hg_lp_t*)y, (hg_lp_t*)dy, rows,
                         F);
}

int hg_embedding_fwd(const void* ids, const void* W, const void* pos_emb, void* out, int tokens, int H, int v0, int v1,
                     int batch, int pos_offset, void* stream) {
  if (tokens <= 0) return 0;
  if (H & 7) return -1;
  embedding_fwd_kernel<<<grid_for(int64_t(tokens) * (H >> 3), 256), 256, 0, (cudaStream_t)stream>>>(
      (const int64_t*)ids, (const hg_lp_t*)W, (const hg_lp_t*)pos_emb, (hg_lp_t*)out, tokens, H, v0,
      v1, batch, pos_offset);
  return int(cudaGetLastError());
}

int hg_embedding_bwd(const void* ids, const void* dout, void* dW, void* dpos, int tokens, int H, int v0, int v1,
                     int batch, int pos_offset, void* stream) {
  if (tokens <= 0) return 0;
  if (H & 7) return -1;
  const int g = grid_for(int64_t(tokens) * (H >> 3), 256);
  if (((uintptr_t(dW) | uintptr_t(dpos)) & 15) == 0)
    embedding_bwd_kernel<true><<<g, 256, 0, (cudaStream_t)stream>>>(
        (const int64_t*)ids, (const hg_lp_t*)dout, (float*)dW, (float*)dpos, tokens, H, v0, v1, batch, pos_offset);
  else
    embedding_bwd_kernel<false><<<g, 256, 0, (cudaStream_t)stream>>>(
        (const int64_t*)ids, (const hg_lp_t*)dout, (float*)dW, (float*)dpos, tokens, H, v0, v1, batch, pos_offset);
  return int(cudaGetLastError());
}

static bool runs_can(const void* dW, int tokens, int H, int rows) {
  return tokens > 0 && tokens <= kSortTokens && H > 0 && H % 8 == 0 && rows > 0 && rows <= (int)(kNoRow >> kSortIndexBits) &&
         (uintptr_t(dW) & 15) == 0;
}
// Whether it pays to bring the tokens together, for a table that holds nothing.  Into one that does, where the sort has nothing to
// hide behind, 8192 tokens take 85 us and 54 scattered.
// The table is cleared at 7.3 TB/s.  The sort is of the next power of two: log2 n (log2 n + 1) / 2 passes of 0.25 us and 0.06 ns a key
// (8192 keys 68 us, 16384 131), a little longer beside the clearing.  Sums of runs instead of a scatter save about 1 ps per element
// of the gradient; clearing in this kernel and the second one cost up to 1 us and a fortieth.  us, cleared and scattered / so: 8192 tokens
// of 24576 rows x 4096 115 / 106, of 32000 132 / 114; 8193 of 32000 140 / 159 (not taken), of 58479 186 / 182; 4097 of 24327 86 / 91 (not
// taken), of 39532 118 / 107; 4096 of 152064 x 3584 318 / 309, of 50304 x 1600 60 / 54, of 50304 x 768 34 / 40 (not taken); 1024 of 3072
// x 4096 20 / 22 (not taken), of 16000 46 / 45, of 128256 288 / 290 (not taken); 256 of 8521 24 / 26 (not taken).
int hg_embedding_bwd_runs_takes(const void* dW, int tokens, int H, int rows) {
  if (!runs_can(dW, tokens, H, rows)) return 0;
  long long n = 1, log2n = 0;
  while (n < tokens) n <<= 1, ++log2n;
  const long long clear = (long long)rows * H / 1825, saved = (long long)tokens * H / 1024;        // ns
  const long long sort = log2n * (log2n + 1) / 2 * (250 + n / 16);
  return clear * 4 / 5 + saved >= sort * 9 / 10 && clear / 40 + 1000 <= saved;
}
// dW [rows, H] = the sums of the gradients of the tokens of rows v0 .. v0 + rows - 1.  keys: scratch of `tokens` words.
int hg_embedding_bwd_runs(const void* ids, const void* dout, void* dW, void* keys, int tokens, int H, int v0, int rows, void* stream) {
  if (!runs_can(dW, tokens, H, rows)) return -1;
  cudaStream_t st = (cudaStream_t)stream;
  int n = 1;
  while (n < tokens) n <<= 1;
  static const cudaError_t rc0 =
      cudaFuncSetAttribute(embedding_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSortTokens * int(sizeof(unsigned)));
  if (rc0 != cudaSuccess) return int(rc0);
  const int64_t n4 = int64_t(rows) * H / 4;
  embedding_sort_kernel<<<unsigned(1 + (n4 + kClearVecs - 1) / kClearVecs), 1024, n * sizeof(unsigned), st>>>(
      (const int64_t*)ids, (unsigned*)keys, tokens, v0, v0 + rows, (float4*)dW, n4);
  embedding_run_kernel<<<dim3((tokens + kRunTokens - 1) / kRunTokens, (H / 8 + 255) / 256), 256, 0, st>>>(
      (const unsigned*)keys, (const hg_lp_t*)dout, (float*)dW, tokens, H);
  return int(cudaGetLastError());
}

// Row ranges the column sums of a [rows, cols] matrix are cut into: about four CTAs per SM, each warp with at least
// four rows.  `partial` of hg_colsum_bf16 holds that many rows of `cols` floats.
int hg_colsum_parts(int rows, int cols) {
  const int blocks = (cols + 255) / 256;
  int parts = (148 * 4 + blocks - 1) / (blocks > 0 ? blocks : 1);
  if (parts > rows / 32) parts = rows / 32;
  return parts < 1 ? 1 : (parts > 64 ? 64 : parts);
}

// out[c] = sum over rows of x[r, c]; x 16-byte aligned, pitch a multiple of 8 elements.  out_lp: 16-bit result; null: out_f32, which
// is added to if `accumulate`.
int hg_colsum(const void* x, long long pitch, int rows, int cols, void* partial, int parts, void* out_lp, void* out_f32,
              int accumulate, void* stream) {
  if (cols <= 0) return 0;
  if ((pitch & 7) || (uintptr_t(x) & 15) || parts < 1 || parts > 65535 || (out_lp == nullptr) == (out_f32 == nullptr)) return -1;
  cudaStream_t st = (cudaStream_t)stream;
  const ColsumOut out{(hg_lp_t*)out_lp, (float*)out_f32, accumulate};
  int rc = hg_host::launch_over(colsum_kernel, dim3((cols + 255) / 256, parts), 256, 0, st, (const hg_lp_t*)x, int64_t(pitch), rows, cols,
                                (float*)partial, out);
  if (rc == 0 && parts > 1)
    rc = hg_host::launch_over(colsum_final_kernel, (cols + 31) / 32, 256, 0, st, (const float*)partial, parts, cols, out);
  return rc;
}
int hg_colsum_bf16(const void* x, long long pitch, int rows, int cols, void* partial, int parts, void* out, void* stream) {
  return hg_colsum(x, pitch, rows, cols, partial, parts, out, nullptr, 0, stream);
}

int hg_cast_f32_bf16(const void* in, void* out, long long n, void* stream) {
  if (n <= 0) return 0;
  cast_f32_to_bf16_kernel<<<grid_for(n >> 3, 256), 256, 0, (cudaStream_t)stream>>>((const float*)in,
                                                                                    (hg_lp_t*)out, n);
  return int(cudaGetLastError());
}

int hg_add_bf16(const void* a, const void* b, void* out, long long n, void* stream) {
  if (n <= 0) return 0;
  return hg_host::launch_over(add_bf16_kernel, grid_for(n >> 3, 256), 256, 0, (cudaStream_t)stream, (const hg_lp_t*)a,
                         (const hg_lp_t*)b, (hg_lp_t*)out, n);
}

// See attn_merge_kernel.  d must be 64 or 128; S * BH rows.
int hg_attn_merge(void* out_acc, void* lse_acc, long long lse_pitch, const void* out_new, const void* lse_new, int S,
                  int BH, int d, void* stream) {
  if (S <= 0 || BH <= 0) return 0;
  if (d != 64 && d != 128) return -1;
  const int lpr = d / 8;
  const int64_t threads = int64_t(S) * BH * lpr;
  const int grid = int((threads + 255) / 256);
  cudaStream_t st = (cudaStream_t)stream;
  if (lpr == 16)
    attn_merge_kernel<16><<<grid, 256, 0, st>>>((float*)out_acc, (float*)lse_acc, lse_pitch, (const hg_lp_t*)out_new,
                                                (const float*)lse_new, S, BH);
  else
    attn_merge_kernel<8><<<grid, 256, 0, st>>>((float*)out_acc, (float*)lse_acc, lse_pitch, (const hg_lp_t*)out_new,
                                               (const float*)lse_new, S, BH);
  return int(cudaGetLastError());
}

}  // extern "C"
