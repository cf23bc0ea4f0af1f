// RMSNorm / LayerNorm forward and backward with the residual add fused in.
// Memory-bound: every element is read once with 16-byte accesses and kept in registers
// between the statistics pass and the normalisation pass.
// Replaces the flash-attn RMSNorm / DropoutAddLayerNorm extension calls of
// galvatron/core/runtime/transformer/norm.py:6-29.
#include "entry_points.h"
#include "sm100_common.cuh"

namespace {

constexpr int kThreads = 256;
// per-thread 8-element chunks kept in registers: MAXV = 2 / 4 / 8 covers H <= 4096 / 8192 / 16384

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (threadIdx.x < kThreads / 32) ? red[threadIdx.x] : 0.f;
  if (w == 0) {
    t = warp_sum(t);
    if (l == 0) red[0] = t;
  }
  __syncthreads();
  return red[0];
}

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

// y = norm(x + residual) * w (+ b);  h_out = x + residual (optional);  stats: rstd (and mean for LN).
template <bool RMS, int kMaxVec>
__global__ void __launch_bounds__(kThreads)
norm_fwd_kernel(const hg_lp_t* __restrict__ x, const hg_lp_t* __restrict__ residual,
                const hg_lp_t* __restrict__ w, const hg_lp_t* __restrict__ b,
                hg_lp_t* __restrict__ y, hg_lp_t* __restrict__ h_out, float* __restrict__ rstd_out,
                float* __restrict__ mean_out, int rows, int H, float eps) {
  __shared__ float red[kThreads / 32];
  hg::chain_release();
  const int zero = hg::chain_wait();
  x += zero;
  residual += zero;
  w += zero;
  b += zero;
  const int nvec = H >> 3;
  // The next row's loads are issued before this row's reductions, so that a block always has a row in flight
  // across its __syncthreads (with one row per trip the memory system idles while the block reduces).
  uint4 xraw[kMaxVec], rraw[kMaxVec];
  auto fetch = [&](int row) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + size_t(row) * H);
    const uint4* rr = residual ? reinterpret_cast<const uint4*>(residual + size_t(row) * H) : nullptr;
#pragma unroll
    for (int i = 0; i < kMaxVec; ++i) {
      const int c = threadIdx.x + i * kThreads;
      if (c < nvec) {
        xraw[i] = xr[c];
        if (rr) rraw[i] = rr[c];
      }
    }
  };
  constexpr bool kPrefetch = kMaxVec <= 4;    // the widest rows keep too much in registers to hold a second row
  if (kPrefetch && int(blockIdx.x) < rows) fetch(blockIdx.x);
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    if (!kPrefetch) fetch(row);
    float v[kMaxVec][8];
    float s = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < kMaxVec; ++i) {
      const int c = threadIdx.x + i * kThreads;
      if (c < nvec) {
        unpack8(xraw[i], v[i]);
        if (residual) {
          float r[8];
          unpack8(rraw[i], r);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] += r[j];
          if (h_out) {
            // round the sum to bf16 so that the saved residual stream and the normalised value agree
            uint4 packed = pack8(v[i]);
            reinterpret_cast<uint4*>(h_out + size_t(row) * H)[c] = packed;
            unpack8(packed, v[i]);
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) { s += v[i][j]; s2 += v[i][j] * v[i][j]; }
      }
    }
    if (kPrefetch && row + int(gridDim.x) < rows) fetch(row + gridDim.x);
    float mean = 0.f, var;
    if (RMS) {
      var = block_sum(s2, red) / H;
    } else {
      mean = block_sum(s, red) / H;
      float d2 = 0.f;
#pragma unroll
      for (int i = 0; i < kMaxVec; ++i) {
        const int c = threadIdx.x + i * kThreads;
        if (c < nvec) {
#pragma unroll
          for (int j = 0; j < 8; ++j) { float d = v[i][j] - mean; d2 += d * d; }
        }
      }
      var = block_sum(d2, red) / H;
    }
    const float rstd = rsqrtf(var + eps);
    if (threadIdx.x == 0) {
      rstd_out[row] = rstd;
      if (!RMS && mean_out) mean_out[row] = mean;
    }
    uint4* yr = reinterpret_cast<uint4*>(y + size_t(row) * H);
#pragma unroll
    for (int i = 0; i < kMaxVec; ++i) {
      const int c = threadIdx.x + i * kThreads;
      if (c < nvec) {
        float wv[8], o[8];
        unpack8(reinterpret_cast<const uint4*>(w)[c], wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (v[i][j] - mean) * rstd * wv[j];
        if (!RMS && b) {
          float bv[8];
          unpack8(reinterpret_cast<const uint4*>(b)[c], bv);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += bv[j];
        }
        yr[c] = pack8(o);
      }
    }
  }
}

// Backward.  dx = rstd * (dy*w - xhat*mean(dy*w*xhat) [- mean(dy*w)]) (+ dres);  partial dw/db per CTA (fp32).
//
// A row belongs to a group of TPR threads with VPT 16-byte chunks each (TPR * VPT >= H / 8), and a CTA of kBwdThreads
// threads holds kBwdThreads / TPR groups that walk the rows on their own: a group meets once per row (one barrier of
// its own warps, the partial sums double-buffered by row parity), never with its neighbours, so that a CTA always has
// rows in different phases and loads in flight.  One chunk per thread for H <= 4096 keeps the weight-gradient
// accumulators, the weights and the prefetched next row within 64 registers, i.e. 1024 threads per SM.  Bound by
// memory for wide rows, by the latency of a row's barrier for narrow ones.  Measured with the reduction of the partials
// (before: 256 threads per row whatever its width, three barriers per reduction): RMSNorm 8192 x 4096 73 -> 61 us (268 MB),
// 8192 x 8192 159 -> 125 us, 1531 x 3584 28 -> 16 us; LayerNorm 2997 x 1600 72 -> 25 us.
constexpr int kBwdThreads = 512;

template <int TPR>
__device__ __forceinline__ void group_sync(int group) {
  if (TPR == 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(TPR) : "memory");
}

// sums of (a, b) over the TPR threads of a group; `red` holds two floats per warp of the CTA
template <int TPR, bool TWO>
__device__ __forceinline__ void group_sum2(float& a, float& b, float2* red, int group) {
  a = warp_sum(a);
  if (TWO) b = warp_sum(b);
  if (TPR == 32) return;
  constexpr int W = TPR / 32;
  const int first = group * W;
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_float2(a, b);
  group_sync<TPR>(group);
  float sa = 0.f, sb = 0.f;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    const float2 v = red[first + i];
    sa += v.x;
    if (TWO) sb += v.y;
  }
  a = sa;
  b = sb;
}

template <bool RMS, int TPR, int VPT>
__global__ void __launch_bounds__(kBwdThreads, VPT == 1 ? 2 : 1)
norm_bwd_kernel(const hg_lp_t* __restrict__ dy, const hg_lp_t* __restrict__ h,
                const hg_lp_t* __restrict__ w, const float* __restrict__ rstd_in,
                const float* __restrict__ mean_in, const hg_lp_t* __restrict__ dres,
                hg_lp_t* __restrict__ dx, float* __restrict__ dw_partial, float* __restrict__ db_partial,
                int rows, int H) {
  constexpr int G = kBwdThreads / TPR;
  hg::chain_release();
  const int zero = hg::chain_wait();
  dy += zero;
  h += zero;
  w += zero;
  rstd_in += zero;
  mean_in += zero;
  dres += dres ? zero : 0;
  __shared__ float2 red[2][kBwdThreads / 32];
  extern __shared__ __align__(16) float comb[];                      // G > 1: [G - 1][H] accumulators of the other groups
  const int group = threadIdx.x / TPR, t = threadIdx.x - group * TPR;
  const int nvec = H >> 3;
  const float inv_h = 1.f / float(H);
  float dw_acc[VPT][8], db_acc[RMS ? 1 : VPT][8];
  uint4 wraw[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = t + i * TPR;
    wraw[i] = c < nvec ? reinterpret_cast<const uint4*>(w)[c] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dw_acc[i][j] = 0.f;
      if (!RMS) db_acc[i][j] = 0.f;
    }
  }
  uint4 dyraw[VPT], hraw[VPT], drraw[VPT];
  float rstd = 0.f, mean = 0.f;
  auto fetch = [&](int row) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = t + i * TPR;
      if (c < nvec) {
        dyraw[i] = __ldcs(reinterpret_cast<const uint4*>(dy + size_t(row) * H) + c);
        hraw[i] = __ldcs(reinterpret_cast<const uint4*>(h + size_t(row) * H) + c);
        if (dres) drraw[i] = __ldcs(reinterpret_cast<const uint4*>(dres + size_t(row) * H) + c);
      } else {
        dyraw[i] = hraw[i] = make_uint4(0, 0, 0, 0);
      }
    }
    rstd = rstd_in[row];
    if (!RMS) mean = mean_in[row];
  };
  constexpr bool kPrefetch = VPT <= 2;                 // the widest rows have no registers left for a second one
  const int step = gridDim.x * G;
  int row = blockIdx.x * G + group;
  if (kPrefetch && row < rows) fetch(row);
  for (int parity = 0; row < rows; row += step, parity ^= 1) {
    if (!kPrefetch) fetch(row);
    uint4 dyc[VPT], hc[VPT], drc[VPT];
    const float rs = rstd, mu = mean;
#pragma unroll
    for (int i = 0; i < VPT; ++i) { dyc[i] = dyraw[i]; hc[i] = hraw[i]; drc[i] = drraw[i]; }
    if (kPrefetch && row + step < rows) fetch(row + step);   // in flight across this row's reduction
    float c1 = 0.f, c2 = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      float d[8], hv[8], wv[8];
      unpack8(dyc[i], d);
      unpack8(hc[i], hv);
      unpack8(wraw[i], wv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = (hv[j] - mu) * rs, g = d[j] * wv[j];
        dw_acc[i][j] += d[j] * xh;
        if (!RMS) db_acc[i][j] += d[j];
        c1 += g * xh;
        if (!RMS) c2 += g;
      }
    }
    group_sum2<TPR, !RMS>(c1, c2, red[parity], group);
    c1 *= inv_h;
    c2 *= inv_h;
    uint4* dxr = reinterpret_cast<uint4*>(dx + size_t(row) * H);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = t + i * TPR;
      if (c < nvec) {
        float d[8], hv[8], wv[8], o[8];
        unpack8(dyc[i], d);
        unpack8(hc[i], hv);
        unpack8(wraw[i], wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = (hv[j] - mu) * rs;
          o[j] = rs * (d[j] * wv[j] - xh * c1 - (RMS ? 0.f : c2));
        }
        if (dres) {
          float r[8];
          unpack8(drc[i], r);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += r[j];
        }
        dxr[c] = pack8(o);
      }
    }
  }
  // the groups' accumulators, added in group order by group 0
  auto combine = [&](float (&acc)[VPT][8], float* out) {
    if (G > 1) {
      __syncthreads();
      if (group > 0) {
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
          const int c = t + i * TPR;
          if (c < nvec) {
            float4* dst = reinterpret_cast<float4*>(comb + size_t(group - 1) * H + c * 8);
            dst[0] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            dst[1] = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
          }
        }
      }
      __syncthreads();
    }
    if (group == 0) {
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int c = t + i * TPR;
        if (c < nvec) {
          for (int k = 0; k + 1 < G; ++k) {
            const float4* src = reinterpret_cast<const float4*>(comb + size_t(k) * H + c * 8);
            const float4 a = src[0], b = src[1];
            acc[i][0] += a.x; acc[i][1] += a.y; acc[i][2] += a.z; acc[i][3] += a.w;
            acc[i][4] += b.x; acc[i][5] += b.y; acc[i][6] += b.z; acc[i][7] += b.w;
          }
          float* dst = out + size_t(blockIdx.x) * H + c * 8;   // caller's scratch: no alignment is asked of it
#pragma unroll
          for (int j = 0; j < 8; ++j) dst[j] = acc[i][j];
        }
      }
    }
  };
  combine(dw_acc, dw_partial);
  if constexpr (!RMS) {
    if (db_partial) combine(db_acc, db_partial);
  }
}

// out[c] (+)= sum_p partial[p, c], parts taken in a fixed order.  A CTA owns 32 columns and its 16 warps share the
// parts; one thread per column with all parts in one chain left most of the chip idle for the whole sum.
__global__ void __launch_bounds__(512)
reduce_partials_kernel(const float* __restrict__ partial, float* __restrict__ out, const float* __restrict__ partial_b,
                       float* __restrict__ out_b, int parts, int H, int accumulate) {
  hg::chain_release();
  const int zero = hg::chain_wait();
  partial += zero;
  out += zero;
  partial_b += zero;
  out_b += zero;
  if (blockIdx.y == 1) {                     // a LayerNorm's bias, in the same launch
    partial = partial_b;
    out = out_b;
  }
  __shared__ float red[16][32];
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < H) {
#pragma unroll 8
    for (int p = wy; p < parts; p += 16) s += partial[size_t(p) * H + c];
  }
  red[wy][lane] = s;
  __syncthreads();
  if (wy == 0 && c < H) {
#pragma unroll
    for (int k = 1; k < 16; ++k) s += red[k][lane];
    out[c] = accumulate ? out[c] + s : s;
  }
}

// Launches the backward and the reduction of its partials.  TPR and VPT: the fewest threads per row that hold it.
template <bool RMS, int TPR, int VPT>
int launch_norm_bwd(const void* dy, const void* h, const void* w, const void* rstd, const void* mean, const void* dres,
                    void* dx, void* dw, void* db, float* P, float* PB, int parts, int rows, int H, int accumulate,
                    cudaStream_t st) {
  constexpr int G = kBwdThreads / TPR;
  const int want = (rows + G - 1) / G;
  const int grid = want < parts ? want : parts;
  const size_t smem = size_t(G - 1) * H * sizeof(float);
  static_assert(size_t(G - 1) * TPR * VPT * 8 * sizeof(float) <= 48 * 1024, "fits without an opt-in");
  int rc = hg_host::launch_over(norm_bwd_kernel<RMS, TPR, VPT>, grid, kBwdThreads, smem, st, (const hg_lp_t*)dy, (const hg_lp_t*)h,
                           (const hg_lp_t*)w, (const float*)rstd, (const float*)mean, (const hg_lp_t*)dres, (hg_lp_t*)dx, P,
                           RMS ? nullptr : PB, rows, H);
  const int cols = (H + 31) / 32;
  if (rc == 0)
    rc = hg_host::launch_over(reduce_partials_kernel, dim3(cols, !RMS && db ? 2 : 1), 512, 0, st, P, (float*)dw, PB, (float*)db, grid, H,
                              accumulate);
  return rc;
}

template <bool RMS, typename... A>
int dispatch_norm_bwd(int H, A... a) {
  if (H <= 256) return launch_norm_bwd<RMS, 32, 1>(a...);
  if (H <= 512) return launch_norm_bwd<RMS, 64, 1>(a...);
  if (H <= 1024) return launch_norm_bwd<RMS, 128, 1>(a...);
  if (H <= 2048) return launch_norm_bwd<RMS, 256, 1>(a...);
  if (H <= 4096) return launch_norm_bwd<RMS, 512, 1>(a...);
  if (H <= 8192) return launch_norm_bwd<RMS, 512, 2>(a...);
  return launch_norm_bwd<RMS, 512, 4>(a...);
}

}  // namespace

extern "C" {

// rms != 0 -> RMSNorm, else LayerNorm.  H must be a multiple of 8 and <= 16384.
int hg_norm_fwd(const void* x, const void* residual, const void* w, const void* b, void* y, void* h_out,
                void* rstd, void* mean, int rows, int H, float eps, int rms, void* stream) {
  if (rows <= 0) return 0;
  if ((H & 7) || H > kThreads * 8 * 8) return -1;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int grid = rows < 148 * 8 ? rows : 148 * 8;
  auto X = reinterpret_cast<const hg_lp_t*>(x);
  auto R = reinterpret_cast<const hg_lp_t*>(residual);
  auto W = reinterpret_cast<const hg_lp_t*>(w);
  auto B = reinterpret_cast<const hg_lp_t*>(b);
  auto Y = reinterpret_cast<hg_lp_t*>(y);
  auto Ho = reinterpret_cast<hg_lp_t*>(h_out);
#define HG_FWD(R_, V_) return hg_host::launch_over(norm_fwd_kernel<R_, V_>, grid, kThreads, 0, st, X, R, W, B, Y, Ho, (float*)rstd, (float*)mean, rows, H, eps)
  if (rms) { if (H <= 4096) HG_FWD(true, 2); else if (H <= 8192) HG_FWD(true, 4); else HG_FWD(true, 8); }
  else     { if (H <= 4096) HG_FWD(false, 2); else if (H <= 8192) HG_FWD(false, 4); else HG_FWD(false, 8); }
#undef HG_FWD
}

// `h` is the tensor that was normalised (x + residual).  `partial` is scratch of parts*H floats
// (and another parts*H for LayerNorm's bias gradient); dw/db are fp32 and are accumulated into when
// `accumulate` != 0.  Returns the number of partial rows used through *parts_used when non-null.
int hg_norm_bwd(const void* dy, const void* h, const void* w, const void* rstd, const void* mean, const void* dres,
                void* dx, void* dw, void* db, void* partial, int parts, int rows, int H, int rms, int accumulate,
                void* stream) {
  if (rows <= 0) return 0;
  if ((H & 7) || H > kThreads * 8 * 8 || parts <= 0) return -1;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  float* P = reinterpret_cast<float*>(partial);
  float* PB = P + size_t(parts) * H;
  return rms ? dispatch_norm_bwd<true>(H, dy, h, w, rstd, mean, dres, dx, dw, db, P, PB, parts, rows, H, accumulate, st)
             : dispatch_norm_bwd<false>(H, dy, h, w, rstd, mean, dres, dx, dw, db, P, PB, parts, rows, H, accumulate, st);
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------
// Allocation-free variant of the norm backward (declared and documented in norm_noalloc.h)
// ---------------------------------------------------------------------------------------------------
#include "norm_noalloc.h"

#include <mutex>

namespace {

constexpr int kNoAllocMaxDevices = HG_NORM_NOALLOC_MAX_DEVICES;
constexpr size_t kNoAllocFloats = size_t(2) * HG_NORM_NOALLOC_PARTS * HG_NORM_NOALLOC_MAX_H;

// Per-CTA partial sums: rows [0, PARTS) for the weight gradient, rows [PARTS, 2*PARTS) for LayerNorm's bias
// gradient, each row H floats wide (H <= MAX_H).  One copy per device, shared by every call on that device.
static __device__ __align__(256) float g_norm_bwd_scratch[kNoAllocFloats];

float* g_scratch_addr[kNoAllocMaxDevices] = {};
std::mutex g_scratch_mu;

// Device address of the array on the current device.  In host code the array's name is only a handle for the
// runtime, not a device pointer, so the address is asked for once per device and cached.
int noalloc_scratch(float** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return -(1000 + int(e));
  if (dev < 0 || dev >= kNoAllocMaxDevices) return HG_NORM_NOALLOC_BAD_DEVICE;
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (g_scratch_addr[dev] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_norm_bwd_scratch);
    if (e != cudaSuccess || p == nullptr) return -(1000 + int(e));
    g_scratch_addr[dev] = p;
  }
  *out = g_scratch_addr[dev];
  return 0;
}

}  // namespace

extern "C" int hg_norm_bwd_noalloc(const void* dy, const void* h, const void* w, const void* rstd, const void* mean,
                                   const void* dres, void* dx, void* dw, void* db, int rows, int H, int rms,
                                   int accumulate, void* stream) {
  if (rows <= 0) return 0;
  if ((H & 7) || H <= 0) return -1;
  if (H > HG_NORM_NOALLOC_MAX_H) return HG_NORM_NOALLOC_TOO_WIDE;
  // a null required pointer would be dereferenced on the device: refuse before anything is launched
  if (!dy || !h || !w || !rstd || !dx || !dw || (!rms && !mean)) return HG_NORM_NOALLOC_NULL_ARG;
  float* P = nullptr;
  if (int rc = noalloc_scratch(&P)) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int parts = HG_NORM_NOALLOC_PARTS;
  float* PB = P + size_t(parts) * HG_NORM_NOALLOC_MAX_H;
  return rms ? dispatch_norm_bwd<true>(H, dy, h, w, rstd, mean, dres, dx, dw, db, P, PB, parts, rows, H, accumulate, st)
             : dispatch_norm_bwd<false>(H, dy, h, w, rstd, mean, dres, dx, dw, db, P, PB, parts, rows, H, accumulate, st);
}
