// Token dispatch and weighted combine of a mixture-of-experts layer whose experts are all on this GPU.
//
//   plan      idx [n = T * k] (expert of every (token, slot) pair, negative = dropped)  ->
//             row_start [E + 1]  aligned segment starts of the experts,
//             dest [n]           row of the pair in the expert buffer (-1: dropped, -2: no such expert),
//             src [bound]        pair that fills a row of the buffer (-1: padding)
//   dispatch  buf[r] = x[src[r] / k] or 0                 backward: dx[t] = sum_j dbuf[dest[t, j]]
//   combine   out[t] = sum_j w[t, j] * y[dest[t, j]]      backward: dy[r] = w[src[r]] * dout[src[r] / k] or 0,
//                                                                   dw[t, j] = <dout[t], y[dest[t, j]]>
//
// Rows of an expert are in pair order (token-minor), so the result does not depend on timing; sums over a token's
// slots are taken in fp32 in slot order and rounded once.  Nothing is read back on the host: the buffer has the static
// bound of rows that any routing of n pairs can need.  All four row passes are bound by memory: every row is moved
// once, 16 bytes per access, where sorting, index_select / index_add and fp32 copies moved it several times.  4096
// tokens x 4096, 8 experts, top-2: forward and backward 120 us around the experts' products, 2.1 ms before (with 110
// launches and two host reads).
#include "sm100_common.cuh"

namespace {

constexpr int kPlanThreads = 1024;   // pairs per CTA of the plan kernels
constexpr int kMaxExperts = 256;
constexpr int kNoSuchExpert = -2;    // a number from E on is a mistake of the caller: its token's result is NaN

__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const hg_lp2_t* p = reinterpret_cast<const hg_lp2_t*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = hg_lp22ff(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(hg::pack_bf16(f[0], f[1]), hg::pack_bf16(f[2], f[3]), hg::pack_bf16(f[4], f[5]),
                    hg::pack_bf16(f[6], f[7]));
}

// counts[chunk, e] = pairs of the chunk routed to e; src[] = -1
__global__ void __launch_bounds__(kPlanThreads)
moe_count_kernel(const int64_t* __restrict__ idx, int n, int E, int* __restrict__ counts, int* __restrict__ src, int bound) {
  __shared__ int hist[kMaxExperts];
  for (int e = threadIdx.x; e < E; e += kPlanThreads) hist[e] = 0;
  __syncthreads();
  const int p = blockIdx.x * kPlanThreads + threadIdx.x;
  if (p < n) {
    const int64_t e = idx[p];
    if (e >= 0 && e < E) atomicAdd(&hist[e], 1);
  }
  for (int r = p; r < bound; r += gridDim.x * kPlanThreads) src[r] = -1;
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += kPlanThreads) counts[blockIdx.x * E + e] = hist[e];
}

// Every CTA derives the segment starts and its chunk's offsets from the counts of all chunks (a few KB from L2), then
// ranks its pairs: inside a warp by matching experts, between the warps of the chunk by a prefix over their counts.
__global__ void __launch_bounds__(kPlanThreads)
moe_place_kernel(const int64_t* __restrict__ idx, int n, int E, int align, const int* __restrict__ counts, int bound,
                 int* __restrict__ row_start, int* __restrict__ dest, int* __restrict__ src, int* status) {
  constexpr int kWarps = kPlanThreads / 32;
  __shared__ int padded[kMaxExperts];            // then: first row of this chunk's pairs of an expert
  __shared__ int warp_cnt[kWarps][kMaxExperts];  // then: rank of a warp's first pair of an expert
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int before = 0;
  if (threadIdx.x < E) {
    int total = 0;
    for (int c = 0; c < int(gridDim.x); ++c) {
      if (c == int(blockIdx.x)) before = total;
      total += counts[c * E + threadIdx.x];
    }
    padded[threadIdx.x] = (total + align - 1) / align * align;
  }
  for (int i = threadIdx.x; i < kWarps * E; i += kPlanThreads) warp_cnt[i / E][i % E] = 0;
  __syncthreads();
  int start = 0;
  if (threadIdx.x < E)
    for (int e = 0; e < int(threadIdx.x); ++e) start += padded[e];
  if (blockIdx.x == 0 && threadIdx.x < E) {
    row_start[threadIdx.x] = start;
    if (threadIdx.x == E - 1) row_start[E] = start + padded[E - 1];
  }
  const int p = blockIdx.x * kPlanThreads + threadIdx.x;
  int e = -1;
  if (p < n) {
    const int64_t v = idx[p];
    if (v >= 0 && v < E) e = int(v);
  }
  const unsigned same = __match_any_sync(0xffffffffu, e);
  const int rank = __popc(same & ((1u << lane) - 1));
  if (e >= 0 && rank == 0) warp_cnt[warp][e] = __popc(same);
  __syncthreads();                               // everybody has read `padded`, every warp has counted
  if (threadIdx.x < E) {
    padded[threadIdx.x] = start + before;
    int run = 0;
    for (int w = 0; w < kWarps; ++w) {
      const int c = warp_cnt[w][threadIdx.x];
      warp_cnt[w][threadIdx.x] = run;
      run += c;
    }
  }
  __syncthreads();
  if (p < n) {
    int row = idx[p] >= E ? kNoSuchExpert : -1;
    if (row == kNoSuchExpert) hg::set_status(status, hg::kBadArgument);
    if (e >= 0) {
      row = padded[e] + warp_cnt[warp][e] + rank;
      if (row < bound) src[row] = p;             // always, for the bound that the host computes
      else row = -1;
    }
    dest[p] = row;
  }
}

// buf[r] = w[src[r]] * x[src[r] / k] (w null: 1), zeros where src[r] < 0
__global__ void __launch_bounds__(256)
moe_scatter_kernel(const hg_lp_t* __restrict__ x, int64_t x_pitch, const int* __restrict__ src,
                   const float* __restrict__ w, int rows, int k, int vec, hg_lp_t* __restrict__ buf) {
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const int p = src[r];
    uint4* out = reinterpret_cast<uint4*>(buf + int64_t(r) * vec * 8);
    if (p < 0) {
      for (int c = threadIdx.x; c < vec; c += 256) out[c] = make_uint4(0, 0, 0, 0);
      continue;
    }
    const uint4* in = reinterpret_cast<const uint4*>(x + int64_t(p / k) * x_pitch);
    if (w == nullptr) {
      for (int c = threadIdx.x; c < vec; c += 256) out[c] = in[c];
    } else {
      const float s = w[p];
      for (int c = threadIdx.x; c < vec; c += 256) {
        float f[8];
        unpack8(in[c], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] *= s;
        out[c] = pack8(f);
      }
    }
  }
}

// out[t] = sum_j w[t, j] * y[dest[t, j]] (w null: 1), dropped pairs skipped, NaN where an expert does not exist
__global__ void __launch_bounds__(256)
moe_gather_kernel(const hg_lp_t* __restrict__ y, const int* __restrict__ dest, const float* __restrict__ w, int T, int k,
                  int vec, hg_lp_t* __restrict__ out) {
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    for (int c = threadIdx.x; c < vec; c += 256) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
      for (int j = 0; j < k; ++j) {
        const int r = dest[t * k + j];
        if (r < 0) {
          if (r == kNoSuchExpert)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] = NAN;
          continue;
        }
        const float s = w ? w[t * k + j] : 1.f;
        float f[8];
        unpack8(reinterpret_cast<const uint4*>(y + int64_t(r) * vec * 8)[c], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += s * f[i];
      }
      reinterpret_cast<uint4*>(out + int64_t(t) * vec * 8)[c] = pack8(acc);
    }
  }
}

// dw[p] = <dout[p / k], y[dest[p]]>, one warp per pair (0 for dropped pairs)
__global__ void __launch_bounds__(256)
moe_dot_kernel(const hg_lp_t* __restrict__ y, const hg_lp_t* __restrict__ dout, int64_t dout_pitch,
               const int* __restrict__ dest, int n, int k, int vec, float* __restrict__ dw) {
  const int p = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (p >= n) return;
  const int r = dest[p];
  float s = 0.f;
  if (r >= 0) {
    const uint4* a = reinterpret_cast<const uint4*>(y + int64_t(r) * vec * 8);
    const uint4* b = reinterpret_cast<const uint4*>(dout + int64_t(p / k) * dout_pitch);
#pragma unroll 4
    for (int c = lane; c < vec; c += 32) {
      float f[8], g[8];
      unpack8(a[c], f);
      unpack8(b[c], g);
#pragma unroll
      for (int i = 0; i < 8; ++i) s += f[i] * g[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  if (lane == 0) dw[p] = s;
}

// Rows outside [row_start[0], row_start[G]) set to zero.
__global__ void __launch_bounds__(256)
zero_outside_kernel(hg_lp_t* __restrict__ buf, const int* __restrict__ row_start, int G, int rows, int64_t vec) {
  const int first = min(max(row_start[0], 0), rows), last = min(max(row_start[G], first), rows);
  const int64_t head = int64_t(first) * vec, total = head + int64_t(rows - last) * vec;
  for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll)
    reinterpret_cast<uint4*>(buf)[i < head ? i : i - head + int64_t(last) * vec] = make_uint4(0, 0, 0, 0);
}

inline bool aligned16(const void* p) { return (uintptr_t(p) & 15) == 0; }
inline int row_grid(int rows) { return rows < 148 * 16 ? rows : 148 * 16; }

}  // namespace

extern "C" {

// `counts`: scratch of ceil(n / 1024) (at least 1) * E ints.  `bound` rows must hold every routing of n pairs:
// n + min(n, E) * (align - 1), rounded down to a multiple of align, is enough.
int hg_moe_plan(const void* idx, int n, int E, int align, int bound, void* counts, void* row_start, void* dest, void* src,
                void* stream) {
  if (n < 0 || E < 1 || E > kMaxExperts || align < 1 || bound < 0) return -1;
  const int chunks = n > 0 ? (n + kPlanThreads - 1) / kPlanThreads : 1;
  cudaStream_t st = (cudaStream_t)stream;
  moe_count_kernel<<<chunks, kPlanThreads, 0, st>>>((const int64_t*)idx, n, E, (int*)counts, (int*)src, bound);
  moe_place_kernel<<<chunks, kPlanThreads, 0, st>>>((const int64_t*)idx, n, E, align, (const int*)counts, bound,
                                                    (int*)row_start, (int*)dest, (int*)src, hg_host::status_ptr());
  return int(cudaGetLastError());
}

// H a multiple of 8, pointers 16-byte aligned, pitches multiples of 8 elements; w (fp32 [n]) may be null.
int hg_moe_scatter(const void* x, long long x_pitch, const void* src, const void* w, int rows, int k, int H, void* buf,
                   void* stream) {
  if (rows <= 0) return 0;
  if (k < 1 || (H & 7) || (x_pitch & 7) || !aligned16(x) || !aligned16(buf)) return -1;
  moe_scatter_kernel<<<row_grid(rows), 256, 0, (cudaStream_t)stream>>>((const hg_lp_t*)x, x_pitch, (const int*)src,
                                                                       (const float*)w, rows, k, H / 8, (hg_lp_t*)buf);
  return int(cudaGetLastError());
}

int hg_moe_gather(const void* y, const void* dest, const void* w, int T, int k, int H, void* out, void* stream) {
  if (T <= 0) return 0;
  if (k < 1 || (H & 7) || !aligned16(y) || !aligned16(out)) return -1;
  moe_gather_kernel<<<row_grid(T), 256, 0, (cudaStream_t)stream>>>((const hg_lp_t*)y, (const int*)dest, (const float*)w, T,
                                                                   k, H / 8, (hg_lp_t*)out);
  return int(cudaGetLastError());
}

int hg_moe_dot(const void* y, const void* dout, long long dout_pitch, const void* dest, int n, int k, int H, void* dw,
               void* stream) {
  if (n <= 0) return 0;
  if (k < 1 || (H & 7) || (dout_pitch & 7) || !aligned16(y) || !aligned16(dout)) return -1;
  moe_dot_kernel<<<(n + 7) / 8, 256, 0, (cudaStream_t)stream>>>((const hg_lp_t*)y, (const hg_lp_t*)dout, dout_pitch,
                                                                (const int*)dest, n, k, H / 8, (float*)dw);
  return int(cudaGetLastError());
}

// buf [rows, width] contiguous, width a multiple of 8: the rows that no segment of row_start (device int[G + 1],
// ascending) covers become zero.
int hg_zero_outside(void* buf, const void* row_start, int G, int rows, int width, void* stream) {
  if (rows <= 0 || width <= 0) return 0;
  if ((width & 7) || !aligned16(buf) || G < 0) return -1;
  zero_outside_kernel<<<148 * 4, 256, 0, (cudaStream_t)stream>>>((hg_lp_t*)buf, (const int*)row_start, G, rows, width / 8);
  return int(cudaGetLastError());
}

}  // extern "C"
