// Attention of a few queries over a long key / value cache (decode steps), forward only.
//
// The tile kernels of attention.cu give a CTA 128 query rows of one head: with one new token a CTA does 1 / 128 of the
// work it is built for, walks all keys of its head alone, and the query heads that share a kv head read its keys once
// each.  What bounds a decode step is reading K and V once, so here a CTA takes one kv head, CH keys and the (at most
// eight) query rows that attend to them; the key ranges of a sequence are spread over the chip and their partial
// results merged by a second small kernel (skipped when one range covers all keys).  Scores and probabilities stay in
// fp32 throughout.  A row that sees no key (its sum l is 0) is written as zeros; a NaN score or one of +inf makes l, and with
// it the row of O, NaN (LSE -inf), as on the tile kernels.
//
// Rows: r = s * qpg + j is query token s of query head g * qpg + j.  A lane holds eight channels, so HD / 8 lanes share a
// key and a warp reads 32 / (HD / 8) keys per 16-byte access.
#include "entry_points.h"
#include "sm100_common.cuh"

namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr int kMaxRows = 8;

struct DecodeParams {
  const hg_lp_t *Q, *K, *V;
  int64_t q_ss, q_sb, k_ss, k_sb, v_ss, v_sb, o_ss, o_sb;
  int q_gs, q_hs, q_off, k_gs, k_off, v_gs, v_off;    // slot of a head, see SlotMap in attention.cu
  hg_lp_t* O;
  float* LSE;               // [B, nheads, Sq]
  float* ws;                // partial results, (HD + 2) floats per (row, key range)
  int Sq, kv_len, B, nheads, nkv, qpg, causal, q_pos0, k_pos0;
  float scale;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const hg_lp2_t* p = reinterpret_cast<const hg_lp2_t*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = hg_lp22ff(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

template <int HD, int R, int CH>
__global__ void __launch_bounds__(128)
flash_decode_kernel(const DecodeParams p) {
  constexpr int LPK = HD / 8, KPW = 32 / LPK, STEPS = CH / (4 * KPW);
  __shared__ float sS[R][CH];
  __shared__ float sML[R][2];
  __shared__ float sAcc[4][R][HD];
  hg::chain_release();
  hg::chain_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / LPK, ch = (lane % LPK) * 8;
  const int g = blockIdx.x, b = blockIdx.y, key0 = blockIdx.z * CH, ranges = gridDim.z;
  const int rows = p.Sq * p.qpg;
  const hg_lp_t* kb = p.K + int64_t(b) * p.k_sb + int64_t(g * p.k_gs + p.k_off) * HD + ch;
  const hg_lp_t* vb = p.V + int64_t(b) * p.v_sb + int64_t(g * p.v_gs + p.v_off) * HD + ch;

  // With one or two rows there are registers for all of a thread's keys and values: both are requested before anything
  // is computed.
  constexpr bool kPreload = R <= 2;
  uint4 ku[kPreload ? STEPS : 1], vu[kPreload ? STEPS : 1];
  if constexpr (kPreload) {
#pragma unroll
    for (int it = 0; it < STEPS; ++it) {
      const int key = key0 + (it * 4 + warp) * KPW + sub;
      ku[it] = key < p.kv_len ? *reinterpret_cast<const uint4*>(kb + int64_t(key) * p.k_ss) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int it = 0; it < STEPS; ++it) {
      const int key = key0 + (it * 4 + warp) * KPW + sub;
      vu[it] = key < p.kv_len ? *reinterpret_cast<const uint4*>(vb + int64_t(key) * p.v_ss) : make_uint4(0, 0, 0, 0);
    }
  }
  {
    float q[R][8];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      uint4 u = make_uint4(0, 0, 0, 0);
      if (r < rows)
        u = *reinterpret_cast<const uint4*>(p.Q + int64_t(r / p.qpg) * p.q_ss + int64_t(b) * p.q_sb +
                                            int64_t(g * p.q_gs + (r % p.qpg) * p.q_hs + p.q_off) * HD + ch);
      unpack8(u, q[r]);
    }
#pragma unroll (kPreload ? STEPS : 4)
    for (int it = 0; it < STEPS; ++it) {
      const int kl = (it * 4 + warp) * KPW + sub, key = key0 + kl;
      uint4 u = make_uint4(0, 0, 0, 0);
      if constexpr (kPreload) u = ku[it];
      else if (key < p.kv_len) u = *reinterpret_cast<const uint4*>(kb + int64_t(key) * p.k_ss);
      float f[8];
      unpack8(u, f);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float d = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) d = fmaf(q[r][i], f[i], d);
#pragma unroll
        for (int o = LPK / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if (lane % LPK == 0) sS[r][kl] = d;
      }
    }
  }
  __syncthreads();
  for (int r = warp; r < R; r += 4) {
    const float sl2 = p.scale * kLog2e;
    const int q_pos = p.q_pos0 + r / p.qpg;
    float s[CH / 32], m = -INFINITY;
#pragma unroll
    for (int i = 0; i < CH / 32; ++i) {
      const int kl = i * 32 + lane, key = key0 + kl;
      const bool seen = r < rows && key < p.kv_len && (!p.causal || p.k_pos0 + key <= q_pos);
      s[i] = seen ? sS[r][kl] * sl2 : -INFINITY;
      m = fmaxf(m, s[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float ref = m == -INFINITY ? 0.f : m;
    float l = 0.f;
#pragma unroll
    for (int i = 0; i < CH / 32; ++i) {
      const float e = ex2(s[i] - ref);
      l += e;
      sS[r][i * 32 + lane] = e;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (lane == 0) {
      sML[r][0] = m;
      sML[r][1] = l;
    }
  }
  __syncthreads();
  float acc[R][8];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[r][i] = 0.f;
#pragma unroll (kPreload ? STEPS : 4)
  for (int it = 0; it < STEPS; ++it) {
    const int kl = (it * 4 + warp) * KPW + sub, key = key0 + kl;
    uint4 u = make_uint4(0, 0, 0, 0);
    if constexpr (kPreload) u = vu[it];
    else if (key < p.kv_len) u = *reinterpret_cast<const uint4*>(vb + int64_t(key) * p.v_ss);
    float f[8];
    unpack8(u, f);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float e = sS[r][kl];
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[r][i] = fmaf(e, f[i], acc[r][i]);
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int o = LPK; o < 32; o <<= 1) acc[r][i] += __shfl_xor_sync(0xffffffffu, acc[r][i], o);
      if (sub == 0) sAcc[warp][r][ch + i] = acc[r][i];
    }
  __syncthreads();
  for (int i = threadIdx.x; i < rows * HD; i += 128) {
    const int r = i / HD, c = i % HD;
    const float v = (sAcc[0][r][c] + sAcc[1][r][c]) + (sAcc[2][r][c] + sAcc[3][r][c]);
    const float m = sML[r][0], l = sML[r][1];
    if (ranges == 1) {
      const int h = g * p.qpg + r % p.qpg, s = r / p.qpg;
      p.O[int64_t(s) * p.o_ss + int64_t(b) * p.o_sb + int64_t(h) * HD + c] = hg_f2lp(l == 0.f ? 0.f : v / l);
      if (c == 0) p.LSE[(size_t(b) * p.nheads + h) * p.Sq + s] = l > 0.f ? (m + log2f(l)) * kLn2 : -INFINITY;
    } else {
      float* w = p.ws + ((int64_t(b) * p.nkv + g) * rows + r) * int64_t(ranges) * (HD + 2) + int64_t(blockIdx.z) * (HD + 2);
      w[c] = v;
      if (c == 0) {
        w[HD] = m;
        w[HD + 1] = l;
      }
    }
  }
}

// One CTA of HD threads per (sequence, kv head, row): the key ranges' partial results, merged in range order.
template <int HD>
__global__ void __launch_bounds__(HD)
flash_decode_merge_kernel(const DecodeParams p, int ranges) {
  hg::chain_release();
  hg::chain_wait();
  const int rows = p.Sq * p.qpg;
  const int r = blockIdx.x % rows, g = (blockIdx.x / rows) % p.nkv, b = blockIdx.x / rows / p.nkv, c = threadIdx.x;
  const float* w = p.ws + int64_t(blockIdx.x) * ranges * (HD + 2);
  float m = -INFINITY;
#pragma unroll 8
  for (int i = 0; i < ranges; ++i) m = fmaxf(m, w[int64_t(i) * (HD + 2) + HD]);
  const float ref = m == -INFINITY ? 0.f : m;
  float v = 0.f, l = 0.f;
#pragma unroll 8
  for (int i = 0; i < ranges; ++i) {
    const float* wi = w + int64_t(i) * (HD + 2);
    const float f = ex2(wi[HD] - ref);
    v = fmaf(f, wi[c], v);
    l = fmaf(f, wi[HD + 1], l);
  }
  const int h = g * p.qpg + r % p.qpg, s = r / p.qpg;
  p.O[int64_t(s) * p.o_ss + int64_t(b) * p.o_sb + int64_t(h) * HD + c] = hg_f2lp(l == 0.f ? 0.f : v / l);
  if (c == 0) p.LSE[(size_t(b) * p.nheads + h) * p.Sq + s] = l > 0.f ? (m + log2f(l)) * kLn2 : -INFINITY;
}

// ---------------------------------------------------------------------------------------------
// One query per head and kv head: a CTA streams the keys of a head, or a run of them, and nothing of it is kept but the running
// maximum, sum and context; the CTAs of a cluster share a head's keys and merge through distributed shared memory, so that
// there is one launch and no scratch.
//
// What bounds it is reading K and V.  A thread copies (cp.async) the 16 bytes of either that it reads itself, kDepth steps
// ahead, into slots of its own: no barrier inside the loop, 64 KB in flight per CTA, three CTAs per SM.  HD / 8 lanes share a
// key; eight warps take 2048 / HD keys a step.  Scores of kBatch steps are formed before one rescale, since the chain of
// shuffles and exponentials of a single key is longer than its bytes take.  In a chain the keys below `settled` are older than
// the chain: the first copies of those are made before the wait.
// ---------------------------------------------------------------------------------------------
constexpr int kDepth = 8, kBatch = 4, kStreamThreads = 256, kMaxCluster = 8;

__device__ __forceinline__ void copy16(void* dst, const void* src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(hg::smem_u32(dst)), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_rank(const float* mine, int rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(hg::smem_u32(mine)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
// What a partial result with maximum m counts beside one with maximum top >= m.
__device__ __forceinline__ float weight_of(float m, float top) { return ex2(m - (top == -INFINITY ? 0.f : top)); }

template <int HD>
struct StreamSmem {
  static constexpr int kRow = HD + 2;                                 // context, maximum, sum
  static constexpr int kRing = kDepth * 2 * kStreamThreads * 16;      // later the warps' results
  static constexpr int kTotal = kRing + kRow * 4;
  static_assert(8 * kRow * 4 <= kRing, "the warps' results reuse the ring");
};

template <int HD>
__global__ void __launch_bounds__(kStreamThreads, 3)
flash_stream_kernel(const DecodeParams p, int settled) {
  using L = StreamSmem<HD>;
  constexpr int LPK = HD / 8, KPW = 32 / LPK, KPS = 8 * KPW;
  extern __shared__ __align__(16) uint8_t smem[];
  uint4* ring = reinterpret_cast<uint4*>(smem);                       // [kDepth][K, V][thread]
  float* sums = reinterpret_cast<float*>(smem);                       // [warp][kRow]
  float* part = reinterpret_cast<float*>(smem + L::kRing);            // [kRow]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int sub = lane / LPK, ch = (lane % LPK) * 8;
  const int rank = blockIdx.x, splits = gridDim.x, g = blockIdx.y, b = blockIdx.z;
  const int steps = (p.kv_len + KPS - 1) / KPS;
  const int first = int((long long)steps * rank / splits), n = int((long long)steps * (rank + 1) / splits) - first;
  const hg_lp_t* kb = p.K + int64_t(b) * p.k_sb + int64_t(g * p.k_gs + p.k_off) * HD + ch;
  const hg_lp_t* vb = p.V + int64_t(b) * p.v_sb + int64_t(g * p.v_gs + p.v_off) * HD + ch;
  hg::chain_release();
  auto copy = [&](int it) {                                           // step `it` of this CTA, or an empty group
    if (it < n) {
      const int key = (first + it) * KPS + warp * KPW + sub;
      const bool on = key < p.kv_len;                                 // otherwise zeros
      const int64_t at = on ? key : 0;
      uint4* slot = ring + (it % kDepth) * 2 * kStreamThreads + tid;
      copy16(slot, kb + at * p.k_ss, on);
      copy16(slot + kStreamThreads, vb + at * p.v_ss, on);
    }
    copies_commit();
  };
  int ahead = 0;
  for (; ahead < kDepth && (first + ahead + 1) * KPS <= settled; ++ahead) copy(ahead);
  hg::chain_wait();
  for (; ahead < kDepth; ++ahead) copy(ahead);

  float q[8], acc[8], m = -INFINITY, l = 0.f;
  const float sl2 = p.scale * kLog2e;
  unpack8(*reinterpret_cast<const uint4*>(p.Q + int64_t(b) * p.q_sb + int64_t(g * p.q_gs + p.q_off) * HD + ch), q);
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  for (int it = 0; it < n; it += kBatch) {
    copies_wait<kDepth - kBatch>();
    float s[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const int key = (first + it + j) * KPS + warp * KPW + sub;
      float f[8], d = 0.f;
      unpack8(ring[((it + j) % kDepth) * 2 * kStreamThreads + tid], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) d = fmaf(q[i], f[i], d);
#pragma unroll
      for (int o = LPK / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      s[j] = it + j < n && key < p.kv_len ? d * sl2 : -INFINITY;
    }
    float top = m;
#pragma unroll
    for (int j = 0; j < kBatch; ++j) top = fmaxf(top, s[j]);
    const float f = weight_of(m, top);
    m = top;
    l *= f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] *= f;
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      if (it + j >= n) break;                                         // slots that were never filled
      const float e = weight_of(s[j], top);
      l += e;
      float v[8];
      unpack8(ring[(((it + j) % kDepth) * 2 + 1) * kStreamThreads + tid], v);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(e, v[i], acc[i]);
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) copy(it + j + kDepth);
  }
  // the key streams of a warp, then the warps, then the cluster, always in the same order
#pragma unroll
  for (int o = LPK; o < 32; o <<= 1) {
    const float top = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o)), f = weight_of(m, top);
    m = top;
    l *= f;
    l += __shfl_xor_sync(0xffffffffu, l, o);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      acc[i] *= f;
      acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
    }
  }
  copies_wait<0>();
  __syncthreads();                                                    // the ring is read out
  if (sub == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) sums[warp * L::kRow + ch + i] = acc[i];
  }
  if (lane == 0) {
    sums[warp * L::kRow + HD] = m;
    sums[warp * L::kRow + HD + 1] = l;
  }
  __syncthreads();
  if (tid < HD) {
    float top = -INFINITY, v = 0.f, sum = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) top = fmaxf(top, sums[k * L::kRow + HD]);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float f = weight_of(sums[k * L::kRow + HD], top);
      v = fmaf(f, sums[k * L::kRow + tid], v);
      sum = fmaf(f, sums[k * L::kRow + HD + 1], sum);
    }
    part[tid] = v;
    if (tid == 0) {
      part[HD] = top;
      part[HD + 1] = sum;
    }
  }
  if (splits > 1) cluster_barrier();
  else __syncthreads();
  if (rank == 0 && tid < HD) {
    float top = part[HD], v = part[tid], sum = part[HD + 1];
    if (splits > 1) {
      float ms[kMaxCluster], vs[kMaxCluster], ls[kMaxCluster];
#pragma unroll
      for (int k = 0; k < kMaxCluster; ++k)
        if (k < splits) {
          ms[k] = ld_rank(part + HD, k);
          vs[k] = ld_rank(part + tid, k);
          ls[k] = ld_rank(part + HD + 1, k);
          top = fmaxf(top, ms[k]);
        }
      v = sum = 0.f;
#pragma unroll
      for (int k = 0; k < kMaxCluster; ++k)
        if (k < splits) {
          const float f = weight_of(ms[k], top);
          v = fmaf(f, vs[k], v);
          sum = fmaf(f, ls[k], sum);
        }
    }
    p.O[int64_t(b) * p.o_sb + int64_t(g) * HD + tid] = hg_f2lp(sum == 0.f ? 0.f : v / sum);
    if (tid == 0) p.LSE[size_t(b) * p.nheads + g] = sum > 0.f ? (top + log2f(sum)) * kLn2 : -INFINITY;
  }
  if (splits > 1) cluster_barrier();                                  // nobody leaves while its part may be read
}

// CTAs that share a head's keys, a power of two.  Two CTAs an SM stream at the memory's rate, so a wave is split until it has
// those, eight steps each at least; heads of more than a wave of three CTAs an SM only where the keys are many enough that a
// nearly empty last wave costs more than the merge.  Us cold, one, two, four, eight CTAs a head, head dim 128: 32 heads x 4000
// keys 49, 33, 25, 23; 64 x 4000 53, 41, 35, 41; 128 x 4000 64, 59, 68, 66; 256 x 4000 102, 107, 107, 109; 512 x 300 29, 33,
// 39, 57; 512 x 1000 72, 66, 68, 82; 512 x 4000 203, 178, 174, 186.
int stream_splits(long long heads, int steps) {
  int s = 1;
  while (s < kMaxCluster && heads * s * 2 <= 296 && steps >= s * 16) s *= 2;
  if (heads > 444) s = steps >= 192 ? 4 : steps >= 48 ? 2 : 1;
  return s;
}

template <int HD>
int launch_stream(const DecodeParams& p, int settled, cudaStream_t st) {
  auto k = flash_stream_kernel<HD>;
  constexpr int kps = 2048 / HD;
  const int splits = stream_splits((long long)p.nkv * p.B, (p.kv_len + kps - 1) / kps);
  if (cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, StreamSmem<HD>::kTotal)) return int(e);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(splits);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(unsigned(splits), unsigned(p.nkv), unsigned(p.B));
  cfg.blockDim = dim3(kStreamThreads, 1, 1);
  cfg.dynamicSmemBytes = StreamSmem<HD>::kTotal;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = hg_host::chain_overlaps() ? 2 : 1;
  return hg_host::launched(cudaLaunchKernelEx(&cfg, k, p, settled));
}

inline int keys_seen(int Sq, int Skv, int causal, int q_pos0, int k_pos0) {
  long long n = Skv;
  if (causal) {
    const long long last = (long long)q_pos0 + Sq - k_pos0;   // keys that the last query may see
    if (last < n) n = last;
  }
  return n < 0 ? 0 : int(n);
}
// Up to two rows: 64 keys per CTA, all loaded at once.  More rows: 128 where that still gives every SM several CTAs.
inline int keys_per_cta(int rows, int kv_len, int nkv, int B) {
  return rows > 2 && (long long)((kv_len + 127) / 128) * nkv * B >= 148 * 8 ? 128 : 64;
}
inline int range_count(int kv_len, int chunk) { return kv_len > chunk ? (kv_len + chunk - 1) / chunk : 1; }

template <int HD, int R>
int launch(const DecodeParams& p, int chunk, int ranges, cudaStream_t st) {
  const dim3 grid(p.nkv, p.B, ranges);   // neighbours read neighbouring heads of the same cache rows
  auto k = flash_decode_kernel<HD, R, 64>;
  if constexpr (R > 2) {
    if (chunk == 128) k = flash_decode_kernel<HD, R, 128>;
  }
  if (int rc = hg_host::launch(k, grid, 128, 0, st, p)) return rc;
  return ranges > 1 ? hg_host::launch(flash_decode_merge_kernel<HD>, p.B * p.nkv * p.Sq * p.qpg, HD, 0, st, p, ranges) : 0;
}

template <int HD>
int launch_rows(const DecodeParams& p, int chunk, int ranges, cudaStream_t st) {
  const int rows = p.Sq * p.qpg;
  if (rows == 1) return launch<HD, 1>(p, chunk, ranges, st);
  if (rows == 2) return launch<HD, 2>(p, chunk, ranges, st);
  if (rows <= 4) return launch<HD, 4>(p, chunk, ranges, st);
  return launch<HD, 8>(p, chunk, ranges, st);
}

}  // namespace

extern "C" {

// Floats of scratch hg_flash_decode needs (0: none), or -1 when it does not take the call: more than eight query rows
// per kv head, another head dim, or rows that are not whole 16-byte groups.
long long hg_flash_decode_scratch(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, int Sq, int Skv, int B,
                                  int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0) {
  if ((hd != 64 && hd != 128) || Sq < 1 || Skv < 1 || B < 1 || nkv < 1 || nheads % nkv) return -1;
  if ((long long)Sq * (nheads / nkv) > kMaxRows || nkv > 65535 || B > 65535) return -1;
  for (const HgAttnTensor* t : {q, k, v})
    if ((uintptr_t(t->ptr) & 15) || (t->ss & 7) || (t->sb & 7)) return -1;
  const int kv_len = keys_seen(Sq, Skv, causal, q_pos0, k_pos0);
  const int ranges = range_count(kv_len, keys_per_cta(Sq * (nheads / nkv), kv_len, nkv, B));
  if (ranges > 65535) return -1;
  return ranges > 1 ? (long long)B * nheads * Sq * ranges * (hd + 2) : 0;
}

// Whether spreading the keys beats the one-tile kernel.  That kernel gives a CTA all queries of one query head and walks
// the head's keys alone: it loses when its heads leave part of the last wave of 148 idle, when a head has many keys, or
// when query heads share a kv head and it reads those keys once for each.  It wins when a few queries of a head share its
// one walk (here each is a row of its own), and below about 500 keys, where its single launch beats a launch and a merge.
// Measured, us cold, here / there:
//   one wave, 1 query   head dim 128: 32 heads (8 kv) x 2000 keys 24 / 32, 1000 24 / 20; 64 x 4000 48 / 54, 96 x 4000 62 / 57,
//                       128 x 1536 36 / 31, 128 (32 kv) x 1536 28 / 27, x 2000 32 / 33; head dim 64: 128 x 1536 24 / 27
//   two waves           head dim 128: 256 (64 kv) x 128 24 / 16, 512 24 / 26, 2000 46 / 60; 192 x 256 20 / 20, 384 25 / 22,
//                       2000 54 / 66; 288 x 2000 75 / 72; head dim 64: 288 x 384 22 / 23, 2000 44 / 59
//   three waves         head dim 128: 384 (96 kv) x 128 24 / 22, 192 26 / 29, 2000 64 / 86; 320 x 256 24 / 27, 2000 79 / 96
//   more                head dim 128: 512 x 64 12 / 31, 1000 65 / 80; 1024 (256 kv) x 1000 62 / 119
//   several queries     head dim 128: 4 x 192 heads x 2000 91 / 66, 8 x 512 x 2000 294 / 127; 2 x 320 (80 kv) x 2000 62 / 84
int hg_flash_decode_pays(int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0) {
  if (nkv < 1) return 0;
  const long long heads = (long long)B * nheads;
  const int keys = keys_seen(Sq, Skv, causal, q_pos0, k_pos0), qpg = nheads / nkv, rows = Sq * qpg;
  if (Sq > 1 && qpg < 2 * Sq) return 0;
  if (heads > 3 * 148) return 1;
  if (heads > 2 * 148) return rows <= 2 || keys >= 192;
  if (heads > 148) return rows > 2 ? keys >= 512 : rows == 2 || hd == 64 || keys <= 256 || (keys >= 512 && heads <= 224);
  if (hd == 128 && rows == 1 && heads > 64) return 0;
  return keys >= (hd == 128 && rows > 2 ? 2000 : 1536);
}

static DecodeParams decode_params(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, const HgAttnTensor* o,
                                  void* lse, int Sq, int Skv, int B, int nheads, int nkv, int causal, int q_pos0, int k_pos0,
                                  float scale) {
  DecodeParams p{};
  p.Q = (const hg_lp_t*)q->ptr; p.K = (const hg_lp_t*)k->ptr; p.V = (const hg_lp_t*)v->ptr; p.O = (hg_lp_t*)o->ptr;
  p.q_ss = q->ss; p.q_sb = q->sb; p.k_ss = k->ss; p.k_sb = k->sb; p.v_ss = v->ss; p.v_sb = v->sb; p.o_ss = o->ss; p.o_sb = o->sb;
  p.q_gs = q->gs; p.q_hs = q->hs; p.q_off = q->off;
  p.k_gs = k->gs; p.k_off = k->off; p.v_gs = v->gs; p.v_off = v->off;
  p.LSE = (float*)lse;
  p.Sq = Sq; p.B = B; p.nheads = nheads; p.nkv = nkv; p.qpg = nheads / nkv; p.causal = causal;
  p.q_pos0 = q_pos0; p.k_pos0 = k_pos0; p.scale = scale;
  p.kv_len = keys_seen(Sq, Skv, causal, q_pos0, k_pos0);
  return p;
}

// Whether hg_flash_fwd gives the call to hg_flash_stream: one query, a kv head of its own for every head, and not what the
// spread keys are taken for.  It wins there but for 129 to 148 heads of many keys, two CTAs a head on two to an SM (144 heads x
// 4000 keys 68 / 68, 16000 197 / 205).  Us cold, tile kernel / here, head dim 128: 32 heads x 100 keys 12 / 8,
// 300 14 / 12, 1000 21 / 14; 64 x 1000 23 / 16; 128 x 100 12 / 10, 1000 25 / 23, 4000 61 / 59, 16000 186 / 174; 256 x 300 27 / 16,
// 1000 45 / 35, 4000 115 / 100; head dim 64: 32 x 1000 21 / 12, 128 x 300 14 / 11, 1000 23 / 16.  Probabilities stay in fp32:
// 0.0017 of the result's norm off 64 bits (the rounding of the result), 0.0023 on the tile kernel.
int hg_flash_stream_takes(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, int Sq, int Skv, int B,
                          int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0) {
  if ((hd != 64 && hd != 128) || Sq != 1 || Skv < 1 || B < 1 || nheads < 1 || nheads != nkv || nkv > 65535 || B > 65535) return 0;
  for (const HgAttnTensor* t : {q, k, v})
    if ((uintptr_t(t->ptr) & 15) || (t->ss & 7) || (t->sb & 7)) return 0;
  const long long heads = (long long)B * nheads;
  if (heads > 128 && heads <= 148 && keys_seen(Sq, Skv, causal, q_pos0, k_pos0) >= 4000) return 0;
  return !hg_flash_decode_pays(Sq, Skv, B, nheads, nkv, hd, causal, q_pos0, k_pos0);
}

// Same contract as hg_flash_fwd for those calls.  settled: keys that no kernel of an open chain writes.
int hg_flash_stream(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, const HgAttnTensor* o, void* lse,
                    int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0, float scale,
                    int settled, void* stream) {
  const DecodeParams p = decode_params(q, k, v, o, lse, Sq, Skv, B, nheads, nkv, causal, q_pos0, k_pos0, scale);
  cudaStream_t st = (cudaStream_t)stream;
  return hd == 128 ? launch_stream<128>(p, settled, st) : launch_stream<64>(p, settled, st);
}

// Same contract as hg_flash_fwd for the calls that hg_flash_decode_scratch accepts; `ws` is its scratch.
int hg_flash_decode(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, const HgAttnTensor* o, void* lse,
                    void* ws, int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0,
                    float scale, void* stream) {
  const long long need = hg_flash_decode_scratch(q, k, v, Sq, Skv, B, nheads, nkv, hd, causal, q_pos0, k_pos0);
  if (need < 0 || (need > 0 && ws == nullptr)) return -1;
  DecodeParams p = decode_params(q, k, v, o, lse, Sq, Skv, B, nheads, nkv, causal, q_pos0, k_pos0, scale);
  p.ws = (float*)ws;
  const int chunk = keys_per_cta(Sq * p.qpg, p.kv_len, nkv, B), ranges = range_count(p.kv_len, chunk);
  cudaStream_t st = (cudaStream_t)stream;
  return hd == 128 ? launch_rows<128>(p, chunk, ranges, st) : launch_rows<64>(p, chunk, ranges, st);
}

}  // extern "C"
