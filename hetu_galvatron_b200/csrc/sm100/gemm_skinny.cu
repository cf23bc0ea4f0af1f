// GEMM for few rows (M <= 128 tokens): decode steps, short prompts and the backward of tiny batches.
//
//   C[M, N] = x[M, K] W (+ bias),  W stored [N, K] (forward) or [K, N] (W_MN: the data gradient's layout)
//
// What bounds it is reading W once from HBM, so the kernel is a weight streamer.  The roles of the operands are
// swapped against the large-M kernels: 128 rows of W are the M side of the tcgen05 tile and the tokens, padded to
// NT = 16, 32, 64 or 128, its N side, so that the tensor core does no more padded work than the token count needs
// and a CTA's accumulator is only NT columns.  A long contraction is cut over the S <= 8 CTAs of a cluster: a 4096 x 4096
// weight has 32 row tiles, which keep 32 SMs busy, and 256 CTAs when each tile is shared by eight.  Two CTAs fit
// an SM (at most 113 KB of shared memory each), which keeps about 200 KB of loads in flight per SM.  The partial
// sums meet through distributed shared memory, added in rank order: no workspace, no atomics, the same bits every time.
// Measured, 4 rows, cold caches: 4096 x 4096 16 us (35 us in 16 tiles of the one-CTA kernel, 5 us for the bytes alone),
// 4096 x 11008 29 us (78), 22016 x 4096 47 us (53), 152064 x 3584 176 us (208; 164 for the bytes); the seventeen
// products of a decode step through four 7B-sized layers and the head 386 us instead of 743.  In a chain (the native decoder
// step) a CTA's first stages of W are requested before the kernel in front has ended, up to 190 KB per SM: such a step as a
// CUDA graph 519 -> 477 us.
//
// Roles (192 threads): warp 0 TMA producer, warp 1 TMEM allocator + UMMA issuer, warps 2-5 epilogue (thread = row of W
// = output column, so a warp stores 32 consecutive elements of a token's row).
#include <mutex>

#include "entry_points.h"
#include "gemm_core.cuh"

namespace hg {
namespace skinny {

using namespace hg::gemm;

constexpr int TM = 128;                      // rows of W per tile
constexpr int W_BYTES = TM * BK * 2;         // 16 KB

template <int NT>
struct Cfg {
  static constexpr int kXBytes = NT * BK * 2;
  static constexpr int kStageBytes = W_BYTES + kXBytes;
  static constexpr int kStages = NT <= 16 ? 6 : NT <= 32 ? 5 : NT <= 64 ? 4 : 3;
  static constexpr int kTmemCols = NT < 32 ? 32 : NT;
  static constexpr int kSmem = kStages * kStageBytes + 1024 + 256;
  static_assert(kSmem <= 113 * 1024, "two CTAs per SM");
  static_assert(NT * TM * 4 <= kStages * kStageBytes, "the partial tile reuses the stages");
};

struct SkinnyParams {
  int M, N, K, ldc;
  void* C;
  const hg_lp_t* bias;
  int out_mode;                              // kOutBf16 or kOutF32
  int* status;
};

__device__ __forceinline__ uint32_t cta_rank_in_cluster() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_addr(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_peer(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ void store_out(const SkinnyParams& p, int m, int n, float v) {
  if (p.out_mode == kOutBf16) reinterpret_cast<hg_lp_t*>(p.C)[size_t(m) * p.ldc + n] = hg_f2lp(v);
  else reinterpret_cast<float*>(p.C)[size_t(m) * p.ldc + n] = v;
}

template <bool W_MN, int NT>
__global__ void __launch_bounds__(192, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                   const SkinnyParams p) {
  using C_ = Cfg<NT>;
  constexpr int ST = C_::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sW = base;
  uint8_t* sX = base + ST * W_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + ST * C_::kStageBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + ST;
  uint64_t* acc_full = bars + 2 * ST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * ST + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int splits = gridDim.x;                               // = cluster size
  const int rank = splits > 1 ? int(cta_rank_in_cluster()) : 0;
  const int n0 = blockIdx.y * TM;
  const int num_kb = (p.K + BK - 1) / BK;
  const int kb0 = int((long long)num_kb * rank / splits), kb1 = int((long long)num_kb * (rank + 1) / splits);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
#pragma unroll
    for (int i = 0; i < ST; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, C_::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  chain_release();                            // after the allocation: see chain_release
  if (warp != 0) chain_wait();

  if (warp == 0) {
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    int issued = 0;
    const bool issuer = elect_one() != 0;
    auto load_w = [&](int st, int kb) {
      uint8_t* w = sW + st * W_BYTES;
      mbar_expect_tx(&full[st], C_::kStageBytes);
      if (W_MN) {
#pragma unroll
        for (int j = 0; j < TM / 64; ++j) tma_load_2d(w + j * SLAB_BYTES, &tmW, &full[st], n0 + j * 64, kb * BK);
      } else {
        tma_load_2d(w, &tmW, &full[st], kb * BK, n0);
      }
    };
    // In a chain nothing writes weights: the first stages of them are on their way while the kernel before this one, which
    // makes x, still runs.
    const int ahead = min(ST, kb1 - kb0);
    if (issuer)
      for (int i = 0; i < ahead; ++i) load_w(i, kb0 + i);
    __syncwarp();
    chain_wait();
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(&empty[stage], phase ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { ok = false; break; }
      if (issuer) {
        if (issued >= ahead) load_w(stage, kb);
        tma_load_2d(sX + stage * C_::kXBytes, &tmX, &full[stage], kb * BK, 0);
      }
      __syncwarp();
      ++issued;
      if (++stage == ST) { stage = 0; phase ^= 1; }
    }
    if (!ok) {
      *abort_flag = 1;
      // our own copies land before this CTA's shared memory is released (bounded)
      const int flying = max(issued, ahead);
      for (int i = 0; i < ST && i < flying; ++i) {
        const int at = flying - 1 - i;
        for (uint32_t spin = 0; spin < (1u << 16); ++spin)
          if (mbar_try_wait(&full[at % ST], uint32_t(at / ST) & 1)) break;
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_lp(TM, NT, W_MN, false);
    constexpr uint32_t lbo = W_MN ? SLAB_BYTES : 16, kadv = W_MN ? 2048 : 32;
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    const bool issuer = elect_one() != 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(&full[stage], phase, p.status, kTimeoutSmemFull, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const uint32_t w = smem_u32(sW + stage * W_BYTES), x = smem_u32(sX + stage * C_::kXBytes);
      if (issuer) {
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_f16_ss(tmem, make_smem_desc(w + k * kadv, lbo, 1024), make_smem_desc(x + k * 32, 16, 1024), idesc,
                      ((kb - kb0) | k) != 0);
        umma_commit(&empty[stage]);
      }
      __syncwarp();
      if (++stage == ST) { stage = 0; phase ^= 1; }
    }
    if (ok && issuer) umma_commit(acc_full);
    __syncwarp();
    if (!ok) *abort_flag = 1;
  } else {
    const int row = (warp & 3) * 32 + int(lane_id());
    const uint32_t lane_off = uint32_t((warp & 3) * 32) << 16;
    const int n = n0 + row;
    // every stage has been read by the tensor core once the accumulator is complete: the partial tile goes over them
    float* part = reinterpret_cast<float*>(base);
    if (mbar_wait_warp(acc_full, 0, p.status, kTimeoutTmemFull, abort_flag)) {
      tc_fence_after();
      const float bias = (splits == 1 && p.bias != nullptr && n < p.N) ? hg_lp2f(p.bias[n]) : 0.f;
#pragma unroll 1
      for (int c = 0; c < NT; c += 16) {
        if (c >= p.M) break;
        uint32_t r[16];
        tmem_ld16(tmem + lane_off + c, r);
        tmem_ld_wait();
        if (splits == 1) {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (c + i < p.M && n < p.N) store_out(p, c + i, n, __uint_as_float(r[i]) + bias);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) part[(c + i) * TM + row] = __uint_as_float(r[i]);
        }
      }
      tc_fence_before();
    } else {
      *abort_flag = 1;
    }
  }

  __syncthreads();
  if (splits > 1) {
    cluster_barrier();                                        // every CTA's partial tile is in its shared memory
    if (warp >= 2) {
      const int row = (warp & 3) * 32 + int(lane_id());
      const int n = n0 + row;
      const uint32_t mine = smem_u32(base) + uint32_t(row) * 4;
      if (!*abort_flag && n < p.N) {
        const float bias = p.bias != nullptr ? hg_lp2f(p.bias[n]) : 0.f;
        for (int m = rank; m < p.M; m += splits) {            // each CTA finishes its share of the tokens
          float part[8];
#pragma unroll
          for (int s = 0; s < 8; ++s)
            if (s < splits) part[s] = ld_peer(peer_addr(mine + uint32_t(m) * (TM * 4), s));
          float v = 0.f;
#pragma unroll
          for (int s = 0; s < 8; ++s)
            if (s < splits) v += part[s];
          store_out(p, m, n, v + bias);
        }
      }
    }
    __syncwarp();
    cluster_barrier();                                        // nobody leaves while its partial tile may be read
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, C_::kTmemCols);
  }
}

}  // namespace skinny
}  // namespace hg

using namespace hg::skinny;

namespace {

constexpr int kMaxSplits = 8;                // portable cluster size

// How many clusters of each size the device holds at once (index: size), asked once per kernel variant and device.
template <bool W_MN, int NT>
int resident_clusters(int splits, int* out) {
  static std::mutex mu;
  static int table[64][kMaxSplits + 1] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return int(e);
  if (dev < 0 || dev >= 64) return -1;
  std::lock_guard<std::mutex> lk(mu);
  if (table[dev][splits] == 0) {
    auto k = gemm_skinny_kernel<W_MN, NT>;
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<NT>::kSmem);
    if (e != cudaSuccess) return int(e);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(splits);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(unsigned(splits), 1024, 1);
    cfg.blockDim = dim3(192, 1, 1);
    cfg.dynamicSmemBytes = Cfg<NT>::kSmem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, k, &cfg);
    if (e != cudaSuccess) return int(e);
    table[dev][splits] = n > 0 ? n : -1;
  }
  *out = table[dev][splits];
  return 0;
}

template <bool W_MN, int NT>
int launch_skinny(const CUtensorMap& tw, const CUtensorMap& tx, const SkinnyParams& p, int want_splits, cudaStream_t st) {
  const int tiles = (p.N + TM - 1) / TM, num_kb = (p.K + BK - 1) / BK;
  // The largest split whose clusters are all resident at once (they then share the memory bandwidth evenly and end
  // together), or none where the contraction is too short for what the split costs, the partial tile's way through
  // shared memory and M / splits rows added one after the other by each CTA: a split by two of a short contraction is the
  // worst of both (64 rows, 512 columns, K = 512: 1, 2, 4, 8 CTAs a tile 8.8, 13.3, 10.8, 8.8 us; K = 1024: 10.8, 14.9, 10.8,
  // 8.8; 8192 columns, four at most, K = 1024 14.1 alone, 14.9 by four, K = 2048 19.9, 17.8; 12288 columns, two at most,
  // 4 rows, K = 2048 18.1 alone, 18.8 by two, K = 4096 29.0, 27.7).
  int splits = 1;
  for (int s = kMaxSplits; s > 1; --s) {
    if (num_kb * s < (s == 2 ? 128 : 96)) continue;
    int resident = 0;
    if (int rc = resident_clusters<W_MN, NT>(s, &resident)) return rc;
    if (tiles <= resident) { splits = s; break; }
  }
  if (splits == 1) {                           // the first launch of a variant sets its shared memory limit here
    int resident = 0;
    if (int rc = resident_clusters<W_MN, NT>(1, &resident)) return rc;
  }
  if (want_splits > 0) splits = want_splits;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(splits);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(unsigned(splits), unsigned(tiles), 1);
  cfg.blockDim = dim3(192, 1, 1);
  cfg.dynamicSmemBytes = Cfg<NT>::kSmem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = hg_host::chain_overlaps() ? 2 : 1;
  return hg_host::launched(cudaLaunchKernelEx(&cfg, gemm_skinny_kernel<W_MN, NT>, tw, tx, p));
}

template <bool W_MN>
int dispatch_skinny(const CUtensorMap& tw, const CUtensorMap& tx, const SkinnyParams& p, int nt, int splits, cudaStream_t st) {
  switch (nt) {
    case 16: return launch_skinny<W_MN, 16>(tw, tx, p, splits, st);
    case 32: return launch_skinny<W_MN, 32>(tw, tx, p, splits, st);
    case 64: return launch_skinny<W_MN, 64>(tw, tx, p, splits, st);
    default: return launch_skinny<W_MN, 128>(tw, tx, p, splits, st);
  }
}

}  // namespace

extern "C" {

// C[M, N] = x[M, K] op(W) (+ bias) for M <= 128, fp32 accumulation; out_mode kOutBf16 or kOutF32.
//   w_mn == 0 : W is [N, K] row-major with pitch ldw;  w_mn == 1 : W is [K, N] row-major.
//   splits: CTAs that share one tile's contraction (1..8), 0 = chosen here.
// Returns 0 on success, a CUDA error code or -1 (bad argument) otherwise.
int hg_gemm_skinny_bf16(const void* x, const void* W, void* C, const void* bias, int M, int N, int K, int ldx, int ldw,
                        int ldc, int w_mn, int out_mode, int splits, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M > 128 || splits < 0 || splits > kMaxSplits || (out_mode != kOutBf16 && out_mode != kOutF32)) return -1;
  if ((ldx & 7) || (ldw & 7) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(W) & 15)) return -1;
  if ((long long)(N + TM - 1) / TM > 65535) return -1;
  if (splits > (K + BK - 1) / BK) splits = (K + BK - 1) / BK;
  const int nt = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  CUtensorMap tw, tx;
  int rc;
  if (w_mn) rc = hg_host::make_tmap_2d_bf16(&tw, W, K, N, ldw, 64, 64);
  else      rc = hg_host::make_tmap_2d_bf16(&tw, W, N, K, ldw, TM, 64);
  if (rc) return rc;
  if ((rc = hg_host::make_tmap_2d_bf16(&tx, x, M, K, ldx, nt, 64))) return rc;
  SkinnyParams p{};
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.C = C;
  p.bias = reinterpret_cast<const hg_lp_t*>(bias);
  p.out_mode = out_mode;
  p.status = hg_host::status_ptr();
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  return w_mn ? dispatch_skinny<true>(tw, tx, p, nt, splits, st) : dispatch_skinny<false>(tw, tx, p, nt, splits, st);
}

}  // extern "C"
