// Device-side building blocks of the CTA-pair (tcgen05.mma.cta_group::2) bf16 GEMM: shared-memory layout, pair
// primitives, TMA producer, UMMA issuer and the row-coalescing epilogue.  Used by gemm2.cu (plain GEMM) and
// fused_tp2.cu (all-gather -> GEMM and GEMM -> reduce-scatter over peer memory on the same tile).
#pragma once
#include "gemm_core.cuh"

namespace hg {
namespace gemm2 {

using namespace hg::gemm;

constexpr int CM = 256;                       // rows of the pair's tile
constexpr int HALF_N = BN / 2;                // B rows staged by one CTA
constexpr int STAGES2 = 6;
constexpr int A2_BYTES = BM * BK * 2;         // 16 KB
constexpr int B2_BYTES = HALF_N * BK * 2;     // 16 KB
// The plain and grouped kernels have one or two epilogue warps per 32 rows; two take turns at the blocks of columns.  A block's
// way out is a chain (tensor memory, registers, shared memory, fence, copy) of about 1000 cycles of which a warp keeps little in
// flight.  us, one / two: fp32 results 37888 x 3584, K = 63 126 / 103 (5.3 TB/s written), 22016 x 4096, K = 128 88 / 73, added to
// what is there, K = 1024 240 / 197; 16 bits 8192 x 22016, K = 512 169 / 158.  Two stages per warp instead of one are worth
// 0 to 10 % where stores bound, and cost 1 to 1.5 % on large products.
constexpr int EPI2_WARPS = 2 * EPI_WARPS;
// Per epilogue warp: a block of 32 rows x 128 bytes on its way to C, as TMA's 128-byte swizzle has it.
constexpr int EPI_STAGE_FLOATS = 32 * 32;
constexpr int SMEM2_BYTES = STAGES2 * (A2_BYTES + B2_BYTES) + EPI2_WARPS * EPI_STAGE_FLOATS * 4 + 1024 + 256;
static_assert(SMEM2_BYTES <= 232448, "one CTA per SM");
constexpr uint16_t kPairMask = 0x3;

struct Smem2 {
  uint8_t* a;
  uint8_t* b;
  uint64_t* full;
  uint64_t* empty;
  uint64_t* tmem_full;
  uint64_t* tmem_empty;
  uint32_t* tmem_base;
  volatile int* abort;
  float* epi_stage;
};

__device__ __forceinline__ Smem2 carve2(uint8_t* raw) {
  Smem2 s;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  s.a = base;
  s.b = base + STAGES2 * A2_BYTES;
  s.epi_stage = reinterpret_cast<float*>(base + STAGES2 * (A2_BYTES + B2_BYTES));   // 1024-byte aligned
  uint64_t* bars = reinterpret_cast<uint64_t*>(s.epi_stage + EPI2_WARPS * EPI_STAGE_FLOATS);
  s.full = bars;
  s.empty = bars + STAGES2;
  s.tmem_full = bars + 2 * STAGES2;
  s.tmem_empty = bars + 2 * STAGES2 + 2;
  s.tmem_base = reinterpret_cast<uint32_t*>(bars + 2 * STAGES2 + 4);
  s.abort = reinterpret_cast<volatile int*>(s.tmem_base + 1);
  return s;
}

// ---- cluster / pair primitives -------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of `local_addr` (a shared::cta address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 2-D tile load into this CTA's shared memory; the bytes complete on the barrier at `bar_cluster_addr`
// (the leader's).  No multicast: the destination is this CTA only.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, uint32_t bar_cluster_addr, int c0,
                                                 int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_f16_ss_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n"
      :
      : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at this shared-memory offset in every CTA of `mask` once the issued MMAs retired.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(mask)
      : "memory");
}

// ---- work units -------------------------------------------------------------------------------------------------
// Pair `first` of `step` walks tiles first, first + step, ...; with the tail split on, every pair has the same number
// of whole tiles (split_tail_begin / step) and the first (tail tiles x split_s) pairs one slice of a tail tile after them.
struct Unit {
  int tile, kb0, kb1, slice;
};
constexpr int kSplitWords = 2 * EPI2_WARPS;              // of a tile: one per epilogue warp of the pair
constexpr unsigned long long kSplitCountMask = 255;      // low bits of a word: slices that have arrived; a token has none of them
// Word `q` (four columns) of 32-column block `c` of this thread's row in a partial tile: neighbouring lanes, neighbouring words.
__device__ __forceinline__ int split_word(int bn, int warp8, int c, int q) {
  return (((warp8 * (bn / 32) + c) * 8 + q) * 32 + int(lane_id())) * 4;
}
__device__ __forceinline__ int unit_count(const Params& p, int first, int step, int num_tiles) {
  if (p.split_s > 1) return p.split_tail_begin / step + (first < (num_tiles - p.split_tail_begin) * p.split_s ? 1 : 0);
  return first < num_tiles ? (num_tiles - first + step - 1) / step : 0;
}
__device__ __forceinline__ Unit unit_at(const Params& p, int first, int step, int u, int num_kb) {
  Unit w;
  if (p.split_s > 1 && u == p.split_tail_begin / step) {
    w.tile = p.split_tail_begin + first / p.split_s;
    w.slice = first % p.split_s;
    w.kb0 = num_kb * w.slice / p.split_s;
    w.kb1 = num_kb * (w.slice + 1) / p.split_s;
  } else {
    w.tile = first + u * step;
    w.slice = 0;
    w.kb0 = 0;
    w.kb1 = num_kb;
  }
  return w;
}

// ---- roles ------------------------------------------------------------------------------------------------------
template <bool A_MN, bool B_MN>
__device__ __forceinline__ void producer2(const CUtensorMap* tmA, const CUtensorMap* tmB, const Params& p, const Smem2& s,
                                          uint32_t rank, int first, int step, int num_tiles) {
  uint32_t stage = 0, phase = 0;
  bool issued[STAGES2];
  uint32_t issued_parity[STAGES2];
#pragma unroll
  for (int i = 0; i < STAGES2; ++i) { issued[i] = false; issued_parity[i] = 0; }
  const int num_kb = (p.K + BK - 1) / BK;
  const int half = p.bn / 2;              // of B's rows (columns) of a tile, each CTA stages one half; whole slabs where N-major
  const uint32_t stage_bytes = 2 * (A2_BYTES + (B_MN ? (half + 63) / 64 * SLAB_BYTES : half * BK * 2));
  bool ok = true;
  const bool issuer = elect_one() != 0;   // the warp walks the loop together; only this lane issues the copies
  const int n_units = unit_count(p, first, step, num_tiles);
  for (int u = 0; ok && u < n_units; ++u) {
    const Unit w = unit_at(p, first, step, u, num_kb);
    int tm, tn;
    tile_coords(p, w.tile, tm, tn);
    const int m0 = tm * CM + int(rank) * BM;
    const int n0 = tn * p.bn + int(rank) * half;
    if (p.ready != nullptr) {
      // readiness gate on this CTA's 128 A rows (all-gather fused variant): one lane polls, bounded, and the verdict
      // is made warp-uniform; the rows were written with ordinary stores, TMA reads through the async proxy
      const int f0 = m0 / p.rows_per_flag;
      const int f1 = (min(m0 + BM, p.M) - 1) / p.rows_per_flag;
      int landed = 1;
      if (lane_id() == 0) {
        for (int f = f0; landed && f <= f1; ++f) {
          const uint64_t t0 = globaltimer_ns();
          while (ld_acquire_sys(p.ready + f) < p.ready_target) {
            if (*s.abort || globaltimer_ns() - t0 > kWaitLimitNs) {
              set_status(p.status, kTimeoutPeerFlag);
              landed = 0;
              break;
            }
            __nanosleep(64);
          }
        }
      }
      landed = __shfl_sync(0xffffffffu, landed, 0);
      __syncwarp();
      if (!landed) { ok = false; break; }
      asm volatile("fence.proxy.async.global;" ::: "memory");
    }
    for (int kb = w.kb0; kb < w.kb1; ++kb) {
      if (!mbar_wait_warp(&s.empty[stage], phase ^ 1, p.status, kTimeoutSmemEmpty, s.abort)) { ok = false; break; }
      const uint32_t bar = map_to_cta(smem_u32(&s.full[stage]), 0);
      uint8_t* sa = s.a + stage * A2_BYTES;
      uint8_t* sb = s.b + stage * B2_BYTES;
      const int k0 = kb * BK;
      if (issuer) {
        if (rank == 0) mbar_expect_tx(&s.full[stage], stage_bytes);
        if (A_MN) {
#pragma unroll
          for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * SLAB_BYTES, tmA, bar, m0 + j * 64, k0);
        } else {
          tma_load_2d_pair(sa, tmA, bar, k0, m0);
        }
        if (B_MN) {
#pragma unroll
          for (int j = 0; j < HALF_N / 64; ++j)
            if (j * 64 < half) tma_load_2d_pair(sb + j * SLAB_BYTES, tmB, bar, n0 + j * 64, k0);
        } else {
          tma_load_2d_pair(sb, tmB, bar, k0, n0);
        }
      }
      __syncwarp();
      issued[stage] = true;
      issued_parity[stage] = phase;
      if (++stage == STAGES2) { stage = 0; phase ^= 1; }
    }
  }
  // The leader's commits arrive on this CTA's barriers: leave only when the last of them has.
  for (int i = 0; ok && i < STAGES2; ++i) {
    ok = mbar_wait_warp(&s.empty[stage], phase ^ 1, p.status, kTimeoutSmemEmpty, s.abort);
    if (++stage == STAGES2) { stage = 0; phase ^= 1; }
  }
  if (!ok) {
    *s.abort = 1;
    if (rank == 0) {
      // the leader can see its own copies land; give them a bounded moment before shared memory is released
#pragma unroll
      for (int i = 0; i < STAGES2; ++i)
        if (issued[i])
          for (uint32_t spin = 0; spin < (1u << 16); ++spin)
            if (mbar_try_wait(&s.full[i], issued_parity[i])) break;
    } else {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);  // 2 ms: far longer than a tile load
    }
  }
}

template <bool A_MN, bool B_MN>
__device__ __forceinline__ void mma2(const Params& p, const Smem2& s, uint32_t tmem_base, int first, int step,
                                     int num_tiles) {
  const uint32_t idesc = make_idesc_lp(CM, p.bn, A_MN, B_MN);
  constexpr uint32_t a_lbo = A_MN ? SLAB_BYTES : 16, a_sbo = 1024, a_kadv = A_MN ? 2048 : 32;
  constexpr uint32_t b_lbo = B_MN ? SLAB_BYTES : 16, b_sbo = 1024, b_kadv = B_MN ? 2048 : 32;
  const int num_kb = (p.K + BK - 1) / BK;
  uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
  bool ok = true;
  const bool issuer = elect_one() != 0;   // the warp walks the loop together; only this lane issues (see gemm_core.cuh)
  const int n_units = unit_count(p, first, step, num_tiles);
  for (int u = 0; ok && u < n_units; ++u) {
    const Unit w = unit_at(p, first, step, u, num_kb);
    if (!mbar_wait_warp(&s.tmem_empty[acc], acc_phase ^ 1, p.status, kTimeoutTmemEmpty, s.abort)) { ok = false; break; }
    tc_fence_after();
    const uint32_t d = tmem_base + acc * BN;
    for (int kb = w.kb0; kb < w.kb1; ++kb) {
      if (!mbar_wait_warp(&s.full[stage], phase, p.status, kTimeoutSmemFull, s.abort)) { ok = false; break; }
      tc_fence_after();
      const uint32_t sa = smem_u32(s.a + stage * A2_BYTES);
      const uint32_t sb = smem_u32(s.b + stage * B2_BYTES);
      if (issuer) {
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {
          const uint64_t da = make_smem_desc(sa + k * a_kadv, a_lbo, a_sbo);
          const uint64_t db = make_smem_desc(sb + k * b_kadv, b_lbo, b_sbo);
          umma_f16_ss_pair(d, da, db, idesc, ((kb - w.kb0) | k) != 0);
        }
        umma_commit_pair(&s.empty[stage], kPairMask);
      }
      __syncwarp();
      if (++stage == STAGES2) { stage = 0; phase ^= 1; }
    }
    if (!ok) break;
    if (issuer) umma_commit_pair(&s.tmem_full[acc], kPairMask);
    __syncwarp();
    if (++acc == 2) { acc = 0; acc_phase ^= 1; }
  }
  if (!ok) *s.abort = 1;
}

// Epilogue.  tcgen05.ld hands every thread one accumulator ROW (32 consecutive columns), but a row per thread is the
// wrong shape for global memory, so each warp turns its blocks through shared memory.
//
// Plain 16-bit and fp32 stores: 32 rows x 128 bytes are written to the warp's stage in the layout of the 128-byte
// swizzle, eight conflict-free 16-byte stores per thread, and leave as one TMA store that clips at the matrix' edges.
// Accumulating modes, a C that no tensor map covers and the ragged end of an expert's rows: a 32 x 32 fp32 block at a time
// through the same stage (conflict-free 16-byte accesses both ways), eight lanes on 32 consecutive columns of a row, four
// elements each, all loads of a block before its first store.
//
// What an epilogue costs is instructions, not bytes, and every decision that can be taken once per tile is taken there:
// whether there is a bias, the output mode, whole or clipped blocks.  Decided per element they were 64 branches around
// loads that never ran, 2700 cycles of a 64-column block (by clock64()), 5.6 us of every tile: 256 x 256 x 64 12.9 us,
// 8192 x 8192 x 512 111 us.
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ float4 lds128(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// H warps share 32 rows: the one with number h takes the blocks h, h + H, ...
struct Share {
  int h, H;
};
// Columns of a block: 128 bytes of a row where C leaves by TMA, else 32.  The parts of a shared tile are stored in the same
// blocks, because a warp that adds them has counted the arrivals of the warps of its own number alone.
__host__ __device__ constexpr int block_columns(bool tma, int out_mode) { return tma && out_mode == kOutBf16 ? 64 : 32; }

// w: the 128 bytes of this thread's row, to columns col0.. of rows y0 .. y0 + 31 of the map.
// Bulk groups belong to a thread: lane 0 issues and waits.
__device__ __forceinline__ void tma_store_rows(const CUtensorMap* tm, uint32_t buf, const uint32_t (&w)[32], int col0, int y0) {
  const uint32_t lane = lane_id();
  if (lane == 0) tma_store_wait_read<0>();          // the last store has left the stage
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 8; ++j)
    sts128(buf + sw128_offset(lane, j), w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                 :
                 : "l"(reinterpret_cast<uint64_t>(tm)), "r"(buf), "r"(col0), "r"(y0)
                 : "memory");
    tma_store_commit();
  }
}

// The slices of a shared tile (n = 0: a tile of one pair), all of them in memory by the time that they are added: the last slice
// first, then the others in order, whoever adds them.
struct Parts {
  const float* base;
  int n, warp8, bn;
  __device__ __forceinline__ void add(int c, uint32_t (&r)[32]) const {
    if (n == 0) return;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float4 v = part(n - 1, c, q);
      r[4 * q] = __float_as_uint(v.x);
      r[4 * q + 1] = __float_as_uint(v.y);
      r[4 * q + 2] = __float_as_uint(v.z);
      r[4 * q + 3] = __float_as_uint(v.w);
    }
#pragma unroll 1
    for (int k = 0; k + 1 < n; ++k) {
      float4 v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = part(k, c, q);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        r[4 * q] = __float_as_uint(__uint_as_float(r[4 * q]) + v[q].x);
        r[4 * q + 1] = __float_as_uint(__uint_as_float(r[4 * q + 1]) + v[q].y);
        r[4 * q + 2] = __float_as_uint(__uint_as_float(r[4 * q + 2]) + v[q].z);
        r[4 * q + 3] = __float_as_uint(__uint_as_float(r[4 * q + 3]) + v[q].w);
      }
    }
  }

 private:
  __device__ __forceinline__ float4 part(int k, int c, int q) const {
    return __ldcg(reinterpret_cast<const float4*>(base + size_t(k) * (CM * bn) + split_word(bn, warp8, c, q)));
  }
};

// One lane, once a warp's part is stored and fenced: whether it is the last of the tile's slices to arrive at `word`.  Whatever the
// word held before this launch is not its token; the last to arrive clears it, since a replayed graph's token is the same.
__device__ __forceinline__ bool split_arrive(unsigned long long* word, unsigned long long token, int slices) {
  unsigned long long seen = *reinterpret_cast<volatile unsigned long long*>(word);
  for (int i = 0; i < slices; ++i) {                   // a slice arrives once, so that no more than slices - 1 tries can fail
    const unsigned long long next = (seen & ~kSplitCountMask) == token ? seen + 1 : token + 1;
    const unsigned long long was = atomicCAS(word, seen, next);
    if (was == seen) {
      if (int(next & kSplitCountMask) != slices) return false;
      *word = 0;
      return true;
    }
    seen = was;
  }
  return false;
}

// The bias of N consecutive columns from col0 on, added to a thread's row.  Every lane reads the same 16 bytes.
template <int N>
__device__ __forceinline__ void add_bias_row(const Params& p, int col0, uint32_t* r) {
  const hg_lp_t* src = p.bias + col0;
  if (col0 + N <= p.N && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
    for (int q = 0; q < N / 8; ++q) {
      const uint4 u = reinterpret_cast<const uint4*>(src)[q];
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 b = hg_unpack2(w[j]);
        r[q * 8 + 2 * j] = __float_as_uint(__uint_as_float(r[q * 8 + 2 * j]) + b.x);
        r[q * 8 + 2 * j + 1] = __float_as_uint(__uint_as_float(r[q * 8 + 2 * j + 1]) + b.y);
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (col0 + i < p.N) r[i] = __float_as_uint(__uint_as_float(r[i]) + hg_lp2f(src[i]));
  }
}

// A 32 x 64 block from registers (thread = row) through the tensor map.
template <bool BIAS>
__device__ __forceinline__ void store_block64_tma(const Params& p, const CUtensorMap* tm, uint32_t stg, int y0, int col0,
                                                  uint32_t (&r0)[32], uint32_t (&r1)[32]) {
  if (BIAS) {
    add_bias_row<32>(p, col0, r0);
    add_bias_row<32>(p, col0 + 32, r1);
  }
  uint32_t w[32];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    w[i] = pack_bf16(__uint_as_float(r0[2 * i]), __uint_as_float(r0[2 * i + 1]));
    w[16 + i] = pack_bf16(__uint_as_float(r1[2 * i]), __uint_as_float(r1[2 * i + 1]));
  }
  tma_store_rows(tm, stg, w, col0, y0);
}

// Columns n0.. of the tile as TMA stores of 128-byte rows: 64 columns of 16 bits, or 32 of fp32.
template <bool BIAS, bool F32>
__device__ __forceinline__ void store_tile_tma(const Params& p, const CUtensorMap* tmC, uint32_t stg, Share w, uint32_t src, int row0,
                                               int y0, int n0, const Parts& parts) {
  constexpr int kBlock = block_columns(true, F32 ? kOutF32 : kOutBf16);
#pragma unroll 1
  for (int c = w.h * kBlock; c < p.bn && n0 + c < p.N; c += w.H * kBlock) {
    uint32_t r0[32], r1[32];
    tmem_ld32(src + c, r0);
    if (!F32) tmem_ld32(src + c + 32, r1);
    tmem_ld_wait();
    if (!HG_BOUNDS_OK(row0 >= 0 && row0 < p.M, p.status)) continue;
    parts.add(c / 32, r0);
    if (!F32) parts.add(c / 32 + 1, r1);
    if constexpr (F32) {
      if (BIAS) add_bias_row<32>(p, n0 + c, r0);
      tma_store_rows(tmC, stg, r0, n0 + c, y0);
    } else {
      store_block64_tma<BIAS>(p, tmC, stg, y0, n0 + c, r0, r1);
    }
  }
}

// Row by row: lane l works on columns 4 (l % 8) .. + 3 of rows l / 8, l / 8 + 4, ... of a 32 x 32 block.
// Whether those four elements can move as one access (C and its pitch multiples of four elements).
__device__ __forceinline__ bool four_aligned(const Params& p) {
  const uint32_t es = p.out_mode == kOutBf16 || p.out_mode == kOutBf16Acc ? 2 : 4;
  return (reinterpret_cast<uintptr_t>(p.C) & (4 * es - 1)) == 0 && (p.ldc & 3) == 0;
}

// What the accumulating modes add to a block (zeros otherwise): all loads in flight together.
__device__ __forceinline__ void load_old(const Params& p, int row0, int col0, float4 (&old)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) old[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (p.out_mode != kOutF32Acc && p.out_mode != kOutBf16Acc) return;
  const int lane = int(lane_id()), col = col0 + (lane & 7) * 4, rows = p.M - row0;
  const bool vec = four_aligned(p) && col + 3 < p.N;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + (lane >> 3);
    if (r >= rows) continue;
    const size_t at = size_t(row0 + r) * p.ldc + col;
    if (p.out_mode == kOutF32Acc) {
      const float* c = reinterpret_cast<const float*>(p.C) + at;
      if (vec) {
        old[i] = *reinterpret_cast<const float4*>(c);
      } else {
        float* o = reinterpret_cast<float*>(&old[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (col + j < p.N) o[j] = c[j];
      }
    } else {
      const hg_lp_t* c = reinterpret_cast<const hg_lp_t*>(p.C) + at;
      if (vec) {
        const uint2 u = *reinterpret_cast<const uint2*>(c);
        const float2 lo = hg_unpack2(u.x), hi = hg_unpack2(u.y);
        old[i] = make_float4(lo.x, lo.y, hi.x, hi.y);
      } else {
        float* o = reinterpret_cast<float*>(&old[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (col + j < p.N) o[j] = hg_lp2f(c[j]);
      }
    }
  }
}

// One 32 x 32 block from registers (thread = row), any output mode.
__device__ __forceinline__ void store_block_rows(const Params& p, uint32_t stg, int row0, int col0, const uint32_t (&src)[32],
                                                 const float4 (&old)[8]) {
  const int lane = int(lane_id());
#pragma unroll
  for (int j = 0; j < 8; ++j)
    sts128(stg + sw128_offset(lane, j), src[4 * j], src[4 * j + 1], src[4 * j + 2], src[4 * j + 3]);
  __syncwarp();
  const int q = (lane & 7) * 4, col = col0 + q;
  float4 v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = lds128(stg + sw128_offset(i * 4 + (lane >> 3), lane & 7));
  __syncwarp();
  if (!HG_BOUNDS_OK(row0 >= 0 && row0 < p.M && col0 >= 0 && col0 < p.N, p.status)) return;
  if (col >= p.N) return;
  float b[4] = {0.f, 0.f, 0.f, 0.f};
  if (p.bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (col + j < p.N) b[j] = hg_lp2f(p.bias[col + j]);
  }
  const bool vec = four_aligned(p) && col + 3 < p.N;
  const int rows = p.M - row0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + (lane >> 3);
    if (r >= rows) continue;
    const float o[4] = {v[i].x + b[0] + old[i].x, v[i].y + b[1] + old[i].y, v[i].z + b[2] + old[i].z, v[i].w + b[3] + old[i].w};
    const size_t at = size_t(row0 + r) * p.ldc + col;
    if (p.out_mode == kOutBf16 || p.out_mode == kOutBf16Acc) {
      hg_lp_t* c = reinterpret_cast<hg_lp_t*>(p.C) + at;
      if (vec) {
        *reinterpret_cast<uint2*>(c) = make_uint2(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]));
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (col + j < p.N) c[j] = hg_f2lp(o[j]);
      }
    } else {
      float* c = reinterpret_cast<float*>(p.C) + at;
      if (vec) {
        *reinterpret_cast<float4*>(c) = make_float4(o[0], o[1], o[2], o[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (col + j < p.N) c[j] = o[j];
      }
    }
  }
}

// One whole 32 x 32 block from registers (thread = row): no edge in it, four elements per access.
template <int MODE>
__device__ __forceinline__ void store_block_whole(const Params& p, uint32_t stg, int row0, int col0, const uint32_t (&src)[32],
                                                  const float4 (&old)[8]) {
  const int lane = int(lane_id());
#pragma unroll
  for (int j = 0; j < 8; ++j)
    sts128(stg + sw128_offset(lane, j), src[4 * j], src[4 * j + 1], src[4 * j + 2], src[4 * j + 3]);
  __syncwarp();
  const int q = (lane & 7) * 4;
  float4 v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = lds128(stg + sw128_offset(i * 4 + (lane >> 3), lane & 7));
  __syncwarp();
  if (!HG_BOUNDS_OK(row0 >= 0 && row0 + 32 <= p.M && col0 >= 0 && col0 + 32 <= p.N, p.status)) return;
  float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
  if (p.bias != nullptr)
    b = make_float4(hg_lp2f(p.bias[col0 + q]), hg_lp2f(p.bias[col0 + q + 1]), hg_lp2f(p.bias[col0 + q + 2]),
                    hg_lp2f(p.bias[col0 + q + 3]));
  const size_t at = size_t(row0 + (lane >> 3)) * p.ldc + col0 + q, step = size_t(4) * p.ldc;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float4 o = make_float4(v[i].x + b.x, v[i].y + b.y, v[i].z + b.z, v[i].w + b.w);
    if (MODE == kOutF32Acc || MODE == kOutBf16Acc) {
      o.x += old[i].x; o.y += old[i].y; o.z += old[i].z; o.w += old[i].w;
    }
    if (MODE == kOutBf16 || MODE == kOutBf16Acc)
      *reinterpret_cast<uint2*>(reinterpret_cast<hg_lp_t*>(p.C) + at + i * step) = make_uint2(pack_bf16(o.x, o.y), pack_bf16(o.z, o.w));
    else
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.C) + at + i * step) = o;
  }
}

template <int MODE>
__device__ __forceinline__ void load_old_whole(const Params& p, int row0, int col0, float4 (&old)[8]) {
  if (MODE != kOutF32Acc && MODE != kOutBf16Acc) return;
  const int lane = int(lane_id());
  const size_t at = size_t(row0 + (lane >> 3)) * p.ldc + col0 + (lane & 7) * 4, step = size_t(4) * p.ldc;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (MODE == kOutF32Acc) {
      old[i] = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.C) + at + i * step);
    } else {
      const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const hg_lp_t*>(p.C) + at + i * step);
      const float2 lo = hg_unpack2(u.x), hi = hg_unpack2(u.y);
      old[i] = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
  }
}

// This warp's whole blocks of a tile part.
template <int MODE>
__device__ __forceinline__ void store_tile_whole(const Params& p, uint32_t stg, Share w, uint32_t src, int row0, int n0, const Parts& parts) {
  const int cols = min(p.bn, (p.N - n0) & ~31);
#pragma unroll 1
  for (int c = w.h * 32; c < cols; c += w.H * 32) {
    float4 old[8];
    load_old_whole<MODE>(p, row0, n0 + c, old);
    uint32_t r0[32];
    tmem_ld32(src + c, r0);
    tmem_ld_wait();
    parts.add(c / 32, r0);
    store_block_whole<MODE>(p, stg, row0, n0 + c, r0, old);
  }
}

// This warp's blocks of the 32 x bn part of a tile that tensor memory holds at `src`: rows row0.. of C (p.M: the first row
// that is not this tile's), rows y0.. of the tensor map.
__device__ __forceinline__ void store_tile_part(const Params& p, const CUtensorMap* tmC, uint32_t stg, Share w, uint32_t src, int row0,
                                                int y0, int n0, bool whole_rows, const Parts& parts = Parts{nullptr, 0, 0, 0}) {
  if (p.c_tma && whole_rows) {
    if (p.out_mode == kOutF32) {
      if (p.bias != nullptr) store_tile_tma<true, true>(p, tmC, stg, w, src, row0, y0, n0, parts);
      else store_tile_tma<false, true>(p, tmC, stg, w, src, row0, y0, n0, parts);
    } else {
      if (p.bias != nullptr) store_tile_tma<true, false>(p, tmC, stg, w, src, row0, y0, n0, parts);
      else store_tile_tma<false, false>(p, tmC, stg, w, src, row0, y0, n0, parts);
    }
    return;
  }
  if (p.c_tma) {                                    // the stage is about to be written past the store that reads it
    if (lane_id() == 0) tma_store_wait_read<0>();
    __syncwarp();
  }
  int c0 = 0;
  if (row0 + 32 <= p.M && four_aligned(p)) {
    switch (p.out_mode) {
      case kOutF32: store_tile_whole<kOutF32>(p, stg, w, src, row0, n0, parts); break;
      case kOutF32Acc: store_tile_whole<kOutF32Acc>(p, stg, w, src, row0, n0, parts); break;
      case kOutBf16Acc: store_tile_whole<kOutBf16Acc>(p, stg, w, src, row0, n0, parts); break;
      default: store_tile_whole<kOutBf16>(p, stg, w, src, row0, n0, parts); break;
    }
    c0 = max(min(p.bn, (p.N - n0) & ~31), 0);       // the columns that are left: one block that the edge of C cuts
  }
#pragma unroll 1
  for (int c = c0 + (w.H - 1 - (c0 / 32 + w.H - 1 - w.h) % w.H) * 32; c < p.bn && n0 + c < p.N; c += w.H * 32) {
    float4 old[8];
    load_old(p, row0, n0 + c, old);
    uint32_t r0[32];
    tmem_ld32(src + c, r0);
    tmem_ld_wait();
    parts.add(c / 32, r0);
    store_block_rows(p, stg, row0, n0 + c, r0, old);
  }
}

// A turned tile part, 16-bit results: a lane holds one column of C, C[n0 + c, row0 + lane] for its columns c, so that a warp's values
// of one c are 32 consecutive elements and need no shared memory.  Neighbouring lanes trade a value, and each stores two columns of
// one row, 16 lanes a row and 64 bytes each.
__device__ __forceinline__ void store_tile_turned(const Params& p, Share w, uint32_t src, int row0, int n0, const Parts& parts) {
  const int lane = int(lane_id()), col = row0 + lane, odd = lane & 1;
  const bool mine = col < p.M;
  const float b = p.bias != nullptr && mine ? hg_lp2f(p.bias[col]) : 0.f;
#pragma unroll 1
  for (int c = w.h * 32; c < p.bn && n0 + c < p.N; c += w.H * 32) {
    uint32_t r[32];
    tmem_ld32(src + c, r);
    tmem_ld_wait();
    if (!HG_BOUNDS_OK(row0 >= 0 && row0 < p.M && n0 >= 0, p.status)) continue;
    parts.add(c / 32, r);
    const int rows = p.N - (n0 + c);
    hg_lp_t* at = reinterpret_cast<hg_lp_t*>(p.C) + size_t(n0 + c + odd) * p.ldc + (col - odd);
#pragma unroll
    for (int i = 0; i < 32; i += 2, at += size_t(2) * p.ldc) {
      const float x = __uint_as_float(r[i]) + b, y = __uint_as_float(r[i + 1]) + b;
      const float z = __shfl_xor_sync(0xffffffffu, odd ? x : y, 1);
      if (mine && i + odd < rows) *reinterpret_cast<uint32_t*>(at) = odd ? pack_bf16(z, y) : pack_bf16(x, z);
    }
  }
}

// H: epilogue warps per 32 rows, warps 2 .. 1 + 4 H of the block.
__device__ __forceinline__ void epilogue2(const Params& p, const CUtensorMap* tmC, const Smem2& s, uint32_t tmem_base,
                                          uint32_t rank, int H, int first, int step, int num_tiles) {
  const int wq = (threadIdx.x >> 5) & 3;
  const int lane = int(lane_id());
  const uint32_t lane_off = uint32_t(wq * 32) << 16;
  const int e = (threadIdx.x >> 5) - 2;
  const Share share{e / EPI_WARPS, H};
  const uint32_t stg = smem_u32(s.epi_stage + e * EPI_STAGE_FLOATS);
  uint32_t acc = 0, acc_phase = 0;
  const int num_kb = (p.K + BK - 1) / BK;
  const int n_units = unit_count(p, first, step, num_tiles);
  for (int u = 0; u < n_units; ++u) {
    const Unit w = unit_at(p, first, step, u, num_kb);
    const int tile = w.tile;
    int tm, tn;
    tile_coords(p, tile, tm, tn);
    const int row0 = tm * CM + int(rank) * BM + wq * 32;   // first of this warp's 32 rows
    const int n0 = tn * p.bn;
    // a tail tile shared with other pairs: whichever of them is done last adds the parts and writes it
    const bool shared_tile = p.split_s > 1 && tile >= p.split_tail_begin;
    const int tail_idx = tile - p.split_tail_begin, warp8 = int(rank) * EPI_WARPS + wq;
    float* ws_tile = shared_tile ? p.split_ws + size_t(tail_idx) * p.split_s * (CM * p.bn) : nullptr;
    const Parts parts{ws_tile, shared_tile ? p.split_s : 0, warp8, p.bn};
    if (!mbar_wait_warp(&s.tmem_full[acc], acc_phase, p.status, kTimeoutTmemFull, s.abort)) {
      *s.abort = 1;
      break;
    }
    tc_fence_after();
    const uint32_t src = tmem_base + lane_off + acc * BN;
    if (row0 < p.M) {   // warp-uniform, and the same for the slices of a tile
      bool writes = true;
      if (shared_tile) {
        // Nobody waits for another pair, whatever the order in which the device runs them.
        float* dst = ws_tile + size_t(w.slice) * (CM * p.bn);
        const int cols = block_columns(p.c_tma != 0, p.out_mode);          // bn is a multiple of it
#pragma unroll 1
        for (int c0 = share.h * cols; c0 < p.bn; c0 += H * cols)
#pragma unroll 1
          for (int c = c0; c < c0 + cols; c += 32) {
            uint32_t r0[32];
            tmem_ld32(src + c, r0);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 8; ++q)
              __stcg(reinterpret_cast<uint4*>(dst + split_word(p.bn, warp8, c / 32, q)),
                     make_uint4(r0[4 * q], r0[4 * q + 1], r0[4 * q + 2], r0[4 * q + 3]));
          }
        __threadfence();
        __syncwarp();
        int last = 0;
        if (lane == 0) last = split_arrive(p.split_words + size_t(tail_idx) * kSplitWords + share.h * 8 + warp8, p.split_token, p.split_s);
        writes = __shfl_sync(0xffffffffu, last, 0) != 0;
        __threadfence();                  // the other slices' parts are read after their arrivals
      }
      if (writes && p.turned) store_tile_turned(p, share, src, row0, n0, parts);
      else if (writes) store_tile_part(p, tmC, stg, share, src, row0, row0, n0, true, parts);
    }
    tc_fence_before();
    // the accumulator buffer is free again once all epilogue threads of the pair have read it
    if (rank == 0) mbar_arrive(&s.tmem_empty[acc]);
    else mbar_arrive_cluster(map_to_cta(smem_u32(&s.tmem_empty[acc]), 0));
    if (++acc == 2) { acc = 0; acc_phase ^= 1; }
  }
  if (p.c_tma && lane == 0) tma_store_wait<0>();     // shared memory is released after this
}


}  // namespace gemm2
}  // namespace hg
