// bf16 GEMM on CTA pairs: tcgen05.mma.cta_group::2 with a 256 x 256 x 64 tile per two-SM cluster.
//
// Compared with the one-CTA kernel (gemm.cu, 128 x 256 tile per SM) each SM stages only half of the B tile: the
// pair's MMA reads A rows [0,128) / [128,256) from the two CTAs' shared memory and the two halves of B's N range
// from both, so a 128 x 256 slice of the output costs 32 KB of operand traffic per k-block per SM instead of 48 KB,
// and six stages fit where four did.
//
// Roles per CTA (192 or 320 threads): warp 0 TMA producer (the warp walks the loop, one elected lane issues), warp 1 TMEM allocator (+ UMMA issuer in the leader
// CTA only: the warp walks the loop, one elected lane issues), warps 2-5 or 2-9 epilogue.  Barriers (same shared-memory offsets in both CTAs):
//   full[s]        leader only; the leader's producer arrives with the byte count of BOTH CTAs' loads, every load
//                  (from either CTA) completes its bytes on the leader's barrier
//   empty[s]       both CTAs; signalled by tcgen05.commit with a cluster mask covering the pair
//   tmem_full[a]   both CTAs; same mechanism, once per tile
//   tmem_empty[a]  leader only; all epilogue threads of the pair arrive (the peer's through its cluster address)
// Every wait is bounded (2 s); a CTA that gives up raises its abort flag and the status word, its partner runs into
// its own limit, and both still meet at the final cluster barrier and free their tensor memory.
// No operand load uses cluster multicast: each CTA loads exactly the bytes it alone needs.
#include <atomic>
#include <chrono>
#include <cstdlib>
#include <utility>

#include "gemm2_core.cuh"

namespace hg {
namespace gemm2 {

constexpr int kThreads2 = 64 + 32 * EPI2_WARPS;      // at most; see threads_for

// Barriers, tensor memory and the first meeting of the pair; returns the tensor-memory base address.
__device__ __forceinline__ uint32_t pair_setup(const Smem2& s, const CUtensorMap* tmA, const CUtensorMap* tmB, int warp) {
  if (threadIdx.x == 0) {
    tma_prefetch_desc(tmA);
    tma_prefetch_desc(tmB);
#pragma unroll
    for (int i = 0; i < STAGES2; ++i) {
      mbar_init(&s.full[i], 1);
      mbar_init(&s.empty[i], 1);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s.tmem_full[i], 1);
      mbar_init(&s.tmem_empty[i], 2 * (blockDim.x - 64));
    }
    *s.abort = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(s.tmem_base, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the partner's barriers exist before anything arrives on them remotely
  tc_fence_after();
  return *s.tmem_base;
}

__device__ __forceinline__ void pair_teardown(uint32_t tmem_base, int warp) {
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA frees tensor memory or leaves while its partner may still touch it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kThreads2, 1)
gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                  const __grid_constant__ CUtensorMap tmC, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  Smem2 s = carve2(smem_raw);
  const int warp = threadIdx.x >> 5;
  const uint32_t rank = cluster_ctarank();
  const int num_tiles = p.tiles_m * p.tiles_n;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  const uint32_t tmem_base = pair_setup(s, &tmA, &tmB, warp);
  chain_release();                            // after the allocation: see chain_release
  chain_wait();

  if (warp == 0) {
    producer2<A_MN, B_MN>(&tmA, &tmB, p, s, rank, pair, pairs, num_tiles);
  } else if (warp == 1) {
    if (rank == 0) mma2<A_MN, B_MN>(p, s, tmem_base, pair, pairs, num_tiles);
  } else {
    epilogue2(p, &tmC, s, tmem_base, rank, int(blockDim.x - 64) / (32 * EPI_WARPS), pair, pairs, num_tiles);
  }

  pair_teardown(tmem_base, warp);
}

// ---- grouped products on the pair's tile (mixture-of-experts layers) ------------------------------------------------
// One launch for the G products of a layer whose sizes only the device knows.  Every role of every pair walks the same
// tile list; `fn(tile)` returns false to stop.
struct GroupedTile {
  int m, m_end, n;        // first row and column of the output tile; rows from m_end on are another group's
  int a_k, b_off;         // offsets into the stacked operands (see the loads below)
  int num_kb;
  int c_row;              // row of the tensor map of C at which this group's rows start
  long long c_off;        // elements of C before this group
  int bn;                 // columns of the tile
};

// C[r0:r1] = A[r0:r1] op(B_g) for the row segments [r0, r1) = row_start[g..g+1].  Inside a segment up to eight row tiles
// of one column tile come first: the weight is then read from HBM once by the pairs that need it at the same time, and
// A, whose eight tiles fit the L2, is what is re-read.  (Walking the columns first streamed an expert's whole weight
// once per row tile.)
struct RowSegments {
  const int* row_start;
  int G, tiles_n, num_kb, b_group_rows, max_rows;
  int* status;
  static constexpr int kGroupM = 8;
  static constexpr bool kTurned = false;
  template <typename F>
  __device__ __forceinline__ void walk(int pair, int pairs, F&& fn) const {
    int counter = 0;
    for (int g = 0; g < G; ++g) {
      const int r0 = row_start[g], r1 = row_start[g + 1];
      // an expert's row range must lie inside the operand and not run backwards (checked in the debug build)
      if (!HG_BOUNDS_OK(r0 >= 0 && r1 >= r0 && r1 <= max_rows, status)) return;
      const int tm_cnt = (r1 - r0 + CM - 1) / CM, cnt = tm_cnt * tiles_n;
      for (int t = (pair - counter % pairs + pairs) % pairs; t < cnt; t += pairs) {
        const int first = t / (kGroupM * tiles_n) * kGroupM, gsize = min(kGroupM, tm_cnt - first);
        const int r = t - first * tiles_n;
        GroupedTile w{r0 + (first + r % gsize) * CM, r1, r / gsize * BN, 0, g * b_group_rows, num_kb, 0, 0, BN};
        if (!fn(w)) return;
      }
      counter += cnt;
    }
  }
};

// The same products with A and B in each other's place: a tile is 256 columns of C (rows of the weight) by up to 256 rows of a
// segment, which is cut into as few equal tiles as it takes, of a multiple of 64 rows each.  Tiles of 256 rows of C by 256
// columns were one in eight padding at segments of about 1024 ragged rows.  Up to kGroupN tiles along the rows are walked
// together, piece of the weight by piece, so that both operands are reused out of L2: with all of a segment's tiles together, more
// rows than L2 holds came from HBM again for every few pieces (sustained, us, all / 8 / 4 together: 16384 rows, 28672 columns, K = 4096
// 3520 / 2855 / 2918; 8192 rows, 4096 columns, K = 14336 786 / 734 / 729; 8 x (4096, 28672, 4096) 5853 / 5979 / 6123).
struct TurnedSegments {
  const int* row_start;
  int G, tiles_m, num_kb, w_group_rows, max_rows;
  int* status;
  static constexpr int kGroupN = 8;
  static constexpr bool kTurned = true;
  template <typename F>
  __device__ __forceinline__ void walk(int pair, int pairs, F&& fn) const {
    int counter = 0;
    for (int g = 0; g < G; ++g) {
      const int r0 = row_start[g], r1 = row_start[g + 1], rows = r1 - r0;
      if (!HG_BOUNDS_OK(r0 >= 0 && r1 >= r0 && r1 <= max_rows, status)) return;
      if (rows <= 0) continue;
      const int pieces = (rows + BN - 1) / BN, bn = ((rows + pieces - 1) / pieces + 63) / 64 * 64;
      const int tn = (rows + bn - 1) / bn, cnt = tn * tiles_m;
      for (int t = (pair - counter % pairs + pairs) % pairs; t < cnt; t += pairs) {
        const int first = t / (kGroupN * tiles_m) * kGroupN, gsize = min(kGroupN, tn - first);
        const int r = t - first * tiles_m;
        GroupedTile w{r / gsize * CM, r1, r0 + (first + r % gsize) * bn, 0, g * w_group_rows, num_kb, 0, 0, bn};
        if (!fn(w)) return;
      }
      counter += cnt;
    }
  }
};

// C_g (+)= A[k0:k1]^T B[k0:k1] for the contraction ranges [k0, k1) = k_start[g..g+1] (multiples of 64).
struct ContractionRanges {
  const int* k_start;
  int G, tiles_m, tiles_n, M;
  long long c_group_stride;
  static constexpr int kGroupM = 4;
  static constexpr bool kTurned = false;
  template <typename F>
  __device__ __forceinline__ void walk(int pair, int pairs, F&& fn) const {
    const int per = tiles_m * tiles_n;
    for (int t = pair; t < per * G; t += pairs) {
      const int g = t / per, u = t - g * per;
      const int first = u / (kGroupM * tiles_n) * kGroupM, gsize = min(kGroupM, tiles_m - first);
      const int r = u - first * tiles_n;
      const int k0 = k_start[g];
      GroupedTile w{(first + r % gsize) * CM, M, r / gsize * BN, k0, k0, (k_start[g + 1] - k0 + BK - 1) / BK,
                    g * M, g * c_group_stride, BN};
      if (!fn(w)) return;
    }
  }
};

template <bool A_MN, bool B_MN, typename Tiles>
__global__ void __launch_bounds__(kThreads2, 1)
grouped_gemm2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, const Params p, const Tiles tiles) {
  extern __shared__ uint8_t smem_raw[];
  Smem2 s = carve2(smem_raw);
  const int warp = threadIdx.x >> 5;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const uint32_t tmem_base = pair_setup(s, &tmA, &tmB, warp);
  chain_release();                            // after the allocation: see chain_release
  chain_wait();

  if (warp == 0) {
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    const bool issuer = elect_one() != 0;
    tiles.walk(pair, pairs, [&](const GroupedTile& w) {
      const int half = w.bn / 2, m = w.m + int(rank) * BM, n = w.n + int(rank) * half;
      for (int kb = 0; kb < w.num_kb; ++kb) {
        if (!mbar_wait_warp(&s.empty[stage], phase ^ 1, p.status, kTimeoutSmemEmpty, s.abort)) { ok = false; return false; }
        const uint32_t bar = map_to_cta(smem_u32(&s.full[stage]), 0);
        uint8_t* sa = s.a + stage * A2_BYTES;
        uint8_t* sb = s.b + stage * B2_BYTES;
        const int k0 = kb * BK;
        if (issuer) {
          if (rank == 0) mbar_expect_tx(&s.full[stage], 2 * (A2_BYTES + half * BK * 2));
          const int a_off = Tiles::kTurned ? w.b_off : w.a_k;      // the weight is the stacked operand
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * SLAB_BYTES, &tmA, bar, m + j * 64, a_off + k0);
          } else {
            tma_load_2d_pair(sa, &tmA, bar, k0, Tiles::kTurned ? a_off + m : m);
          }
          if (B_MN) {
#pragma unroll
            for (int j = 0; j < HALF_N / 64; ++j) tma_load_2d_pair(sb + j * SLAB_BYTES, &tmB, bar, n + j * 64, w.b_off + k0);
          } else if (Tiles::kTurned) {
#pragma unroll
            for (int j = 0; j < HALF_N / 32; ++j)
              if (j * 32 < half) tma_load_2d_pair(sb + j * (32 * BK * 2), &tmB, bar, k0, n + j * 32);
          } else {
            tma_load_2d_pair(sb, &tmB, bar, k0, w.b_off + n);
          }
        }
        __syncwarp();
        if (++stage == STAGES2) { stage = 0; phase ^= 1; }
      }
      return true;
    });
    for (int i = 0; ok && i < STAGES2; ++i) {       // as in producer2
      ok = mbar_wait_warp(&s.empty[stage], phase ^ 1, p.status, kTimeoutSmemEmpty, s.abort);
      if (++stage == STAGES2) { stage = 0; phase ^= 1; }
    }
    if (!ok) {
      *s.abort = 1;
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);  // 2 ms: far longer than a tile load
    }
  } else if (warp == 1) {
    if (rank == 0) {
      constexpr uint32_t a_lbo = A_MN ? SLAB_BYTES : 16, a_kadv = A_MN ? 2048 : 32;
      constexpr uint32_t b_lbo = B_MN ? SLAB_BYTES : 16, b_kadv = B_MN ? 2048 : 32;
      uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
      bool ok = true;
      const bool issuer = elect_one() != 0;
      tiles.walk(pair, pairs, [&](const GroupedTile& w) {
        if (w.num_kb <= 0) return true;   // nothing to contract: the epilogue writes the result
        if (!mbar_wait_warp(&s.tmem_empty[acc], acc_phase ^ 1, p.status, kTimeoutTmemEmpty, s.abort)) { ok = false; return false; }
        tc_fence_after();
        const uint32_t d = tmem_base + acc * BN, idesc = make_idesc_lp(CM, w.bn, A_MN, B_MN);
        for (int kb = 0; kb < w.num_kb; ++kb) {
          if (!mbar_wait_warp(&s.full[stage], phase, p.status, kTimeoutSmemFull, s.abort)) { ok = false; return false; }
          tc_fence_after();
          const uint32_t sa = smem_u32(s.a + stage * A2_BYTES);
          const uint32_t sb = smem_u32(s.b + stage * B2_BYTES);
          if (issuer) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_f16_ss_pair(d, make_smem_desc(sa + k * a_kadv, a_lbo, 1024), make_smem_desc(sb + k * b_kadv, b_lbo, 1024),
                               idesc, (kb | k) != 0);
            umma_commit_pair(&s.empty[stage], kPairMask);
          }
          __syncwarp();
          if (++stage == STAGES2) { stage = 0; phase ^= 1; }
        }
        if (issuer) umma_commit_pair(&s.tmem_full[acc], kPairMask);
        __syncwarp();
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        return true;
      });
      if (!ok) *s.abort = 1;
    }
  } else {
    const int wq = warp & 3, lane = int(lane_id());
    const uint32_t lane_off = uint32_t(wq * 32) << 16;
    const int e = warp - 2;
    const Share share{e / EPI_WARPS, int(blockDim.x - 64) / (32 * EPI_WARPS)};
    const uint32_t stg = smem_u32(s.epi_stage + e * EPI_STAGE_FLOATS);
    uint32_t acc = 0, acc_phase = 0;
    tiles.walk(pair, pairs, [&](const GroupedTile& w) {
      const int row0 = w.m + int(rank) * BM + wq * 32;
      Params q = p;
      if (Tiles::kTurned) {
        q.bn = w.bn;
        q.N = w.m_end;
        if (!mbar_wait_warp(&s.tmem_full[acc], acc_phase, p.status, kTimeoutTmemFull, s.abort)) { *s.abort = 1; return false; }
        tc_fence_after();
        if (row0 < q.M) store_tile_turned(q, share, tmem_base + lane_off + acc * BN, row0, w.n, Parts{nullptr, 0, 0, 0});
        tc_fence_before();
        if (rank == 0) mbar_arrive(&s.tmem_empty[acc]);
        else mbar_arrive_cluster(map_to_cta(smem_u32(&s.tmem_empty[acc]), 0));
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        return true;
      }
      q.M = w.m_end;
      q.C = p.out_mode == kOutF32 || p.out_mode == kOutF32Acc ? static_cast<void*>(reinterpret_cast<float*>(p.C) + w.c_off)
                                                              : static_cast<void*>(reinterpret_cast<hg_lp_t*>(p.C) + w.c_off);
      if (w.num_kb <= 0) {                          // nothing contracted: zeros (or C unchanged)
        if (p.c_tma) {
          if (lane == 0) tma_store_wait_read<0>();
          __syncwarp();
        }
        const uint32_t zero[32] = {};
        for (int c = share.h * 32; c < BN && row0 < w.m_end && w.n + c < p.N; c += share.H * 32) {
          float4 old[8];
          load_old(q, row0, w.n + c, old);
          store_block_rows(q, stg, row0, w.n + c, zero, old);
        }
        return true;
      }
      if (!mbar_wait_warp(&s.tmem_full[acc], acc_phase, p.status, kTimeoutTmemFull, s.abort)) { *s.abort = 1; return false; }
      tc_fence_after();
      if (row0 < w.m_end)   // warp-uniform; a block that reaches into the next group's rows is stored row by row
        store_tile_part(q, &tmC, stg, share, tmem_base + lane_off + acc * BN, row0, w.c_row + row0, w.n, row0 + 32 <= w.m_end);
      tc_fence_before();
      if (rank == 0) mbar_arrive(&s.tmem_empty[acc]);
      else mbar_arrive_cluster(map_to_cta(smem_u32(&s.tmem_empty[acc]), 0));
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      return true;
    });
    if (p.c_tma && lane == 0) tma_store_wait<0>();   // shared memory is released after this
  }
  pair_teardown(tmem_base, warp);
}

}  // namespace gemm2
}  // namespace hg

using namespace hg::gemm;
using namespace hg::gemm2;

namespace {

// HG_GEMM_SPLIT_TAIL: 0 never, 1 wherever a slice keeps eight k-blocks, unset: by the cost of the plan.
int split_mode() {
  static const int mode = [] {
    const char* e = getenv("HG_GEMM_SPLIT_TAIL");
    return e == nullptr || e[0] == 0 ? -1 : int(e[0] != '0');
  }();
  return mode;
}

// How a product is cut: columns of a tile, whether A and B change places (the tile's 256 rows are then columns of C and its `bn`
// columns rows of C), and how many pairs share each tile of the last wave (s < 2: none do), `tail` of them.
struct TilePlan {
  int bn, turned, s, tail;
  long long word_bytes() const { return ((long long)tail * kSplitWords * sizeof(unsigned long long) + 255) / 256 * 256; }
  long long bytes() const { return s < 2 ? 0 : word_bytes() + (long long)tail * s * (CM * bn) * sizeof(float); }
};

// Costs in cycles of 1.6 GHz, fitted to 50 products of the three layouts, 128 to 152064 rows and columns, K = 63 to 152064 (kStore
// later, by the two given beside it).
// A k-block moves 16 KB of A and 64 bn bytes of B into each SM, which takes 64 bytes a cycle from L2, and 2 bn cycles on the
// tensor core: 256 + bn cycles, in which narrower tiles leave the tensor core idle.
constexpr int kBlockCost = 256;
// With every SM at work for long it is the power limit that bounds, and with it the products themselves: 2 bn cycles of a
// k-block at five sixths of the clock, the part of the last wave that idles not counted (1554 x 37888, K = 3584: 1036 tiles of
// 256 columns 310 us, as many of 224 278, 1332 of 192 295).  An idle last wave still costs a little there: 4096 x 4096, K = 32000,
// 256 tiles 760 us, the last 34 shared by two 703.
// A tile's way out of tensor memory: it counts once per launch, and in every wave where it is longer than the products.  One
// tile of K = 512, bn = 64 to 256, us: 16 bits 6.0 to 8.1, fp32 7.7 to 11.2, turned 6.5 to 11.5.  A part is not the columns' (fp32,
// 11008 x 4096, K = 300, all stores, with one epilogue warp per 32 rows: bn = 256 50 us, bn = 128 62; 37888 x 3584, K = 63, 28 waves:
// 126 us and 103 with two, 5900 cycles a wave).
constexpr int kStore = 1400, kStore16 = 10, kStore32 = 21, kStoreTurned = 34, kTurned = 1000;
// A shared tile, per column: the parts' way to L2 and the arrivals, and each part that is added (200 x 3584, K = 18944: 256
// columns by five 52 us, 192 by three 44, not shared 89).
constexpr int kSplitCost = 48, kPartCost = 20;
// A plan other than whole tiles of 256 columns has to promise a gain of one part in this many: turned tiles, which never lost, and
// narrower ones that are not turned, whose small promises do not hold over several waves (of 2 to 6 % in the cost, us, whole / narrower:
// 12288 x 1600, K = 808 30.8 / 34.0, fp32 K = 1168 49.5 / 56.0, fp32 15360 x 3584, K = 72 46.8 / 48.9).
constexpr int kWorth = 64, kWorthNarrow = 20;

long long plan_cost(long long tiles, int num_kb, int pairs, int bn, int store, int s) {
  const long long main = num_kb * (kBlockCost + bn), epi = kStore + bn * store, wave = main > epi ? main : epi;
  const long long waves = tiles / pairs, tail = tiles % pairs;
  const long long power = tiles * num_kb * bn * 12 / (5 * pairs) + epi;
  long long cost = waves * wave + main + epi;
  if (tail == 0) cost = (waves - 1) * wave + main + epi;
  else if (s > 1) cost = waves * wave + (num_kb + s - 1) / s * (kBlockCost + bn) + bn * (kSplitCost + kPartCost * (s - 1)) + epi;
  return cost > power ? cost : (3 * power + cost) / 4;
}
int split_most(int tail, int num_kb, int pairs) {
  const int s = tail == 0 ? 0 : pairs / tail < num_kb / 8 ? pairs / tail : num_kb / 8;
  return s > int(kSplitCountMask) ? int(kSplitCountMask) : s;
}

// The cheapest cut of C[M, N] for `max_pairs` pairs.  What there is to gain: rows of tiles that hang over the edge of C (tokens
// are ragged, the columns of a weight hardly ever are: turned, the tokens are cut into equal tiles of as few columns as they
// need), a last wave with few tiles in it, and pairs without a tile.
TilePlan cheapest_plan(int M, int N, int K, bool wide, bool may_turn, int max_pairs) {
  const int num_kb = (K + BK - 1) / BK;
  TilePlan best{BN, 0, 0, 0};
  long long best_cost = 0, whole_cost = 0;              // whole: tiles of 256 columns, not turned, which come first
  for (int turned = 0; turned <= (may_turn ? 1 : 0); ++turned) {
    const int rows = turned ? N : M, cols = turned ? M : N;
    const int step = turned || wide ? 32 : 64;           // 16-bit blocks leave 64 columns at a time
    for (int bn = BN; bn >= 64; bn -= step) {
      const long long tiles = (long long)((rows + CM - 1) / CM) * ((cols + bn - 1) / bn);
      const int tail = int(tiles % max_pairs);
      const int store = turned ? kStoreTurned : wide ? kStore32 : kStore16;
      int most = split_mode() == 0 ? 0 : split_most(tail, num_kb, max_pairs), least = 0;
      if (split_mode() > 0 && most > 1) least = most = most > 4 ? 4 : most;
      long long before = 0;
      for (int s = least; s == 0 || s <= most; s += s == 0 ? 2 : 1) {
        const long long cost = plan_cost(tiles, num_kb, max_pairs, bn, store, s) + (turned ? kTurned : 0);
        if (s > 2 && cost > before && split_mode() < 0) break;      // more slices only cost more from here on
        before = cost;
        const bool first = best_cost == 0, whole = bn == BN && !turned;
        if (!turned && !whole && cost * kWorthNarrow >= whole_cost * (kWorthNarrow - 1)) continue;
        if (first || (whole ? cost < best_cost : cost * kWorth < best_cost * (kWorth - 1))) {
          if (whole) whole_cost = cost;
          best = TilePlan{bn, turned, s, tail};
          best_cost = cost;
        }
      }
    }
  }
  return best;
}

// The same; a thread's last few are kept, because the layers of a model ask for the same ones again and a search takes a
// microsecond or two.
TilePlan tile_plan(int M, int N, int K, int out_mode, bool may_turn, int max_pairs) {
  struct Kept {
    int m, n, k, kind, pairs;
    TilePlan plan;
  };
  constexpr unsigned kSlots = 64;
  static thread_local Kept kept[kSlots] = {};
  const bool wide = out_mode == kOutF32 || out_mode == kOutF32Acc;
  const int kind = wide ? 2 : may_turn ? 1 : 0;
  Kept& e = kept[(unsigned(M) * 31u + unsigned(N) * 17u + unsigned(K) / 8u * 7u + unsigned(kind)) % kSlots];
  if (e.m != M || e.n != N || e.k != K || e.kind != kind || e.pairs != max_pairs)
    e = Kept{M, N, K, kind, max_pairs, cheapest_plan(M, N, K, wide, !wide && may_turn, max_pairs)};
  return e.plan;
}

// Starts at the clock: no launch of this process has the token of another, and nothing here can throw at a C entry.
unsigned long long split_token() {
  constexpr unsigned long long kStep = kSplitCountMask + 1;
  static std::atomic<unsigned long long> next{
      (unsigned long long)std::chrono::system_clock::now().time_since_epoch().count() * kStep + kStep};
  return next.fetch_add(kStep, std::memory_order_relaxed);
}

}  // namespace

// Threads of a CTA: with two epilogue warps per 32 rows where a tile's way out counts beside its products, which take `main`
// cycles (see plan_cost), with one elsewhere: on large products, which the power limit bounds, the four more warps cost
// 1 to 3 % (sustained, us, one and two: 4096 x 32000, K = 4096 827 -> 850 us; 22016 x 4096, K = 8192, added to C 1217 -> 1258; 28672 x 4096, fp32, K = 1024 236 ->
// 238, K = 512 164 -> 157; added to C, K = 2048 460 -> 453).  16-bit results of two operands that are M- and N-major pay it sooner
// (4608 x 37888, K = 760 241 -> 257; 13824 x 27648, K = 800 545 -> 589; K = 520 and 640 still gain 3 to 4 %).
static int threads_for(int out_mode, long long main, bool mn) {
  const bool adds = out_mode == kOutF32Acc || out_mode == kOutBf16Acc;
  return main < (adds ? 20000 : mn && out_mode == kOutBf16 ? 5300 : 8000) ? kThreads2 : 64 + 32 * EPI_WARPS;
}

// Launch attributes of a kernel of CTA pairs, and how many pairs of it the device holds at once (-2: none).
template <typename K>
static int pair_config(K kernel, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int* max_pairs, bool overlaps, cudaStream_t st, int threads = kThreads2) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = 2;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg->blockDim = dim3(kThreads2, 1, 1);
  cfg->dynamicSmemBytes = SMEM2_BYTES;
  cfg->stream = st;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
  if (*max_pairs < 0) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM2_BYTES);
    if (e != cudaSuccess) return int(e);
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cfg->gridDim = dim3(unsigned(sms / 2 * 2), 1, 1);
    int n = 0;
    e = cudaOccupancyMaxActiveClusters(&n, kernel, cfg);
    if (e != cudaSuccess) return int(e);
    if (n <= 0) return -2;
    *max_pairs = n;
  }
  if (overlaps) cfg->numAttrs = 2;
  cfg->blockDim = dim3(unsigned(threads), 1, 1);
  return 0;
}

template <bool A_MN, bool B_MN, typename Tiles>
static int launch_grouped2(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const Params& p,
                           const Tiles& tiles, int want_pairs, int threads, cudaStream_t st) {
  static int max_pairs = -1;
  auto k = grouped_gemm2_kernel<A_MN, B_MN, Tiles>;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  if (int rc = pair_config(k, &cfg, attr, &max_pairs, hg_host::launch_overlaps(), st, threads)) return rc;
  const int pairs = want_pairs < max_pairs ? want_pairs : max_pairs;
  cfg.gridDim = dim3(unsigned(2 * pairs), 1, 1);
  return hg_host::launched(cudaLaunchKernelEx(&cfg, k, ta, tb, tc, p, tiles));
}

template <bool A_MN, bool B_MN>
static int launch2(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const Params& p_in, const TilePlan& plan,
                   int max_pairs, int want_pairs, void* ws, long long ws_bytes, cudaStream_t st) {
  Params p = p_in;
  static int co_resident = -1;
  auto k = gemm2_bf16_kernel<A_MN, B_MN>;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  const int threads = threads_for(p.out_mode, (long long)((p.K + BK - 1) / BK) * (kBlockCost + p.bn), A_MN && B_MN);
  if (int rc = pair_config(k, &cfg, attr, &co_resident, hg_host::launch_overlaps(), st, threads)) return rc;
  int pairs = want_pairs < co_resident ? want_pairs : co_resident;
  p.split_s = 0;
  if (ws != nullptr && plan.s > 1 && ws_bytes >= plan.bytes()) {     // see Params::split_s
    p.split_s = plan.s;
    p.split_tail_begin = p.tiles_m * p.tiles_n - plan.tail;
    p.split_words = static_cast<unsigned long long*>(ws);
    p.split_ws = reinterpret_cast<float*>(static_cast<char*>(ws) + plan.word_bytes());
    p.split_token = split_token();
    pairs = p.split_tail_begin > 0 ? max_pairs : plan.tail * plan.s;   // the plan's pairs, co-resident or not: none waits for another
  }
  cfg.gridDim = dim3(unsigned(2 * pairs), 1, 1);
  return hg_host::launched(cudaLaunchKernelEx(&cfg, k, ta, tb, tc, p));
}

// Pairs of the plain kernels that the device holds at once (the four layouts take the same shared memory and threads).
static int plain_pairs(int* pairs) {
  static int max_pairs = -1;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  const int rc = max_pairs > 0 ? 0 : pair_config(gemm2_bf16_kernel<false, false>, &cfg, attr, &max_pairs, false, nullptr);
  *pairs = max_pairs;
  return rc;
}

// The tensor map of C for the plain stores (p.c_tma says whether it is used; `any` fills the kernel's parameter else).
static int store_map(CUtensorMap* tc, const CUtensorMap& any, Params& p, uint64_t rows) {
  p.c_tma = 0;
  *tc = any;
  if (p.out_mode != kOutBf16 && p.out_mode != kOutF32) return 0;
  const int rc = p.out_mode == kOutF32 ? hg_host::make_tmap_2d_store_f32(tc, p.C, rows, uint64_t(p.N), uint64_t(p.ldc))
                                       : hg_host::make_tmap_2d_store(tc, p.C, rows, uint64_t(p.N), uint64_t(p.ldc));
  if (rc == 0) p.c_tma = 1;
  else *tc = any;
  return rc < 0 ? rc : 0;
}

// Whether C can be stored from turned tiles: 16-bit results, two of a row at a time.  (Turned fp32 tiles were up to half slower:
// 32000 x 5120, K = 670 219 -> 350 us.)
static bool turns(const void* C, int N, int ldc, int out_mode) {
  return out_mode == kOutBf16 && N % 2 == 0 && ldc % 2 == 0 && (reinterpret_cast<uintptr_t>(C) & 3) == 0;
}

extern "C" {

// Same contract as hg_gemm_bf16 (gemm.cu), computed by CTA pairs.  Returns -2 when the device cannot co-schedule a
// pair of these CTAs (the caller then uses the one-CTA kernel).
// ws: scratch of ws_bytes bytes, 256-byte aligned (contents do not matter); with less than hg_gemm2_scratch bytes every tile
// has one pair.
int hg_gemm2_bf16(const void* A, const void* B, void* C, const void* bias, int M, int N, int K, int lda, int ldb,
                  int ldc, int a_mn, int b_mn, int out_mode, int max_ctas, void* ws, long long ws_bytes, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda & 7) || (ldb & 7) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15))
    return -1;
  int max_pairs, rc = plain_pairs(&max_pairs);
  if (rc) return rc;
  TilePlan plan{BN, 0, 0, 0};
  if (max_ctas == 0) plan = tile_plan(M, N, K, out_mode, turns(C, N, ldc, out_mode), max_pairs);
  if (plan.turned) {
    std::swap(A, B);
    std::swap(M, N);
    std::swap(lda, ldb);
    std::swap(a_mn, b_mn);
  }
  CUtensorMap ta, tb;
  if (a_mn) rc = hg_host::make_tmap_2d_bf16(&ta, A, K, M, lda, 64, 64);
  else      rc = hg_host::make_tmap_2d_bf16(&ta, A, M, K, lda, BM, 64);
  if (rc) return rc;
  if (b_mn) rc = hg_host::make_tmap_2d_bf16(&tb, B, K, N, ldb, 64, 64);
  else      rc = hg_host::make_tmap_2d_bf16(&tb, B, N, K, ldb, plan.bn / 2, 64);
  if (rc) return rc;
  Params p{};
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.C = C;
  p.bias = reinterpret_cast<const hg_lp_t*>(bias);
  p.out_mode = out_mode;
  p.bn = plan.bn;
  p.turned = plan.turned;
  p.tiles_m = (M + CM - 1) / CM;
  p.tiles_n = (N + plan.bn - 1) / plan.bn;
  p.group_m = 4;
  p.status = hg_host::status_ptr();
  p.ready = nullptr; p.rows_per_flag = 1; p.ready_target = 0; p.m_tile_shift = 0;
  p.k_ranges = nullptr; p.groups = 1; p.c_group_stride = 0;
  int pairs = p.tiles_m * p.tiles_n;
  if (max_ctas > 1 && max_ctas / 2 < pairs) pairs = max_ctas / 2;
  CUtensorMap tc = ta;
  if (!plan.turned && (rc = store_map(&tc, ta, p, M))) return rc;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (a_mn && b_mn) return launch2<true, true>(ta, tb, tc, p, plan, max_pairs, pairs, ws, ws_bytes, st);
  if (a_mn) return launch2<true, false>(ta, tb, tc, p, plan, max_pairs, pairs, ws, ws_bytes, st);
  if (b_mn) return launch2<false, true>(ta, tb, tc, p, plan, max_pairs, pairs, ws, ws_bytes, st);
  return launch2<false, false>(ta, tb, tc, p, plan, max_pairs, pairs, ws, ws_bytes, st);
}

// How hg_gemm2_bf16 cuts a product for `pairs` pairs: columns of a tile, whether A and B change places (`may_turn`: if C allows it),
// pairs per tile of the last wave (below 2: one), its tiles, epilogue warps per 32 rows (`mn`: of M- and N-major operands).
// Needs no device.
int hg_gemm2_plan(int M, int N, int K, int out_mode, int may_turn, int mn, int pairs, int* plan) {
  const TilePlan t = tile_plan(M, N, K, out_mode, may_turn && out_mode == kOutBf16, pairs);
  const int threads = threads_for(out_mode, (long long)((K + BK - 1) / BK) * (kBlockCost + t.bn), mn);
  const int of_plan[5] = {t.bn, t.turned, t.s, t.tail, (threads - 64) / (32 * EPI_WARPS)};
  for (int i = 0; i < 5; ++i) plan[i] = of_plan[i];
  return 0;
}

// Bytes of scratch that hg_gemm2_bf16 may ask for on the current device, whatever the type of the result (0: none).
long long hg_gemm2_scratch(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  int max_pairs;
  if (plain_pairs(&max_pairs)) return 0;
  long long most = 0;
  for (int kind = 0; kind < 3; ++kind) {
    const long long need = tile_plan(M, N, K, kind == 2 ? kOutF32 : kOutBf16, kind == 1, max_pairs).bytes();
    if (need > most) most = need;
  }
  return most;
}

// Same contracts as hg_grouped_gemm_bf16 and hg_grouped_wgrad_bf16 (gemm.cu), computed by CTA pairs; -2 as above.
int hg_grouped_gemm2_bf16(const void* A, const void* B, void* C, const void* row_start, int G, int max_rows, int N,
                          int K, int lda, int ldb, int ldc, int b_mn, int out_mode, void* stream) {
  if (G <= 0 || max_rows <= 0) return 0;
  if ((lda & 7) || (ldb & 7)) return -1;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap ta, tb, tc;
  int rc;
  Params p{};
  p.K = K; p.ldc = ldc; p.C = C; p.out_mode = out_mode; p.bn = BN; p.status = hg_host::status_ptr();
  const int* starts = reinterpret_cast<const int*>(row_start);
  const int num_kb = (K + BK - 1) / BK, threads = threads_for(out_mode, (long long)num_kb * (kBlockCost + BN), false);
  if (turns(C, N, ldc, out_mode)) {
    p.M = N; p.N = max_rows;
    if (b_mn) rc = hg_host::make_tmap_2d_bf16(&ta, B, uint64_t(G) * K, N, ldb, 64, 64);
    else      rc = hg_host::make_tmap_2d_bf16(&ta, B, uint64_t(G) * N, K, ldb, BM, 64);
    if (!rc) rc = hg_host::make_tmap_2d_bf16(&tb, A, max_rows, K, lda, 32, 64);
    if (rc) return rc;
    const TurnedSegments t{starts, G, (N + CM - 1) / CM, num_kb, b_mn ? K : N, max_rows, p.status};
    return b_mn ? launch_grouped2<true, false>(ta, tb, ta, p, t, 1 << 20, threads, st)
                : launch_grouped2<false, false>(ta, tb, ta, p, t, 1 << 20, threads, st);
  }
  if ((rc = hg_host::make_tmap_2d_bf16(&ta, A, max_rows, K, lda, BM, 64))) return rc;
  if (b_mn) rc = hg_host::make_tmap_2d_bf16(&tb, B, uint64_t(G) * K, N, ldb, 64, 64);
  else      rc = hg_host::make_tmap_2d_bf16(&tb, B, uint64_t(G) * N, K, ldb, HALF_N, 64);
  if (rc) return rc;
  p.M = max_rows; p.N = N;
  RowSegments t{starts, G, (N + BN - 1) / BN, num_kb, b_mn ? K : N, max_rows, p.status};
  if ((rc = store_map(&tc, ta, p, max_rows))) return rc;
  return b_mn ? launch_grouped2<false, true>(ta, tb, tc, p, t, 1 << 20, threads, st)
              : launch_grouped2<false, false>(ta, tb, tc, p, t, 1 << 20, threads, st);
}

int hg_grouped_wgrad2_bf16(const void* dy, const void* x, void* out, const void* row_start, int G, int rows, int N,
                           int K, int lddy, int ldx, int out_mode, int max_ctas, void* stream) {
  if (G <= 0 || rows <= 0) return 0;
  if ((lddy & 7) || (ldx & 7)) return -1;
  CUtensorMap ta, tb;
  int rc = hg_host::make_tmap_2d_bf16(&ta, dy, rows, N, lddy, 64, 64);
  if (rc) return rc;
  rc = hg_host::make_tmap_2d_bf16(&tb, x, rows, K, ldx, 64, 64);
  if (rc) return rc;
  Params p{};
  p.M = N; p.N = K; p.K = rows; p.ldc = K; p.C = out; p.out_mode = out_mode; p.bn = BN; p.status = hg_host::status_ptr();
  ContractionRanges t{reinterpret_cast<const int*>(row_start), G, (N + CM - 1) / CM, (K + BN - 1) / BN, N, (long long)N * K};
  int pairs = t.tiles_m * t.tiles_n * G;
  if (max_ctas > 1 && max_ctas / 2 < pairs) pairs = max_ctas / 2;
  CUtensorMap tc;
  if ((rc = store_map(&tc, ta, p, uint64_t(G) * N))) return rc;
  const int threads = threads_for(out_mode, ((long long)rows / G + BK - 1) / BK * (kBlockCost + BN), true);    // a group's, on average
  return launch_grouped2<true, true>(ta, tb, tc, p, t, pairs, threads, reinterpret_cast<cudaStream_t>(stream));
}

}  // extern "C"
