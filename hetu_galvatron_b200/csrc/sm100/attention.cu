// Flash attention for sm_100a on tcgen05 / TMEM: forward (O, LSE), and a two-kernel backward
// (dK,dV per key block; dQ per query block) that recomputes the scores.  Causal or full, GQA,
// head dim 64 or 128, arbitrary (s, b, head) strides so that Q/K/V are read straight out of the
// packed QKV projection and O is written in [tokens, heads*hd] layout for the output projection.
//
// Every score-like product runs as  tcgen05.mma (SS, both operands K-major, TMA-loaded),
// accumulators live in TMEM, each softmax thread owns one accumulator row (tcgen05.ld 32x32b),
// probabilities go back to shared memory as the bf16 K-major A operand of the second product,
// whose B operand is the same TMA tile of V / dO / Q / K read through an MN-major descriptor.
//
// Replaces flash_attn_varlen_func / _flash_attn_forward / _flash_attn_backward as called from
// galvatron/core/runtime/transformer/attention_impl.py:55-111,587-616,696-727.
#include <atomic>
#include <type_traits>

#include "entry_points.h"
#include "sm100_common.cuh"

namespace hg {
namespace attn {

constexpr int kThreads = 192;  // warp 0: TMA, warp 1: UMMA, warps 2-5: softmax / epilogue
// Backward kernels: two softmax warpgroups (warps 2-5 and 6-9).  Thread == accumulator row in both; warpgroup g owns
// columns [32g, 32g+32) of every 64-column score step, which halves the exp2 / FMA work per thread so that the
// score pipeline keeps up with the tensor core.  (TMEM lanes a warp may touch are 32*(warp%4)..: warps w and w+4
// share a lane quarter.)
constexpr int kBwdThreads = 320;
constexpr int kBwdSoftmaxThreads = 256;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;
constexpr int kSmCount = 148;

// 2^x on the special-function unit: one instruction, results below 2^-126 flush to zero, 2^-inf = 0.
// (exp2f() wraps the same instruction in range handling that costs several more per element, and the score
// loops below run it tens of thousands of times per step.)
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two fp32 operations per instruction, each rounded as alone.  A pair of neighbouring registers is one operand.  The softmax of the
// forward is bound by the instructions of its threads beside the exponentials: 2 x 4096 tokens and 32 heads of 128 317 us without,
// 301 with these and max3; 8 x 1024 and 25 heads of 64 100, 97; 1531 and 28 heads on 4 46.9, 44.9.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n.reg .b64 a, b, c, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %7};\n"
      "fma.rn.f32x2 d, a, b, c;\nmov.b64 {%0, %1}, d;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n.reg .b64 a, b, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nadd.rn.f32x2 d, a, b;\nmov.b64 {%0, %1}, d;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n.reg .b64 a, b, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmul.rn.f32x2 d, a, b;\nmov.b64 {%0, %1}, d;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

// The larger of three: one instruction.
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Softmax warpgroups of the 128-query dK/dV kernel.
constexpr int kDkvWarpgroups = 4;
// Softmax warpgroups of the 128-key dQ kernel (2 or 4).
#ifndef HG_DQ_WARPGROUPS
#define HG_DQ_WARPGROUPS 4
#endif
constexpr int kDqWarpgroups = HG_DQ_WARPGROUPS;
// Per-role cycle counts of CTA (0, 0, 0), for builds with -DHG_ATTN_TIMING: where a step's time goes (waiting for the
// other role, or working).  Lane 0 of the first softmax warp writes words 16..20 of the device status buffer
// (steps, wait for S^T, probabilities, wait for dP^T, dS^T and stores), lane 0 of the MMA warp words 24..28 (steps, wait
// for free S^T columns, wait for P^T, wait for dS^T, time spent issuing).  The dQ kernel reports in words 40..44 and
// 48..52: softmax (steps, wait for S, loads, arithmetic, dS store), MMA (steps, S + dP issue including
// its waits, wait for dS, dQ issue).  The counts are clock64() differences; nothing is compiled in without
// the define.
#ifdef HG_ATTN_TIMING
#define HG_DKV_TIMERS(a, b, c, d) long long a = 0, b = 0, c = 0, d = 0
#define HG_DKV_TICK(t) long long t = clock64()
#define HG_DKV_TOCK(acc, t)          \
  do {                               \
    const long long now_ = clock64(); \
    acc += now_ - t;                 \
    t = now_;                        \
  } while (0)
#define HG_DKV_REPORT(off, n, a, b, c, d)                                                                   \
  do {                                                                                                      \
    if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && lane_id() == 0 && (warp == 1 || warp == 2 || warp == 4)) { \
      p.status[16 + off] = n;                                                                               \
      p.status[17 + off] = int(a);                                                                          \
      p.status[18 + off] = int(b);                                                                          \
      p.status[19 + off] = int(c);                                                                          \
      p.status[20 + off] = int(d);                                                                          \
    }                                                                                                       \
  } while (0)
#else
#define HG_DKV_TIMERS(a, b, c, d)
#define HG_DKV_TICK(t)
#define HG_DKV_TOCK(acc, t)
#define HG_DKV_REPORT(off, n, a, b, c, d)
#endif

// Head -> slot mapping inside the (possibly packed) tensor:  slot = (h / qpg) * gs + (h % qpg) * hs + off
struct SlotMap {
  int gs, hs, off;
  __device__ __forceinline__ int slot(int h, int qpg) const { return (h / qpg) * gs + (h % qpg) * hs + off; }
};

struct FwdParams {
  int Sq, Skv, B, nheads, qpg;  // qpg = query heads per kv head
  int causal;
  int q_pos0, k_pos0;           // global positions of row 0 / key 0 (ring / context-parallel steps)
  float scale;                  // softmax scale (1/sqrt(hd))
  SlotMap qmap, kmap, vmap;
  hg_lp_t* O;             // element (s, b, h, d) at O + s*o_ss + b*o_sb + h*hd + d
  int64_t o_ss, o_sb;
  float* LSE;                   // [B, nheads, Sq]
  int* status;
};

// K-major operand: `rows` x (64*slabs) bf16 stored as slabs of [rows x 128 B]; descriptor for k-step kk.
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t base, int rows, int kk) {
  return make_smem_desc(base + (kk >> 2) * rows * 128 + (kk & 3) * 32, 16, 1024);
}
// The same buffer viewed as an MN-major operand (MN = the 64*slabs columns, K = rows); k-step kk = rows 16kk..
__device__ __forceinline__ uint64_t mnmajor_desc(uint32_t base, int rows, int kk) {
  return make_smem_desc(base + kk * 2048, rows * 128, 1024);
}

// =================================================================================================
// Forward
// =================================================================================================
template <int HD>
struct FwdSmem {
  static constexpr int kQ = 128 * HD * 2;
  static constexpr int kKV = 128 * HD * 2;
  static constexpr int kP = 128 * 128 * 2;
  static constexpr int kTotal = kQ + 4 * kKV + kP + 1024 + 256;
};

template <int HD>
__global__ void __launch_bounds__(kThreads, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = base;
  uint8_t* sK = sQ + FwdSmem<HD>::kQ;              // 2 stages
  uint8_t* sV = sK + 2 * FwdSmem<HD>::kKV;         // 2 stages
  uint8_t* sP = sV + 2 * FwdSmem<HD>::kKV;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sP + FwdSmem<HD>::kP);
  uint64_t* q_full = bars;          // 1
  uint64_t* k_full = bars + 1;      // 2
  uint64_t* k_empty = bars + 3;     // 2
  uint64_t* v_full = bars + 5;      // 2
  uint64_t* v_empty = bars + 7;     // 2
  uint64_t* s_full = bars + 9;      // 2
  uint64_t* s_empty = bars + 11;    // 2
  uint64_t* p_full = bars + 13;     // 1
  uint64_t* o_done = bars + 14;     // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int qb = gridDim.x - 1 - blockIdx.x;  // heavy (late) query blocks first under a causal mask
  const int h = blockIdx.y, b = blockIdx.z;
  const int q0 = qb * 128;

  // key blocks this query block attends to
  int kv_len = p.Skv;
  if (p.causal) {
    const int last = p.q_pos0 + q0 + 127 - p.k_pos0;  // last visible key index for the last row
    kv_len = min(p.Skv, last + 1);
  }
  const int n_kv = kv_len > 0 ? (kv_len + 127) / 128 : 0;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&s_empty[i], 4);     // one arrival per softmax warp (mbar_arrive_warp)
    }
    mbar_init(p_full, 4);
    mbar_init(o_done, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  chain_release();                            // after the allocation: see chain_release
  chain_wait();
  const uint32_t tS[2] = {tmem, tmem + 128};
  const uint32_t tO = tmem + 256;

  const int qslot = p.qmap.slot(h, p.qpg), kslot = p.kmap.slot(h, p.qpg), vslot = p.vmap.slot(h, p.qpg);

  if (warp == 0) {
    if (n_kv > 0) {
      // the whole warp walks the loop, one elected lane issues the copies (see producer_loop in gemm_core.cuh)
      const bool issuer = elect_one() != 0;
      if (issuer) mbar_expect_tx(q_full, FwdSmem<HD>::kQ);
#pragma unroll
      for (int j = 0; j < HD / 64; ++j) if (issuer) tma_load_4d(sQ + j * 128 * 128, &tmQ, q_full, j * 64, qslot, q0, b);
      for (int j = 0; j < n_kv; ++j) {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        if (!mbar_wait_warp(&k_empty[st], ph ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { *abort_flag = 1; break; }
        if (issuer) mbar_expect_tx(&k_full[st], FwdSmem<HD>::kKV);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          if (issuer) tma_load_4d(sK + st * FwdSmem<HD>::kKV + c * 128 * 128, &tmK, &k_full[st], c * 64, kslot, j * 128, b);
        if (!mbar_wait_warp(&v_empty[st], ph ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { *abort_flag = 1; break; }
        if (issuer) mbar_expect_tx(&v_full[st], FwdSmem<HD>::kKV);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          if (issuer) tma_load_4d(sV + st * FwdSmem<HD>::kKV + c * 128 * 128, &tmV, &v_full[st], c * 64, vslot, j * 128, b);
      }
    }
  } else if (warp == 1) {
    if (n_kv > 0) {
      // the whole warp walks the loop, one elected lane issues (see mma_loop in gemm_core.cuh)
      const bool issuer = elect_one() != 0;
      constexpr uint32_t idesc_s = make_idesc_lp(128, 128, false, false);
      constexpr uint32_t idesc_o = make_idesc_lp(128, HD, false, true);
      const uint32_t aQ = smem_u32(sQ), aP = smem_u32(sP);
      bool ok = mbar_wait_warp(q_full, 0, p.status, kTimeoutSmemFull, abort_flag);
      auto issue_s = [&](int j) -> bool {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        if (!mbar_wait_warp(&k_full[st], ph, p.status, kTimeoutSmemFull, abort_flag)) return false;
        if (!mbar_wait_warp(&s_empty[st], ph ^ 1, p.status, kTimeoutTmemEmpty, abort_flag)) return false;
        tc_fence_after();
        const uint32_t aK = smem_u32(sK + st * FwdSmem<HD>::kKV);
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk)
            umma_f16_ss(tS[st], kmajor_desc(aQ, 128, kk), kmajor_desc(aK, 128, kk), idesc_s, kk != 0);
          umma_commit(&s_full[st]);
          umma_commit(&k_empty[st]);
        }
        __syncwarp();
        return true;
      };
      if (ok) ok = issue_s(0);
      for (int j = 0; ok && j < n_kv; ++j) {
        if (j + 1 < n_kv) { ok = issue_s(j + 1); if (!ok) break; }
        const int st = j & 1;
        if (!mbar_wait_warp(p_full, j & 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
        if (!mbar_wait_warp(&v_full[st], (j >> 1) & 1, p.status, kTimeoutSmemFull, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t aV = smem_u32(sV + st * FwdSmem<HD>::kKV);
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_f16_ss(tO, kmajor_desc(aP, 128, kk), mnmajor_desc(aV, 128, kk), idesc_o, (j | kk) != 0);
          umma_commit(&v_empty[st]);
          umma_commit(o_done);
        }
        __syncwarp();
      }
      if (!ok) *abort_flag = 1;
    }
  } else {
    // ---- softmax: thread == query row ----
    const int wq = warp & 3;
    const int row = wq * 32 + lane_id();
    const uint32_t lane_off = uint32_t(wq * 32) << 16;
    const float sl2 = p.scale * kLog2e;
    const int q_pos = p.q_pos0 + q0 + row;
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_kv; ++j) {
      const int st = j & 1;
      if (!mbar_wait_warp(&s_full[st], (j >> 1) & 1, p.status, kTimeoutTmemFull, abort_flag)) { ok = false; break; }
      tc_fence_after();
      float s[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t r[32];
        tmem_ld32(tS[st] + lane_off + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) s[c * 32 + i] = __uint_as_float(r[i]);
      }
      tc_fence_before();
      mbar_arrive_warp(&s_empty[st]);
      // masking (only blocks that cross the diagonal or the ragged end need it)
      const int k_base = p.k_pos0 + j * 128;
      const bool need_mask = (p.causal && (k_base + 127 > p.q_pos0 + q0)) || (j * 128 + 128 > p.Skv);
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < 128; ++i) {
          const bool dead = (j * 128 + i >= p.Skv) || (p.causal && (k_base + i > q_pos));
          if (dead) s[i] = -INFINITY;
        }
      }
      float mx4[4] = {s[0], s[1], s[2], s[3]};   // four chains: a single one is 63 dependent instructions long
#pragma unroll
      for (int i = 4; i < 124; i += 8) {
#pragma unroll
        for (int u = 0; u < 4; ++u) mx4[u] = max3(mx4[u], s[i + u], s[i + 4 + u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) mx4[u] = fmaxf(mx4[u], s[124 + u]);
      float mx = max3(mx4[0], mx4[1], fmaxf(mx4[2], mx4[3]));
      mx *= sl2;
      // lazy rescale: keep the running reference max unless the new max exceeds it by more than 2^8
      float alpha = 1.f;
      bool rescale = false;
      if (mx > m_used + 8.f) {
        alpha = (m_used == -INFINITY) ? 0.f : ex2(m_used - mx);
        m_used = mx;
        rescale = (j > 0);
      }
      const float nmref = (m_used == -INFINITY) ? 0.f : -m_used;
      float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int i = 0; i < 128; i += 2) {
        const float2 x = fma2(make_float2(s[i], s[i + 1]), make_float2(sl2, sl2), make_float2(nmref, nmref));
        s[i] = ex2(x.x);
        s[i + 1] = ex2(x.y);
        sum2[(i >> 1) & 1] = add2(sum2[(i >> 1) & 1], make_float2(s[i], s[i + 1]));
      }
      l = l * alpha + ((sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y));
      if (j > 0) {
        if (!mbar_wait_warp(o_done, (j - 1) & 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
        tc_fence_after();
      }
      if (__any_sync(0xffffffffu, rescale)) {
#pragma unroll
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t r[32];
          tmem_ld32(tO + lane_off + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
          tmem_st32(tO + lane_off + c * 32, r);
        }
        tmem_st_wait();
      }
      // P -> shared memory, bf16, 128B-swizzled K-major (two 64-column slabs)
#pragma unroll
      for (int cc = 0; cc < 16; ++cc) {
        uint4 u;
        u.x = pack_bf16(s[cc * 8 + 0], s[cc * 8 + 1]);
        u.y = pack_bf16(s[cc * 8 + 2], s[cc * 8 + 3]);
        u.z = pack_bf16(s[cc * 8 + 4], s[cc * 8 + 5]);
        u.w = pack_bf16(s[cc * 8 + 6], s[cc * 8 + 7]);
        *reinterpret_cast<uint4*>(sP + (cc >> 3) * 128 * 128 + sw128_offset(row, cc & 7)) = u;
      }
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive_warp(p_full);
    }
    // ---- epilogue: O / l -> global, LSE ----
    const int srow = q0 + row;
    if (n_kv == 0) {
      if (srow < p.Sq) {
        hg_lp_t* o = p.O + int64_t(srow) * p.o_ss + int64_t(b) * p.o_sb + h * HD;
#pragma unroll
        for (int i = 0; i < HD / 8; ++i) reinterpret_cast<uint4*>(o)[i] = make_uint4(0, 0, 0, 0);
        p.LSE[(size_t(b) * p.nheads + h) * p.Sq + srow] = -INFINITY;
      }
    } else if (ok && !*abort_flag && mbar_wait_warp(o_done, (n_kv - 1) & 1, p.status, kTimeoutOther, abort_flag)) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t r[32];
        tmem_ld32(tO + lane_off + c * 32, r);
        tmem_ld_wait();
        if (srow < p.Sq) {
          hg_lp_t* o = p.O + int64_t(srow) * p.o_ss + int64_t(b) * p.o_sb + h * HD + c * 32;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 u;
            u.x = pack_bf16(__uint_as_float(r[q * 8 + 0]) * inv, __uint_as_float(r[q * 8 + 1]) * inv);
            u.y = pack_bf16(__uint_as_float(r[q * 8 + 2]) * inv, __uint_as_float(r[q * 8 + 3]) * inv);
            u.z = pack_bf16(__uint_as_float(r[q * 8 + 4]) * inv, __uint_as_float(r[q * 8 + 5]) * inv);
            u.w = pack_bf16(__uint_as_float(r[q * 8 + 6]) * inv, __uint_as_float(r[q * 8 + 7]) * inv);
            reinterpret_cast<uint4*>(o)[q] = u;
          }
        }
      }
      if (srow < p.Sq)
        p.LSE[(size_t(b) * p.nheads + h) * p.Sq + srow] = (l > 0.f) ? (m_used + log2f(l)) * kLn2 : -INFINITY;
    } else {
      *abort_flag = 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// =================================================================================================
// Forward with two query tiles per CTA and P in tensor memory (both head dims).
// In the one-tile kernel a scheduler hosts a single softmax warp, so every latency of its step (the loads from tensor
// memory, the maximum, the exp2 / convert chains) is exposed, and the tensor core idles while the softmax of its only
// tile runs.  Here a CTA owns 256 queries as two tiles of 128, one softmax warpgroup per tile: while one tile's
// threads work on their scores, the tensor core runs the other tile's products, and every scheduler has two softmax
// warps to switch between.  P never goes through shared memory: the threads store it, packed, over the first 64 of
// the 128 S columns they have just read, and the PV product takes its A operand from tensor memory.
//
// Tensor memory (512 columns): S of tile 0 / 1 at 0 / 128, O of tile 0 / 1 at 256 / 384.  Per tile the order is
// S(j) -> softmax(j) -> P(j) -> PV(j) -> S(j+1): S(j+1) overwrites the columns PV(j) reads, and the tensor core
// executes in issue order, so the MMA warp issues PV(t, j) and S(t, j+1) back to back when P(t, j) is stored.
// K and V stages are shared by the two tiles; a stage is released after the last product that reads it.
// =================================================================================================
template <int HD>
struct Fwd2Smem {
  static constexpr int kQ = 128 * HD * 2;     // one query tile
  static constexpr int kKV = 128 * HD * 2;    // one stage of K or V
  static constexpr int kTotal = 2 * kQ + 4 * kKV + 1024 + 256;
};

// Registers.  A softmax thread holds its 128 scores and a half row of packed probabilities, more than the 168 registers
// an even share of twelve warps leaves; the warpgroup of the TMA and MMA warps (warps 0-3, two of them idle) gives most
// of its share away.  setmaxnreg moves registers inside what the block was launched with: 384 threads x 168 = 64512
// (as ptxas reports for this kernel) >= 128 x 56 + 256 x 216 = 62464.
constexpr int kFwd2Threads = 384;
constexpr int kFwd2AuxRegs = 56, kFwd2SoftmaxRegs = 216;
template <int N>
__device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

template <int HD>
__global__ void __launch_bounds__(kFwd2Threads, 1)
flash_fwd2_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                  const __grid_constant__ CUtensorMap tmV, const FwdParams p) {
  static_assert(HD == 64 || HD == 128, "tensor memory holds two S tiles and two O tiles of up to 128 columns");
  extern __shared__ uint8_t smem_raw[];
  using L = Fwd2Smem<HD>;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = base;                     // 2 tiles
  uint8_t* sK = sQ + 2 * L::kQ;           // 2 stages
  uint8_t* sV = sK + 2 * L::kKV;          // 2 stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 2 * L::kKV);
  uint64_t* q_full = bars;          // 1
  uint64_t* k_full = bars + 1;      // 2
  uint64_t* k_empty = bars + 3;     // 2
  uint64_t* v_full = bars + 5;      // 2
  uint64_t* v_empty = bars + 7;     // 2
  uint64_t* s_full = bars + 9;      // 2 (per tile)
  uint64_t* p_full = bars + 11;     // 4 (per tile and half of the key block)
  uint64_t* o_done = bars + 15;     // 2 (per tile)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int qb = gridDim.x - 1 - blockIdx.x;  // heavy (late) query blocks first under a causal mask
  const int h = blockIdx.y, b = blockIdx.z;
  const int q0 = qb * 256;

  // key blocks each tile attends to (tile 1 never fewer than tile 0)
  int n_kv_t[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    int kv_len = p.Skv;
    if (p.causal) kv_len = min(p.Skv, p.q_pos0 + q0 + t * 128 + 127 - p.k_pos0 + 1);
    n_kv_t[t] = (kv_len > 0 && q0 + t * 128 < p.Sq) ? (kv_len + 127) / 128 : 0;
  }
  const int n_kv = max(n_kv_t[0], n_kv_t[1]);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[2 * i], 4);  // one arrival per softmax warp of the tile (mbar_arrive_warp)
      mbar_init(&p_full[2 * i + 1], 4);
      mbar_init(&o_done[i], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  chain_release();                            // after the allocation: see chain_release
  chain_wait();
  const uint32_t tS[2] = {tmem, tmem + 128};
  const uint32_t tO[2] = {tmem + 256, tmem + 384};

  const int qslot = p.qmap.slot(h, p.qpg), kslot = p.kmap.slot(h, p.qpg), vslot = p.vmap.slot(h, p.qpg);

  if (warp < 4) {
  regs_dec<kFwd2AuxRegs>();
  if (warp == 0) {
    if (n_kv > 0) {
      // the whole warp walks the loop, one elected lane issues the copies (see producer_loop in gemm_core.cuh)
      const bool issuer = elect_one() != 0;
      if (issuer) mbar_expect_tx(q_full, 2 * L::kQ);   // rows past the end of the tensor arrive as zeros
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          if (issuer) tma_load_4d(sQ + t * L::kQ + c * 128 * 128, &tmQ, q_full, c * 64, qslot, q0 + t * 128, b);
      for (int j = 0; j < n_kv; ++j) {
        const int st = j & 1;
        const uint32_t ph = (j >> 1) & 1;
        if (!mbar_wait_warp(&k_empty[st], ph ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { *abort_flag = 1; break; }
        if (issuer) mbar_expect_tx(&k_full[st], L::kKV);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          if (issuer) tma_load_4d(sK + st * L::kKV + c * 128 * 128, &tmK, &k_full[st], c * 64, kslot, j * 128, b);
        if (!mbar_wait_warp(&v_empty[st], ph ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { *abort_flag = 1; break; }
        if (issuer) mbar_expect_tx(&v_full[st], L::kKV);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          if (issuer) tma_load_4d(sV + st * L::kKV + c * 128 * 128, &tmV, &v_full[st], c * 64, vslot, j * 128, b);
      }
    }
  } else if (warp == 1) {
    if (n_kv > 0) {
      // the whole warp walks the loop, one elected lane issues (see mma_loop in gemm_core.cuh)
      const bool issuer = elect_one() != 0;
      constexpr uint32_t idesc_s = make_idesc_lp(128, 128, false, false);
      constexpr uint32_t idesc_o = make_idesc_lp(128, HD, false, true);
      bool ok = mbar_wait_warp(q_full, 0, p.status, kTimeoutSmemFull, abort_flag);
      // the last tile (in issue order) that has a step j: it releases the K / V stage of that step
      auto last_user = [&](int j) -> int { return j < n_kv_t[1] ? 1 : 0; };
      auto issue_s = [&](int t, int j) -> bool {
        const int st = j & 1;
        if (!mbar_wait_warp(&k_full[st], (j >> 1) & 1, p.status, kTimeoutSmemFull, abort_flag)) return false;
        tc_fence_after();
        const uint32_t aQ = smem_u32(sQ + t * L::kQ), aK = smem_u32(sK + st * L::kKV);
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk)
            umma_f16_ss(tS[t], kmajor_desc(aQ, 128, kk), kmajor_desc(aK, 128, kk), idesc_s, kk != 0);
          umma_commit(&s_full[t]);
          if (t == last_user(j)) umma_commit(&k_empty[st]);
        }
        __syncwarp();
        return true;
      };
#pragma unroll
      for (int t = 0; t < 2; ++t)
        if (ok && n_kv_t[t] > 0) ok = issue_s(t, 0);
      HG_DKV_TIMERS(tm_wait_p0, tm_wait_p1, tm_issue, tm_unused);
      HG_DKV_TICK(t0);
      for (int j = 0; ok && j < n_kv; ++j) {
        const int st = j & 1;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (!ok || j >= n_kv_t[t]) continue;
          if (!mbar_wait_warp(&p_full[2 * t], j & 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
          if (t == 0) { HG_DKV_TOCK(tm_wait_p0, t0); } else { HG_DKV_TOCK(tm_wait_p1, t0); }
          if (!mbar_wait_warp(&v_full[st], (j >> 1) & 1, p.status, kTimeoutSmemFull, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t aV = smem_u32(sV + st * L::kKV);
          if (issuer) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)   // k-step kk = keys 16kk..16kk+15 = 8 packed columns of P
              umma_f16_ts(tO[t], tS[t] + kk * 8, mnmajor_desc(aV, 128, kk), idesc_o, (j | kk) != 0);
          }
          __syncwarp();
          if (!mbar_wait_warp(&p_full[2 * t + 1], j & 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
          tc_fence_after();
          if (issuer) {
#pragma unroll
            for (int kk = 4; kk < 8; ++kk)
              umma_f16_ts(tO[t], tS[t] + kk * 8, mnmajor_desc(aV, 128, kk), idesc_o, true);
            if (t == last_user(j)) umma_commit(&v_empty[st]);
            if (j + 1 >= n_kv_t[t]) umma_commit(&o_done[t]);
          }
          __syncwarp();
          if (j + 1 < n_kv_t[t]) ok = issue_s(t, j + 1);
          HG_DKV_TOCK(tm_issue, t0);
        }
      }
      HG_DKV_REPORT(8, n_kv, tm_wait_p0, tm_wait_p1, tm_issue, tm_unused);
      if (!ok) *abort_flag = 1;
    }
  }
  } else {
    regs_inc<kFwd2SoftmaxRegs>();
    // ---- softmax: one warpgroup per tile, thread == query row ----
    const int t = (warp - 4) >> 2;
    const int wq = warp & 3;
    const int row = wq * 32 + lane_id();
    const uint32_t lane_off = uint32_t(wq * 32) << 16;
    const float sl2 = p.scale * kLog2e;
    const int qt0 = q0 + t * 128;
    const int q_pos = p.q_pos0 + qt0 + row;
    const int my_kv = n_kv_t[t];
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    HG_DKV_TIMERS(tm_wait_s, tm_ld, tm_math, tm_st);
    for (int j = 0; j < my_kv; ++j) {
      HG_DKV_TICK(t0);
      if (!mbar_wait_warp(&s_full[t], j & 1, p.status, kTimeoutTmemFull, abort_flag)) { ok = false; break; }
      tc_fence_after();
      HG_DKV_TOCK(tm_wait_s, t0);
      float s[128];
      {
        uint32_t r[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(tS[t] + lane_off + c * 32, r[c]);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i) s[c * 32 + i] = __uint_as_float(r[c][i]);
      }
      HG_DKV_TOCK(tm_ld, t0);
      // masking (only blocks that cross the diagonal or the ragged end need it)
      const int k_base = p.k_pos0 + j * 128;
      const bool need_mask = (p.causal && (k_base + 127 > p.q_pos0 + qt0)) || (j * 128 + 128 > p.Skv);
      if (need_mask) {
#pragma unroll
        for (int i = 0; i < 128; ++i) {
          const bool dead = (j * 128 + i >= p.Skv) || (p.causal && (k_base + i > q_pos));
          if (dead) s[i] = -INFINITY;
        }
      }
      float mx4[4] = {s[0], s[1], s[2], s[3]};   // four chains: a single one is 63 dependent instructions long
#pragma unroll
      for (int i = 4; i < 124; i += 8) {
#pragma unroll
        for (int u = 0; u < 4; ++u) mx4[u] = max3(mx4[u], s[i + u], s[i + 4 + u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) mx4[u] = fmaxf(mx4[u], s[124 + u]);
      float mx = max3(mx4[0], mx4[1], fmaxf(mx4[2], mx4[3]));
      mx *= sl2;
      // lazy rescale: keep the running reference max unless the new max exceeds it by more than 2^8
      float alpha = 1.f;
      bool rescale = false;
      if (mx > m_used + 8.f) {
        alpha = (m_used == -INFINITY) ? 0.f : ex2(m_used - mx);
        m_used = mx;
        rescale = (j > 0);
      }
      const float nmref = (m_used == -INFINITY) ? 0.f : -m_used;
      // S(t, j) was issued after PV(t, j-1), and the tensor core executes in order: O holds steps 0..j-1 by now
      if (__any_sync(0xffffffffu, rescale)) {
#pragma unroll
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t r[32];
          tmem_ld32(tO[t] + lane_off + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
          tmem_st32(tO[t] + lane_off + c * 32, r);
        }
      }
      // P, packed, over the first 64 of this row's S columns, in two halves: the PV product of keys 0..63 runs while
      // the exponentials of keys 64..127 are taken
      float2 sum2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          const float2 x = fma2(make_float2(s[hh * 64 + i], s[hh * 64 + i + 1]), make_float2(sl2, sl2), make_float2(nmref, nmref));
          const float2 e = make_float2(ex2(x.x), ex2(x.y));
          sum2[(i >> 1) & 1] = add2(sum2[(i >> 1) & 1], e);
          pk[i >> 1] = pack_bf16(e.x, e.y);
        }
        tmem_st32(tS[t] + lane_off + hh * 32, pk);
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive_warp(&p_full[2 * t + hh]);
        if (hh == 0) { HG_DKV_TOCK(tm_math, t0); }
      }
      l = l * alpha + ((sum2[0].x + sum2[0].y) + (sum2[1].x + sum2[1].y));
      HG_DKV_TOCK(tm_st, t0);
    }
    if (t == 0) { HG_DKV_REPORT(0, my_kv, tm_wait_s, tm_ld, tm_math, tm_st); }
    // ---- epilogue: O / l -> global, LSE ----
    const int srow = qt0 + row;
    if (my_kv == 0) {
      if (srow < p.Sq) {
        hg_lp_t* o = p.O + int64_t(srow) * p.o_ss + int64_t(b) * p.o_sb + h * HD;
#pragma unroll
        for (int i = 0; i < HD / 8; ++i) reinterpret_cast<uint4*>(o)[i] = make_uint4(0, 0, 0, 0);
        p.LSE[(size_t(b) * p.nheads + h) * p.Sq + srow] = -INFINITY;
      }
    } else if (ok && !*abort_flag && mbar_wait_warp(&o_done[t], 0, p.status, kTimeoutOther, abort_flag)) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t r[32];
        tmem_ld32(tO[t] + lane_off + c * 32, r);
        tmem_ld_wait();
        if (srow < p.Sq) {
          hg_lp_t* o = p.O + int64_t(srow) * p.o_ss + int64_t(b) * p.o_sb + h * HD + c * 32;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 u;
            u.x = pack_bf16(__uint_as_float(r[q * 8 + 0]) * inv, __uint_as_float(r[q * 8 + 1]) * inv);
            u.y = pack_bf16(__uint_as_float(r[q * 8 + 2]) * inv, __uint_as_float(r[q * 8 + 3]) * inv);
            u.z = pack_bf16(__uint_as_float(r[q * 8 + 4]) * inv, __uint_as_float(r[q * 8 + 5]) * inv);
            u.w = pack_bf16(__uint_as_float(r[q * 8 + 6]) * inv, __uint_as_float(r[q * 8 + 7]) * inv);
            reinterpret_cast<uint4*>(o)[q] = u;
          }
        }
      }
      if (srow < p.Sq)
        p.LSE[(size_t(b) * p.nheads + h) * p.Sq + srow] = (l > 0.f) ? (m_used + log2f(l)) * kLn2 : -INFINITY;
    } else {
      *abort_flag = 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// =================================================================================================
// Backward, part 0:  D[b,h,s] = sum_d dO * O
// =================================================================================================
// O and dO are read once, 16 bytes per lane: HD / 8 lanes share a (token, head) row and meet in log2(HD / 8) shuffles.
// (A warp per row with 4-byte loads had half a kilobyte in flight per warp and reached a third of the memory rate:
// 64 us for the 134 MB of 8192 tokens x 32 heads x 128.)
// VEC = false: for an O or dO whose rows are not 16-byte aligned.
template <bool VEC>
__device__ __forceinline__ uint4 dot_load8(const hg_lp_t* p) {
  if (VEC) return __ldcs(reinterpret_cast<const uint4*>(p));
  uint4 u;
  hg_lp_t* e = reinterpret_cast<hg_lp_t*>(&u);
#pragma unroll
  for (int i = 0; i < 8; ++i) e[i] = p[i];
  return u;
}
template <int HD, bool VEC>
__global__ void __launch_bounds__(256)
attn_bwd_dot_kernel(const hg_lp_t* __restrict__ O, const hg_lp_t* __restrict__ dO, int64_t ss, int64_t sb, int64_t dss,
                    int64_t dsb, int S, int B, int nheads, float* __restrict__ D) {
  constexpr int LPR = HD / 8, U = 4;              // lanes per row, rows in flight per thread
  // 2^31 rows of 64 channels would be 275 GB: rows are counted in 32 bits, since a 64-bit division per row is most of the kernel's
  // instructions, which bound it (us with / without: 2 x 4096 tokens and 32 heads of 128 34 / 29, 8 x 1024 and 25 of 64 16.5 / 14.3)
  const unsigned total = unsigned(S) * unsigned(B) * unsigned(nheads);
  const int sub = threadIdx.x % LPR;
  const unsigned stride = gridDim.x * (256 / LPR);
  for (unsigned r0 = blockIdx.x * (256 / LPR) + threadIdx.x / LPR; r0 - threadIdx.x / LPR < total; r0 += U * stride) {
    uint4 a[U], c[U];
    float* dst[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned row = r0 + u * stride;
      dst[u] = nullptr;
      a[u] = c[u] = make_uint4(0, 0, 0, 0);
      if (row < total) {
        const unsigned tok = row / unsigned(nheads);
        const int h = int(row - tok * unsigned(nheads)), s = int(tok / unsigned(B)), b = int(tok) - s * B;
        a[u] = dot_load8<VEC>(O + s * ss + b * sb + h * HD + sub * 8);
        c[u] = dot_load8<VEC>(dO + s * dss + b * dsb + h * HD + sub * 8);
        dst[u] = D + (size_t(b) * nheads + h) * S + s;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t* x = reinterpret_cast<const uint32_t*>(&a[u]);
      const uint32_t* y = reinterpret_cast<const uint32_t*>(&c[u]);
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 p = hg_unpack2(x[i]), q = hg_unpack2(y[i]);
        acc += p.x * q.x + p.y * q.y;
      }
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (sub == 0 && dst[u] != nullptr) *dst[u] = acc;
    }
  }
}

// =================================================================================================
// Backward parameters (shared by the dK/dV and the dQ kernels)
// =================================================================================================
struct BwdParams {
  int Sq, Skv, B, nheads, qpg;
  int causal;
  int q_pos0, k_pos0;
  float scale;
  SlotMap qmap, kmap, vmap, domap;  // dO uses slot = h (gs = qpg, hs = 1, off = 0)
  const float* LSE;                 // [B, nheads, Sq]
  const float* D;                   // [B, nheads, Sq]
  // outputs: element (s, b, slot, d) at base + s*ss + b*sb + slot*hd + d
  hg_lp_t* dQ; int64_t dq_ss, dq_sb; SlotMap dqmap;
  hg_lp_t* dK; int64_t dk_ss, dk_sb; SlotMap dkmap;
  hg_lp_t* dV; int64_t dv_ss, dv_sb; SlotMap dvmap;
  int* status;
  // dK/dV of a key block shared by several CTAs (see dkv_chunk_steps): at most `chunk` query steps each (0: off), their
  // fp32 parts in `part`, [CTA][dV, dK][128][HD]
  int chunk;
  float* part;
  // A launch covers nh_c heads from h0_c on (and their kv heads from g0_c on) of the sequences from b0_c on: grids count from there.
  int b0_c, g0_c, h0_c, nh_c;
};

// Tiles of dS of key blocks 0 .. kb - 1 of one head.  Key block j is seen by the query blocks from max(0, j + d) on, d being
// the distance of the first key behind the first query in blocks, rounded down.
__host__ __device__ __forceinline__ long long ds_tiles_before(const BwdParams& p, int kb) {
  const long long n_qs = (p.Sq + 127) / 128;
  if (!p.causal) return kb * n_qs;
  const int behind = p.k_pos0 - p.q_pos0, d = behind >= 0 ? behind / 128 : -((127 - behind) / 128);
  const long long a = kb < -d ? kb : d < 0 ? -d : 0;                   // blocks that every query block sees
  const long long e = kb < n_qs - d ? kb : n_qs - d;                   // blocks from e on are seen by none
  const long long n = e > a ? e - a : 0;
  return a * n_qs + n * n_qs - n * (a + e - 1) / 2 - n * d;
}
// dS as the dK/dV kernel leaves it for the dQ product: 128 x 128 tiles of the pairs of a key block and a query block that see each
// other, in the order of ds_tiles_before, `heads` heads of the launch one after the other in each of up to kDsPieces pieces (0: dS is
// not stored).  A tile is what the tensor core reads as an M-major operand without swizzle, [2 x 64 keys][16 x 8 queries][64 keys][8
// queries]: a warp's store of eight queries of 32 keys is 512 bytes in a row (as rows of 128 queries, 32 pieces of 32 bytes, these
// stores doubled the kernel's time), and half a tile one copy.
constexpr int kDsPieces = kHgDsPieces;
struct DsPieces {
  hg_lp_t* at[kDsPieces];
  int heads;
};
// Tile `tile` of a head, counted from the launch's first; `head_tiles`: of each.
__device__ __forceinline__ hg_lp_t* ds_tile(const DsPieces& ds, int head, int64_t head_tiles, int64_t tile) {
  const int piece = head / ds.heads;
  return ds.at[piece] + ((head - piece * ds.heads) * head_tiles + tile) * (128 * 128);
}

// First query block that sees key block kb.
__host__ __device__ __forceinline__ int ds_first_query_block(const BwdParams& p, int kb) {
  const int first = p.causal ? p.k_pos0 + kb * 128 - p.q_pos0 : 0;
  return first > 0 ? first / 128 : 0;
}

// 128-query steps of key block kb, all query heads of its kv head together
__host__ __device__ __forceinline__ int dkv_block_steps(const BwdParams& p, int kb) {
  const int n = (p.Sq + 127) / 128 - ds_first_query_block(p, kb);
  return n > 0 ? n * p.qpg : 0;
}
// CTAs that share key block kb, `steps` being its query steps
__host__ __device__ __forceinline__ int dkv_block_ctas(const BwdParams& p, int steps) {
  return p.chunk > 0 && steps > p.chunk ? (steps + p.chunk - 1) / p.chunk : 1;
}

// =================================================================================================
// Backward, part 1: one CTA per (key block of 128, kv head, batch); loops over the query heads of the
// group and over 64-row query steps.  Thread == key row.
//   S^T = K Q^T, dP^T = V dO^T  (M = 128 keys, N = 64 queries)
//   P^T = exp2(S^T*c - lse), dS^T = P^T * (dP^T - D)
//   dV += P^T dO, dK += dS^T Q   (A from shared memory written by the threads; B = the dO / Q tile, MN-major)
// =================================================================================================
template <int HD>
struct DkvSmem {
  static constexpr int kKV = 128 * HD * 2;     // resident K or V
  static constexpr int kQD = 64 * HD * 2;      // one stage of Q or dO
  static constexpr int kQDStages = 3;          // a stage is held from its S^T product to its dK product, i.e. for more
                                               // than a step: with two stages every load was waited for in full
  static constexpr int kPT = 128 * 64 * 2;     // one P^T or dS^T buffer (two of each: written for step i+1 while step i is multiplied)
  static constexpr int kStats = 2 * 2 * 64 * 4;  // lse2/D, double buffered
  static constexpr int kTotal = 2 * kKV + 2 * kQDStages * kQD + 4 * kPT + kStats + 1024 + 256;
};

template <int HD>
__global__ void __launch_bounds__(kBwdThreads, 1)
flash_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                     const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = base;
  uint8_t* sV = sK + DkvSmem<HD>::kKV;
  constexpr int NQ = DkvSmem<HD>::kQDStages;
  uint8_t* sQ = sV + DkvSmem<HD>::kKV;            // NQ stages
  uint8_t* sDO = sQ + NQ * DkvSmem<HD>::kQD;      // NQ stages
  uint8_t* sPT = sDO + NQ * DkvSmem<HD>::kQD;
  uint8_t* sDST = sPT + 2 * DkvSmem<HD>::kPT;
  float* sStats = reinterpret_cast<float*>(sDST + 2 * DkvSmem<HD>::kPT);  // [2][2][64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sStats) + DkvSmem<HD>::kStats);
  uint64_t* kv_full = bars;        // 1
  uint64_t* qd_full = bars + 1;    // 3
  uint64_t* qd_empty = bars + 4;   // 3
  uint64_t* st_full = bars + 7;    // 2
  uint64_t* st_empty = bars + 9;   // 2
  uint64_t* pds_full = bars + 11;  // 2
  uint64_t* pds_empty = bars + 13; // 2
  uint64_t* stats_full = bars + 15; // 2
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int kb = blockIdx.x, g = blockIdx.y, b = blockIdx.z;  // g = kv head
  const int k0 = kb * 128;
  // first query row that can see this key block
  int q_first = 0;
  if (p.causal) q_first = max(0, p.k_pos0 + k0 - p.q_pos0);
  const int qs0 = (q_first / 64);                       // first 64-row query step
  const int n_qs = (p.Sq + 63) / 64;
  const int steps_per_head = max(0, n_qs - qs0);
  const int n_it = steps_per_head * p.qpg;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmDO);
    mbar_init(kv_full, 1);
    for (int i = 0; i < NQ; ++i) {
      mbar_init(&qd_full[i], 1);
      mbar_init(&qd_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&st_full[i], 1);
      mbar_init(&st_empty[i], kBwdSoftmaxThreads);
      mbar_init(&pds_full[i], kBwdSoftmaxThreads);
      mbar_init(&pds_empty[i], 1);
    }
    mbar_init(&stats_full[0], kBwdSoftmaxThreads);
    mbar_init(&stats_full[1], kBwdSoftmaxThreads);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // columns: S^T[0] 0..63, dP^T[0] 64..127, S^T[1] 128..191, dP^T[1] 192..255, dV 256.., dK 384..
  const uint32_t tST[2] = {tmem, tmem + 128};
  const uint32_t tDPT[2] = {tmem + 64, tmem + 192};
  const uint32_t tDV = tmem + 256, tDK = tmem + 384;

  const int h0 = g * p.qpg;  // first query head of the group
  const int kslot = p.kmap.slot(h0, p.qpg), vslot = p.vmap.slot(h0, p.qpg);

  if (warp == 0) {
    if (n_it > 0) {
      // the whole warp walks the loop, one elected lane issues the copies (see producer_loop in gemm_core.cuh)
      const bool issuer = elect_one() != 0;
      if (issuer) mbar_expect_tx(kv_full, 2 * DkvSmem<HD>::kKV);
#pragma unroll
      for (int c = 0; c < HD / 64; ++c) {
        if (issuer) tma_load_4d(sK + c * 128 * 128, &tmK, kv_full, c * 64, kslot, k0, b);
        if (issuer) tma_load_4d(sV + c * 128 * 128, &tmV, kv_full, c * 64, vslot, k0, b);
      }
      int st = 0;            // ring slot and its phase, and the (head, query step) of the iteration
      uint32_t ph = 0;
      int h = h0, qs = qs0;
      for (int it = 0; it < n_it; ++it) {
        const int qrow = qs * 64;
        if (!mbar_wait_warp(&qd_empty[st], ph ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { *abort_flag = 1; break; }
        if (issuer) mbar_expect_tx(&qd_full[st], 2 * DkvSmem<HD>::kQD);
        const int qslot = p.qmap.slot(h, p.qpg), doslot = p.domap.slot(h, p.qpg);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) {
          if (issuer) tma_load_4d(sQ + st * DkvSmem<HD>::kQD + c * 64 * 128, &tmQ, &qd_full[st], c * 64, qslot, qrow, b);
          if (issuer) tma_load_4d(sDO + st * DkvSmem<HD>::kQD + c * 64 * 128, &tmDO, &qd_full[st], c * 64, doslot, qrow, b);
        }
        if (++st == NQ) { st = 0; ph ^= 1; }
        if (++qs == n_qs) { qs = qs0; ++h; }
      }
    }
  } else if (warp == 1) {
    if (n_it > 0) {
      // the whole warp walks the loop, one elected lane issues (see mma_loop in gemm_core.cuh)
      const bool issuer = elect_one() != 0;
      constexpr uint32_t idesc_st = make_idesc_lp(128, 64, false, false);
      constexpr uint32_t idesc_acc = make_idesc_lp(128, HD, false, true);
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aPT = smem_u32(sPT), aDST = smem_u32(sDST);
      bool ok = mbar_wait_warp(kv_full, 0, p.status, kTimeoutSmemFull, abort_flag);
      int qs_s = 0, qs_d = 0;          // Q / dO ring slot of the next S^T issue and of the next dV / dK issue
      uint32_t qph_s = 0;
      auto issue_st = [&](int it) -> bool {
        const int st = it & 1;
        const uint32_t ph = (it >> 1) & 1;
        if (!mbar_wait_warp(&qd_full[qs_s], qph_s, p.status, kTimeoutSmemFull, abort_flag)) return false;
        if (!mbar_wait_warp(&st_empty[st], ph ^ 1, p.status, kTimeoutTmemEmpty, abort_flag)) return false;
        tc_fence_after();
        const uint32_t aQ = smem_u32(sQ + qs_s * DkvSmem<HD>::kQD), aDO = smem_u32(sDO + qs_s * DkvSmem<HD>::kQD);
        if (++qs_s == NQ) { qs_s = 0; qph_s ^= 1; }
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk)
            umma_f16_ss(tST[st], kmajor_desc(aK, 128, kk), kmajor_desc(aQ, 64, kk), idesc_st, kk != 0);
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk)
            umma_f16_ss(tDPT[st], kmajor_desc(aV, 128, kk), kmajor_desc(aDO, 64, kk), idesc_st, kk != 0);
          umma_commit(&st_full[st]);
        }
        __syncwarp();
        return true;
      };
      if (ok) ok = issue_st(0);
      for (int it = 0; ok && it < n_it; ++it) {
        if (it + 1 < n_it) { ok = issue_st(it + 1); if (!ok) break; }
        const int st = it & 1;
        if (!mbar_wait_warp(&pds_full[st], (it >> 1) & 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t aQ = smem_u32(sQ + qs_d * DkvSmem<HD>::kQD), aDO = smem_u32(sDO + qs_d * DkvSmem<HD>::kQD);
        const uint32_t aPTs = aPT + st * DkvSmem<HD>::kPT, aDSTs = aDST + st * DkvSmem<HD>::kPT;
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_f16_ss(tDV, kmajor_desc(aPTs, 128, kk), mnmajor_desc(aDO, 64, kk), idesc_acc, (it | kk) != 0);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            umma_f16_ss(tDK, kmajor_desc(aDSTs, 128, kk), mnmajor_desc(aQ, 64, kk), idesc_acc, (it | kk) != 0);
          umma_commit(&qd_empty[qs_d]);
          umma_commit(&pds_empty[st]);
        }
        __syncwarp();
        if (++qs_d == NQ) qs_d = 0;
      }
      if (!ok) *abort_flag = 1;
    }
  } else {
    const int wq = warp & 3;
    const int half = (warp - 2) >> 2;     // which 32 of the step's 64 query columns this warpgroup owns
    const int c0 = half * 32;
    const int row = wq * 32 + lane_id();  // key row inside the block
    const int tid = threadIdx.x - 64;     // 0..255 among the softmax threads
    const uint32_t lane_off = uint32_t(wq * 32) << 16;
    const float sl2 = p.scale * kLog2e;
    const int k_pos = p.k_pos0 + k0 + row;
    const bool k_valid = (k0 + row) < p.Skv;
    bool ok = true;
    // Per-query statistics (-LSE * log2 e and D) of a step, fetched one step ahead so that the global-memory
    // latency is hidden behind the previous step's work: thread t < 64 carries -lse2 of query t, 64 <= t < 128 D.
    int ld_h = h0, ld_qs = qs0, ld_it = 0;   // (head, query step) of the next statistics fetch; no division in the loop
    auto load_stat = [&]() -> float {
      float v = 0.f;
      if (tid < 128 && ld_it < n_it) {
        const int q = ld_qs * 64 + (tid & 63);
        if (q >= p.Sq) {
          v = (tid < 64) ? INFINITY : 0.f;    // rows past the end: -inf after scaling, 2^-inf = 0
        } else {
          const float* src = (tid < 64) ? p.LSE : p.D;
          v = src[(size_t(b) * p.nheads + ld_h) * p.Sq + q];   // raw; scaled by stat_scale when it is stored, so
        }                                                        // that nothing waits for the load here
      }
      ++ld_it;
      if (++ld_qs == n_qs) { ld_qs = qs0; ++ld_h; }
      return v;
    };
    const float stat_scale = (tid < 64) ? -kLog2e : 1.f;   // -LSE * log2 e for the first 64 threads, D as it is
    float stat_next = load_stat();
    if (n_it > 0) {
      if (tid < 128) sStats[tid] = stat_next * stat_scale;
      mbar_arrive(&stats_full[0]);
      stat_next = load_stat();
    }
    int cur_qs = qs0;
    for (int it = 0; it < n_it; ++it) {
      const int st = it & 1;
      const int qrow = cur_qs * 64;
      if (++cur_qs == n_qs) cur_qs = qs0;
      if (!mbar_wait_warp(&stats_full[st], (it >> 1) & 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
      if (!mbar_wait_warp(&st_full[st], (it >> 1) & 1, p.status, kTimeoutTmemFull, abort_flag)) { ok = false; break; }
      tc_fence_after();
      float pt[32], ds[32];
      {
        uint32_t r0[32], r1[32];
        tmem_ld32(tST[st] + lane_off + c0, r0);
        tmem_ld32(tDPT[st] + lane_off + c0, r1);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) { pt[i] = __uint_as_float(r0[i]); ds[i] = __uint_as_float(r1[i]); }
      }
      tc_fence_before();
      mbar_arrive(&st_empty[st]);
      {
        const float4* nl4 = reinterpret_cast<const float4*>(sStats + st * 128 + c0);   // -lse2
        const float4* dd4 = nl4 + 16;                                                  // D
        // only steps that touch the diagonal, or a key block with rows past the end, need the mask
        const bool need_mask = !k_valid || (p.causal && (p.q_pos0 + qrow < p.k_pos0 + k0 + 127));
        const int q_base = p.q_pos0 + qrow + c0;
        if (!need_mask) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 nl = nl4[i >> 2], dd = dd4[i >> 2];
            const float nlv[4] = {nl.x, nl.y, nl.z, nl.w}, ddv[4] = {dd.x, dd.y, dd.z, dd.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              pt[i + u] = ex2(fmaf(pt[i + u], sl2, nlv[u]));
              ds[i + u] = pt[i + u] * (ds[i + u] - ddv[u]);   // in the same loop: these overlap with the exp2 unit
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 nl = nl4[i >> 2], dd = dd4[i >> 2];
            const float nlv[4] = {nl.x, nl.y, nl.z, nl.w}, ddv[4] = {dd.x, dd.y, dd.z, dd.w};
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const bool dead = !k_valid || (p.causal && k_pos > q_base + i + u);
              pt[i + u] = dead ? 0.f : ex2(fmaf(pt[i + u], sl2, nlv[u]));
              ds[i + u] = pt[i + u] * (ds[i + u] - ddv[u]);
            }
          }
        }
      }
      // the next step's statistics go to the other buffer: every thread is past its reads of that buffer (they
      // all arrived on this step's stats barrier after finishing the previous step)
      if (it + 1 < n_it) {
        if (tid < 128) sStats[(st ^ 1) * 128 + tid] = stat_next * stat_scale;
        mbar_arrive(&stats_full[st ^ 1]);
        stat_next = load_stat();
      }
      if (it >= 2) {   // these buffers were last read by the dV / dK products of step it-2
        if (!mbar_wait_warp(&pds_empty[st], ((it >> 1) & 1) ^ 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
      }
      uint8_t* sPTs = sPT + st * DkvSmem<HD>::kPT;
      uint8_t* sDSTs = sDST + st * DkvSmem<HD>::kPT;
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        uint4 u, w;
        u.x = pack_bf16(pt[cc * 8 + 0], pt[cc * 8 + 1]); u.y = pack_bf16(pt[cc * 8 + 2], pt[cc * 8 + 3]);
        u.z = pack_bf16(pt[cc * 8 + 4], pt[cc * 8 + 5]); u.w = pack_bf16(pt[cc * 8 + 6], pt[cc * 8 + 7]);
        w.x = pack_bf16(ds[cc * 8 + 0], ds[cc * 8 + 1]); w.y = pack_bf16(ds[cc * 8 + 2], ds[cc * 8 + 3]);
        w.z = pack_bf16(ds[cc * 8 + 4], ds[cc * 8 + 5]); w.w = pack_bf16(ds[cc * 8 + 6], ds[cc * 8 + 7]);
        *reinterpret_cast<uint4*>(sPTs + sw128_offset(row, half * 4 + cc)) = u;
        *reinterpret_cast<uint4*>(sDSTs + sw128_offset(row, half * 4 + cc)) = w;
      }
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(&pds_full[st]);
    }
    // ---- epilogue ----
    const int krow = k0 + row;
    const int dkslot = p.dkmap.slot(h0, p.qpg), dvslot = p.dvmap.slot(h0, p.qpg);
    hg_lp_t* dk = p.dK + int64_t(krow) * p.dk_ss + int64_t(b) * p.dk_sb + int64_t(dkslot) * HD;
    hg_lp_t* dv = p.dV + int64_t(krow) * p.dv_ss + int64_t(b) * p.dv_sb + int64_t(dvslot) * HD;
    if (n_it == 0) {
      if (krow < p.Skv) {
#pragma unroll
        for (int i = half; i < HD / 8; i += 2) {
          reinterpret_cast<uint4*>(dk)[i] = make_uint4(0, 0, 0, 0);
          reinterpret_cast<uint4*>(dv)[i] = make_uint4(0, 0, 0, 0);
        }
      }
    } else if (ok && !*abort_flag &&
               mbar_wait_warp(&pds_empty[(n_it - 1) & 1], ((n_it - 1) >> 1) & 1, p.status, kTimeoutOther, abort_flag)) {
      tc_fence_after();
#pragma unroll
      for (int c = half; c < HD / 32; c += 2) {   // the two warpgroups take alternate 32-column chunks
        uint32_t r0[32], r1[32];
        tmem_ld32(tDV + lane_off + c * 32, r0);
        tmem_ld32(tDK + lane_off + c * 32, r1);
        tmem_ld_wait();
        if (krow < p.Skv) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 u, w;
            u.x = pack_bf16(__uint_as_float(r0[q * 8 + 0]), __uint_as_float(r0[q * 8 + 1]));
            u.y = pack_bf16(__uint_as_float(r0[q * 8 + 2]), __uint_as_float(r0[q * 8 + 3]));
            u.z = pack_bf16(__uint_as_float(r0[q * 8 + 4]), __uint_as_float(r0[q * 8 + 5]));
            u.w = pack_bf16(__uint_as_float(r0[q * 8 + 6]), __uint_as_float(r0[q * 8 + 7]));
            w.x = pack_bf16(__uint_as_float(r1[q * 8 + 0]) * p.scale, __uint_as_float(r1[q * 8 + 1]) * p.scale);
            w.y = pack_bf16(__uint_as_float(r1[q * 8 + 2]) * p.scale, __uint_as_float(r1[q * 8 + 3]) * p.scale);
            w.z = pack_bf16(__uint_as_float(r1[q * 8 + 4]) * p.scale, __uint_as_float(r1[q * 8 + 5]) * p.scale);
            w.w = pack_bf16(__uint_as_float(r1[q * 8 + 6]) * p.scale, __uint_as_float(r1[q * 8 + 7]) * p.scale);
            reinterpret_cast<uint4*>(dv + c * 32)[q] = u;
            reinterpret_cast<uint4*>(dk + c * 32)[q] = w;
          }
        }
      }
    } else {
      *abort_flag = 1;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// =================================================================================================
// Backward, part 1 with 128-query steps and the probabilities kept in tensor memory (both head dims; gpt2-xl sized,
// 8 x 1024 x 25 heads of 64: 170 -> 152 us against the 64-query kernel).
// The 64-query version issues its score products with N = 64, which occupy the tensor core as long as N = 128 would,
// and stages P^T / dS^T through 64 KB of shared memory.  Here a step covers 128 queries:
//   S^T = K Q^T and dP^T = V dO^T are 128 x 128 products (8 MMAs each);
//   the softmax threads turn them into P^T = exp2(S^T c - lse) and dS^T = P^T (dP^T - D) and store both back into
//   tensor memory as packed 16-bit pairs;
//   dV += P^T dO and dK += dS^T Q take their A operand from tensor memory (8 MMAs each, K = 128 queries).
// Per 128 queries that is 32 MMAs instead of 48, no shared-memory traffic from the softmax threads, and the 64 KB
// of staging buffers become Q / dO ring slots (three of Q, two of dO: a Q tile lives from its S^T product to its
// dK product, a dO tile from dP^T to dV).
//
// Tensor memory (512 columns): S^T 0..127, dP^T 128..255, dV 256..383, dK 384..511.  A softmax thread (one key row,
// the 128 / NWG query columns of its warpgroup) loads its S^T values and releases the S^T columns at once, so that
// S^T of the next step is computed while this step's exponentials run; once dP^T has arrived it loads its dP^T
// values and then owns those columns: the packed P^T goes over their first half, the packed dS^T over the second.
// The tensor core executes MMAs in issue order, which makes the reuse safe: dP^T(i+1) is issued after dV(i) and
// dK(i), the readers of P^T(i) and dS^T(i).  Per step the MMA warp issues S^T(i+1) when the S^T(i) columns are
// free, dV(i) when P^T(i) is stored, dK(i) and dP^T(i+1) when dS^T(i) is stored.
//
// Two warps fetch the statistics of the queries a step ahead.  In the softmax threads that cost registers: taken out, with the
// probabilities kept in fp32, head dim 64, 8 x 1024 tokens and 25 heads 141 -> 106 us.  Where ds has pieces the threads also store
// dS for the dQ product, half of it between the two halves of their arithmetic (all at the end: 629 against 603 us at 2 x 4096,
// 32 heads of 128; none: 518).
// =================================================================================================

constexpr int kDkvAuxRegs = 64, kDkvSoftmaxRegs = 104;
static_assert(128 * kDkvAuxRegs + 512 * kDkvSoftmaxRegs <= 640 * 96, "setmaxnreg deals out what the block was launched with");
__device__ __forceinline__ float4 lds_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}

template <int HD>
struct Dkv128Smem {
  static constexpr int kKV = 128 * HD * 2;       // resident K or V
  static constexpr int kQD = 128 * HD * 2;       // one Q or dO tile
  static constexpr int kQStages = 3;
  static constexpr int kDOStages = 2;
  static constexpr int kStats = 2 * 2 * 128 * 4;  // -lse*log2e and -D of a step, double buffered
  static constexpr int kBars = 256;
  static constexpr int kUsed = 2 * kKV + (kQStages + kDOStages) * kQD + kStats + kBars;
  // head dim 128: everything a CTA can have; the 1024-byte alignment of the tiles comes out of the rest
  static constexpr int kTotal = HD == 128 ? 232448 : kUsed + 1024;
};

// NWG = 4 softmax warpgroups: thread == key row, warpgroup g owns query columns [g * 128 / NWG, (g + 1) * 128 / NWG)
// of every step.  Four warpgroups put four warps on every scheduler, which is what keeps the exp2 unit and the FMA
// pipe busy through the latencies of the loads from tensor memory and of the dependent exp2 / convert chains.
// SHARED: key blocks may be shared between CTAs (p.chunk > 0).
template <int HD, int NWG, bool SHARED>
__global__ void __launch_bounds__(128 + 128 * NWG, 1)
flash_bwd_dkv128_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                        const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                        const BwdParams p, const __grid_constant__ DsPieces ds) {
  static_assert(HD == 64 || HD == 128, "tensor memory holds S^T, dP^T and two accumulators of up to 128 columns");
  static_assert(NWG == 4, "a thread's 32 columns: two halves of 16");
  constexpr int kSoftmaxWarps = 4 * NWG;
  constexpr int CPT = 128 / NWG;               // query columns per thread and step
  // A CTA works on further blocks of the grid (WorkSlot).  Whole backward, us, one block a CTA / so, causal: head dim 64, 16 x 256
  // tokens and 25 heads 94 / 78, 8 x 1024 283 / 250, 4 x 2048 418 / 383, 1 x 8192 1205 / 1151, 12 heads 4096 210 / 203, 8192 634 /
  // 608, 32 heads on 8 4 x 2048 525 / 491; head dim 128, 32 heads 16 x 256 168 / 138, 8 x 1024 433 / 389, 4 x 2048 610 / 574,
  // 2 x 4096 967 / 949, 1 x 8192 1689 / 1688, 28 on 4 8 x 1024 360 / 341.  A grid of one wave pays: 12 heads of 64, 300 tokens
  // 23.1 / 23.5.
  extern __shared__ uint8_t smem_raw[];
  using L = Dkv128Smem<HD>;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (base + L::kUsed > smem_raw + L::kTotal) {   // the same for every thread: nothing has been set up yet
    if (threadIdx.x == 0) set_status(p.status, kTimeoutOther);
    return;
  }
  uint8_t* sK = base;
  uint8_t* sV = sK + L::kKV;
  constexpr int NQ = L::kQStages, ND = L::kDOStages;
  uint8_t* sQ = sV + L::kKV;                 // NQ tiles
  uint8_t* sDO = sQ + NQ * L::kQD;           // ND tiles
  float* sStats = reinterpret_cast<float*>(sDO + ND * L::kQD);   // [2][256]: 128 x -lse2, 128 x -D
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sStats) + L::kStats);
  uint64_t* kv_full = bars;          // 1
  uint64_t* q_full = bars + 1;       // 3
  uint64_t* q_empty = bars + 4;      // 3
  uint64_t* do_full = bars + 7;      // 2
  uint64_t* do_empty = bars + 9;     // 2
  uint64_t* st_full = bars + 11;     // S^T of a step is in tensor memory
  uint64_t* dpt_full = bars + 12;    // dP^T of a step is in tensor memory
  uint64_t* p_full = bars + 13;      // every thread has stored its part of P^T
  uint64_t* ds_full = bars + 14;     // every thread has stored its part of dS^T
  uint64_t* acc_full = bars + 15;    // the last dK product has completed
  uint64_t* stats_full = bars + 16;  // 2
  uint64_t* x_free = bars + 18;      // every thread has loaded its S^T values: the S^T columns may be overwritten
  uint64_t* kv_empty = bars + 19;    // the last products that read K and V have completed
  uint64_t* acc_empty = bars + 20;   // the epilogue has read dV and dK
  uint64_t* stats_empty = bars + 27; // 2
  // [2], beside a step's statistics: its tile of dS, its first query row
  hg_lp_t** sTile = reinterpret_cast<hg_lp_t**>(bars + 29);
  int* sRow = reinterpret_cast<int*>(bars + 31);
  const WorkSlot work{reinterpret_cast<uint4*>(bars + 24), bars + 21, bars + 22};
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 26);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int n_qs = (p.Sq + 127) / 128;
  // What a block of the grid is: a kv head's key block and some of its query steps, heads outside, queries inside.
  struct Steps {
    int g, b, k0, sharers;       // kv head, sequence, first key; blocks of the grid that share this key block
    int h0, qs0, h, qs, n_it;    // first query head, first 128-row step; head and query step of the first step; steps
  };
  auto steps_of = [&](const Block& w) {
    int kb = w.x, mine = 0, sharers = 1;
    if constexpr (SHARED) {
      int left = w.x;
      for (kb = 0;; ++kb) {
        sharers = dkv_block_ctas(p, dkv_block_steps(p, kb));
        if (left < sharers) break;
        left -= sharers;
      }
      mine = left;
    }
    Steps t;
    t.g = w.y + p.g0_c; t.b = w.z + p.b0_c; t.k0 = kb * 128; t.sharers = sharers;
    int q_first = 0;                                          // first query row that can see this key block
    if (p.causal) q_first = max(0, p.k_pos0 + t.k0 - p.q_pos0);
    t.qs0 = q_first / 128;
    const int per_head = max(0, n_qs - t.qs0), n_steps = per_head * p.qpg;
    const int it0 = SHARED ? n_steps * mine / sharers : 0;
    t.n_it = SHARED ? n_steps * (mine + 1) / sharers - it0 : n_steps;
    t.h0 = t.g * p.qpg;
    t.h = t.h0 + (SHARED && per_head > 0 ? it0 / per_head : 0);
    t.qs = t.qs0 + (SHARED && per_head > 0 ? it0 % per_head : 0);
    return t;
  };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmDO);
    mbar_init(kv_full, 1);
    for (int i = 0; i < NQ; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
    for (int i = 0; i < ND; ++i) { mbar_init(&do_full[i], 1); mbar_init(&do_empty[i], 1); }
    mbar_init(st_full, 1);
    mbar_init(dpt_full, 1);
    mbar_init(p_full, kSoftmaxWarps);       // one arrival per softmax warp (mbar_arrive_warp)
    mbar_init(ds_full, kSoftmaxWarps);
    mbar_init(x_free, kSoftmaxWarps);
    mbar_init(acc_full, 1);
    mbar_init(kv_empty, 1);
    mbar_init(acc_empty, kSoftmaxWarps);
    mbar_init(work.full, 1);
    mbar_init(work.empty, 4 + kSoftmaxWarps);
    for (int i = 0; i < 2; ++i) { mbar_init(&stats_full[i], 2); mbar_init(&stats_empty[i], kSoftmaxWarps); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tST = tmem, tDPT = tmem + 128, tDV = tmem + 256, tDK = tmem + 384;

  Block blk{int(blockIdx.x), int(blockIdx.y), int(blockIdx.z)};
  // 640 threads start with 96 registers each.  A spilled one costs a trip to L2: head dim 128 leaves no L1 beside its shared memory
  // (spills of the step loop doubled the kernel's time).
  if (warp < 4) regs_dec<kDkvAuxRegs>();

  if (warp == 0) {
    // the whole warp walks the loop, one elected lane issues the copies (see producer_loop in gemm_core.cuh)
    const bool issuer = elect_one() != 0;
    int qs_slot = 0, ds_slot = 0, nkv = 0, n = 0;    // ring positions, K / V tiles loaded so far, blocks done
    uint32_t qph = 0, dph = 0;
    bool ok = true, asked = false;
    for (; ok; ++n) {
      asked = false;
      const Steps t = steps_of(blk);
      const int kslot = p.kmap.slot(t.h0, p.qpg), vslot = p.vmap.slot(t.h0, p.qpg), b = t.b;
      if (t.n_it > 0) {
        if (!mbar_wait_warp(kv_empty, (nkv & 1) ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { ok = false; break; }
        ++nkv;
        if (issuer) mbar_expect_tx(kv_full, 2 * L::kKV);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) {
          if (issuer) tma_load_4d(sK + c * 128 * 128, &tmK, kv_full, c * 64, kslot, t.k0, b);
          if (issuer) tma_load_4d(sV + c * 128 * 128, &tmV, kv_full, c * 64, vslot, t.k0, b);
        }
        int h = t.h, qs = t.qs;
        for (int it = 0; it < t.n_it; ++it) {
          const int qrow = qs * 128;
          const int qslot = p.qmap.slot(h, p.qpg), doslot = p.domap.slot(h, p.qpg);
          if (!mbar_wait_warp(&q_empty[qs_slot], qph ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { ok = false; break; }
          if (issuer) mbar_expect_tx(&q_full[qs_slot], L::kQD);
#pragma unroll
          for (int c = 0; c < HD / 64; ++c)
            if (issuer) tma_load_4d(sQ + qs_slot * L::kQD + c * 128 * 128, &tmQ, &q_full[qs_slot], c * 64, qslot, qrow, b);
          if (!mbar_wait_warp(&do_empty[ds_slot], dph ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { ok = false; break; }
          if (issuer) mbar_expect_tx(&do_full[ds_slot], L::kQD);
#pragma unroll
          for (int c = 0; c < HD / 64; ++c)
            if (issuer) tma_load_4d(sDO + ds_slot * L::kQD + c * 128 * 128, &tmDO, &do_full[ds_slot], c * 64, doslot, qrow, b);
          if (++qs_slot == NQ) { qs_slot = 0; qph ^= 1; }
          if (++ds_slot == ND) { ds_slot = 0; dph ^= 1; }
          if (++qs == n_qs) { qs = t.qs0; ++h; }
        }
      }
      if (!ok) break;
      // The next block is asked for once this one's loads are all on their way.  Asked for earlier it waits for a CTA that is busy
      // while others run dry (12 heads of 64, 4096 tokens: 203 -> 233 us).  The answer slot is free once every warp has this block.
      if (n > 0 && !mbar_wait_warp(work.empty, (n - 1) & 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
      if (issuer) work_request(work);
      __syncwarp();
      asked = true;
      if (!work_take(work, n, blk, p.status, abort_flag)) break;
    }
    if (!ok) {
      *abort_flag = 1;
      if (asked) work_drain(work, n);
    }
  } else if (warp == 1) {
      // the whole warp walks the loop, one elected lane issues (see mma_loop in gemm_core.cuh)
      const bool issuer = elect_one() != 0;
      constexpr uint32_t idesc_st = make_idesc_lp(128, 128, false, false);
      constexpr uint32_t idesc_acc = make_idesc_lp(128, HD, false, true);
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aQ0 = smem_u32(sQ), aDO0 = smem_u32(sDO);
      // queries 16kk.. belong to warpgroup 16kk / CPT; its packed P^T values start at the first of its CPT columns of
      // the dP^T range, its packed dS^T values CPT / 2 columns further
      auto packed_col = [](int kk) -> uint32_t { return uint32_t((16 * kk / CPT) * CPT + (16 * kk % CPT) / 2); };
      // ring positions: Q / dO tile of the next S^T / dP^T issue, and of the next dK / dV issue
      int q_s = 0, q_k = 0, d_p = 0, d_v = 0;
      uint32_t qph_s = 0, dph_p = 0;
      auto issue_st = [&]() -> bool {     // S^T of the next step
        if (!mbar_wait_warp(&q_full[q_s], qph_s, p.status, kTimeoutSmemFull, abort_flag)) return false;
        tc_fence_after();
        const uint32_t aQ = aQ0 + q_s * L::kQD;
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk)
            umma_f16_ss(tST, kmajor_desc(aK, 128, kk), kmajor_desc(aQ, 128, kk), idesc_st, kk != 0);
          umma_commit(st_full);
        }
        __syncwarp();
        if (++q_s == NQ) { q_s = 0; qph_s ^= 1; }
        return true;
      };
      auto issue_dpt = [&]() -> bool {    // dP^T of the next step
        if (!mbar_wait_warp(&do_full[d_p], dph_p, p.status, kTimeoutSmemFull, abort_flag)) return false;
        tc_fence_after();
        const uint32_t aDO = aDO0 + d_p * L::kQD;
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk)
            umma_f16_ss(tDPT, kmajor_desc(aV, 128, kk), kmajor_desc(aDO, 128, kk), idesc_st, kk != 0);
          umma_commit(dpt_full);
        }
        __syncwarp();
        if (++d_p == ND) { d_p = 0; dph_p ^= 1; }
        return true;
      };
      bool ok = true;
      int nkv = 0;                        // blocks with steps so far
      uint32_t ph = 1;                    // of a step's barriers
      for (int n = 0; ok; ++n) {
      const int n_it = steps_of(blk).n_it;
      if (n_it > 0) {
      ok = mbar_wait_warp(kv_full, nkv & 1, p.status, kTimeoutSmemFull, abort_flag);
      if (ok) ok = issue_st();
      if (ok) ok = issue_dpt();
      if (ok && n_it == 1 && issuer) umma_commit(kv_empty);
      __syncwarp();
      HG_DKV_TIMERS(tm_wait_x, tm_wait_p, tm_wait_ds, tm_issue);
      for (int it = 0; ok && it < n_it; ++it) {
        ph ^= 1;
        HG_DKV_TICK(t0);
        // ---- S^T(it+1), as soon as the S^T(it) values are in the threads' registers
        if (!mbar_wait_warp(x_free, ph, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
        tc_fence_after();
        HG_DKV_TOCK(tm_wait_x, t0);
        if (it + 1 < n_it) { ok = issue_st(); if (!ok) break; }
        HG_DKV_TOCK(tm_issue, t0);
        // ---- dV(it); dV and dK still hold the last block's sums until its epilogue has read them
        if (it == 0 && !mbar_wait_warp(acc_empty, (nkv & 1) ^ 1, p.status, kTimeoutTmemEmpty, abort_flag)) { ok = false; break; }
        if (!mbar_wait_warp(p_full, ph, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
        tc_fence_after();
        HG_DKV_TOCK(tm_wait_p, t0);
        if (issuer) {
          const uint32_t aDO = aDO0 + d_v * L::kQD;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)     // k-step kk = queries 16kk..16kk+15 = 8 packed columns of their warpgroup's range
            umma_f16_ts(tDV, tDPT + packed_col(kk), mnmajor_desc(aDO, 128, kk), idesc_acc, (it | kk) != 0);
          umma_commit(&do_empty[d_v]);
        }
        __syncwarp();
        if (++d_v == ND) d_v = 0;
        HG_DKV_TOCK(tm_issue, t0);
        // ---- dK(it), then dP^T(it+1) over the columns dV and dK have just read
        if (!mbar_wait_warp(ds_full, ph, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
        tc_fence_after();
        HG_DKV_TOCK(tm_wait_ds, t0);
        if (issuer) {
          const uint32_t aQ = aQ0 + q_k * L::kQD;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_f16_ts(tDK, tDPT + CPT / 2 + packed_col(kk), mnmajor_desc(aQ, 128, kk), idesc_acc, (it | kk) != 0);
          umma_commit(&q_empty[q_k]);
        }
        __syncwarp();
        if (++q_k == NQ) q_k = 0;
        if (it + 1 < n_it) {
          ok = issue_dpt();
          if (!ok) break;
          if (it + 2 == n_it && issuer) umma_commit(kv_empty);     // the last of the block's products that read K and V
          __syncwarp();
        }
        HG_DKV_TOCK(tm_issue, t0);
      }
      HG_DKV_REPORT(8, n_it, tm_wait_x, tm_wait_p, tm_wait_ds, tm_issue);
      if (ok && issuer) umma_commit(acc_full);
      __syncwarp();
      ++nkv;
      }
      if (ok && !work_take(work, n, blk, p.status, abort_flag)) break;
      }
      if (!ok) *abort_flag = 1;
  } else if (warp < 4) {
    // Per-query statistics of the steps, fetched one ahead: a thread carries -lse * log2 e and -D of two queries of a step.
    const int q2 = threadIdx.x - 64;
    bool ok = true;
    uint32_t done = 0;                    // steps so far
    for (int n = 0; ok; ++n) {
      const Steps t = steps_of(blk);
      int h = t.h, qs = t.qs, ld_h = t.h, ld_qs = t.qs;
      auto head_tile = [&]() {             // the first of this key block's and head's
        return ds_tile(ds, (t.b - p.b0_c) * p.nh_c + h - p.h0_c, ds_tiles_before(p, (p.Skv + 127) / 128), ds_tiles_before(p, t.k0 / 128));
      };
      hg_lp_t* tile = nullptr;
      if (ds.heads > 0 && t.n_it > 0) tile = head_tile() + (qs - t.qs0) * (128 * 128);
      float lse[2], d[2];
      auto fetch = [&]() {
        const size_t at = (size_t(t.b) * p.nheads + ld_h) * p.Sq;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int q = ld_qs * 128 + q2 + i * 64;
          lse[i] = q < p.Sq ? p.LSE[at + q] : INFINITY;      // rows past the end: 2^-inf = 0
          d[i] = q < p.Sq ? p.D[at + q] : 0.f;
        }
        if (++ld_qs == n_qs) { ld_qs = t.qs0; ++ld_h; }
      };
      if (t.n_it > 0) fetch();
      for (int it = 0; it < t.n_it; ++it, ++done) {
        const uint32_t sb = done & 1;
        if (!mbar_wait_warp(&stats_empty[sb], ((done >> 1) & 1) ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { ok = false; break; }
        float* st = sStats + sb * 256;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          st[q2 + i * 64] = -lse[i] * kLog2e;
          st[128 + q2 + i * 64] = -d[i];
        }
        if (q2 == 0) {
          sTile[sb] = tile;
          sRow[sb] = qs * 128;
        }
        mbar_arrive_warp(&stats_full[sb]);
        tile += 128 * 128;
        if (++qs == n_qs) {
          qs = t.qs0;
          ++h;
          if (ds.heads > 0 && it + 1 < t.n_it) tile = head_tile();
        }
        if (it + 1 < t.n_it) fetch();
      }
      if (ok && !work_take(work, n, blk, p.status, abort_flag)) break;
    }
    if (!ok) *abort_flag = 1;
  } else {
    regs_inc<kDkvSoftmaxRegs>();
    const int wq = warp & 3;
    const int half = (warp - 4) >> 2;     // warpgroup: which CPT of the step's 128 query columns these threads own
    const int c0 = half * CPT;
    const int row = wq * 32 + lane_id();  // key row inside the block
    const uint32_t lane_off = uint32_t(wq * 32) << 16;
    const float sl2 = p.scale * kLog2e;
    bool ok = true;
    int nkv = 0;                          // blocks with steps so far
    uint32_t done = 0;                    // steps so far
    for (int n = 0; ok; ++n) {
    int steps = steps_of(blk).n_it, k_row;
    {
      const Steps t = steps_of(blk);
      k_row = t.k0 + row;
    }
    HG_DKV_TIMERS(tm_wait_a, tm_a, tm_wait_b, tm_b);
    for (int it = 0; it < steps; ++it, ++done) {
      const uint32_t sb = done & 1, ph = done & 1;
      HG_DKV_TICK(t0);
      const uint32_t st = smem_u32(sStats) + sb * 1024 + c0 * 4;
      float pf[CPT];                      // this thread's probabilities, kept for the second phase
      // ---------------- S^T -> probabilities (kept in registers; the S^T columns are released at once)
      if (!mbar_wait_warp(&stats_full[sb], (done >> 1) & 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
      if (!mbar_wait_warp(st_full, ph, p.status, kTimeoutTmemFull, abort_flag)) { ok = false; break; }
      tc_fence_after();
      HG_DKV_TOCK(tm_wait_a, t0);
      {
        uint32_t r[CPT];
        tmem_ld32(tST + lane_off + c0, r);
        tmem_ld_wait();
        tc_fence_before();
        mbar_arrive_warp(x_free);
        // Only steps that touch the diagonal, or a key block with rows past the end, need the mask: columns before `seen` are 0.
        // The masked and the plain form are two straight-line bodies: a branch inside the element loop would cut it
        // into sixteen basic blocks, and the compiler schedules (overlaps the loads, FMAs and exp2 of different
        // elements) only inside one.
        const int behind = p.k_pos0 + k_row - p.q_pos0 - sRow[sb];       // of this row's key and the step's first query
        const int seen = k_row >= p.Skv ? CPT : p.causal ? behind - c0 : 0;
        const bool need_mask = (k_row - row + 128 > p.Skv) || (p.causal && behind - row + 127 > 0);
        auto probabilities = [&](auto masked) {
#pragma unroll
          for (int i = 0; i < CPT; i += 4) {
            const float4 nl = lds_f4(st + i * 4);
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
              const float2 x = fma2(make_float2(__uint_as_float(r[i + u]), __uint_as_float(r[i + u + 1])), make_float2(sl2, sl2),
                                    u == 0 ? make_float2(nl.x, nl.y) : make_float2(nl.z, nl.w));
              const float e0 = ex2(x.x), e1 = ex2(x.y);
              pf[i + u] = decltype(masked)::value && i + u < seen ? 0.f : e0;
              pf[i + u + 1] = decltype(masked)::value && i + u + 1 < seen ? 0.f : e1;
            }
          }
        };
        if (need_mask) probabilities(std::true_type{});
        else probabilities(std::false_type{});
      }
      HG_DKV_TOCK(tm_a, t0);
      // ---------------- dP^T -> dS^T; P^T and dS^T go, packed, over this thread's own dP^T columns
      if (!mbar_wait_warp(dpt_full, ph, p.status, kTimeoutTmemFull, abort_flag)) { ok = false; break; }
      tc_fence_after();
      HG_DKV_TOCK(tm_wait_b, t0);
      static_assert(CPT == 32, "P^T takes the columns of the first half of dP^T, dS^T those of the second");
      uint32_t dsp[CPT / 2];
      {
        const uint32_t dpt = tDPT + lane_off + c0;
        uint32_t ra[16], rb[16];
        auto half_ds = [&](const uint32_t(&r)[16], int at) {
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const float4 nd = lds_f4(st + 512 + (at + i) * 4);
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
              const float2 d = mul2(make_float2(pf[at + i + u], pf[at + i + u + 1]),
                                    add2(make_float2(__uint_as_float(r[i + u]), __uint_as_float(r[i + u + 1])),
                                         u == 0 ? make_float2(nd.x, nd.y) : make_float2(nd.z, nd.w)));
              dsp[(at + i + u) >> 1] = pack_bf16(d.x, d.y);
            }
          }
        };
        tmem_ld16(dpt, ra);
        tmem_ld_wait();
        {
          uint32_t pp[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) pp[i] = pack_bf16(pf[2 * i], pf[2 * i + 1]);
          tmem_st16(dpt, pp);
        }
        tmem_ld16(dpt + 16, rb);
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive_warp(p_full);
        half_ds(ra, 0);
        if (ds.heads > 0) {
          hg_lp_t* out = sTile[sb] + ((row >> 6) * (64 * 128) + c0 * 64 + (row & 63) * 8);
#pragma unroll
          for (int i = 0; i < 2; ++i)
            *reinterpret_cast<uint4*>(out + i * 512) = make_uint4(dsp[4 * i], dsp[4 * i + 1], dsp[4 * i + 2], dsp[4 * i + 3]);
        }
        tmem_ld_wait();
        half_ds(rb, 16);
        tmem_st16(dpt + 16, dsp);
        if (ds.heads > 0) {
          hg_lp_t* out = sTile[sb] + ((row >> 6) * (64 * 128) + c0 * 64 + (row & 63) * 8);
#pragma unroll
          for (int i = 2; i < 4; ++i)
            *reinterpret_cast<uint4*>(out + i * 512) = make_uint4(dsp[4 * i], dsp[4 * i + 1], dsp[4 * i + 2], dsp[4 * i + 3]);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive_warp(ds_full);
      mbar_arrive_warp(&stats_empty[sb]);
      HG_DKV_TOCK(tm_b, t0);
    }
    // the epilogue's numbers are worked out again instead of being kept through the steps, where registers are short
    asm volatile("" : "+r"(blk.x), "+r"(blk.y), "+r"(blk.z));
    const Steps t = steps_of(blk);
    const int k0 = t.k0, b = t.b, g = t.g, n_it = t.n_it, h0 = t.h0, sharers = t.sharers;
    HG_DKV_REPORT(0, n_it, tm_wait_a, tm_a, tm_wait_b, tm_b);
    // ---- epilogue ----
    const int krow = k0 + row;
    const int dkslot = p.dkmap.slot(h0, p.qpg), dvslot = p.dvmap.slot(h0, p.qpg);
    hg_lp_t* dk = p.dK + int64_t(krow) * p.dk_ss + int64_t(b) * p.dk_sb + int64_t(dkslot) * HD;
    hg_lp_t* dv = p.dV + int64_t(krow) * p.dv_ss + int64_t(b) * p.dv_sb + int64_t(dvslot) * HD;
    if (n_it == 0) {
      if (krow < p.Skv) {
#pragma unroll
        for (int i = half; i < HD / 8; i += NWG) {
          reinterpret_cast<uint4*>(dk)[i] = make_uint4(0, 0, 0, 0);
          reinterpret_cast<uint4*>(dv)[i] = make_uint4(0, 0, 0, 0);
        }
      }
    } else if (ok && !*abort_flag && mbar_wait_warp(acc_full, nkv & 1, p.status, kTimeoutOther, abort_flag)) {
      tc_fence_after();
#pragma unroll
      for (int c = half; c < HD / 32; c += NWG) {   // the warpgroups take alternate 32-column chunks
        uint32_t r0[32], r1[32];
        tmem_ld32(tDV + lane_off + c * 32, r0);
        tmem_ld32(tDK + lane_off + c * 32, r1);
        tmem_ld_wait();
        if (SHARED && sharers > 1) {                // summed, scaled and rounded by dkv_sum_kernel
          float* part = p.part + ((size_t(b) * gridDim.y + g) * gridDim.x + blk.x) * (2 * 128 * HD) + row * HD + c * 32;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            reinterpret_cast<uint4*>(part)[q] = make_uint4(r0[q * 4], r0[q * 4 + 1], r0[q * 4 + 2], r0[q * 4 + 3]);
            reinterpret_cast<uint4*>(part + 128 * HD)[q] = make_uint4(r1[q * 4], r1[q * 4 + 1], r1[q * 4 + 2], r1[q * 4 + 3]);
          }
        } else if (krow < p.Skv) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 u, w;
            u.x = pack_bf16(__uint_as_float(r0[q * 8 + 0]), __uint_as_float(r0[q * 8 + 1]));
            u.y = pack_bf16(__uint_as_float(r0[q * 8 + 2]), __uint_as_float(r0[q * 8 + 3]));
            u.z = pack_bf16(__uint_as_float(r0[q * 8 + 4]), __uint_as_float(r0[q * 8 + 5]));
            u.w = pack_bf16(__uint_as_float(r0[q * 8 + 6]), __uint_as_float(r0[q * 8 + 7]));
            w.x = pack_bf16(__uint_as_float(r1[q * 8 + 0]) * p.scale, __uint_as_float(r1[q * 8 + 1]) * p.scale);
            w.y = pack_bf16(__uint_as_float(r1[q * 8 + 2]) * p.scale, __uint_as_float(r1[q * 8 + 3]) * p.scale);
            w.z = pack_bf16(__uint_as_float(r1[q * 8 + 4]) * p.scale, __uint_as_float(r1[q * 8 + 5]) * p.scale);
            w.w = pack_bf16(__uint_as_float(r1[q * 8 + 6]) * p.scale, __uint_as_float(r1[q * 8 + 7]) * p.scale);
            reinterpret_cast<uint4*>(dv + c * 32)[q] = u;
            reinterpret_cast<uint4*>(dk + c * 32)[q] = w;
          }
        }
      }
      tc_fence_before();
      mbar_arrive_warp(acc_empty);
      ++nkv;
    } else {
      ok = false;
    }
    if (ok && !work_take(work, n, blk, p.status, abort_flag)) break;
    }
    if (!ok) *abort_flag = 1;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// dK and dV of the key blocks that several CTAs share: their parts added in CTA order, scaled, rounded once.  A CTA takes
// 16 rows of a key block, a thread eight columns of one row of dV or dK.
template <int HD>
__global__ void __launch_bounds__(4 * HD)
dkv_sum_kernel(const BwdParams p, int ctas) {
  const int g = blockIdx.y, b = blockIdx.z, kb = blockIdx.x >> 3;
  int first = 0;
  for (int i = 0; i < kb; ++i) first += dkv_block_ctas(p, dkv_block_steps(p, i));
  const int sharers = dkv_block_ctas(p, dkv_block_steps(p, kb));
  const int which = threadIdx.x / (2 * HD), t = threadIdx.x % (2 * HD);        // 0: dV, 1: dK
  const int row = (blockIdx.x & 7) * 16 + t / (HD / 8), c = t % (HD / 8) * 8;
  const int krow = kb * 128 + row;
  if (sharers < 2 || krow >= p.Skv) return;
  const float* part = p.part + ((size_t(b) * gridDim.y + g) * ctas + first) * (2 * 128 * HD) + (which * 128 + row) * HD + c;
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int i = 0; i < sharers; ++i) {
    const float4 u = __ldcs(reinterpret_cast<const float4*>(part + size_t(i) * (2 * 128 * HD)));
    const float4 w = __ldcs(reinterpret_cast<const float4*>(part + size_t(i) * (2 * 128 * HD)) + 1);
    s[0] += u.x; s[1] += u.y; s[2] += u.z; s[3] += u.w;
    s[4] += w.x; s[5] += w.y; s[6] += w.z; s[7] += w.w;
  }
  const float f = which ? p.scale : 1.f;
  const int h0 = g * p.qpg;
  hg_lp_t* out = which ? p.dK + int64_t(krow) * p.dk_ss + int64_t(b) * p.dk_sb + int64_t(p.dkmap.slot(h0, p.qpg)) * HD
                       : p.dV + int64_t(krow) * p.dv_ss + int64_t(b) * p.dv_sb + int64_t(p.dvmap.slot(h0, p.qpg)) * HD;
  *reinterpret_cast<uint4*>(out + c) = make_uint4(pack_bf16(s[0] * f, s[1] * f), pack_bf16(s[2] * f, s[3] * f),
                                                  pack_bf16(s[4] * f, s[5] * f), pack_bf16(s[6] * f, s[7] * f));
}

// =================================================================================================
// Backward, part 2 with 128-key steps (both head dims; head dim 64, 8 x 1024 x 25 heads: 182 us with 64-key steps
// staged through shared memory, 107 us).  A tcgen05.mma of shape 128 x N x 16 occupies the tensor core
// for the same time whatever N <= 256 is, so the score products are issued with N = 128 instead of 64: per 128 keys
// the kernel issues 24 MMAs (8 S, 8 dP, 8 dQ) where the 64-key version issues 40.  Shared memory holds three K
// stages and one V stage of 128 rows (128 KB) and Q and dO (64 KB); tensor memory holds one S / dP pair (256 columns),
// dQ (128) and two dS buffers (64 columns each): the softmax threads store dS there as packed 16-bit pairs and the
// dQ product takes it as its A operand, so nothing of a step goes through shared memory.  The S and dP products of
// step i+1 are issued as soon as the softmax threads have loaded step i into registers, so they overlap the
// arithmetic.  NWG softmax warpgroups (2 or 4): thread == query row, warpgroup g owns key columns
// [g * 128 / NWG, (g + 1) * 128 / NWG) of every step; four warpgroups put four warps on every scheduler, which is
// what covers the latencies of the tensor-memory loads and of the exp2 / convert chains.
// =================================================================================================
template <int HD>
struct Dq128Smem {
  static constexpr int kQ = 128 * HD * 2;      // resident Q or dO
  static constexpr int kKV = 128 * HD * 2;     // one stage of K or V
  // K is read by the first and by the last product of a step (S = Q K^T, dQ += dS K), so a K slot is held for more
  // than a step: three slots let the load of step i+2 start while step i is still being multiplied.  V is read by
  // dP = dO V^T only, early in the step, so one slot suffices: its reload has the rest of the step to land.
  static constexpr int kKStages = 3;
  static constexpr int kTotal = 2 * kQ + (kKStages + 1) * kKV + 1024 + 256;
};

template <int HD, int NWG>
__global__ void __launch_bounds__(64 + 128 * NWG, 1)
flash_bwd_dq128_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                       const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                       const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  using L = Dq128Smem<HD>;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = base;
  uint8_t* sDO = sQ + L::kQ;
  constexpr int NK = L::kKStages;
  uint8_t* sK = sDO + L::kQ;            // NK stages
  uint8_t* sV = sK + NK * L::kKV;       // 1 stage
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + L::kKV);
  static_assert(NWG == 2 || NWG == 4, "two or four softmax warpgroups");
  constexpr int kSoftmaxWarps = 4 * NWG;
  constexpr int CPT = 128 / NWG;        // key columns per thread and step
  uint64_t* qdo_full = bars;       // 1
  uint64_t* k_full = bars + 1;     // 3
  uint64_t* k_empty = bars + 4;    // 3
  uint64_t* v_full = bars + 7;     // 1
  uint64_t* v_empty = bars + 8;    // 1
  uint64_t* s_full = bars + 9;     // 1
  uint64_t* s_empty = bars + 10;   // 1
  uint64_t* ds_full = bars + 22;   // 2, by step parity: a warp may store the next step's dS before another has stored this one's
  uint64_t* ds_empty = bars + 12;  // 2
  uint64_t* qdo_empty = bars + 14; // 1: the last products that read Q and dO have completed
  uint64_t* acc_empty = bars + 15; // 1: the epilogue has read dQ
  const WorkSlot work{reinterpret_cast<uint4*>(bars + 18), bars + 16, bars + 17};
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  auto query_row = [&](const Block& w) { return (int(gridDim.x) - 1 - w.x) * 128; };
  auto steps_of = [&](const Block& w) {
    int kv_len = p.Skv;
    if (p.causal) kv_len = min(p.Skv, p.q_pos0 + query_row(w) + 127 - p.k_pos0 + 1);
    return kv_len > 0 ? (kv_len + 127) / 128 : 0;
  };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmDO);
    mbar_init(qdo_full, 1);
    for (int i = 0; i < NK; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
    }
    mbar_init(v_full, 1);
    mbar_init(v_empty, 1);
    mbar_init(s_full, 1);
    mbar_init(s_empty, kSoftmaxWarps);   // one arrival per softmax warp (mbar_arrive_warp)
    mbar_init(&ds_full[0], kSoftmaxWarps);
    mbar_init(&ds_full[1], kSoftmaxWarps);
    mbar_init(&ds_empty[0], 1);
    mbar_init(&ds_empty[1], 1);
    mbar_init(qdo_empty, 1);
    mbar_init(acc_empty, kSoftmaxWarps);
    mbar_init(work.full, 1);
    mbar_init(work.empty, 2 + kSoftmaxWarps);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem, tDP = tmem + 128, tDQ = tmem + 256;
  const uint32_t tDS[2] = {tmem + 384, tmem + 448};   // packed dS, step parity

  Block blk{int(blockIdx.x), int(blockIdx.y), int(blockIdx.z)};

  if (warp == 0) {
    // the whole warp walks the loop, one elected lane issues the copies (see producer_loop in gemm_core.cuh)
    const bool issuer = elect_one() != 0;
    int ks = 0, nq = 0, n = 0;                       // K ring position, Q tiles loaded so far, blocks done
    uint32_t kph = 0, vph = 0;
    bool ok = true, asked = false;
    for (; ok; ++n) {
      asked = false;
      const int q0 = query_row(blk), h = blk.y, b = blk.z, n_it = steps_of(blk);
      const int qslot = p.qmap.slot(h, p.qpg), kslot = p.kmap.slot(h, p.qpg), vslot = p.vmap.slot(h, p.qpg),
                doslot = p.domap.slot(h, p.qpg);
      if (n_it > 0) {
        if (!mbar_wait_warp(qdo_empty, (nq & 1) ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { ok = false; break; }
        ++nq;
        if (issuer) mbar_expect_tx(qdo_full, 2 * L::kQ);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c) {
          if (issuer) tma_load_4d(sQ + c * 128 * 128, &tmQ, qdo_full, c * 64, qslot, q0, b);
          if (issuer) tma_load_4d(sDO + c * 128 * 128, &tmDO, qdo_full, c * 64, doslot, q0, b);
        }
        for (int it = 0; it < n_it; ++it) {
          if (!mbar_wait_warp(&k_empty[ks], kph ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { ok = false; break; }
          if (issuer) mbar_expect_tx(&k_full[ks], L::kKV);
#pragma unroll
          for (int c = 0; c < HD / 64; ++c)
            if (issuer) tma_load_4d(sK + ks * L::kKV + c * 128 * 128, &tmK, &k_full[ks], c * 64, kslot, it * 128, b);
          if (!mbar_wait_warp(v_empty, vph ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { ok = false; break; }
          if (issuer) mbar_expect_tx(v_full, L::kKV);
#pragma unroll
          for (int c = 0; c < HD / 64; ++c)
            if (issuer) tma_load_4d(sV + c * 128 * 128, &tmV, v_full, c * 64, vslot, it * 128, b);
          if (++ks == NK) { ks = 0; kph ^= 1; }
          vph ^= 1;
        }
      }
      if (!ok) break;
      // The next block is asked for once this one's loads are all on their way.  Asked for earlier it waits for a CTA that is busy
      // while others run dry (12 heads of 64, 4096 tokens: 203 -> 233 us).  The answer slot is free once every warp has this block.
      if (n > 0 && !mbar_wait_warp(work.empty, (n - 1) & 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
      if (issuer) work_request(work);
      __syncwarp();
      asked = true;
      if (!work_take(work, n, blk, p.status, abort_flag)) break;
    }
    if (!ok) {
      *abort_flag = 1;
      if (asked) work_drain(work, n);
    }
  } else if (warp == 1) {
      // the whole warp walks the loop, one elected lane issues (see mma_loop in gemm_core.cuh)
      const bool issuer = elect_one() != 0;
      constexpr uint32_t idesc_s = make_idesc_lp(128, 128, false, false);
      constexpr uint32_t idesc_dq = make_idesc_lp(128, HD, false, true);
      const uint32_t aQ = smem_u32(sQ), aDO = smem_u32(sDO);
      bool ok = true;
      uint32_t step_s = 0, step_d = 0;   // S / dP and dQ products issued so far
      int nq = 0;                        // blocks with steps so far
      int ks_s = 0, ks_d = 0;          // K slot of the next S issue and of the next dQ issue
      uint32_t kph_s = 0;
      const uint32_t aV = smem_u32(sV);
      auto issue_s = [&](bool last) -> bool {
        if (!mbar_wait_warp(&k_full[ks_s], kph_s, p.status, kTimeoutSmemFull, abort_flag)) return false;
        if (!mbar_wait_warp(s_empty, (step_s & 1) ^ 1, p.status, kTimeoutTmemEmpty, abort_flag)) return false;
        tc_fence_after();
        const uint32_t aK = smem_u32(sK + ks_s * L::kKV);
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk)
            umma_f16_ss(tS, kmajor_desc(aQ, 128, kk), kmajor_desc(aK, 128, kk), idesc_s, kk != 0);
        }
        __syncwarp();
        if (!mbar_wait_warp(v_full, step_s & 1, p.status, kTimeoutSmemFull, abort_flag)) return false;
        tc_fence_after();
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk)
            umma_f16_ss(tDP, kmajor_desc(aDO, 128, kk), kmajor_desc(aV, 128, kk), idesc_s, kk != 0);
          umma_commit(v_empty);
          umma_commit(s_full);
          if (last) umma_commit(qdo_empty);
        }
        __syncwarp();
        ++step_s;
        if (++ks_s == NK) { ks_s = 0; kph_s ^= 1; }
        return true;
      };
      for (int n = 0; ok; ++n) {
      const int n_it = steps_of(blk);
      if (n_it > 0) {
      ok = mbar_wait_warp(qdo_full, nq & 1, p.status, kTimeoutSmemFull, abort_flag);
      if (ok) ok = issue_s(n_it == 1);
      HG_DKV_TIMERS(tm_s, tm_wait_ds, tm_dq, tm_unused);
      for (int it = 0; ok && it < n_it; ++it) {
        HG_DKV_TICK(t0);
        if (it + 1 < n_it) { ok = issue_s(it + 2 == n_it); if (!ok) break; }
        HG_DKV_TOCK(tm_s, t0);
        // dQ still holds the last block's sums until its epilogue has read them
        if (it == 0 && !mbar_wait_warp(acc_empty, (nq & 1) ^ 1, p.status, kTimeoutTmemEmpty, abort_flag)) { ok = false; break; }
        if (!mbar_wait_warp(&ds_full[step_d & 1], (step_d >> 1) & 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
        tc_fence_after();
        HG_DKV_TOCK(tm_wait_ds, t0);
        const uint32_t aK = smem_u32(sK + ks_d * L::kKV);
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)   // k-step kk = keys 16kk..16kk+15 = 8 packed columns
            umma_f16_ts(tDQ, tDS[step_d & 1] + kk * 8, mnmajor_desc(aK, 128, kk), idesc_dq, (it | kk) != 0);
          umma_commit(&k_empty[ks_d]);
          umma_commit(&ds_empty[step_d & 1]);
        }
        __syncwarp();
        ++step_d;
        if (++ks_d == NK) ks_d = 0;
        HG_DKV_TOCK(tm_dq, t0);
      }
      HG_DKV_REPORT(32, n_it, tm_s, tm_wait_ds, tm_dq, tm_unused);
      ++nq;
      }
      if (ok && !work_take(work, n, blk, p.status, abort_flag)) break;
      }
      if (!ok) *abort_flag = 1;
  } else {
    const int wq = warp & 3;
    const int half = (warp - 2) >> 2;     // warpgroup: which CPT of the step's 128 key columns these threads own
    const int c0 = half * CPT;
    const int row = wq * 32 + lane_id();
    const uint32_t lane_off = uint32_t(wq * 32) << 16;
    const float sl2 = p.scale * kLog2e;
    bool ok = true;
    uint32_t done = 0;                    // steps so far
    for (int n = 0; ok; ++n) {
    const int q0 = query_row(blk), h = blk.y, b = blk.z, n_it = steps_of(blk);
    const int srow = q0 + row;
    const int q_pos = p.q_pos0 + srow;
    float lse2 = INFINITY, dsum = 0.f;
    if (srow < p.Sq) {
      const size_t idx = (size_t(b) * p.nheads + h) * p.Sq + srow;
      lse2 = p.LSE[idx] * kLog2e;
      dsum = p.D[idx];
    }
    const float nlse2 = -lse2;
    HG_DKV_TIMERS(tm_wait_s, tm_ld, tm_math, tm_st);
    for (int it = 0; it < n_it; ++it, ++done) {
      HG_DKV_TICK(t0);
      if (!mbar_wait_warp(s_full, done & 1, p.status, kTimeoutTmemFull, abort_flag)) { ok = false; break; }
      tc_fence_after();
      HG_DKV_TOCK(tm_wait_s, t0);
      float ds[CPT];
      {
        float sv[CPT];
#pragma unroll
        for (int c = 0; c < CPT / 32; ++c) {
          uint32_t r0[32], r1[32];
          tmem_ld32(tS + lane_off + c0 + c * 32, r0);
          tmem_ld32(tDP + lane_off + c0 + c * 32, r1);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) { sv[c * 32 + i] = __uint_as_float(r0[i]); ds[c * 32 + i] = __uint_as_float(r1[i]); }
        }
        tc_fence_before();
        mbar_arrive_warp(s_empty);
        HG_DKV_TOCK(tm_ld, t0);
        const int kbase = it * 128 + c0;
        const bool need_mask = (p.causal && (p.k_pos0 + kbase + CPT - 1 > p.q_pos0 + q0)) || (kbase + CPT > p.Skv);
        if (!need_mask) {
#pragma unroll
          for (int i = 0; i < CPT; ++i) ds[i] = ex2(fmaf(sv[i], sl2, nlse2)) * (ds[i] - dsum);
        } else {
#pragma unroll
          for (int i = 0; i < CPT; ++i) {
            const bool dead = (kbase + i >= p.Skv) || (p.causal && (p.k_pos0 + kbase + i > q_pos));
            ds[i] = dead ? 0.f : ex2(fmaf(sv[i], sl2, nlse2)) * (ds[i] - dsum);
          }
        }
      }
      HG_DKV_TOCK(tm_math, t0);
      if (done >= 2) {   // this dS buffer was last read by the dQ product of step it-2
        if (!mbar_wait_warp(&ds_empty[done & 1], ((done >> 1) & 1) ^ 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
        tc_fence_after();
      }
      {
        uint32_t w[CPT / 2];
#pragma unroll
        for (int i = 0; i < CPT / 2; ++i) w[i] = pack_bf16(ds[2 * i], ds[2 * i + 1]);
        if constexpr (CPT == 64) tmem_st32(tDS[done & 1] + lane_off + half * (CPT / 2), w);
        else tmem_st16(tDS[done & 1] + lane_off + half * (CPT / 2), w);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive_warp(&ds_full[done & 1]);
      HG_DKV_TOCK(tm_st, t0);
    }
    HG_DKV_REPORT(24, n_it, tm_wait_s, tm_ld, tm_math, tm_st);
    const int dqslot = p.dqmap.slot(h, p.qpg);
    hg_lp_t* dq = p.dQ + int64_t(srow) * p.dq_ss + int64_t(b) * p.dq_sb + int64_t(dqslot) * HD;
    if (n_it == 0) {
      if (srow < p.Sq) {
#pragma unroll
        for (int i = half; i < HD / 8; i += NWG) reinterpret_cast<uint4*>(dq)[i] = make_uint4(0, 0, 0, 0);
      }
    } else if (ok && !*abort_flag &&
               mbar_wait_warp(&ds_empty[(done - 1) & 1], ((done - 1) >> 1) & 1, p.status, kTimeoutOther, abort_flag)) {
      tc_fence_after();
#pragma unroll
      for (int c = half; c < HD / 32; c += NWG) {
        uint32_t r[32];
        tmem_ld32(tDQ + lane_off + c * 32, r);
        tmem_ld_wait();
        if (srow < p.Sq) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 u;
            u.x = pack_bf16(__uint_as_float(r[q * 8 + 0]) * p.scale, __uint_as_float(r[q * 8 + 1]) * p.scale);
            u.y = pack_bf16(__uint_as_float(r[q * 8 + 2]) * p.scale, __uint_as_float(r[q * 8 + 3]) * p.scale);
            u.z = pack_bf16(__uint_as_float(r[q * 8 + 4]) * p.scale, __uint_as_float(r[q * 8 + 5]) * p.scale);
            u.w = pack_bf16(__uint_as_float(r[q * 8 + 6]) * p.scale, __uint_as_float(r[q * 8 + 7]) * p.scale);
            reinterpret_cast<uint4*>(dq + c * 32)[q] = u;
          }
        }
      }
      tc_fence_before();
      mbar_arrive_warp(acc_empty);
    } else {
      ok = false;
    }
    if (ok && !work_take(work, n, blk, p.status, abort_flag)) break;
    }
    if (!ok) *abort_flag = 1;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// =================================================================================================
// Backward, part 2 where the dK/dV kernel has left dS in memory: dQ = dS K, a product with nothing to recompute.  Against S, dP
// and the exponentials a second time (flash_bwd_dq128_kernel: 24 MMAs and 16384 exponentials per 128 x 128 pair) it takes 8 MMAs
// and reads 32 KB of dS, which bounds it: HBM, and 64 bytes a cycle into an SM, for which a CTA takes 256 queries whose two tiles
// share the keys (48 KB a pair).  us, causal, dK/dV kernel + dQ kernel, without dS in memory / with: head dim 128, 2 x 4096 and 32
// heads 518 + 381 / 603 + 203 (the power limit holds the clock at 1.7 GHz, and the stores cost power), 1531 and 28 heads on 4
// 49 + 42 / 57 + 20; head dim 64, 8 x 1024 and 25 heads 106 + 89 / 113 + 51.  dS is read at 5.4 TB/s at the first of these.
// A unit of work is 256 queries of a head, a block of the grid, longest first; CTAs take further ones (WorkSlot; dealt out in turn,
// a CTA had up to 1.3 times the mean), and the four stages of 64 keys run on across them.  Two accumulators of two tiles fill tensor memory (head dim 128), so that a unit's results leave under the next one's
// products.  Roles: warp 0 TMA, warp 1 MMA, warps 2-5 epilogue.
// =================================================================================================
// 128 queries x 16 keys of a half tile of dS (see BwdParams::dS) at `saddr`: 8 x 8 blocks of 128 bytes, 128 bytes apart along the
// keys and 1024 along the queries, no swizzle.
__device__ __forceinline__ uint64_t plain_mn_desc(uint32_t saddr) {
  return (uint64_t(1) << 46) | uint64_t((saddr & 0x3FFFF) >> 4) | (uint64_t(128 >> 4) << 16) | (uint64_t(1024 >> 4) << 32);
}
// `bytes` in a row into shared memory; both addresses and the size are multiples of 16.
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               :
               : "r"(smem_u32(smem_dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

template <int HD>
struct DqDsSmem {
  static constexpr int kTile = 128 * 64 * 2;       // dS^T of 64 keys x 128 queries
  static constexpr int kK = 64 * HD * 2;
  static constexpr int kStages = 4;
  static constexpr int kStage = 2 * kTile + kK;
  static constexpr int kTotal = kStages * kStage + 1024 + 256;
};

template <int HD>
__global__ void __launch_bounds__(192, 1)
flash_bwd_dq_ds_kernel(const __grid_constant__ CUtensorMap tmK, const BwdParams p, int heads, const __grid_constant__ DsPieces ds) {
  extern __shared__ uint8_t smem_raw[];
  using L = DqDsSmem<HD>;
  constexpr int NS = L::kStages;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + NS * L::kStage);
  uint64_t* full = bars;                 // 4
  uint64_t* empty = bars + 4;            // 4
  uint64_t* acc_full = bars + 8;         // 2
  uint64_t* acc_empty = bars + 10;       // 2
  const WorkSlot work{reinterpret_cast<uint4*>(bars + 14), bars + 12, bars + 13};
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5;
  const int n_qs = (p.Sq + 127) / 128, n_kb = (p.Skv + 127) / 128, n_pairs = (n_qs + 1) / 2;
  const int64_t head_tiles = ds_tiles_before(p, n_kb);

  struct Unit {
    int qb, h, b, kbs[2];        // first query block, head, sequence; key blocks that each of the two query blocks sees
    int head;                    // among the heads of this launch
  };
  auto key_blocks = [&](int qb) {
    if (qb >= n_qs) return 0;
    if (!p.causal) return n_kb;
    const int keys = p.q_pos0 + qb * 128 + 128 - p.k_pos0;       // before the first that no row of the block sees
    return keys <= 0 ? 0 : min(n_kb, (keys + 127) / 128);
  };
  auto unit_at = [&](int u) {
    Unit w;
    // some heads at a time, the last ones, whose dS may still be in L2, first
    const int some = (2 * kSmCount + n_pairs - 1) / n_pairs, first = u / (some * n_pairs) * some, n = min(some, heads - first);
    const int r = u - first * n_pairs, pair = n_pairs - 1 - r / n, hb = heads - 1 - first - r % n;
    w.qb = 2 * pair;
    w.head = hb;
    w.b = p.b0_c + hb / p.nh_c;
    w.h = p.h0_c + hb % p.nh_c;
    w.kbs[0] = key_blocks(w.qb);
    w.kbs[1] = key_blocks(w.qb + 1);
    return w;
  };
  // Key blocks of a unit in the order of both roles: the second query block sees at least those of the first, where it exists.
  auto most = [](const Unit& w) { return max(w.kbs[0], w.kbs[1]); };

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmK);
    for (int i = 0; i < NS; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 4); }
    mbar_init(work.full, 1);
    mbar_init(work.empty, 6);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 4 * HD);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  Block blk{int(blockIdx.x), 0, 0};

  if (warp == 0) {
    const bool issuer = elect_one() != 0;
    uint32_t stage = 0, phase = 0;
    bool ok = true, asked = false;
    int n_done = 0;
    for (; ok; ++n_done) {
      asked = false;
      const Unit w = unit_at(blk.x);
      const int kslot = p.kmap.slot(w.h, p.qpg), n = most(w);
      const hg_lp_t* tiles = ds_tile(ds, w.head, head_tiles, 0);
      for (int kb = 0; ok && kb < n; ++kb) {
        // a first query block that does not see this key block has no tile: this is then the one before the second's
        const hg_lp_t* src = tiles + (ds_tiles_before(p, kb) + w.qb - ds_first_query_block(p, kb)) * (128 * 128);
        for (int half = 0; half < 2; ++half) {
          if (!mbar_wait_warp(&empty[stage], phase ^ 1, p.status, kTimeoutSmemEmpty, abort_flag)) { ok = false; break; }
          uint8_t* s = base + stage * L::kStage;
          if (issuer) {
            mbar_expect_tx(&full[stage], (int(kb < w.kbs[0]) + int(kb < w.kbs[1])) * L::kTile + L::kK);
#pragma unroll
            for (int j = 0; j < 2; ++j)
              if (kb < w.kbs[j]) bulk_load(s + j * L::kTile, src + (2 * j + half) * (64 * 128), L::kTile, &full[stage]);
#pragma unroll
            for (int c = 0; c < HD / 64; ++c)
              tma_load_4d(s + 2 * L::kTile + c * 64 * 128, &tmK, &full[stage], c * 64, kslot, kb * 128 + half * 64, w.b);
          }
          __syncwarp();
          if (++stage == NS) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) break;
      if (n_done > 0 && !mbar_wait_warp(work.empty, (n_done - 1) & 1, p.status, kTimeoutOther, abort_flag)) { ok = false; break; }
      if (issuer) work_request(work);
      __syncwarp();
      asked = true;
      if (!work_take(work, n_done, blk, p.status, abort_flag)) break;
    }
    for (int i = 0; ok && i < NS; ++i) {          // leave when the last commits have arrived
      ok = mbar_wait_warp(&empty[stage], phase ^ 1, p.status, kTimeoutSmemEmpty, abort_flag);
      if (++stage == NS) { stage = 0; phase ^= 1; }
    }
    if (!ok) {
      *abort_flag = 1;
      if (asked) work_drain(work, n_done);
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);  // 2 ms for copies in flight: far longer than a tile load
    }
  } else if (warp == 1) {
    const bool issuer = elect_one() != 0;
    constexpr uint32_t idesc = make_idesc_lp(128, HD, true, true);
    uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
    bool ok = true;
    for (int n_done = 0; ok; ++n_done) {
      const Unit w = unit_at(blk.x);
      const int n = most(w);
      if (n > 0) {
      if (!mbar_wait_warp(&acc_empty[acc], acc_phase ^ 1, p.status, kTimeoutTmemEmpty, abort_flag)) { ok = false; break; }
      tc_fence_after();
      for (int hs = 0; hs < 2 * n; ++hs) {
        if (!mbar_wait_warp(&full[stage], phase, p.status, kTimeoutSmemFull, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t s = smem_u32(base + stage * L::kStage), k = s + 2 * L::kTile;
        if (issuer) {
#pragma unroll
          for (int j = 0; j < 2; ++j)
            if (hs < 2 * w.kbs[j]) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                umma_f16_ss(tmem + (acc * 2 + j) * HD, plain_mn_desc(s + j * L::kTile + kk * 256),
                            make_smem_desc(k + kk * 2048, 64 * 128, 1024), idesc, (hs | kk) != 0);
            }
          umma_commit(&empty[stage]);
        }
        __syncwarp();
        if (++stage == NS) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      if (issuer) umma_commit(&acc_full[acc]);
      __syncwarp();
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      if (!work_take(work, n_done, blk, p.status, abort_flag)) break;
    }
    if (!ok) *abort_flag = 1;
  } else {
    const int wq = warp & 3, row = wq * 32 + lane_id();
    const uint32_t lane_off = uint32_t(wq * 32) << 16;
    uint32_t acc = 0, acc_phase = 0;
    for (int n_done = 0;; ++n_done) {
      const Unit w = unit_at(blk.x);
      const bool any = most(w) > 0;
      if (any && !mbar_wait_warp(&acc_full[acc], acc_phase, p.status, kTimeoutTmemFull, abort_flag)) { *abort_flag = 1; break; }
      tc_fence_after();
#pragma unroll 1
      for (int j = 0; j < 2; ++j) {
        const int q = (w.qb + j) * 128 + row;
        hg_lp_t* dq = p.dQ + int64_t(q) * p.dq_ss + int64_t(w.b) * p.dq_sb + int64_t(p.dqmap.slot(w.h, p.qpg)) * HD;
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t r[32];
          tmem_ld32(tmem + lane_off + (acc * 2 + j) * HD + c * 32, r);
          tmem_ld_wait();
          if (q < p.Sq) {
            const float scale = p.scale;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint4 v = make_uint4(0, 0, 0, 0);                      // queries that see no key
              if (w.kbs[j] > 0) {
                v.x = pack_bf16(__uint_as_float(r[i * 8 + 0]) * scale, __uint_as_float(r[i * 8 + 1]) * scale);
                v.y = pack_bf16(__uint_as_float(r[i * 8 + 2]) * scale, __uint_as_float(r[i * 8 + 3]) * scale);
                v.z = pack_bf16(__uint_as_float(r[i * 8 + 4]) * scale, __uint_as_float(r[i * 8 + 5]) * scale);
                v.w = pack_bf16(__uint_as_float(r[i * 8 + 6]) * scale, __uint_as_float(r[i * 8 + 7]) * scale);
              }
              reinterpret_cast<uint4*>(dq + c * 32)[i] = v;
            }
          }
          __syncwarp();
        }
      }
      if (any) {
        tc_fence_before();
        mbar_arrive_warp(&acc_empty[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      if (!work_take(work, n_done, blk, p.status, abort_flag)) break;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 4 * HD);
  }
}

}  // namespace attn
}  // namespace hg

// ------------------------------------------------------------------------------------------------
// Host launchers
// ------------------------------------------------------------------------------------------------
using namespace hg::attn;

namespace {

// 4-D tensor map over (d, slot, s, b) of a bf16 tensor whose element (s, b, slot, d) sits at
// base + s*ss + b*sb + slot*hd + d.  Box = (64, 1, box_rows, 1).
int make_map(CUtensorMap* out, const void* base, int hd, int slots, int S, int B, int64_t ss, int64_t sb,
             int box_rows) {
  const uint64_t key[8] = {4, uint64_t(reinterpret_cast<uintptr_t>(base)), (uint64_t(uint32_t(hd)) << 32) | uint32_t(slots),
                           (uint64_t(uint32_t(S)) << 32) | uint32_t(B), uint64_t(ss), uint64_t(sb), uint64_t(box_rows), 0};
  if (const CUtensorMap* hit = hg_host::tmap_cache_find(key)) {
    *out = *hit;
    return 0;
  }
  auto enc = hg_host::get_encode_fn();
  if (enc == nullptr) return -2;
  cuuint64_t dims[4] = {cuuint64_t(hd), cuuint64_t(slots), cuuint64_t(S), cuuint64_t(B)};
  cuuint64_t strides[3] = {cuuint64_t(hd) * 2, cuuint64_t(ss) * 2, cuuint64_t(sb) * 2};
  cuuint32_t box[4] = {64, 1, cuuint32_t(box_rows), 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  if (B == 1) strides[2] = strides[1] * cuuint64_t(S);  // any legal value; the coordinate is always 0
  CUresult r = enc(out, HG_TMAP_LP, 4, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_SUCCESS) hg_host::tmap_cache_store(key, *out);
  return r == CUDA_SUCCESS ? 0 : -(1000 + int(r));
}

// dK/dV kernel: 0 = 128-query steps with P^T / dS^T in tensor memory, 1 = 64-query steps staged
// through shared memory (kept for side-by-side tests and timing).
int g_dkv_variant = 0;
// Forward kernel: 0 = the rule of two_tile_forward, 1 = one tile per CTA with P staged in shared memory, 2 = two query
// tiles per CTA with P in tensor memory wherever a sequence is longer than one tile (1, 2: side-by-side tests and timing).
int g_fwd_variant = 0;

constexpr int kDkvMinChunk = 4;   // fewest query steps of a CTA that shares its key block: about what its start and end cost

template <typename K>
int set_smem(K kernel, int bytes) {
  return int(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

// Which calls take two query tiles per CTA: sequences longer than one tile.  With head dim 64 the one-tile kernel is the
// faster one as long as all its CTAs run at once (heads x queries, us, two tiles / one: 1 x 4096 64 / 51, 12 x 512 18 / 14,
// 12 x 1536 33 / 27, 48 x 384 16 / 16; beyond a wave 12 x 2048 39 / 41, 25 x 1024 27 / 31, 48 x 512 20 / 22, 74 x 257 16 / 22,
// 200 x 1024 98 / 127).
template <int HD>
bool two_tile_forward(const FwdParams& p) {
  if (p.Sq <= 128 || g_fwd_variant == 1) return false;
  return HD == 128 || g_fwd_variant == 2 || (long long)((p.Sq + 127) / 128) * p.nheads * p.B > kSmCount;
}

template <int HD>
int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p, cudaStream_t st) {
  int rc;
  if (two_tile_forward<HD>(p)) {
    static bool cfg = false;
    if (!cfg) { if ((rc = set_smem(flash_fwd2_kernel<HD>, Fwd2Smem<HD>::kTotal))) return rc; cfg = true; }
    const dim3 grid((p.Sq + 255) / 256, p.nheads, p.B);
    return hg_host::launch(flash_fwd2_kernel<HD>, grid, kFwd2Threads, Fwd2Smem<HD>::kTotal, st, tq, tk, tv, p);
  } else {
    static bool cfg = false;
    if (!cfg) { if ((rc = set_smem(flash_fwd_kernel<HD>, FwdSmem<HD>::kTotal))) return rc; cfg = true; }
    const dim3 grid((p.Sq + 127) / 128, p.nheads, p.B);
    return hg_host::launch(flash_fwd_kernel<HD>, grid, kThreads, FwdSmem<HD>::kTotal, st, tq, tk, tv, p);
  }
}

// CTAs per kv head and sequence of the 128-query dK/dV kernel
int dkv_ctas(const BwdParams& p, int blocks) {
  int n = 0;
  for (int kb = 0; kb < blocks; ++kb) n += dkv_block_ctas(p, dkv_block_steps(p, kb));
  return n;
}

// Query steps per CTA when the key blocks are too few for the chip, 0 where each has one CTA.  A grouped layer has a dK/dV
// CTA per key block and KV head: four kv heads of 1531 tokens are 48 CTAs, and under a causal mask the first of them walks
// twelve times the steps of the last.  The smallest chunk whose CTAs all run at once is taken: their longest is what counts.
// It has to end at least six steps (of 2 us) before the longest block alone, which pays for the parts' way through memory and
// the kernel that adds them.  Whole backward, us, one CTA a block / shared: head dim 128, 28 heads on 4, 1531 tokens 194 / 100,
// 512 tokens 69 / 40, 256 tokens 44 / 34; 8 heads on 1, 4096 tokens 499 / 153; 4 heads, 2048 tokens 63 / 58; fewer steps saved:
// 4 heads, 1024 tokens 40 / 41, 16 heads 41 / 45; head dim 64, 28 on 4, 1531 tokens 190 / 82, 32 on 8, 1024 tokens 87 / 55.
int dkv_chunk_steps(BwdParams p, int Skv, int nkv) {
  const int blocks = (Skv + 127) / 128, heads = nkv * p.B;
  if ((long long)blocks * heads > kSmCount) return 0;
  int longest = 0;
  for (int kb = 0; kb < blocks; ++kb) longest = dkv_block_steps(p, kb) > longest ? dkv_block_steps(p, kb) : longest;
  int lo = kDkvMinChunk - 1, hi = longest;            // the CTAs of chunk `hi` run at once, those of `lo` may not
  while (hi - lo > 1) {
    p.chunk = (lo + hi) / 2;
    if (dkv_ctas(p, blocks) * heads <= kSmCount) hi = p.chunk;
    else lo = p.chunk;
  }
  return hi + 6 <= longest ? hi : 0;
}

template <int HD>
int launch_dkv(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
               const BwdParams& p, const DsPieces& ds, int Skv, int nkv, int nb, bool wide, cudaStream_t st) {
  int rc;
  dim3 grid((Skv + 127) / 128, nkv, nb);
  if (wide) {
    const int blocks = int(grid.x);
    if (p.chunk > 0) grid.x = unsigned(dkv_ctas(p, blocks));
    static bool cfg[2] = {};
    const bool shared = p.chunk > 0;
    auto k = shared ? flash_bwd_dkv128_kernel<HD, kDkvWarpgroups, true> : flash_bwd_dkv128_kernel<HD, kDkvWarpgroups, false>;
    if (!cfg[shared]) { if ((rc = set_smem(k, Dkv128Smem<HD>::kTotal))) return rc; cfg[shared] = true; }
    k<<<grid, 128 + 128 * kDkvWarpgroups, Dkv128Smem<HD>::kTotal, st>>>(tq, tk, tv, tdo, p, ds);
    if (p.chunk > 0) dkv_sum_kernel<HD><<<dim3(blocks * 8, nkv, nb), 4 * HD, 0, st>>>(p, int(grid.x));
  } else {
    static bool cfg = false;
    if (!cfg) { if ((rc = set_smem(flash_bwd_dkv_kernel<HD>, DkvSmem<HD>::kTotal))) return rc; cfg = true; }
    flash_bwd_dkv_kernel<HD><<<grid, kBwdThreads, DkvSmem<HD>::kTotal, st>>>(tq, tk, tv, tdo, p);
  }
  return int(cudaGetLastError());
}

template <int HD>
int launch_dq(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
              const BwdParams& p, cudaStream_t st) {
  int rc;
  static bool cfg = false;
  auto k = flash_bwd_dq128_kernel<HD, kDqWarpgroups>;
  if (!cfg) { if ((rc = set_smem(k, Dq128Smem<HD>::kTotal))) return rc; cfg = true; }
  k<<<dim3((p.Sq + 127) / 128, p.nheads, p.B), 64 + 128 * kDqWarpgroups, Dq128Smem<HD>::kTotal, st>>>(tq, tk, tv, tdo, p);
  return int(cudaGetLastError());
}

template <int HD>
int launch_dq_ds(const CUtensorMap& tk, const BwdParams& p, const DsPieces& ds, int nb, cudaStream_t st) {
  int rc;
  static bool cfg = false;
  auto k = flash_bwd_dq_ds_kernel<HD>;
  if (!cfg) { if ((rc = set_smem(k, DqDsSmem<HD>::kTotal))) return rc; cfg = true; }
  const int heads = p.nh_c * nb, units = ((p.Sq + 255) / 256) * heads;
  k<<<units, 192, DqDsSmem<HD>::kTotal, st>>>(tk, p, heads, ds);
  return int(cudaGetLastError());
}

// How the heads of a backward are cut where dS^T goes through memory: launches of `nb` sequences and `ng` kv heads each, whose
// tiles fit kDsMost.  ng = 0: not even one kv head's do, and the dQ kernel recomputes S and dP.
// The tiles are kept in pieces of `heads` heads and at most kDsPiece bytes (one head, if that has more): a caching allocator finds them
// among the blocks that it holds, where one block for all had to be had from the device for every few new layers (1531 tokens, 28
// heads: the first pass of a layer 0.97 instead of 0.60 ms).  More than half of kDsPiece in each, so that there are kDsPieces at most.
constexpr long long kDsTile = 128 * 128 * 2, kDsMost = 3ll << 29, kDsPiece = 48ll << 20;
static_assert(kDsMost / (kDsPiece / 2) <= kDsPieces, "the table of pieces");
struct DsCut {
  int nb, ng;
  long long bytes;
  int pieces, heads;
};
DsCut ds_cut(const BwdParams& p, int Skv, int nkv) {
  const long long group = ds_tiles_before(p, (Skv + 127) / 128) * p.qpg * kDsTile;
  if (g_dkv_variant != 0 || group > kDsMost) return {};
  if (group == 0) return {p.B, nkv, 0, 0, 0};
  const long long groups = kDsMost / group;
  DsCut c{};
  c.ng = groups < nkv ? int(groups) : nkv;
  c.nb = groups < nkv ? 1 : groups / nkv < p.B ? int(groups / nkv) : p.B;
  if (p.chunk > 0 && (c.ng < nkv || c.nb < p.B)) return {};     // shared key blocks are few: they are launched at once
  auto even = [](int n, int most) {                                     // launches of about the same size
    const int times = (n + most - 1) / most;
    return (n + times - 1) / times;
  };
  c.ng = even(nkv, c.ng);
  c.nb = even(p.B, c.nb);
  c.bytes = group * c.ng * c.nb;
  const long long head = group / p.qpg;
  const int all = c.ng * c.nb * p.qpg;
  c.heads = head < kDsPiece ? even(all, int(kDsPiece / head)) : 1;
  c.pieces = (all + c.heads - 1) / c.heads;
  return c;
}
// Whether storing dS pays.  In one launch it does.  Several end one by one, with fewer and fewer CTAs at work, which costs more than
// dS saves unless the smallest has five key blocks per SM, and with head dim 64 whatever it has.  Whole backward, us, dS stored / S and
// dP again: head dim 128, 8192 tokens, 32 heads (launches of 1024 key blocks) 1814 / 1935, 40 heads (1280) 2210 / 2378, 2 x 8192, 32 heads
// (1024) 3590 / 3730; 16384, 32 heads (640) 7060 / 7000; 8192, 32 heads on 8 (256) 1980 / 1955, 28 on 4 (128) 2165 / 1815; 16384, 32 on 8
// (128) 9705 / 7000; head dim 64, 2 x 8192, 25 heads (768) 2116 / 1942, 16384 4010 / 3731.
bool ds_pays(const DsCut& c, const BwdParams& p, int Skv, int nkv, int hd) {
  if (c.bytes == 0 || (c.ng == nkv && c.nb == p.B)) return c.bytes > 0;
  const int last = c.ng < nkv ? (nkv - 1) % c.ng + 1 : ((p.B - 1) % c.nb + 1) * nkv;
  return hd == 128 && (long long)((Skv + 127) / 128) * last >= 5 * kSmCount;
}
// The scratch of a backward, in floats: row sums of dO * O, parts of dK and dV, and each piece of the tiles of dS^T.
struct BwdScratch {
  long long sums, parts, piece;
  int chunk;
  DsCut cut;
};
BwdScratch bwd_scratch(BwdParams p, int Skv, int nkv, int hd) {
  BwdScratch w{};
  w.sums = ((long long)p.B * p.nheads * p.Sq + 63) / 64 * 64;
  if (g_dkv_variant != 0) return w;
  w.chunk = p.chunk = dkv_chunk_steps(p, Skv, nkv);
  if (w.chunk) w.parts = (long long)dkv_ctas(p, (Skv + 127) / 128) * nkv * p.B * 2 * 128 * hd;
  w.cut = ds_cut(p, Skv, nkv);
  if (w.cut.bytes > 0) w.piece = w.cut.bytes / (w.cut.nb * w.cut.ng * p.qpg) * w.cut.heads / 4;
  return w;
}

}  // namespace

extern "C" {

int hg_flash_fwd(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, const HgAttnTensor* o,
                 void* lse, int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0,
                 float scale, void* stream) {
  if (hd != 64 && hd != 128) return -1;
  if (Sq <= 0 || Skv <= 0 || B <= 0) return 0;
  if (g_fwd_variant == 0 && hg_flash_stream_takes(q, k, v, Sq, Skv, B, nheads, nkv, hd, causal, q_pos0, k_pos0))
    return hg_flash_stream(q, k, v, o, lse, Sq, Skv, B, nheads, nkv, hd, causal, q_pos0, k_pos0, scale, 0, stream);
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_map(&tq, q->ptr, hd, q->slots, Sq, B, q->ss, q->sb, 128))) return rc;
  if ((rc = make_map(&tk, k->ptr, hd, k->slots, Skv, B, k->ss, k->sb, 128))) return rc;
  if ((rc = make_map(&tv, v->ptr, hd, v->slots, Skv, B, v->ss, v->sb, 128))) return rc;
  FwdParams p{};
  p.Sq = Sq; p.Skv = Skv; p.B = B; p.nheads = nheads; p.qpg = nheads / nkv; p.causal = causal;
  p.q_pos0 = q_pos0; p.k_pos0 = k_pos0; p.scale = scale;
  p.qmap = {q->gs, q->hs, q->off}; p.kmap = {k->gs, k->hs, k->off}; p.vmap = {v->gs, v->hs, v->off};
  p.O = reinterpret_cast<hg_lp_t*>(o->ptr); p.o_ss = o->ss; p.o_sb = o->sb;
  p.LSE = reinterpret_cast<float*>(lse);
  p.status = hg_host::status_ptr();
  cudaStream_t st = (cudaStream_t)stream;
  return hd == 128 ? launch_fwd<128>(tq, tk, tv, p, st) : launch_fwd<64>(tq, tk, tv, p, st);
}

// Selects the forward kernel (see g_fwd_variant); returns the previous value.
int hg_attn_set_fwd_variant(int v) {
  const int old = g_fwd_variant;
  g_fwd_variant = v == 1 || v == 2 ? v : 0;
  return old;
}

// Selects the dK/dV kernel (see g_dkv_variant); returns the previous value.
int hg_attn_set_dkv_variant(int v) {
  const int old = g_dkv_variant;
  g_dkv_variant = v ? 1 : 0;
  return old;
}

static BwdParams bwd_sizes(int Sq, int Skv, int B, int nheads, int nkv, int causal, int q_pos0, int k_pos0) {
  BwdParams p{};
  p.Sq = Sq; p.Skv = Skv; p.B = B; p.nheads = nheads; p.qpg = nheads / nkv; p.causal = causal; p.q_pos0 = q_pos0; p.k_pos0 = k_pos0;
  return p;
}

// Floats of scratch that hg_flash_bwd_ws can use: the row sums of dO * O, [B, nheads, Sq], where key blocks are shared the parts
// of dK and dV, and, if `tiles`, all pieces of dS^T, of up to kDsMost bytes (see hg_flash_bwd_pieces).
long long hg_flash_bwd_scratch_of(int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0, int tiles) {
  if (Sq <= 0 || Skv <= 0 || B <= 0 || nheads <= 0 || nkv <= 0) return 0;
  const BwdScratch w = bwd_scratch(bwd_sizes(Sq, Skv, B, nheads, nkv, causal, q_pos0, k_pos0), Skv, nkv, hd);
  return w.sums + w.parts + (tiles ? w.piece * w.cut.pieces : 0);
}
long long hg_flash_bwd_scratch(int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0) {
  return hg_flash_bwd_scratch_of(Sq, Skv, B, nheads, nkv, hd, causal, q_pos0, k_pos0, 1);
}
// Pieces of scratch that hg_flash_bwd_ws can use for dS^T, and the floats of each.
int hg_flash_bwd_pieces(int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0, long long* floats) {
  *floats = 0;
  if (Sq <= 0 || Skv <= 0 || B <= 0 || nheads <= 0 || nkv <= 0) return 0;
  const BwdScratch w = bwd_scratch(bwd_sizes(Sq, Skv, B, nheads, nkv, causal, q_pos0, k_pos0), Skv, nkv, hd);
  *floats = w.piece;
  return w.cut.pieces;
}
// What a caller should give hg_flash_bwd_ws: floats of scratch, pieces for dS (0 where storing it does not pay), floats of each.
int hg_flash_bwd_wants(int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0, long long* wants) {
  wants[0] = wants[1] = wants[2] = 0;
  if (Sq <= 0 || Skv <= 0 || B <= 0 || nheads <= 0 || nkv <= 0) return 0;
  const BwdParams p = bwd_sizes(Sq, Skv, B, nheads, nkv, causal, q_pos0, k_pos0);
  const BwdScratch w = bwd_scratch(p, Skv, nkv, hd);
  wants[0] = w.sums + w.parts;
  if (ds_pays(w.cut, p, Skv, nkv, hd)) {
    wants[1] = w.cut.pieces;
    wants[2] = w.piece;
  }
  return 0;
}

// Where the caller's allocator had no room for dS, the next kNoRoomCalls backwards of that device do not ask it again: a caching
// allocator gives all that it holds back to the device before it says so, and every buffer then has to be had anew.
static std::atomic<int> g_no_room[64];
constexpr int kNoRoomCalls = 256;
int hg_flash_bwd_no_room(int device) {
  g_no_room[unsigned(device) % 64].store(kNoRoomCalls, std::memory_order_relaxed);
  return 0;
}
// Whether the allocator is to be asked; counts a call that is not.
int hg_flash_bwd_has_room(int device) {
  std::atomic<int>& left = g_no_room[unsigned(device) % 64];
  return left.load(std::memory_order_relaxed) <= 0 || left.fetch_sub(1, std::memory_order_relaxed) <= 0;
}

// ws: scratch of ws_floats fp32 values, 16-byte aligned, at least [B, nheads, Sq] (filled here with rowsum(dO*O)).  With less than
// hg_flash_bwd_scratch_of(.., 0) floats every key block has one CTA.  tiles: n_tiles pieces of tile_floats fp32 values, 16-byte
// aligned; with fewer or smaller ones than hg_flash_bwd_pieces says, S and dP are computed again for dQ.
// launched (may be null): the kernels that were launched.
int hg_flash_bwd_ws(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, const HgAttnTensor* o,
                    const HgAttnTensor* d_o, const void* lse, void* ws, long long ws_floats, void* const* tiles, int n_tiles,
                    long long tile_floats, const HgAttnTensor* dq, const HgAttnTensor* dk, const HgAttnTensor* dv, int Sq, int Skv,
                    int B, int nheads, int nkv, int hd, int causal, int q_pos0, int k_pos0, float scale, int* launched,
                    void* stream) {
  void* dsum = ws;
  if (launched != nullptr) *launched = 0;
  if (hd != 64 && hd != 128) return -1;
  if (Sq <= 0 || Skv <= 0 || B <= 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  int rc, kernels = 1;
  {
    const bool vec = (((uintptr_t(o->ptr) | uintptr_t(d_o->ptr)) & 15) | ((o->ss | o->sb | d_o->ss | d_o->sb) & 7)) == 0;
    const int64_t rows = int64_t(Sq) * B * nheads;
    const int64_t want = (rows * (hd / 8) + 256 * 4 - 1) / (256 * 4);
    const int blocks = int(want < kSmCount * 8 ? want : kSmCount * 8);
    auto k = hd == 128 ? (vec ? attn_bwd_dot_kernel<128, true> : attn_bwd_dot_kernel<128, false>)
                       : (vec ? attn_bwd_dot_kernel<64, true> : attn_bwd_dot_kernel<64, false>);
    k<<<blocks, 256, 0, st>>>((const hg_lp_t*)o->ptr, (const hg_lp_t*)d_o->ptr, o->ss, o->sb, d_o->ss, d_o->sb, Sq, B,
                              nheads, (float*)dsum);
  }
  BwdParams p{};
  p.Sq = Sq; p.Skv = Skv; p.B = B; p.nheads = nheads; p.qpg = nheads / nkv; p.causal = causal;
  p.q_pos0 = q_pos0; p.k_pos0 = k_pos0; p.scale = scale;
  p.qmap = {q->gs, q->hs, q->off}; p.kmap = {k->gs, k->hs, k->off}; p.vmap = {v->gs, v->hs, v->off};
  p.domap = {d_o->gs, d_o->hs, d_o->off};
  p.LSE = (const float*)lse; p.D = (const float*)dsum;
  p.dQ = (hg_lp_t*)dq->ptr; p.dq_ss = dq->ss; p.dq_sb = dq->sb; p.dqmap = {dq->gs, dq->hs, dq->off};
  p.dK = (hg_lp_t*)dk->ptr; p.dk_ss = dk->ss; p.dk_sb = dk->sb; p.dkmap = {dk->gs, dk->hs, dk->off};
  p.dV = (hg_lp_t*)dv->ptr; p.dv_ss = dv->ss; p.dv_sb = dv->sb; p.dvmap = {dv->gs, dv->hs, dv->off};
  p.status = hg_host::status_ptr();
  const BwdScratch w = bwd_scratch(p, Skv, nkv, hd);
  if (w.parts > 0 && (reinterpret_cast<uintptr_t>(ws) & 15) == 0 && ws_floats >= w.sums + w.parts) {
    p.chunk = w.chunk;
    p.part = static_cast<float*>(ws) + w.sums;
  }
  bool stored = w.cut.pieces > 0 && n_tiles >= w.cut.pieces && tile_floats >= w.piece;
  for (int i = 0; stored && i < w.cut.pieces; ++i) stored = tiles[i] != nullptr && (reinterpret_cast<uintptr_t>(tiles[i]) & 15) == 0;
  DsPieces ds{};
  if (stored) {
    ds.heads = w.cut.heads;
    for (int i = 0; i < w.cut.pieces; ++i) ds.at[i] = static_cast<hg_lp_t*>(tiles[i]);
  }
  const DsCut cut = stored ? w.cut : DsCut{B, nkv, 0, 0, 0};
  CUtensorMap tq, tk, tv, tdo, tk64;
  const bool wide = g_dkv_variant == 0;   // 128-query steps, P^T / dS^T in tensor memory
  const int q_rows = wide ? 128 : 64;
  if ((rc = make_map(&tq, q->ptr, hd, q->slots, Sq, B, q->ss, q->sb, q_rows))) return rc;
  if ((rc = make_map(&tk, k->ptr, hd, k->slots, Skv, B, k->ss, k->sb, 128))) return rc;
  if ((rc = make_map(&tv, v->ptr, hd, v->slots, Skv, B, v->ss, v->sb, 128))) return rc;
  if ((rc = make_map(&tdo, d_o->ptr, hd, d_o->slots, Sq, B, d_o->ss, d_o->sb, q_rows))) return rc;
  if (stored && (rc = make_map(&tk64, k->ptr, hd, k->slots, Skv, B, k->ss, k->sb, 64))) return rc;
  for (int b0 = 0; b0 < B; b0 += cut.nb)
    for (int g0 = 0; g0 < nkv; g0 += cut.ng) {
      const int nb = B - b0 < cut.nb ? B - b0 : cut.nb, ng = nkv - g0 < cut.ng ? nkv - g0 : cut.ng;
      p.b0_c = b0; p.g0_c = g0; p.h0_c = g0 * p.qpg; p.nh_c = ng * p.qpg;
      if ((rc = hd == 128 ? launch_dkv<128>(tq, tk, tv, tdo, p, ds, Skv, ng, nb, wide, st)
                          : launch_dkv<64>(tq, tk, tv, tdo, p, ds, Skv, ng, nb, wide, st))) return rc;
      kernels += p.chunk > 0 ? 2 : 1;
      if (!stored) continue;
      if ((rc = hd == 128 ? launch_dq_ds<128>(tk64, p, ds, nb, st) : launch_dq_ds<64>(tk64, p, ds, nb, st))) return rc;
      ++kernels;
    }
  if (!stored) {
    if ((rc = make_map(&tq, q->ptr, hd, q->slots, Sq, B, q->ss, q->sb, 128))) return rc;
    if ((rc = make_map(&tdo, d_o->ptr, hd, d_o->slots, Sq, B, d_o->ss, d_o->sb, 128))) return rc;
    if ((rc = hd == 128 ? launch_dq<128>(tq, tk, tv, tdo, p, st) : launch_dq<64>(tq, tk, tv, tdo, p, st))) return rc;
    ++kernels;
  }
  if (launched != nullptr) *launched = kernels;
  return 0;
}

// dsum: scratch [B, nheads, Sq] fp32 (filled here with rowsum(dO*O)); every key block has one CTA.
int hg_flash_bwd(const HgAttnTensor* q, const HgAttnTensor* k, const HgAttnTensor* v, const HgAttnTensor* o,
                 const HgAttnTensor* d_o, const void* lse, void* dsum, const HgAttnTensor* dq, const HgAttnTensor* dk,
                 const HgAttnTensor* dv, int Sq, int Skv, int B, int nheads, int nkv, int hd, int causal, int q_pos0,
                 int k_pos0, float scale, void* stream) {
  return hg_flash_bwd_ws(q, k, v, o, d_o, lse, dsum, 0, nullptr, 0, 0, dq, dk, dv, Sq, Skv, B, nheads, nkv, hd, causal, q_pos0,
                         k_pos0, scale, nullptr, stream);
}

}  // extern "C"
