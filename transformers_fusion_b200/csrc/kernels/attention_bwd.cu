// Flash attention backward for sm_100a: exact gradients, probabilities recomputed from the saved
// log-sum-exp (nothing of size S x S is ever stored).  Two tcgen05 kernels, no atomics.
//
//   attn_bwd_dkdv : one CTA per (batch, kv head, 128-key block); loops over the query heads of the group and the
//                   half blocks (64 queries) that see these keys.  Per half block h:
//                     S^T_h = K Q_h^T, dP^T_h = V dO_h^T                       (shared-memory operands, 128 x 64)
//                     P^T_h = exp(S^T_h - lse), dS^T_h = P^T_h * (dP^T_h - delta)    (one key row per thread)
//                     dV += P^T_h dO_h, dK += dS^T_h Q_h     (A operand from TMEM, B MN-major), accumulated in TMEM
//   attn_bwd_dq   : one CTA per (batch, query head, 128-query block); loops over half blocks of 64 keys:
//                     S_h = Q K_h^T, dP_h = dO V_h^T, dS_h = P_h * (dP_h - delta), dQ += dS_h K_h
//   attn_delta    : delta[b,h,s] = sum_d dO * O
// Scores live in a ring of tensor-memory slots (128 columns: S / P in the first 64, dP / dS in the others); the tensor core runs
// products and scores in issue order, so a slot may be refilled right behind the products that read it.  The operand tiles of the
// loop come in half blocks too, through a ring that runs ahead of the slots.
//   Heads of 128: two compute warpgroups take the half blocks in turn, over three slots (dK / dV: two, their accumulators fill 256
// columns), so that the scores of the next half block are there when a warpgroup is done.
//   Heads of 64: loops are short (nine half blocks on average at 1024 tokens) and a CTA's start and end cost as much as they do; one
// warpgroup and one slot in 256 columns, two CTAs per SM, one working while the other starts, waits or writes.  Launches of few CTAs have no
// second one for an SM and take two warpgroups over three slots (launch_bwd).
// Both kernels and attn_delta, us, two warpgroups with a slot each, one CTA per SM -> now: 64 x 1024, 8 heads of 64 769 -> 601, of which the ring
// of slots 747; 8 x 1024 118 -> 100; 4096, 32 / 8 heads of 128 703 -> 645 (the key blocks in head order before: 876).
// The softmax scale multiplies dK and dQ once, when they are written out.
//
// The reference's memory-efficient attention backward is approximate
// (src/trainer/zero_optimizer_mem.cpp:496-574); its autograd attention op (src/model/autograd_functions.cpp:17-226)
// materialises the S x S matrix.  This computes the exact gradient without either.
#include "tfb_host.h"
#include "tfb_ptx.cuh"

namespace tfb {

// warp 0 TMA, warp 1 MMA, warps 2-5 and (heads of 128) 6-9: compute warpgroups
constexpr int AB_BOX = 128 * 64 * 2;
constexpr int AB_HBOX = 64 * 64 * 2;   // 64 columns of a half block (64 rows)
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float bwd_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

struct AttnBwdParams {
  int B, S, Hq, Hkv;
  float scale;
  int causal;
  int q_col0, k_col0, v_col0;       // head-0 column of q / k / v in their source rows
  const float* lse;                 // [B, Hq, S]
  const float* delta;               // [B, Hq, S]
  __nv_bfloat16* dq; long long lddq; int dq_col0;
  __nv_bfloat16* dk; long long lddk; int dk_col0;
  __nv_bfloat16* dv; long long lddv; int dv_col0;
  int* status;
};

template <int D, bool DKDV, int WARPGROUPS>
struct BwdSmem {
  static constexpr int NB = D / 64;
  static constexpr int TILE = NB * AB_BOX, HALF = NB * AB_HBOX;     // a resident tile, a half block
  static constexpr int WG = WARPGROUPS;                             // compute warpgroups; one: two blocks per SM (heads of 64)
  static constexpr int THREADS = 64 + 128 * WG;
  static constexpr int SLOTS = WG == 1 ? 1 : D == 128 && DKDV ? 2 : 3;      // tensor-memory slots
  static constexpr int ACC_COL = SLOTS * 128, TMEM = WG == 1 ? 256 : 512;
  static constexpr int STAGES = WG == 1 ? 4 : D == 64 ? 6 : DKDV ? 4 : 5;   // half blocks (two operands each) in flight
  static constexpr int RING_OFF = 2 * TILE;                         // behind two resident tiles
  static constexpr int STAT_OFF = RING_OFF + STAGES * 2 * HALF;     // [warpgroups][2 turns][64 -lse | 64 -delta] floats
  static constexpr int BAR_OFF = STAT_OFF + (DKDV ? WG * 2 * 128 * 4 : 0);
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
  static_assert(ACC_COL + (DKDV ? 2 : 1) * D <= TMEM && TOTAL <= (WG == 1 ? 115712 : 232448), "tensor and shared memory");
};

// 16 output rows x 128 bf16 columns of an accumulator, written by one thread (its row)
__device__ __forceinline__ void store_row32(__nv_bfloat16* dst, const uint32_t (&v)[32], float sc) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint4 u;
    u.x = pack_bf16(__uint_as_float(v[q * 8 + 0]) * sc, __uint_as_float(v[q * 8 + 1]) * sc);
    u.y = pack_bf16(__uint_as_float(v[q * 8 + 2]) * sc, __uint_as_float(v[q * 8 + 3]) * sc);
    u.z = pack_bf16(__uint_as_float(v[q * 8 + 4]) * sc, __uint_as_float(v[q * 8 + 5]) * sc);
    u.w = pack_bf16(__uint_as_float(v[q * 8 + 6]) * sc, __uint_as_float(v[q * 8 + 7]) * sc);
    *reinterpret_cast<uint4*>(dst + q * 8) = u;
  }
}

// ------------------------------------------------------------------------------------------------
// dK / dV
// ------------------------------------------------------------------------------------------------
template <int D, int WARPGROUPS>
__global__ void __launch_bounds__(BwdSmem<D, true, WARPGROUPS>::THREADS, WARPGROUPS == 1 ? 2 : 1)
attn_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                     const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo,
                     const AttnBwdParams p) {
  using L = BwdSmem<D, true, WARPGROUPS>;
  constexpr int NB = L::NB, NS = L::SLOTS, ST = L::STAGES, WG = L::WG;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sK = sbase, sV = sbase + L::TILE;
  float* stats = reinterpret_cast<float*>(smem + L::STAT_OFF);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  const uint32_t bar_kv = smem_u32(bars);
  const uint32_t bar_full = bar_kv + 8;             // [ST] Q / dO half block loaded
  const uint32_t bar_empty = bar_full + ST * 8;     // [ST] consumed
  const uint32_t bar_s = bar_empty + ST * 8;        // [NS] S^T and dP^T ready
  const uint32_t bar_pds = bar_s + NS * 8;          // [NS] P^T and dS^T written (128 arrivals)
  const uint32_t bar_stat = bar_pds + NS * 8;       // [2] statistics of a warpgroup's half block staged (128 arrivals)
  const uint32_t bar_acc = bar_stat + 16;           // all accumulation done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 + 2 * ST + 2 * NS + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // causal: the first key blocks see the most queries; all of them start first, so that no long block is left for the end (4096 tokens,
  // 32 / 8 heads of 128, both gradient kernels: 874 -> 703 us)
  const int jb = int(blockIdx.x) / (p.Hkv * p.B);
  const int rem = int(blockIdx.x) % (p.Hkv * p.B);
  const int hk = rem % p.Hkv, b = rem / p.Hkv;
  const int G = p.Hq / p.Hkv;
  const int i0 = p.causal ? 2 * jb : 0;             // first half block of queries
  const int n_i = (p.S + 63) / 64 - i0;
  const int n = G * n_i;

  if (threadIdx.x == 0) {
    mbar_init(bar_kv, 1);
    for (int s = 0; s < ST; ++s) {
      mbar_init(bar_full + s * 8, 1);
      mbar_init(bar_empty + s * 8, 1);
    }
    for (int s = 0; s < NS; ++s) {
      mbar_init(bar_s + s * 8, 1);
      mbar_init(bar_pds + s * 8, 128);
    }
    for (int s = 0; s < 2; ++s) mbar_init(bar_stat + s * 8, 128);
    mbar_init(bar_acc, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), L::TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  tfb::pdl_sync();   // after the allocation: a block of the next kernel may be placed from here on, and must not get the columns first
  const uint32_t tDV = tmem_base + L::ACC_COL, tDK = tDV + D;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(bar_kv, 2 * L::TILE);
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        tma_load_3d(sK + c * AB_BOX, &tk, bar_kv, p.k_col0 + hk * D + c * 64, jb * 128, b);
        tma_load_3d(sV + c * AB_BOX, &tv, bar_kv, p.v_col0 + hk * D + c * 64, jb * 128, b);
      }
      int st = 0, h = hk * G, i = i0;
      uint32_t ph = 1;
      for (int hs = 0; hs < n; ++hs) {
        if (!mbar_wait(bar_empty + st * 8, ph, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
        const uint32_t fb = bar_full + st * 8;
        mbar_expect_tx(fb, 2 * L::HALF);
        const uint32_t sQ = sbase + L::RING_OFF + st * 2 * L::HALF, sDO = sQ + L::HALF;
#pragma unroll
        for (int c = 0; c < NB; ++c) {
          tma_load_3d(sQ + c * AB_HBOX, &tq, fb, p.q_col0 + h * D + c * 64, i * 64, b);
          tma_load_3d(sDO + c * AB_HBOX, &tdo, fb, h * D + c * 64, i * 64, b);
        }
        if (++i == i0 + n_i) { i = i0; ++h; }
        if (++st == ST) { st = 0; ph ^= 1; }
      }
      if (*abort_flag) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) {}
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = umma_idesc(FMT_BF16, FMT_BF16, false, false, 128, 64);
      constexpr uint32_t idesc_acc = umma_idesc(FMT_BF16, FMT_BF16, false, true, 128, D);
      const uint32_t dK = umma_desc_lo(sK, 16), dV = umma_desc_lo(sV, 16);
      // scores of the half block in stage st into slot sl
      auto issue_scores = [&](int sl, int st) {
        const uint32_t sQ = sbase + L::RING_OFF + st * 2 * L::HALF;
        const uint32_t dQ = umma_desc_lo(sQ, 16), dDO = umma_desc_lo(sQ + L::HALF, 16);
        const uint32_t tS = tmem_base + sl * 128, tDP = tS + 64;
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          umma_f16_ss_lo(tS, dK + (((k >> 2) * AB_BOX + (k & 3) * 32) >> 4), dQ + (((k >> 2) * AB_HBOX + (k & 3) * 32) >> 4), idesc_s, k > 0);
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          umma_f16_ss_lo(tDP, dV + (((k >> 2) * AB_BOX + (k & 3) * 32) >> 4), dDO + (((k >> 2) * AB_HBOX + (k & 3) * 32) >> 4), idesc_s, k > 0);
        umma_commit(bar_s + sl * 8);
      };
      bool ok = mbar_wait(bar_kv, 0, abort_flag, p.status, ST_TIMEOUT_FULL);
      int nst = 0;                      // stage and turn of the next scores
      uint32_t nph = 0;
      auto next_scores = [&](int sl) {
        if (!mbar_wait(bar_full + nst * 8, nph, abort_flag, p.status, ST_TIMEOUT_FULL)) { ok = false; return; }
        tc_fence_after();
        issue_scores(sl, nst);
        if (++nst == ST) { nst = 0; nph ^= 1; }
      };
      for (int hs = 0; hs < NS && hs < n && ok; ++hs) next_scores(hs);
      int sl = 0, st = 0;
      uint32_t sph = 0;
      for (int hs = 0; hs < n && ok; ++hs) {
        if (!mbar_wait(bar_pds + sl * 8, sph, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t sQ = sbase + L::RING_OFF + st * 2 * L::HALF;
        const uint32_t dQ = umma_desc_lo(sQ, AB_HBOX), dDO = umma_desc_lo(sQ + L::HALF, AB_HBOX);
        const uint32_t tS = tmem_base + sl * 128, tDP = tS + 64;
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_f16_ts_lo(tDV, tS + k * 8, dDO + k * (2048 >> 4), idesc_acc, hs > 0 || k > 0);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_f16_ts_lo(tDK, tDP + k * 8, dQ + k * (2048 >> 4), idesc_acc, hs > 0 || k > 0);
        umma_commit(bar_empty + st * 8);
        if (hs + NS < n) next_scores(sl);
        if (++sl == NS) { sl = 0; sph ^= 1; }
        if (++st == ST) st = 0;
      }
      umma_commit(bar_acc);
    }
  } else {
    const int w = (warp - 2) >> 2;
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const int key_idx = jb * 128 + r;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    const float2 sl2 = make_float2(p.scale * LOG2E, p.scale * LOG2E);
    bool ok = true;
    // thread r stages one statistic of the half block's 64 queries, negated: r < 64 the pre-scaled log-sum-exp of query r, else the
    // delta of query r - 64.  Loaded one turn ahead so that the global-memory latency hides behind the arithmetic.
    auto load_stat = [&](int g, int i) -> float {
      const int qi = (i0 + i) * 64 + (r & 63);
      const long long o = ((long long)b * p.Hq + hk * G + g) * p.S + qi;
      if (r < 64) return qi < p.S ? -p.lse[o] * LOG2E : -INFINITY;   // probability 0 for padded queries
      return qi < p.S ? -p.delta[o] : 0.f;
    };
    auto advance = [&](int& g, int& i) {      // to this warpgroup's next half block
      i += WG;
      while (i >= n_i) { i -= n_i; ++g; }
    };
    int g = 0, i = w, slot = w;
    uint32_t turn = 0, sph = 0;
    while (i >= n_i) { i -= n_i; ++g; }
    float nxt = w < n ? load_stat(g, i) : 0.f;
    for (int hs = w; hs < n; hs += WG, turn ^= 1) {
      const int q0 = (i0 + i) * 64;
      const uint32_t tS = tmem_base + slot * 128 + lane_off, tDP = tS + 64;
      const uint32_t bar_ready = bar_s + slot * 8, bar_done = bar_pds + slot * 8, par = sph;
      slot += WG;
      if (slot >= NS) { slot -= NS; sph ^= 1; }
      float* s_lse = stats + (w * 2 + turn) * 128;
      float* s_dl = s_lse + 64;
      s_lse[r] = nxt;
      mbar_arrive(bar_stat + w * 8);
      advance(g, i);
      if (hs + WG < n) nxt = load_stat(g, i);
      if (!mbar_wait_warp(bar_stat + w * 8, turn, abort_flag, p.status, ST_TIMEOUT_FLAG)) { ok = false; break; }
      if (!mbar_wait_warp(bar_ready, par, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const bool diag = p.causal && q0 < jb * 128 + 128;
      uint32_t sv[2][32], dv[2][32];
      tmem_ld_32x32(tS, sv[0]);
      tmem_ld_32x32(tDP, dv[0]);
      tmem_ld_wait_regs(sv[0]);
      tmem_ld_wait_regs(dv[0]);
      tmem_ld_32x32(tS + 32, sv[1]);          // in flight behind the arithmetic of the first half
      tmem_ld_32x32(tDP + 32, dv[1]);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (c == 1) {
          tmem_ld_wait_regs(sv[1]);
          tmem_ld_wait_regs(dv[1]);
        }
        uint32_t pk[16], ds[16];
#pragma unroll
        for (int e = 0; e < 16; e += 2) {
          const float4 l4 = *reinterpret_cast<const float4*>(s_lse + c * 32 + e * 2);   // same address in every lane: broadcast
          const float4 d4 = *reinterpret_cast<const float4*>(s_dl + c * 32 + e * 2);
          float2 a = fma2(make_float2(__uint_as_float(sv[c][2 * e]), __uint_as_float(sv[c][2 * e + 1])), sl2, make_float2(l4.x, l4.y));
          float2 e2 = fma2(make_float2(__uint_as_float(sv[c][2 * e + 2]), __uint_as_float(sv[c][2 * e + 3])), sl2, make_float2(l4.z, l4.w));
          a.x = bwd_exp2(a.x);
          a.y = bwd_exp2(a.y);
          e2.x = bwd_exp2(e2.x);
          e2.y = bwd_exp2(e2.y);
          if (diag) {
            const int q = q0 + c * 32 + 2 * e;
            if (q < key_idx) a.x = 0.f;
            if (q + 1 < key_idx) a.y = 0.f;
            if (q + 2 < key_idx) e2.x = 0.f;
            if (q + 3 < key_idx) e2.y = 0.f;
          }
          pk[e] = pack_bf16(a.x, a.y);
          pk[e + 1] = pack_bf16(e2.x, e2.y);
          a = mul2(a, add2(make_float2(__uint_as_float(dv[c][2 * e]), __uint_as_float(dv[c][2 * e + 1])), make_float2(d4.x, d4.y)));
          e2 = mul2(e2, add2(make_float2(__uint_as_float(dv[c][2 * e + 2]), __uint_as_float(dv[c][2 * e + 3])), make_float2(d4.z, d4.w)));
          ds[e] = pack_bf16(a.x, a.y);
          ds[e + 1] = pack_bf16(e2.x, e2.y);
        }
        tmem_st_32x16(tS + c * 16, pk);
        tmem_st_32x16(tDP + c * 16, ds);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(bar_done);
    }
    if (ok && mbar_wait_warp(bar_acc, 0, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
      const bool valid = key_idx < p.S;
      const long long row = (long long)b * p.S + (valid ? key_idx : 0);
      // warpgroup 0 writes dV, warpgroup 1 (or the only one) dK, scaled.  The tensor-memory loads are warp-collective: every
      // lane executes them, only the stores are predicated.
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (WG == 2 && k != w) continue;
        __nv_bfloat16* dst = k == 0 ? p.dv + row * p.lddv + p.dv_col0 + hk * D : p.dk + row * p.lddk + p.dk_col0 + hk * D;
        const uint32_t tA = (k == 0 ? tDV : tDK) + lane_off;
        const float sc = k == 0 ? 1.f : p.scale;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t v[32];
          tmem_ld_32x32(tA + c * 32, v);
          tmem_ld_wait_regs(v);
          if (valid) store_row32(dst + c * 32, v, sc);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, L::TMEM);
  }
}

// ------------------------------------------------------------------------------------------------
// dQ
// ------------------------------------------------------------------------------------------------
// dS = P * (dP - delta) for one query row and one half block (64 keys): reads S and dP from tensor memory, writes dS
// (bf16 pairs) over the dP columns.  nlse2, ndl: negated log-sum-exp (base 2) and delta of the row.
template <bool MASK>
__device__ __forceinline__ void dq_half_block(uint32_t tS, uint32_t tDP, float scale2, float nlse2, float ndl, int k0, int k_lim) {
  uint32_t sv[2][32], dv[2][32];
  const float2 sl2 = make_float2(scale2, scale2), l2 = make_float2(nlse2, nlse2), d2 = make_float2(ndl, ndl);
  tmem_ld_32x32(tS, sv[0]);
  tmem_ld_32x32(tDP, dv[0]);
  tmem_ld_wait_regs(sv[0]);
  tmem_ld_wait_regs(dv[0]);
  tmem_ld_32x32(tS + 32, sv[1]);             // in flight behind the arithmetic of the first half
  tmem_ld_32x32(tDP + 32, dv[1]);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t ds[16];
    if (c == 1) {
      tmem_ld_wait_regs(sv[1]);
      tmem_ld_wait_regs(dv[1]);
    }
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      float2 a = fma2(make_float2(__uint_as_float(sv[c][2 * e]), __uint_as_float(sv[c][2 * e + 1])), sl2, l2);
      a.x = bwd_exp2(a.x);
      a.y = bwd_exp2(a.y);
      if (MASK) {
        if (k0 + c * 32 + 2 * e > k_lim) a.x = 0.f;
        if (k0 + c * 32 + 2 * e + 1 > k_lim) a.y = 0.f;
      }
      a = mul2(a, add2(make_float2(__uint_as_float(dv[c][2 * e]), __uint_as_float(dv[c][2 * e + 1])), d2));
      ds[e] = pack_bf16(a.x, a.y);
    }
    tmem_st_32x16(tDP + c * 16, ds);
  }
}

template <int D, int WARPGROUPS>
__global__ void __launch_bounds__(BwdSmem<D, false, WARPGROUPS>::THREADS, WARPGROUPS == 1 ? 2 : 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                   const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo,
                   const AttnBwdParams p) {
  using L = BwdSmem<D, false, WARPGROUPS>;
  constexpr int NB = L::NB, NS = L::SLOTS, ST = L::STAGES, WG = L::WG;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase, sDO = sbase + L::TILE;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  const uint32_t bar_q = smem_u32(bars);
  const uint32_t bar_full = bar_q + 8;             // [ST]
  const uint32_t bar_empty = bar_full + ST * 8;    // [ST]
  const uint32_t bar_s = bar_empty + ST * 8;       // [NS] S and dP ready
  const uint32_t bar_ds = bar_s + NS * 8;          // [NS] dS written (128 arrivals)
  const uint32_t bar_acc = bar_ds + NS * 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 + 2 * ST + 2 * NS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nqb = (p.S + 127) / 128, nkh = (p.S + 63) / 64;
  const int bh = p.B * p.Hq;
  const int qb = nqb - 1 - int(blockIdx.x) / bh;
  const int rem = int(blockIdx.x) % bh;
  const int b = rem / p.Hq, h = rem % p.Hq;
  const int hk = h / (p.Hq / p.Hkv);
  const int n = p.causal ? min(2 * qb + 2, nkh) : nkh;

  if (threadIdx.x == 0) {
    mbar_init(bar_q, 1);
    for (int s = 0; s < ST; ++s) {
      mbar_init(bar_full + s * 8, 1);
      mbar_init(bar_empty + s * 8, 1);
    }
    for (int s = 0; s < NS; ++s) {
      mbar_init(bar_s + s * 8, 1);
      mbar_init(bar_ds + s * 8, 128);
    }
    mbar_init(bar_acc, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), L::TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  tfb::pdl_sync();   // after the allocation: a block of the next kernel may be placed from here on, and must not get the columns first
  const uint32_t tDQ = tmem_base + L::ACC_COL;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(bar_q, 2 * L::TILE);
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        tma_load_3d(sQ + c * AB_BOX, &tq, bar_q, p.q_col0 + h * D + c * 64, qb * 128, b);
        tma_load_3d(sDO + c * AB_BOX, &tdo, bar_q, h * D + c * 64, qb * 128, b);
      }
      int st = 0;
      uint32_t ph = 1;
      for (int hs = 0; hs < n; ++hs) {
        if (!mbar_wait(bar_empty + st * 8, ph, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
        const uint32_t fb = bar_full + st * 8;
        mbar_expect_tx(fb, 2 * L::HALF);
        const uint32_t sK = sbase + L::RING_OFF + st * 2 * L::HALF, sV = sK + L::HALF;
#pragma unroll
        for (int c = 0; c < NB; ++c) {
          tma_load_3d(sK + c * AB_HBOX, &tk, fb, p.k_col0 + hk * D + c * 64, hs * 64, b);
          tma_load_3d(sV + c * AB_HBOX, &tv, fb, p.v_col0 + hk * D + c * 64, hs * 64, b);
        }
        if (++st == ST) { st = 0; ph ^= 1; }
      }
      if (*abort_flag) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) {}
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = umma_idesc(FMT_BF16, FMT_BF16, false, false, 128, 64);
      constexpr uint32_t idesc_acc = umma_idesc(FMT_BF16, FMT_BF16, false, true, 128, D);
      const uint32_t dQ = umma_desc_lo(sQ, 16), dDO = umma_desc_lo(sDO, 16);
      auto issue_scores = [&](int sl, int st) {
        const uint32_t sK = sbase + L::RING_OFF + st * 2 * L::HALF;
        const uint32_t dK = umma_desc_lo(sK, 16), dV = umma_desc_lo(sK + L::HALF, 16);
        const uint32_t tS = tmem_base + sl * 128, tDP = tS + 64;
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          umma_f16_ss_lo(tS, dQ + (((k >> 2) * AB_BOX + (k & 3) * 32) >> 4), dK + (((k >> 2) * AB_HBOX + (k & 3) * 32) >> 4), idesc_s, k > 0);
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          umma_f16_ss_lo(tDP, dDO + (((k >> 2) * AB_BOX + (k & 3) * 32) >> 4), dV + (((k >> 2) * AB_HBOX + (k & 3) * 32) >> 4), idesc_s, k > 0);
        umma_commit(bar_s + sl * 8);
      };
      bool ok = mbar_wait(bar_q, 0, abort_flag, p.status, ST_TIMEOUT_FULL);
      int nst = 0;                      // stage and turn of the next scores
      uint32_t nph = 0;
      auto next_scores = [&](int sl) {
        if (!mbar_wait(bar_full + nst * 8, nph, abort_flag, p.status, ST_TIMEOUT_FULL)) { ok = false; return; }
        tc_fence_after();
        issue_scores(sl, nst);
        if (++nst == ST) { nst = 0; nph ^= 1; }
      };
      for (int hs = 0; hs < NS && hs < n && ok; ++hs) next_scores(hs);
      int sl = 0, st = 0;
      uint32_t sph = 0;
      for (int hs = 0; hs < n && ok; ++hs) {
        if (!mbar_wait(bar_ds + sl * 8, sph, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t dK = umma_desc_lo(sbase + L::RING_OFF + st * 2 * L::HALF, AB_HBOX);
        const uint32_t tDP = tmem_base + sl * 128 + 64;
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_f16_ts_lo(tDQ, tDP + k * 8, dK + k * (2048 >> 4), idesc_acc, hs > 0 || k > 0);
        umma_commit(bar_empty + st * 8);
        if (hs + NS < n) next_scores(sl);
        if (++sl == NS) { sl = 0; sph ^= 1; }
        if (++st == ST) st = 0;
      }
      umma_commit(bar_acc);
    }
  } else {
    const int w = (warp - 2) >> 2;
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const int q_idx = qb * 128 + r;
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    const float sl2 = p.scale * LOG2E;
    const long long so = ((long long)b * p.Hq + h) * p.S + q_idx;
    const float nlse2 = q_idx < p.S ? -p.lse[so] * LOG2E : -INFINITY;
    const float ndl = q_idx < p.S ? -p.delta[so] : 0.f;
    bool ok = true;
    for (int hs = w; hs < n; hs += WG) {
      const int slot = hs % NS;
      const uint32_t tS = tmem_base + slot * 128 + lane_off, tDP = tS + 64;
      if (!mbar_wait_warp(bar_s + slot * 8, (hs / NS) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      const int k0 = hs * 64;
      const bool need_mask = (p.causal && k0 + 63 > qb * 128) || (k0 + 64 > p.S);
      const int k_lim = p.causal ? min(q_idx, p.S - 1) : p.S - 1;
      if (need_mask) dq_half_block<true>(tS, tDP, sl2, nlse2, ndl, k0, k_lim);
      else dq_half_block<false>(tS, tDP, sl2, nlse2, ndl, k0, k_lim);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(bar_ds + slot * 8);
    }
    if (ok && mbar_wait_warp(bar_acc, 0, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
      // each warpgroup writes its share of the row's columns
      __nv_bfloat16* dqp = p.dq + ((long long)b * p.S + q_idx) * p.lddq + p.dq_col0 + h * D + w * (D / WG);
#pragma unroll
      for (int c = 0; c < D / 32 / WG; ++c) {
        uint32_t v[32];
        tmem_ld_32x32(tDQ + lane_off + w * (D / WG) + c * 32, v);
        tmem_ld_wait();
        if (q_idx < p.S) store_row32(dqp + c * 32, v, p.scale);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, L::TMEM);
  }
}

// delta[b,h,s] = sum_d dO[t, h*D + d] * O[t, h*D + d].  One thread per 8 consecutive elements of a token row (16-byte
// loads, consecutive lanes on consecutive addresses); the D / 8 lanes of a head reduce with shuffles.
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ o, long long ldo,
                                                         const __nv_bfloat16* __restrict__ dout, long long lddo,
                                                         float* __restrict__ delta, int B, int S, int Hq, int D) {
  tfb::pdl_sync();
  const int per_row = Hq * D / 8;                       // threads per token row
  const long long total = (long long)B * S * per_row;
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const bool live = i < total;
  const long long t = live ? i / per_row : 0;
  const int c = live ? int(i - t * per_row) * 8 : 0;    // first column of this thread
  float acc = 0.f;
  if (live) {
    const uint4 a = *reinterpret_cast<const uint4*>(o + t * ldo + c);
    const uint4 g = *reinterpret_cast<const uint4*>(dout + t * lddo + c);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, gw[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = unpack_bf16(aw[j]), y = unpack_bf16(gw[j]);
      acc += x.x * y.x + x.y * y.y;
    }
  }
  const int group = D / 8;                              // 8 or 16 lanes per head, aligned inside the warp
  for (int off = group >> 1; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (live && (threadIdx.x & (group - 1)) == 0) {
    const int h = c / D;
    const long long bb = t / S, s_ = t % S;
    delta[(bb * Hq + h) * S + s_] = acc;
  }
}

template <int D, int WARPGROUPS>
static int launch_dkdv(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo, const AttnBwdParams& p, int blocks,
                       cudaStream_t st) {
  using L = BwdSmem<D, true, WARPGROUPS>;
  static DeviceOnce once;   // kernel attributes are per device: set on the first launch on each one
  auto kern = attn_bwd_dkdv_kernel<D, WARPGROUPS>;
  if (int e = ensure_dyn_smem(once, kern, L::TOTAL)) return e;
  tfb::launch_k(kern, blocks, L::THREADS, L::TOTAL, st, tq, tk, tv, tdo, p);
  return int(cudaGetLastError());
}
template <int D, int WARPGROUPS>
static int launch_dq(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo, const AttnBwdParams& p, int blocks,
                     cudaStream_t st) {
  using L = BwdSmem<D, false, WARPGROUPS>;
  static DeviceOnce once;
  auto kern = attn_bwd_dq_kernel<D, WARPGROUPS>;
  if (int e = ensure_dyn_smem(once, kern, L::TOTAL)) return e;
  tfb::launch_k(kern, blocks, L::THREADS, L::TOTAL, st, tq, tk, tv, tdo, p);
  return int(cudaGetLastError());
}

static int launch_bwd(int D, const CUtensorMap (&m)[8], const AttnBwdParams& p, cudaStream_t st) {
  // boxes of 128 rows (resident tiles) and of 64 (half blocks)
  const CUtensorMap &tq = m[0], &tk = m[1], &tv = m[2], &tdo = m[3], &q_half = m[4], &k_half = m[5], &v_half = m[6], &do_half = m[7];
  const int nqb = (p.S + 127) / 128, b1 = nqb * p.Hkv * p.B, b2 = nqb * p.Hq * p.B;
  if (D == 128) {
    if (int e = launch_dkdv<128, 2>(q_half, tk, tv, do_half, p, b1, st)) return e;
    return launch_dq<128, 2>(tq, k_half, v_half, tdo, p, b2, st);
  }
  // Heads of 64: one warpgroup and two blocks per SM only pay where a second block is there to fill the first one's waits.  us, all gradient kernels,
  // one warpgroup / two: 36 blocks (1 x 300, 12 heads) 24.6 / 20.2, 64 (1 x 2048, 4) 99.6 / 69.9, 128 (16 x 128, 8) 18.2 / 16.7, 192 (3 x 1024, 8) 58.7 /
  // 42.4, 256 (4 x 1024, 8) 61.0 / 50.6, but 256 short ones (32 x 128, 8) 23.2 / 28.5, 320 (5 x 1024, 8) 62.9 / 65.5, 512 (8 x 1024, 8) 88.6 / 97.2.
  const int sms = sm_count(), alone = p.S >= 512 ? 2 * sms : sms;
  if (int e = b1 <= alone ? launch_dkdv<64, 2>(q_half, tk, tv, do_half, p, b1, st) : launch_dkdv<64, 1>(q_half, tk, tv, do_half, p, b1, st)) return e;
  return b2 <= alone ? launch_dq<64, 2>(tq, k_half, v_half, tdo, p, b2, st) : launch_dq<64, 1>(tq, k_half, v_half, tdo, p, b2, st);
}

}  // namespace tfb

// Gradients of tfb_attn_fwd.  q/k/v as in the forward; o and dout are [B*S, ld] with head h at column
// h*D; lse from the forward; delta is [B,Hq,S] fp32 scratch filled here.  dq/dk/dv are written (not
// accumulated) at column offsets d*_col0 + head*D of rows with pitches ldd* - they may all point into
// one fused [T, (Hq + 2 Hkv) D] gradient buffer.
TFB_API int tfb_attn_bwd(const void* q, long long ldq, int q_col0, const void* k, long long ldk, int k_col0,
                         const void* v, long long ldv, int v_col0, const void* o, long long ldo, const void* dout,
                         long long lddo, const float* lse, float* delta, void* dq, long long lddq, int dq_col0,
                         void* dk, long long lddk, int dk_col0, void* dv, long long lddv, int dv_col0, int B, int S,
                         int Hq, int Hkv, int D, float scale, int causal, int* status, void* stream) {
  using namespace tfb;
  if ((D != 64 && D != 128) || Hkv <= 0 || Hq % Hkv || B <= 0 || S <= 0) return TFB_ERR_ARG;
  if ((q_col0 | k_col0 | v_col0 | dq_col0 | dk_col0 | dv_col0) & 7) return TFB_ERR_ARG;
  if ((lddq | lddk | lddv) & 7) return TFB_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv)) & 15)
    return TFB_ERR_ARG;
  if (((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(dout)) & 15) || (ldo & 7) || (lddo & 7)) return TFB_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  {
    const long long threads = (long long)B * S * Hq * D / 8;
    const int blocks = int((threads + 255) / 256);
    tfb::launch_k(attn_delta_kernel, blocks, 256, 0, st, static_cast<const __nv_bfloat16*>(o), ldo,
                                              static_cast<const __nv_bfloat16*>(dout), lddo, delta, B, S, Hq, D);
  }
  CUtensorMap maps[8];
  for (int i = 0; i < 8; ++i) {
    const void* base[4] = {q, k, v, dout};
    const long long ld[4] = {ldq, ldk, ldv, lddo};
    const long long l = ld[i & 3];
    if (int rc = make_tmap_3d(&maps[i], base[i & 3], 2, l, S, B, l * 2, l * 2 * S, 64, i < 4 ? 128 : 64, 1)) return rc;
  }
  AttnBwdParams p;
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv; p.scale = scale; p.causal = causal;
  p.q_col0 = q_col0; p.k_col0 = k_col0; p.v_col0 = v_col0;
  p.lse = lse; p.delta = delta;
  p.dq = static_cast<__nv_bfloat16*>(dq); p.lddq = lddq; p.dq_col0 = dq_col0;
  p.dk = static_cast<__nv_bfloat16*>(dk); p.lddk = lddk; p.dk_col0 = dk_col0;
  p.dv = static_cast<__nv_bfloat16*>(dv); p.lddv = lddv; p.dv_col0 = dv_col0;
  p.status = status;
  return launch_bwd(D, maps, p, st);
}
