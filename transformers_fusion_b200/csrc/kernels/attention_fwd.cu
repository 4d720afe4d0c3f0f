// Flash attention forward for sm_100a (causal or full, grouped-query heads, head_dim 64 or 128).
//
// One CTA per (batch, query head, block of 128 * TILES queries):
//   warp 0        TMA producer: the Q tiles once, then K_j / V_j tiles (128 keys) through a shared-memory ring
//   warp 1        MMA issuer:   S_t = Q_t K_j^T  (tcgen05.mma, both operands in shared memory, fp32 in TMEM)
//                               O_t += P_t V_j   (A operand = bf16 probabilities read from TMEM, B = V_j MN-major)
//   warps 2..5    softmax of tile 0, warps 6..9 of tile 1: one query row per thread - the score row comes out of tensor memory
//                 once and stays in registers through maximum, exponentials and sum; P goes back as bf16 pairs.
// O accumulates in tensor memory relative to a reference maximum that only moves when a row's maximum has grown by more than
// 2^8 (probabilities are then below 256, which bf16 and the fp32 sums hold as exactly as values below one); a move rescales
// the accumulator.  The result divides by the sum relative to the same reference.
// Error of O against float64, of its norm (bf16 rounding of the probabilities and of O): 1.777e-3 at 4 x 1024, heads of 64, 1.793e-3 at 4096, heads of
// 128; 1.774e-3 and 1.792e-3 with a product per tile, added in registers, and a row's largest probability exactly one.
//
// Head size 64: one tile per CTA in 256 columns of tensor memory (scores 0..127, O 128..191, P 192..255), so that two CTAs share an
// SM and one computes while the other starts or ends; P has columns of its own, so S(j+1) is computed while the
// exponentials of S(j) are.  Head size 128: two tiles per CTA that share K and V and take turns on the tensor core (scores and P
// of tile t at 128 t, O at 256 + 128 t); P overwrites S, S_t(j+1) is issued after P_t(j) V_j, and its commit covers both.
//
// At head size 64 the exponentials bound the kernel (128 x 128 of them, 16 per clock, against 384 cycles of tensor time).  Before: two
// passes over the scores in tensor memory, O in registers with a rescale per key tile, 256 queries and one CTA per SM at
// both head sizes.
//
// Reference counterparts: attention_kernel (src/backend/gpu_compute_cuda.cpp:296, one thread per
// query, three passes, non-causal), CPU flash attention (src/kernel/flash_attention.cpp:38-225).
#include "tfb_host.h"
#include "tfb_ptx.cuh"

namespace tfb {

constexpr int ATT_BM = 128;   // queries per tile
constexpr int ATT_BN = 128;   // keys per step
constexpr int BOX_BYTES = 128 * 64 * 2;

struct AttnFwdParams {
  int B, S, Hq, Hkv;
  int Skv, q_off;  // keys per sequence; causal: query i sees keys <= i + q_off (q_off = Skv - S: the queries are the last S positions)
  float scale;
  int causal;
  int q_col0, k_col0, v_col0;
  __nv_bfloat16* O;
  long long ldo;
  float* lse;  // [B, Hq, S]
  const int4* work;  // packed form: (first row, length, pair of query tiles, unused) of every work item, longest first
  int* status;
};

template <int D>
struct AttnSmem {
  static constexpr int TILES = D == 64 ? 1 : 2;
  static constexpr int THREADS = 64 + 128 * TILES;
  static constexpr bool OWN_P = D == 64;                       // P in columns of its own
  static constexpr int TMEM = TILES == 1 ? 256 : 512;
  static constexpr int O_COL = 128 * TILES, P_COL = OWN_P ? 192 : 0;
  static constexpr int NB = D / 64;  // 64-column boxes per tile
  static constexpr int TILE = NB * BOX_BYTES;
  static constexpr int STAGES = 2;
  static constexpr int KV_OFF = TILES * TILE;
  static constexpr int BAR_OFF = KV_OFF + STAGES * 2 * TILE;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// p = 2^(s * sl2 - mb) for the 128 scores of this thread's row (registers), written to tensor memory as bf16 pairs; returns the row
// sum (fp32, four partial sums).  MASK: keys after k_lim count as zero.
template <bool MASK>
__device__ __forceinline__ float row_probs(const uint32_t (&v)[4][32], uint32_t tP, float sl2, float mb, int k0, int k_lim) {
  float2 sum0 = make_float2(0.f, 0.f), sum1 = sum0;
  const float2 sc = make_float2(sl2, sl2), off = make_float2(-mb, -mb);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t pk[16];
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      float2 a = fma2(make_float2(__uint_as_float(v[c][2 * i]), __uint_as_float(v[c][2 * i + 1])), sc, off);
      float2 b = fma2(make_float2(__uint_as_float(v[c][2 * i + 2]), __uint_as_float(v[c][2 * i + 3])), sc, off);
      a.x = fast_exp2(a.x);
      a.y = fast_exp2(a.y);
      b.x = fast_exp2(b.x);
      b.y = fast_exp2(b.y);
      if (MASK) {
        if (k0 + c * 32 + 2 * i > k_lim) a.x = 0.f;
        if (k0 + c * 32 + 2 * i + 1 > k_lim) a.y = 0.f;
        if (k0 + c * 32 + 2 * i + 2 > k_lim) b.x = 0.f;
        if (k0 + c * 32 + 2 * i + 3 > k_lim) b.y = 0.f;
      }
      sum0 = add2(sum0, a);
      sum1 = add2(sum1, b);
      pk[i] = pack_bf16(a.x, a.y);
      pk[i + 1] = pack_bf16(b.x, b.y);
    }
    tmem_st_32x16(tP + c * 16, pk);
  }
  return (sum0.x + sum0.y) + (sum1.x + sum1.y);
}

// PACKED: sequences of any lengths stand one after the other in the rows (prompts that are run together); a work item names its
// sequence.  A tile of keys may then reach into the rows of the next sequence: its scores are masked as at the end of a
// tensor, and its V rows, whose probabilities are zero, are cleared in shared memory (zero times infinity is not zero).
template <int D, bool PACKED>
__global__ void __launch_bounds__(AttnSmem<D>::THREADS, AttnSmem<D>::TILES == 1 ? 2 : 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                const __grid_constant__ CUtensorMap tv, const AttnFwdParams p) {
  using L = AttnSmem<D>;
  constexpr int NB = L::NB;
  constexpr int ST = L::STAGES, TILES = L::TILES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(smem);
  const uint32_t sQ = sbase;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  const uint32_t bar_q = smem_u32(bars);
  const uint32_t bar_kv_full = bar_q + 8;
  const uint32_t bar_kv_empty = bar_kv_full + ST * 8;
  const uint32_t bar_s_full = bar_kv_empty + ST * 8;
  const uint32_t bar_p_ready = bar_s_full + 16;
  const uint32_t bar_o_full = bar_p_ready + 16;
  const uint32_t bar_tail = bar_o_full + 16;
  const uint32_t bar_s_free = bar_tail + 8;      // own P columns: the scores are in registers
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1 + 2 * ST + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(bar_q, 1);
    for (int s = 0; s < ST; ++s) {
      mbar_init(bar_kv_full + s * 8, 1);
      mbar_init(bar_kv_empty + s * 8, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_s_full + i * 8, 1);
      mbar_init(bar_p_ready + i * 8, 128);
      mbar_init(bar_o_full + i * 8, 1);
    }
    mbar_init(bar_tail, 1);
    mbar_init(bar_s_free, 128);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tq);
    tma_prefetch_desc(&tk);
    tma_prefetch_desc(&tv);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), L::TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  tfb::pdl_sync();   // set-up above touches no global memory; operands written by the previous kernel are read below
  int S = p.S, Skv = p.Skv, row0 = 0, b, h, qb0;      // qb0: first 128-query tile of this block
  if constexpr (PACKED) {
    constexpr int PER = 2 / TILES;                     // blocks per work item
    const int i = int(blockIdx.x) / p.Hq;
    const int4 w = p.work[i / PER];
    row0 = w.x;
    S = Skv = w.y;
    qb0 = w.z * 2 + (PER - 1 - i % PER);
    b = 0;
    h = int(blockIdx.x) % p.Hq;
  } else {
    const int nblk = (S + TILES * ATT_BM - 1) / (TILES * ATT_BM);
    const int bh = p.B * p.Hq;
    qb0 = (nblk - 1 - int(blockIdx.x) / bh) * TILES;   // longest (latest) query blocks are scheduled first
    const int rem = int(blockIdx.x) % bh;
    b = rem / p.Hq;
    h = rem % p.Hq;
  }
  const int nkb = (Skv + ATT_BN - 1) / ATT_BN;
  const int hk = h / (p.Hq / p.Hkv);
  // number of key blocks each tile visits (0: the tile lies past the end of the sequence)
  int n_t[TILES];
#pragma unroll
  for (int t = 0; t < TILES; ++t) {
    const int qb = qb0 + t;
    const int q_last = min(qb * ATT_BM + ATT_BM - 1, S - 1);   // last query row of the tile
    n_t[t] = qb * ATT_BM >= S ? 0 : (p.causal ? min((q_last + p.q_off) / ATT_BN + 1, nkb) : nkb);
  }
  const int n_kv = max(n_t[0], n_t[TILES - 1]);
  const bool tail = PACKED && n_kv * ATT_BN > Skv;             // the last key tile ends inside the next sequence's rows
  const uint32_t tS0 = tmem_base, tO0 = tmem_base + L::O_COL;

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(bar_q, TILES * L::TILE);
#pragma unroll
      for (int t = 0; t < TILES; ++t)
#pragma unroll
        for (int i = 0; i < NB; ++i)
          tma_load_3d(sQ + t * L::TILE + i * BOX_BYTES, &tq, bar_q, p.q_col0 + h * D + i * 64, row0 + (qb0 + t) * ATT_BM, b);
      for (int j = 0; j < n_kv; ++j) {
        const int st = j % ST;
        if (!mbar_wait(bar_kv_empty + st * 8, ((j / ST) & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
        const uint32_t fb = bar_kv_full + st * 8;
        mbar_expect_tx(fb, 2 * L::TILE);
        const uint32_t sK = sbase + L::KV_OFF + st * 2 * L::TILE, sV = sK + L::TILE;
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          tma_load_3d(sK + i * BOX_BYTES, &tk, fb, p.k_col0 + hk * D + i * 64, row0 + j * ATT_BN, b);
          tma_load_3d(sV + i * BOX_BYTES, &tv, fb, p.v_col0 + hk * D + i * 64, row0 + j * ATT_BN, b);
        }
      }
      if (*abort_flag) {  // unwinding: bounded wait for copies already issued
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) {}
      }
    }
    if (PACKED && tail) {
      __syncwarp();
      const int j = n_kv - 1, st = j % ST;
      if (mbar_wait_warp(bar_kv_full + st * 8, (j / ST) & 1, abort_flag, p.status, ST_TIMEOUT_FULL)) {
        const uint32_t sV = sbase + L::KV_OFF + st * 2 * L::TILE + L::TILE;
        const int live = (Skv - j * ATT_BN) * 128, all = ATT_BN * 128;                 // bytes of a 64-column box
#pragma unroll
        for (int i = 0; i < NB; ++i)
          for (int o = live + lane * 16; o < all; o += 512) st_shared_v4(sV + i * BOX_BYTES + o, 0u, 0u, 0u, 0u);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_tail);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = umma_idesc(FMT_BF16, FMT_BF16, false, false, ATT_BM, ATT_BN);
      constexpr uint32_t idesc_o = umma_idesc(FMT_BF16, FMT_BF16, false, true, ATT_BM, D);
      auto issue_s = [&](int t, int j) {
        const uint32_t sK = sbase + L::KV_OFF + (j % ST) * 2 * L::TILE;
        const uint32_t dQ = umma_desc_lo(sQ + t * L::TILE, 16), dK = umma_desc_lo(sK, 16);
        const uint32_t tS = tS0 + t * 128;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const uint32_t off = (k >> 2) * BOX_BYTES + (k & 3) * 32;
          umma_f16_ss_lo(tS, dQ + (off >> 4), dK + (off >> 4), idesc_s, k > 0);
        }
        umma_commit(bar_s_full + t * 8);
      };
      auto issue_pv = [&](int t, int j) {
        const uint32_t sV = sbase + L::KV_OFF + (j % ST) * 2 * L::TILE + L::TILE;
        const uint32_t tP = tS0 + t * 128 + L::P_COL, tO = tO0 + t * D, dV = umma_desc_lo(sV, BOX_BYTES);
#pragma unroll
        for (int k = 0; k < ATT_BN / 16; ++k)
          // V_j tile is [key rows][64-col boxes]: MN-major B; 16 keys = 2048 B further, next 64 columns one box on
          umma_f16_ts_lo(tO, tP + k * 8, dV + k * (2048 >> 4), idesc_o, j > 0 || k > 0);
      };
      bool ok = mbar_wait(bar_q, 0, abort_flag, p.status, ST_TIMEOUT_FULL) &&
                (n_kv == 0 || mbar_wait(bar_kv_full, 0, abort_flag, p.status, ST_TIMEOUT_FULL));
      if (ok && n_kv > 0) {
        tc_fence_after();
#pragma unroll
        for (int t = 0; t < TILES; ++t)
          if (n_t[t] > 0) issue_s(t, 0);
      }
      for (int j = 0; j < n_kv && ok; ++j) {
        if (j + 1 < n_kv) {
          const int st1 = (j + 1) % ST;
          if (!mbar_wait(bar_kv_full + st1 * 8, ((j + 1) / ST) & 1, abort_flag, p.status, ST_TIMEOUT_FULL)) break;
          tc_fence_after();
          if constexpr (L::OWN_P) {
            if (!mbar_wait(bar_s_free, j & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY)) break;
            tc_fence_after();
            issue_s(0, j + 1);
          }
        }
        if (PACKED && tail && j == n_kv - 1) {
          if (!mbar_wait(bar_tail, 0, abort_flag, p.status, ST_TIMEOUT_FULL)) break;
          tc_fence_after();
        }
#pragma unroll
        for (int t = 0; t < TILES; ++t) {
          if (!ok || j >= n_t[t]) continue;
          if (!mbar_wait(bar_p_ready + t * 8, j & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY)) {
            ok = false;
            continue;
          }
          tc_fence_after();
          issue_pv(t, j);
          if (L::OWN_P || j + 1 == n_t[t]) umma_commit(bar_o_full + t * 8);
          else issue_s(t, j + 1);                             // its commit also covers the P V product above
        }
        if (ok) umma_commit(bar_kv_empty + (j % ST) * 8);
      }
    }
  } else {
    const int t = (warp - 2) >> 2;
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const int qb = qb0 + t;
    const int q_idx = qb * ATT_BM + r;
    const int n_mine = t ? n_t[TILES - 1] : n_t[0];
    const uint32_t lane_off = uint32_t(quad * 32) << 16;
    const uint32_t tS = tS0 + t * 128 + lane_off;
    const uint32_t tP = tS + L::P_COL;
    const uint32_t tO = tO0 + t * D + lane_off;
    const float sl2 = p.scale * 1.4426950408889634f;
    float m = -INFINITY, l = 0.f;      // reference maximum of this row, sum relative to it
    bool ok = true;
    for (int j = 0; j < n_mine; ++j) {
      if (!mbar_wait_warp(bar_s_full + t * 8, j & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) {
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t v[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(tS + c * 32, v[c]);
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_wait_regs(v[c]);
      if constexpr (L::OWN_P) {
        tc_fence_before();
        mbar_arrive(bar_s_free);
      }
      const int k0 = j * ATT_BN;
      const bool need_mask = (p.causal && k0 + ATT_BN - 1 > qb * ATT_BM + p.q_off) || (k0 + ATT_BN > Skv);
      const int k_lim = p.causal ? min(q_idx + p.q_off, Skv - 1) : (Skv - 1);  // last visible key index for this row
      if (need_mask) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (k0 + c * 32 + i > k_lim) v[c][i] = 0xff800000u;  // -inf
      }
      // four independent chains of three-input max keep the dependent-issue latency off the critical path
      float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          mx0 = fmax3(mx0, __uint_as_float(v[c][i]), __uint_as_float(v[c][i + 1]));
          mx1 = fmax3(mx1, __uint_as_float(v[c][i + 2]), __uint_as_float(v[c][i + 3]));
          mx2 = fmax3(mx2, __uint_as_float(v[c][i + 4]), __uint_as_float(v[c][i + 5]));
          mx3 = fmax3(mx3, __uint_as_float(v[c][i + 6]), __uint_as_float(v[c][i + 7]));
        }
      const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
      if (L::OWN_P && j > 0) {                               // P(j-1) V is done: its P columns are free and O is complete
        if (!mbar_wait_warp(bar_o_full + t * 8, (j - 1) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) {
          ok = false;
          break;
        }
        tc_fence_after();
      }
      if (j == 0) {
        m = mx;
      } else {
        const bool move = (mx - m) * sl2 > 8.f;              // from -inf: infinitely much
        if (__any_sync(0xffffffffu, move)) {
          const float alpha = move ? fast_exp2((m - mx) * sl2) : 1.f;
          if (move) m = mx;
          l *= alpha;
#pragma unroll 1
          for (int c = 0; c < D / 16; ++c) {
            uint32_t w[16];
            tmem_ld_32x16(tO + c * 16, w);
            tmem_ld_wait_regs(w);
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(__uint_as_float(w[i]) * alpha);
            tmem_st_32x16(tO + c * 16, w);
          }
        }
      }
      const float mb = (m == -INFINITY) ? 0.f : m * sl2;
      l += need_mask ? row_probs<true>(v, tP, sl2, mb, k0, k_lim) : row_probs<false>(v, tP, sl2, mb, k0, k_lim);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(bar_p_ready + t * 8);
    }
    if (ok && n_mine > 0) {
      if (mbar_wait_warp(bar_o_full + t * 8, L::OWN_P ? (n_mine - 1) & 1 : 0, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) {
        tc_fence_after();
        const float inv = l > 0.f ? 1.f / l : 0.f;
        __nv_bfloat16* op = p.O + ((long long)b * S + row0 + q_idx) * p.ldo + h * D;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t w[32];
          tmem_ld_32x32(tO + c * 32, w);
          tmem_ld_wait_regs(w);
          if (q_idx < S) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint4 u;
              u.x = pack_bf16(__uint_as_float(w[i * 8 + 0]) * inv, __uint_as_float(w[i * 8 + 1]) * inv);
              u.y = pack_bf16(__uint_as_float(w[i * 8 + 2]) * inv, __uint_as_float(w[i * 8 + 3]) * inv);
              u.z = pack_bf16(__uint_as_float(w[i * 8 + 4]) * inv, __uint_as_float(w[i * 8 + 5]) * inv);
              u.w = pack_bf16(__uint_as_float(w[i * 8 + 6]) * inv, __uint_as_float(w[i * 8 + 7]) * inv);
              *reinterpret_cast<uint4*>(op + c * 32 + i * 8) = u;
            }
          }
        }
        if (!PACKED && p.lse && q_idx < S) p.lse[((long long)b * p.Hq + h) * S + q_idx] = m * p.scale + logf(l);
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

template <int D, bool PACKED>
static int launch_attn_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnFwdParams& p,
                           int blocks, cudaStream_t st) {
  using L = AttnSmem<D>;
  static DeviceOnce once;
  auto kern = attn_fwd_kernel<D, PACKED>;
  if (int e = ensure_dyn_smem(once, kern, L::TOTAL)) return e;
  tfb::launch_k(kern, blocks * p.Hq, L::THREADS, L::TOTAL, st, tq, tk, tv, p);
  return int(cudaGetLastError());
}

}  // namespace tfb

// q, k, v: bf16 buffers whose rows are tokens (b * S + s) with pitches ldq / ldk / ldv (elements);
// head h of q starts at column q_col0 + h * D of its row (likewise k, v with the kv head index), so
// the three pointers may be the same fused [T, (Hq + 2 Hkv) D] projection output.
// o: [B*S, ldo] bf16, head h at column h * D.  lse: [B, Hq, S] fp32 (may be null).
//
// tfb_attn_fwd_kv: the keys / values have Skv >= S rows per sequence (k, v rows are b * Skv + s) and the S queries are the
// last S positions: with `causal`, query i sees keys 0 .. i + (Skv - S).  This is the prefill of a prompt suffix behind a
// cached prefix (the prefix keys come out of the paged cache, see tfb_kv_gather).
TFB_API int tfb_attn_fwd_kv(const void* q, long long ldq, int q_col0, const void* k, long long ldk, int k_col0,
                            const void* v, long long ldv, int v_col0, void* o, long long ldo, float* lse, int B, int S,
                            int Skv, int Hq, int Hkv, int D, float scale, int causal, int* status, void* stream);

TFB_API int tfb_attn_fwd(const void* q, long long ldq, int q_col0, const void* k, long long ldk, int k_col0,
                         const void* v, long long ldv, int v_col0, void* o, long long ldo, float* lse, int B, int S,
                         int Hq, int Hkv, int D, float scale, int causal, int* status, void* stream) {
  return tfb_attn_fwd_kv(q, ldq, q_col0, k, ldk, k_col0, v, ldv, v_col0, o, ldo, lse, B, S, S, Hq, Hkv, D, scale, causal, status,
                         stream);
}

TFB_API int tfb_attn_fwd_kv(const void* q, long long ldq, int q_col0, const void* k, long long ldk, int k_col0,
                            const void* v, long long ldv, int v_col0, void* o, long long ldo, float* lse, int B, int S,
                            int Skv, int Hq, int Hkv, int D, float scale, int causal, int* status, void* stream) {
  using namespace tfb;
  if ((D != 64 && D != 128) || Hkv <= 0 || Hq % Hkv || B <= 0 || S <= 0 || Skv < S) return TFB_ERR_ARG;
  if ((q_col0 | k_col0 | v_col0) & 7 || (ldo & 7) || (reinterpret_cast<uintptr_t>(o) & 15)) return TFB_ERR_ARG;
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_tmap_3d(&tq, q, 2, ldq, S, B, ldq * 2, ldq * 2 * S, 64, 128, 1))) return rc;
  if ((rc = make_tmap_3d(&tk, k, 2, ldk, Skv, B, ldk * 2, ldk * 2 * Skv, 64, 128, 1))) return rc;
  if ((rc = make_tmap_3d(&tv, v, 2, ldv, Skv, B, ldv * 2, ldv * 2 * Skv, 64, 128, 1))) return rc;
  AttnFwdParams p;
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv;
  p.Skv = Skv; p.q_off = Skv - S;
  p.scale = scale; p.causal = causal;
  p.q_col0 = q_col0; p.k_col0 = k_col0; p.v_col0 = v_col0;
  p.O = static_cast<__nv_bfloat16*>(o); p.ldo = ldo; p.lse = lse; p.work = nullptr; p.status = status;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rows = D == 64 ? ATT_BM : 2 * ATT_BM, blocks = (S + rows - 1) / rows * B;
  return D == 64 ? launch_attn_fwd<64, false>(tq, tk, tv, p, blocks, st) : launch_attn_fwd<128, false>(tq, tk, tv, p, blocks, st);
}

// Sequences of any lengths packed one after the other: q, k, v, o rows 0 .. rows - 1, every sequence attends to itself.  `work`
// (device, [items] of four ints): first row, length and pair of 128-query tiles of every work item; a sequence of n rows has
// ceil(n / 256) of them.  One launch over all prompts of a batch instead of one per prompt: what a short prompt cannot
// fill (a prompt of 160 tokens has 32 blocks at 32 heads) its neighbours do.
TFB_API int tfb_attn_fwd_packed(const void* q, long long ldq, int q_col0, const void* k, long long ldk, int k_col0,
                                const void* v, long long ldv, int v_col0, void* o, long long ldo, const void* work, int items,
                                long long rows, int Hq, int Hkv, int D, float scale, int causal, int* status, void* stream) {
  using namespace tfb;
  if ((D != 64 && D != 128) || Hkv <= 0 || Hq <= 0 || Hq % Hkv || rows <= 0 || rows > 0x7fffff00ll || items <= 0 || !work) return TFB_ERR_ARG;
  if ((q_col0 | k_col0 | v_col0) & 7 || (ldo & 7) || (reinterpret_cast<uintptr_t>(o) & 15) || (reinterpret_cast<uintptr_t>(work) & 15) ||
      (long long)items * Hq > 0x3fffffffll)
    return TFB_ERR_ARG;
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_tmap_3d(&tq, q, 2, ldq, rows, 1, ldq * 2, ldq * 2 * rows, 64, 128, 1))) return rc;
  if ((rc = make_tmap_3d(&tk, k, 2, ldk, rows, 1, ldk * 2, ldk * 2 * rows, 64, 128, 1))) return rc;
  if ((rc = make_tmap_3d(&tv, v, 2, ldv, rows, 1, ldv * 2, ldv * 2 * rows, 64, 128, 1))) return rc;
  AttnFwdParams p;
  p.B = 1; p.S = p.Skv = 0; p.q_off = 0; p.Hq = Hq; p.Hkv = Hkv;
  p.scale = scale; p.causal = causal;
  p.q_col0 = q_col0; p.k_col0 = k_col0; p.v_col0 = v_col0;
  p.O = static_cast<__nv_bfloat16*>(o); p.ldo = ldo; p.lse = nullptr; p.work = static_cast<const int4*>(work); p.status = status;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return D == 64 ? launch_attn_fwd<64, true>(tq, tk, tv, p, 2 * items, st) : launch_attn_fwd<128, true>(tq, tk, tv, p, items, st);
}
