// Products of few rows: out[M, N] = act(alpha * x[M, K] . W[N, K]^T + bias) + residual for M <= 128 with W in bf16, M <= 32 with W in the packed
// formats of wq_decode.cuh.  Such a product streams the weights once; everything here serves that stream.
//
//   - Operands swapped: the 128 weight rows of a tile are the M side of tcgen05.mma and the batch (padded to 16, 32, 64 or 128) its
//     N side, so shared memory and tensor time go to weights and not to padding, and the ring holds 110 - 190 KB of weights per SM.
//   - The work is the list of (tile of 128 weight rows, k-block of 64) units, cut into one contiguous run per block: every SM streams
//     the same number of bytes, whatever N and K are.  A tile that several blocks share meets in a workspace: each stores
//     its partial sums, and the block that arrives last adds them in the order of the blocks (the result does not depend on who
//     that is), applies the epilogue and resets the tile's counter.  No block waits for another; no second kernel.
//   - The weights of a model do not change while it serves: with `w_static` their first ring of tiles is fetched before the
//     previous kernel of the stream has ended (programmatic launch), under the norms and the attention between two products.
//   - Packed weights: bulk copies bring the codes into a ring of their own, converter warps (four groups on k-blocks in turn, one
//     weight row per thread) write them as bf16 into tensor memory, which is where the instruction then reads its A operand:
//     no shared-memory image, no proxy fence.
//
// warp 0 loads x, warp 1 issues the MMAs, warp 2 loads the weights, warps 4-7 are the epilogue, warps 8-23 convert packed weights.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <vector>

#include "tfb_host.h"
#include "tfb_ptx.cuh"
#include "wq_decode.cuh"

namespace tfb {

constexpr int RW_BN = 128, RW_BK = 64, RW_W_BYTES = RW_BN * RW_BK * 2, RW_RAW = 128 * 64 + 128 * 2 * 2;
constexpr int RW_MAX_CTAS = 160, RW_MAX_M = 128, RW_MAX_TILES = 8192;

template <int FMT, int MP>
struct RowsPlan {
  static constexpr bool QUANT = FMT >= 0;
  static constexpr int X_BYTES = MP * RW_BK * 2;
  static constexpr int STAGE = X_BYTES + (QUANT ? 0 : RW_W_BYTES);
  // tensor memory: two accumulators of MP columns, then 32 columns of converted weights per stage
  static constexpr int STAGES = QUANT ? 12 : (MP == 16 ? 12 : MP == 32 ? 11 : MP == 64 ? 9 : 6);
  static constexpr int RAW_STAGES = QUANT ? 12 : 0;
  static constexpr int TMEM_COLS = QUANT ? 512 : 2 * MP;
  static constexpr int RAW_OFF = STAGES * STAGE;
  static constexpr int BAR_OFF = RAW_OFF + RAW_STAGES * RW_RAW;
  static constexpr int EX_OFF = BAR_OFF + 512;      // 16 rows of x by 64 "up" columns on their way to the "gate" lanes
  static constexpr int SMEM = EX_OFF + (QUANT ? 0 : 4096) + 1024;
  static constexpr int THREADS = QUANT ? 768 : 256;
  static_assert(2 * MP + (QUANT ? 32 * STAGES : 0) <= 512, "tensor memory");
  static_assert(SMEM <= 232448, "shared memory");
};

struct RowsParams {
  int M, N, K, KB, tiles;   // KB: k-blocks; tiles: tiles of 128 weight rows
  void* C;
  long long ldc;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  long long ldr;
  float alpha;
  int act, out_f32, w_static;
  int glu;                             // > 0: a tile is 64 rows of W and the 64 rows `glu` further on; out = act(first) * second
  const uint8_t* codes;                // packed weights: tile-major codes and scales
  const __nv_bfloat16* scales;
  int group;
  float* ws;                           // [grid][2][MP][128] partial sums
  int* count;                          // [tiles] arrivals, zero between launches
  int* status;
#ifdef TFB_BOUNDS_CHECK
  int give_up;                         // block whose epilogue behaves as if its first wait had run out; -1: none
#endif
};

template <int FMT, int MP>
__global__ void __launch_bounds__(RowsPlan<FMT, MP>::THREADS, 1)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_w, const RowsParams p) {
  using L = RowsPlan<FMT, MP>;
  constexpr bool QUANT = L::QUANT;
  constexpr int S = L::STAGES, R = QUANT ? L::RAW_STAGES : 1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t base = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  const uint32_t bar_full = smem_u32(bars);            // [S] x tile + weights of a k-block are in place
  const uint32_t bar_empty = bar_full + S * 8;         // [S] MMA commit
  const uint32_t bar_tfull = bar_empty + S * 8;        // [2]
  const uint32_t bar_tempty = bar_tfull + 16;          // [2]
  const uint32_t bar_rfull = bar_tempty + 16;          // [R] codes and scales have landed
  const uint32_t bar_rempty = bar_rfull + R * 8;       // [R] ... and are in registers
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * S + 4 + 2 * R);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* last_flag = abort_flag + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = gridDim.x, cta = blockIdx.x;
  const long long U = (long long)p.tiles * p.KB;
  const int u0 = int(cta * U / G), u1 = int((cta + 1) * U / G);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(bar_full + s * 8, QUANT ? 5 : 2);
      mbar_init(bar_empty + s * 8, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_tfull + s * 8, 1);
      mbar_init(bar_tempty + s * 8, 128);
    }
    if (QUANT)
      for (int s = 0; s < R; ++s) {
        mbar_init(bar_rfull + s * 8, 1);
        mbar_init(bar_rempty + s * 8, 4);
      }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tma_x);
    if (!QUANT) tma_prefetch_desc(&tma_w);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), L::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // every warp but the weight loader works on what earlier kernels wrote, or writes what they read
  if (warp != 2) pdl_sync();
  // a role that gave up lets the copies that it has issued land before the block's shared memory goes away
  auto drain = [&]() {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) {}
  };

  // The single-thread roles set the pace of a k-block (a few hundred cycles): no divisions and no descriptor assembly in their
  // loops.
  const int n = u1 - u0, kb_first = u0 % p.KB;
  if (warp == 0) {
    if (lane == 0) {
      int s = 0, kb = kb_first;
      uint32_t ph = 1;
      for (int i = 0; i < n; ++i) {
        if (!mbar_wait(bar_empty + s * 8, ph, abort_flag, p.status, ST_TIMEOUT_EMPTY)) { drain(); break; }
        mbar_expect_tx(bar_full + s * 8, L::X_BYTES);
        tma_load_2d(base + s * L::STAGE, &tma_x, bar_full + s * 8, kb * RW_BK, 0);
        if (++kb == p.KB) kb = 0;
        if (++s == S) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 2) {
    if (lane == 0) {
      if (!p.w_static) pdl_wait();
      const int rows_w = p.glu ? RW_BN / 2 : RW_BN;
      int s = 0, kb = kb_first, row = u0 / p.KB * rows_w;
      uint32_t ph = 1;
      if constexpr (QUANT) {
        constexpr uint32_t code_bytes = 128 * wq_row_bytes(QUANT ? FMT : 0);
        const uint32_t scale_bytes = 128 * (RW_BK / p.group) * 2;
        const uint8_t* cp = p.codes + (long long)u0 * code_bytes;                                       // unit u is blob u
        const uint8_t* sp = reinterpret_cast<const uint8_t*>(p.scales) + (long long)u0 * scale_bytes;
        for (int i = 0; i < n; ++i, cp += code_bytes, sp += scale_bytes) {
          if (!mbar_wait(bar_rempty + s * 8, ph, abort_flag, p.status, ST_TIMEOUT_EMPTY)) { drain(); break; }
          const uint32_t dst = base + L::RAW_OFF + s * RW_RAW, fb = bar_rfull + s * 8;
          mbar_expect_tx(fb, code_bytes + scale_bytes);
          bulk_load(dst, cp, code_bytes, fb);
          bulk_load(dst + 8192, sp, scale_bytes, fb);
          if (++s == R) { s = 0; ph ^= 1; }
        }
      } else {
        for (int i = 0; i < n; ++i) {
          if (!mbar_wait(bar_empty + s * 8, ph, abort_flag, p.status, ST_TIMEOUT_EMPTY)) { drain(); break; }
          mbar_expect_tx(bar_full + s * 8, RW_W_BYTES);
          const uint32_t sw = base + s * L::STAGE + L::X_BYTES;
          tma_load_2d(sw, &tma_w, bar_full + s * 8, kb * RW_BK, row);
          if (p.glu) tma_load_2d(sw + RW_W_BYTES / 2, &tma_w, bar_full + s * 8, kb * RW_BK, p.glu + row);
          if (++kb == p.KB) { kb = 0; row += rows_w; }
          if (++s == S) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc(FMT_BF16, FMT_BF16, false, false, RW_BN, MP);
      const uint64_t xdesc0 = umma_smem_desc(base, 16, 1024), wdesc0 = umma_smem_desc(base + L::X_BYTES, 16, 1024);
      int s = 0, kb = kb_first, ab = 0;
      uint32_t ph = 0, aph = 1;
      bool first = true;
      for (int i = 0; i < n; ++i) {
        if (first && !mbar_wait(bar_tempty + ab * 8, aph, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY)) break;
        if (!mbar_wait(bar_full + s * 8, ph, abort_flag, p.status, ST_TIMEOUT_FULL)) break;
        tc_fence_after();
        const uint32_t d = tmem + ab * MP;
        const uint64_t at = uint64_t(s * (L::STAGE >> 4));         // addresses in a descriptor count 16 bytes
#pragma unroll
        for (int k = 0; k < RW_BK / 16; ++k) {
          const uint64_t xdesc = xdesc0 + at + k * 2;
          if constexpr (QUANT) umma_f16_ts(d, tmem + 2 * MP + s * 32 + k * 8, xdesc, idesc, !first || k > 0);
          else umma_f16_ss(d, wdesc0 + at + k * 2, xdesc, idesc, !first || k > 0);
        }
        umma_commit(bar_empty + s * 8);
        first = ++kb == p.KB || i == n - 1;
        if (first) {
          umma_commit(bar_tfull + ab * 8);
          kb = 0;
          ab ^= 1;
          aph ^= uint32_t(ab == 0);
        }
        if (++s == S) { s = 0; ph ^= 1; }
      }
    }
  } else if (QUANT && warp >= 8) {
    if constexpr (QUANT) {
      // ------------------------------ converters: a whole weight row of a k-block per thread ------------------------------
      const int g = (warp - 8) >> 2, r = (warp & 3) * 32 + lane;
      const uint32_t lane_off = uint32_t((warp & 3) * 32) << 16;
      for (int i = g; i < u1 - u0; i += 4) {
        const int rs = i % R, s = i % S;
        if (!mbar_wait_warp(bar_rfull + rs * 8, (i / R) & 1, abort_flag, p.status, ST_TIMEOUT_FULL)) break;
        const uint32_t raw = base + L::RAW_OFF + rs * RW_RAW;
        uint32_t w0[8], w1[8];
        wq_load_codes<FMT>(raw, r, 0, w0);
        wq_load_codes<FMT>(raw, r, 1, w1);
        uint32_t s0, s1;
        if (p.group == 32) {
          const uint32_t both = ld_shared_u32(raw + 8192 + r * 4);
          s0 = both & 0xffffu;
          s1 = both >> 16;
        } else {
          s0 = s1 = ld_shared_u16(raw + 8192 + r * 2);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_rempty + rs * 8);
        uint32_t o0[16], o1[16];
        wq_convert<FMT>(w0, s0, o0);
        wq_convert<FMT>(w1, s1, o1);
        if (!mbar_wait_warp(bar_empty + s * 8, ((i / S) & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) break;
        tc_fence_after();
        const uint32_t ta = tmem + 2 * MP + s * 32 + lane_off;
        tmem_st_32x16(ta, o0);
        tmem_st_32x16(ta + 16, o1);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_full + s * 8);
      }
    }
  } else if (warp >= 4) {
    // ------------------------------ epilogue: lane = weight row of the tile, columns = rows of x ------------------------------
    const int quad = warp & 3, nl = quad * 32 + lane;
    float* ex = reinterpret_cast<float*>(smem + L::EX_OFF);
    // sixteen rows of x from row c on: the residual's loads are in flight together.  All 128 lanes call it.
    auto finish = [&](const float (&acc)[16], int c, int n, float bias, bool live) {
      if (!QUANT && p.glu) {
        if (nl >= 64) {
#pragma unroll
          for (int j = 0; j < 16; ++j) ex[j * 64 + nl - 64] = acc[j];
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (nl < 64 && live) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c + j < p.M) static_cast<__nv_bfloat16*>(p.C)[(c + j) * p.ldc + n] = __float2bfloat16(apply_act(acc[j], p.act) * ex[j * 64 + nl]);
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        return;
      }
      if (!live) return;
      float v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = fmaf(acc[j], p.alpha, bias);
      if (p.act) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = apply_act(v[j], p.act);
      }
      if (p.residual) {
        __nv_bfloat16 r[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) r[j] = p.residual[min(c + j, p.M - 1) * p.ldr + n];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] += __bfloat162float(r[j]);
      }
      if (p.out_f32) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (c + j < p.M) static_cast<float*>(p.C)[(c + j) * p.ldc + n] = v[j];
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (c + j < p.M) static_cast<__nv_bfloat16*>(p.C)[(c + j) * p.ldc + n] = __float2bfloat16(v[j]);
      }
    };
    bool gave_up = false;
    int seg = 0;
    for (int u = u0; u < u1; ++seg) {
      const int t = u / p.KB, kb0 = u - t * p.KB, end = min(u1, (t + 1) * p.KB), ab = seg & 1;
      const bool whole = kb0 == 0 && end == (t + 1) * p.KB;
      const int n = p.glu ? t * (RW_BN / 2) + (nl & 63) : t * RW_BN + nl;
      const bool live = n < p.N;
      const float bias = p.bias && live ? __bfloat162float(p.bias[n]) : 0.f;
      // A warp whose wait ran out (the status word says so, the block's results are wrong) goes on with what the accumulator holds: the
      // other three meet it at the barriers below, and the block has to arrive at every tile that it shares - the counters outlive the
      // launch, and one left above zero would let a later product add sums that are not there yet.
      gave_up |= !mbar_wait_sleep_warp(bar_tfull + ab * 8, (seg >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL, 20);
#ifdef TFB_BOUNDS_CHECK
      if (cta == p.give_up) {
        gave_up = true;
        *abort_flag = 1;
        report(p.status, ST_TIMEOUT_TMEM_FULL);
      }
#endif
      tc_fence_after();
      // partial sums: [four rows of x][128 weight rows] of four floats
      float4* slot = reinterpret_cast<float4*>(p.ws + ((long long)cta * 2 + (u == u0 ? 0 : 1)) * (MP * 128)) + nl;
#pragma unroll 1
      for (int c = 0; c < MP && c < p.M; c += 16) {
        uint32_t v[16];
        tmem_ld_32x16(tmem + ab * MP + c + (uint32_t(quad * 32) << 16), v);
        tmem_ld_wait();
        float f[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(v[j]);
        if (!whole) {
#pragma unroll
          for (int j = 0; j < 4; ++j) __stcg(slot + (c / 4 + j) * 128, make_float4(f[4 * j], f[4 * j + 1], f[4 * j + 2], f[4 * j + 3]));
        } else {
          finish(f, c, n, bias, live);
        }
      }
      tc_fence_before();
      mbar_arrive(bar_tempty + ab * 8);
      if (!whole) {
        // blocks that share the tile: the ones whose runs hold its first and its last unit, and those in between
        const int c0 = int((((long long)t * p.KB + 1) * G - 1) / U), c1 = int(((long long)(t + 1) * p.KB * G - 1) / U);
        __threadfence();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (nl == 0) {
          const int before = atomicAdd(p.count + t, 1);
          *last_flag = before == c1 - c0;
          if (before == c1 - c0) p.count[t] = 0;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (*last_flag) {
          __threadfence();
          {
            // only the first block can have the tile in its second slot: every later one starts inside the tile
            const long long first = (int(c0 * U / G) / p.KB == t ? 0 : 1);
            const float4* src0 = reinterpret_cast<const float4*>(p.ws) + nl;
            constexpr int CH = MP < 32 ? MP : 32;      // rows per pass: 8 loads of 16 bytes per block in flight, two blocks at a time
#pragma unroll 1
            for (int c = 0; c < p.M; c += CH) {
              float4 v[CH / 4];
              const float4* s = src0 + ((long long)c0 * 2 + first) * (MP * 32) + c / 4 * 128;
#pragma unroll
              for (int j = 0; j < CH / 4; ++j) v[j] = __ldcg(s + j * 128);
              for (int b = c0 + 1; b <= c1; ++b) {
                float4 w[CH / 4];
                s = src0 + (long long)b * 2 * (MP * 32) + c / 4 * 128;
#pragma unroll
                for (int j = 0; j < CH / 4; ++j) w[j] = __ldcg(s + j * 128);
#pragma unroll
                for (int j = 0; j < CH / 4; ++j) {
                  v[j].x += w[j].x;
                  v[j].y += w[j].y;
                  v[j].z += w[j].z;
                  v[j].w += w[j].w;
                }
              }
#pragma unroll
              for (int h = 0; h < CH / 16; ++h) {
                float f[16];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  f[4 * j] = v[4 * h + j].x;
                  f[4 * j + 1] = v[4 * h + j].y;
                  f[4 * j + 2] = v[4 * h + j].z;
                  f[4 * j + 3] = v[4 * h + j].w;
                }
                if (c + h * 16 < p.M) finish(f, c + h * 16, n, bias, live);
              }
            }
          }
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");     // last_flag is read before the next tile writes it
      }
      u = end;
    }
    if (gave_up && lane == 0) drain();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, L::TMEM_COLS);
  }
}

// Partial sums and counters: a workspace belongs to one stream, or to one stream of one capture, so that no two products that may run
// at the same time share any (two graphs on two streams, branches of a graph, threads with streams of their own).  That of a capture is held by
// the graph (a user object) and free for the next owner when graph and executables are gone; that of a stream stays with it, and passes on
// only when the pool is at its bound and the stream has been quiet for RW_QUIET products.  Where none is to be had the general path runs.
// (Two executables made of one graph share its workspace: as for all memory of a graph, they are not to run at the same time.)
constexpr size_t RW_POOL_BYTES = size_t(512) << 20;
constexpr int RW_POOL_SLABS = 64;
constexpr unsigned long long RW_QUIET = 4096;
struct RowsWs {
  float* ws;
  int* count;                         // zero between products
  size_t bytes;                       // of ws
  unsigned long long stream, capture; // owner; capture 0: products issued eagerly
  unsigned long long used;            // number of the last product
  std::atomic<bool> busy;
};
struct RowsPool {
  std::mutex mu;
  std::vector<RowsWs*> slabs[64];     // by device
  size_t bytes[64] = {};
  unsigned long long products = 0;
};
static RowsPool& rows_pool() {
  static RowsPool* p = new RowsPool;  // outlives the graphs that a process still holds at its end
  return *p;
}
static void CUDART_CB rows_give_back(void* slab) { static_cast<RowsWs*>(slab)->busy = false; }      // called by the driver: no CUDA call, no lock
static RowsWs* rows_make(size_t bytes) {
  const size_t cb = RW_MAX_TILES * sizeof(int);
  char* q = nullptr;
  cudaStream_t st = nullptr;
  const bool ok = cudaMalloc(reinterpret_cast<void**>(&q), bytes + cb) == cudaSuccess && cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess &&
                  cudaMemsetAsync(q + bytes, 0, cb, st) == cudaSuccess && cudaStreamSynchronize(st) == cudaSuccess;
  if (st) (void)cudaStreamDestroy(st);
  if (!ok) {
    if (q) (void)cudaFree(q);
    (void)cudaGetLastError();
    return nullptr;
  }
  return new RowsWs{reinterpret_cast<float*>(q), reinterpret_cast<int*>(q + bytes), bytes, 0, 0, 0, false};
}
// The workspace of this stream (of its capture) with room for `need` bytes of partial sums, or null.
static const RowsWs* rows_workspace(cudaStream_t stream, size_t need) {
  int dev = 0;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  unsigned long long cap = 0, sid = 0;
  cudaGraph_t graph = nullptr;
  // nothing here is ordered with the stream or waits for it: allowed while this or another thread captures
  struct Relaxed {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Relaxed() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Relaxed() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
  } relaxed;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 ||
      cudaStreamGetCaptureInfo(stream, &cs, &cap, &graph, nullptr, nullptr) != cudaSuccess || cs == cudaStreamCaptureStatusInvalidated) {
    (void)cudaGetLastError();
    return nullptr;
  }
  // handles are used again for later streams, ids are not; a capturing stream may not be asked for its id, but keeps its handle
  if (cs == cudaStreamCaptureStatusActive) {
    sid = reinterpret_cast<unsigned long long>(stream);
  } else {
    cap = 0;
    if (cudaStreamGetId(stream, &sid) != cudaSuccess) {
      (void)cudaGetLastError();
      return nullptr;
    }
  }
  RowsPool& pool = rows_pool();
  std::lock_guard<std::mutex> lock(pool.mu);
  std::vector<RowsWs*>& all = pool.slabs[dev];
  const unsigned long long now = ++pool.products;
  RowsWs *best = nullptr, *quiet = nullptr;
  for (RowsWs* w : all) {
    if (w->bytes < need) continue;
    if (w->busy && w->stream == sid && w->capture == cap) {
      w->used = now;
      return w;
    }
    if (!w->busy && (!best || w->bytes < best->bytes)) best = w;
    if (w->busy && !w->capture && now - w->used > RW_QUIET && (!quiet || w->used < quiet->used)) quiet = w;
  }
  if (!best && int(all.size()) < RW_POOL_SLABS && pool.bytes[dev] + need <= RW_POOL_BYTES) {
    best = rows_make(need);
    if (best) {
      all.push_back(best);
      pool.bytes[dev] += need;
    }
  }
  if (!best && quiet && !cap) {
    if (cudaDeviceSynchronize() == cudaSuccess) best = quiet;       // what its old owner has launched is done
    else (void)cudaGetLastError();
  }
  if (best) {
    best->stream = sid;
    best->capture = cap;
    best->used = now;
    best->busy = true;
    cudaUserObject_t obj = nullptr;
    if (cap && cudaUserObjectCreate(&obj, best, rows_give_back, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
      best->busy = false;
      best = nullptr;
    } else if (cap && cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove) != cudaSuccess) {
      (void)cudaUserObjectRelease(obj, 1);                           // gives the workspace back
      best = nullptr;
    }
  }
  if (!best) (void)cudaGetLastError();
  return best;
}

#ifdef TFB_BOUNDS_CHECK
static int g_give_up = -1;
#endif

template <int FMT, int MP>
static int launch_rows(const CUtensorMap& tx, const CUtensorMap& tw, const RowsParams& p, int grid, cudaStream_t st) {
  using L = RowsPlan<FMT, MP>;
  static DeviceOnce once;
  auto kern = gemm_rows_kernel<FMT, MP>;
  if (int e = ensure_dyn_smem(once, kern, L::SMEM)) return e;
  launch_k_pdl(kern, grid, L::THREADS, L::SMEM, st, tx, tw, p);
  return int(cudaGetLastError());
}

template <int FMT>
static int launch_rows_m(int M, const CUtensorMap& tx, const CUtensorMap& tw, const RowsParams& p, int grid, cudaStream_t st) {
  if (M <= 16) return launch_rows<FMT, 16>(tx, tw, p, grid, st);
  if (M <= 32) return launch_rows<FMT, 32>(tx, tw, p, grid, st);
  if constexpr (FMT >= 0) return TFB_NOT_TAKEN;      // packed weights: the converters set the pace, more rows only lengthen the drain
  else if (M <= 64) return launch_rows<FMT, 64>(tx, tw, p, grid, st);
  else return launch_rows<FMT, 128>(tx, tw, p, grid, st);
}

static int run_rows(const void* x, long long ldx, const void* W, long long ldw, const void* codes, const void* scales, int fmt, int group, void* C,
                    long long ldc, int M, int N, int K, int Kw, const void* bias, const void* residual, long long ldr, float alpha, int act,
                    int out_f32, int glu, int w_static, int* status, void* stream) {
  if (M <= 0 || M > RW_MAX_M || N <= 0 || K <= 0) return TFB_NOT_TAKEN;
  RowsParams p = {};
  p.M = M; p.N = N; p.K = K;
  p.KB = ((fmt >= 0 ? Kw : K) + RW_BK - 1) / RW_BK;
  const int rows_w = glu ? RW_BN / 2 : RW_BN;      // outputs of a tile
  p.tiles = (N + rows_w - 1) / rows_w;
  p.glu = glu;
  if (p.tiles > RW_MAX_TILES || (long long)p.tiles * p.KB > 0x7fffffffll / RW_MAX_CTAS) return TFB_NOT_TAKEN;
  CUtensorMap tx, tw;
  const int mp = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  if (make_tmap_2d(&tx, x, 2, K, M, ldx * 2, RW_BK, mp)) return TFB_NOT_TAKEN;
  if (fmt < 0 && make_tmap_2d(&tw, W, 2, K, glu ? 2 * N : N, ldw * 2, RW_BK, rows_w)) return TFB_NOT_TAKEN;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int sms = std::min(sm_count(), RW_MAX_CTAS);
  const RowsWs* w = rows_workspace(st, size_t(sms) * 2 * mp * 128 * sizeof(float));
  if (!w) return TFB_NOT_TAKEN;
  p.C = C; p.ldc = ldc;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.ldr = ldr; p.alpha = alpha; p.act = act; p.out_f32 = out_f32; p.w_static = w_static;
  p.codes = static_cast<const uint8_t*>(codes);
  p.scales = static_cast<const __nv_bfloat16*>(scales);
  p.group = group;
  p.ws = w->ws; p.count = w->count; p.status = status;
#ifdef TFB_BOUNDS_CHECK
  p.give_up = g_give_up;
#endif
  // at least four units per block: below that a block's fill, drain and its part in the meeting cost more than the bytes it streams
  const long long units = (long long)p.tiles * p.KB;
  const int grid = int(std::max(1ll, std::min<long long>(sms, units / 4)));
  switch (fmt) {
    case -1: return launch_rows_m<-1>(M, tx, tw, p, grid, st);
    case 0: return launch_rows_m<0>(M, tx, tx, p, grid, st);
    case 1: return launch_rows_m<1>(M, tx, tx, p, grid, st);
    case 2: return launch_rows_m<2>(M, tx, tx, p, grid, st);
    case 3: return launch_rows_m<3>(M, tx, tx, p, grid, st);
    case 4: return launch_rows_m<4>(M, tx, tx, p, grid, st);
    default: return TFB_NOT_TAKEN;
  }
}

int gemm_rows(const void* x, long long ldx, const void* W, long long ldw, const void* codes, const void* scales, int fmt, int group, void* C,
              long long ldc, int M, int N, int K, int Kw, const void* bias, const void* residual, long long ldr, float alpha, int act, int out_f32,
              int w_static, int* status, void* stream) {
  return run_rows(x, ldx, W, ldw, codes, scales, fmt, group, C, ldc, M, N, K, Kw, bias, residual, ldr, alpha, act, out_f32, 0, w_static, status, stream);
}

int gemm_rows_glu(const void* x, long long ldx, const void* W, long long ldw, void* C, long long ldc, int M, int F, int K, int act, int w_static,
                  int* status, void* stream) {
  return run_rows(x, ldx, W, ldw, nullptr, nullptr, -1, 0, C, ldc, M, F, K, K, nullptr, nullptr, 0, 1.f, act, 0, F, w_static, status, stream);
}

}  // namespace tfb

// Workspaces of the current device: 0 all, 1 held by captures and graphs, 2 held by streams, 3 MB allocated.
TFB_API int tfb_rows_workspaces(int what) {
  using namespace tfb;
  int dev = 0, n[3] = {0, 0, 0};
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  RowsPool& pool = rows_pool();
  std::lock_guard<std::mutex> lock(pool.mu);
  for (const RowsWs* w : pool.slabs[dev]) {
    ++n[0];
    if (w->busy) ++n[w->capture ? 1 : 2];
  }
  return what >= 0 && what < 3 ? n[what] : int(pool.bytes[dev] >> 20);
}

#ifdef TFB_BOUNDS_CHECK
// Bounds-check build: the epilogue of block `cta` of every product that follows gives up at its first tile, as if its wait had run out.
TFB_API int tfb_test_rows_give_up(int cta) {
  tfb::g_give_up = cta;
  return 0;
}
#endif

// out [M, N] = act(alpha * x [M, K] . W [N, K]^T + bias) + residual, M <= 128; out bf16, or fp32 with out_f32.  w_static: the caller promises
// that the kernel launched just before this one on the stream does not write W.  (The models' products come through gemm_bf16.cu, which
// chooses; this entry takes the streaming form at every size, for tests and measurements.)
TFB_API int tfb_gemm_rows(const void* x, long long ldx, const void* w, long long ldw, void* out, long long ldo, int M, int N, int K, const void* bias,
                          const void* residual, long long ldr, float alpha, int act, int out_f32, int w_static, int* status, void* stream) {
  const int rc = tfb::gemm_rows(x, ldx, w, ldw, nullptr, nullptr, -1, 0, out, ldo, M, N, K, K, bias, residual, ldr, alpha, act, out_f32, w_static,
                                status, stream);
  return rc == tfb::TFB_NOT_TAKEN ? int(TFB_ERR_ARG) : rc;
}

// The same with packed weights (codes and scales tile-major, N rows padded to a multiple of 128 and Kw >= K entries, a multiple of 64).
TFB_API int tfb_gemm_rows_wq(const void* x, long long ldx, const void* codes, const void* scales, int fmt, int group, void* out, long long ldo, int M,
                             int N, int K, int Kw, const void* bias, const void* residual, long long ldr, int w_static, int* status, void* stream) {
  if (fmt < 0 || fmt > 4 || (group != 32 && group != 64) || Kw % 64 || Kw < K || (reinterpret_cast<uintptr_t>(codes) & 15) ||
      (reinterpret_cast<uintptr_t>(scales) & 15))
    return TFB_ERR_ARG;
  const int rc = tfb::gemm_rows(x, ldx, nullptr, 0, codes, scales, fmt, group, out, ldo, M, N, K, Kw, bias, residual, ldr, 1.f, 0, 0, w_static, status,
                                stream);
  return rc == tfb::TFB_NOT_TAKEN ? int(TFB_ERR_ARG) : rc;
}
