// bf16 GEMM for sm_100a: C[M,N] = epilogue(A * B), fp32 accumulation in tensor memory.
//
// Design (one persistent CTA per SM, 320 threads, warp-specialised):
//   warp 0      TMA producer  : cp.async.bulk.tensor tiles of A and B into a 4-stage shared-memory ring
//   warp 1      MMA issuer    : one thread issues tcgen05.mma (128 x BN x 16) per 32 bytes of K and
//                               commits stage-release / accumulator-ready mbarriers
//   warps 2..9  epilogue      : tcgen05.ld the 128 x BN fp32 accumulator (one row per thread, two warps per TMEM lane
//                               quadrant, each taking half of the columns),
//                               apply alpha / bias / activation / residual, stage 32-row x 128-byte slabs in
//                               shared memory (128-byte swizzle, conflict-free) and hand them to TMA: a tiled
//                               store for bf16 / fp32 outputs, a tiled fp32 reduce-add for accumulating outputs
//                               (weight gradients, split-K).  Ragged edges are clipped by the tensor map.
// The accumulator is double-buffered in TMEM (2 x BN columns), so the epilogue of tile i overlaps
// the main loop of tile i+1.  Either operand may be K-major (reduction dim contiguous) or MN-major
// (output dim contiguous): the forward, data-gradient and weight-gradient GEMMs of a linear layer
// all run without a transpose copy.  Small-output / long-K problems (weight gradients) are split
// along K across CTAs and summed into the fp32 gradient buffer by TMA reduce-add from the staged epilogue.
//
// This replaces the reference's scalar one-thread-per-output kernels
// (src/backend/gpu_compute_cuda.cpp:68 gemm_kernel; src/kernel/kernel_gemm.cpp:26 scalar_gemm_bt).
#include <string.h>

#include <mutex>
#include "tfb_host.h"
#include "tfb_ptx.cuh"

TFB_BOUNDS_DEFINE(gemm_bf16)

namespace tfb {

constexpr int BM = 128;
constexpr int BK = 64;  // 64 bf16 = 128 bytes = one swizzle row
constexpr int STAGES = 4;
constexpr int EPI_WARPS = 8;   // two warps per TMEM lane quadrant, each draining half of the tile's columns
constexpr int GEMM_THREADS = 64 + 32 * EPI_WARPS;

enum : int { TP_AG = 1, TP_RS = 2, TP_WG = 4 };

// Rows of one operand that live as row shards on `world` ranks and are copied into a local buffer in 128-row blocks.
struct GatherSpec {
  int rank, world, rows_per_shard, row_len, epoch, rows;  // rows: rows of the operand that the product touches
  int src_is_full;   // 1: src[r] is rank r's whole gathered buffer (block b at b * 128 * ld); 0: rank r's shard only
  int skip_local;    // 1: this rank's rows are already in place in dst
  int* ready;        // local int[padded rows / 128]: ready[b] >= epoch once block b has landed in dst
  const __nv_bfloat16* const* src;   // [world] base pointers (peer memory)
  __nv_bfloat16* dst;
  long long ld;
};

// C tensor maps of the reduce-scatter form: one per destination rank's staging buffer (peer memory).
constexpr int RS_TMA_MAX_WORLD = 8;
struct PeerMaps {
  CUtensorMap m[RS_TMA_MAX_WORLD];
};

struct GemmParams {
  int M, N, K;
  void* C;
  long long ldc;
  const __nv_bfloat16* bias;      // [N] or null
  const __nv_bfloat16* residual;  // [M, ldr] or null (bf16 output mode only)
  long long ldr;
  float alpha;
  int act;       // 0 none, 1 relu, 2 gelu(tanh), 3 silu, 4 relu squared
  int out_mode;  // 0 bf16 store, 1 fp32 store, 2 fp32 atomic accumulate
  int splits, kb_per_split, tiles_m, tiles_n;
  int raster_gn;   // tile order: groups of raster_gn tile columns; inside a group n runs fastest, then m
  // grouped (mixture-of-experts) modes; expert segments are padded to multiples of 128 rows
  //   1: rows of A / C grouped by expert, B = [E, ...] picked per 128-row tile (forward, data gradient)
  //   2: reduction dimension grouped by expert, C = [E, M, N] (weight gradient of every expert in one launch)
  int group_mode, num_experts;
  const int* expert_of_mtile;   // mode 1: expert of every 128-row tile (-1 = padding, skipped)
  const int* seg_start;         // mode 2: [E + 1] first row of every expert segment
  long long c_expert_stride;    // mode 2: elements between the C matrices of consecutive experts
  // fusion with the collective that precedes / follows the GEMM (see tp_fused.cu); tp_mode is a set of bits:
  //   TP_AG (1): all-gather -> GEMM.  A is the gathered [M, K] buffer in symmetric memory; this rank's rows are in
  //      place, the first `copy_ctas` CTAs of the grid pull the other ranks' rows over NVLink in 128-row blocks
  //      and raise ready[block] = epoch; the TMA producer waits for a block's flag before loading from it.
  //   TP_RS (2): GEMM -> reduce-scatter.  Output rows of shard d are stored straight into rank d's staging buffer
  //      [world, rows_per_shard, N] at slot `rank` (peer stores from the epilogue); remote shards first.
  //   TP_WG (4): weight all-gather -> GEMM (ZeRO-3 / FSDP).  Every rank of the data-parallel group keeps one row
  //      shard of B (128-row blocks) in symmetric memory; the copy CTAs pull all shards (the local one first) into the
  //      local gather buffer B and the TMA producer waits for the flag of every block a B tile touches.  Tiles
  //      (K-major B) or k-blocks (MN-major B) that use the local shard come first.
  //   TP_AG and TP_WG may be combined (column-parallel product of a sharded weight), and so may TP_RS and TP_WG.
  int tp_mode, tp_copy_ctas;
  GatherSpec ag, wg;
  int wg_n_shift, wg_k_shift;   // TP_WG: first n tile / k block of the local shard
  int rs_rank, rs_world, rs_rows_per_shard;
  __nv_bfloat16* const* rs_peer_c;
  int glu;       // pair form: > 0: the first CTA's 128 columns of B are rows n of W, the second's rows glu + n; C = act(first) * second
  int c_tma;     // 1: the epilogue goes through shared memory and the C tensor map (aligned, dense C)
  int* status;
};

// Decodes work item w into tile coordinates / k-block range / expert.  Returns false when there is nothing to do.
struct WorkItem {
  int m0, n0, kb0, kb1, expert;  // n0 is the tile index along N (the kernel scales it by its BN)
};
__device__ __forceinline__ bool decode_work(const GemmParams& p, int w, int total_kb, WorkItem& it) {
  if (p.group_mode == 2) {
    const int tiles = p.tiles_m * p.tiles_n;
    it.expert = w / tiles;
    const int tile = w - it.expert * tiles;
    it.m0 = (tile / p.tiles_n) * BM;
    it.kb0 = p.seg_start[it.expert] / BK;
    it.kb1 = p.seg_start[it.expert + 1] / BK;
    it.n0 = tile % p.tiles_n;
    return it.kb1 > it.kb0;
  }
  const int tile = w / p.splits, split = w - tile * p.splits;
  // Grouped raster.  A wave of 148 tiles in plain row-major order spans every tile column, i.e. reads all of B once per
  // wave; with a wide N (B larger than L2) that is one DRAM pass over B per wave.  In groups of raster_gn columns a wave
  // covers a roughly square patch, the group's slice of B stays in L2 for the whole sweep over M, and A is streamed once
  // per group.  raster_gn == tiles_n is the plain row-major order, raster_gn == 1 column-major.
  const int per_group = p.raster_gn * p.tiles_m;
  const int grp = tile / per_group, within = tile - grp * per_group;
  const int gn = min(p.raster_gn, p.tiles_n - grp * p.raster_gn);
  const int m_idx = within / gn, n_idx = grp * p.raster_gn + (within - m_idx * gn);
  it.m0 = m_idx * BM;
  it.n0 = n_idx;
  it.kb0 = split * p.kb_per_split;
  it.kb1 = min(total_kb, it.kb0 + p.kb_per_split);
  it.expert = 0;
  if (p.group_mode == 1) {
    it.expert = p.expert_of_mtile[m_idx];
    if (it.expert < 0) return false;
    TFB_BOUNDS(it.expert < p.num_experts, 12, it.expert, p.num_experts);
    if (it.expert >= p.num_experts) return false;
  }
  if ((p.tp_mode & TP_WG) && p.wg_n_shift >= 0) {
    // K-major gathered B: the column groups are visited starting at the local shard's columns, in the order in which
    // the copy CTAs deliver the peers' rows
    it.n0 = (n_idx + p.wg_n_shift) % p.tiles_n;
  }
  if (p.tp_mode & TP_AG) {
    // rotate the row-block order: start with the local shard (already in place)
    it.m0 = ((it.m0 / BM + p.ag.rank * (p.ag.rows_per_shard / BM)) % p.tiles_m) * BM;
  } else if (p.tp_mode & TP_RS) {
    // ... and for the reduce-scatter end with it: remote shards are stored first
    it.m0 = ((it.m0 / BM + (p.rs_rank + 1) * (p.rs_rows_per_shard / BM)) % p.tiles_m) * BM;
  }
  return true;
}

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Copy role of the gather -> GEMM fusions: pulls 128-row blocks of the ranks' shards into the local gathered buffer
// and publishes each block with a release store.  Contiguous blocks (row pitch == row length) travel as untiled bulk
// copies through a shared-memory ring driven by one thread: 16 KB chunks in the CTA's operand-stage memory (8 slots for
// the 128-wide tile configuration, 12 for the 256-wide one), all but two slots' worth of loads in flight, so that about
// a dozen CTAs keep more than a megabyte in flight, which is what a ~2 us NVLink round trip needs to run near link
// bandwidth.  Strided rows fall back to per-thread 16-byte copies.
constexpr int COPY_CHUNK = 16384;
constexpr int COPY_MAX_SLOTS = 12;

__device__ __forceinline__ bool copy_block_bulk(const __nv_bfloat16* src, __nv_bfloat16* dst, long long bytes, uint32_t ring,
                                                uint32_t bars, uint32_t& seq, volatile int* abort_flag, int* status,
                                                const uint32_t COPY_SLOTS) {
  const int nt = int((bytes + COPY_CHUNK - 1) / COPY_CHUNK);
  const char* s8 = reinterpret_cast<const char*>(src);
  char* d8 = reinterpret_cast<char*>(dst);
  int nl = 0, ns = 0;
  const uint32_t seq0 = seq;
  while (ns < nt) {
    while (nl < nt && nl - ns < int(COPY_SLOTS) - 2) {
      tma_store_wait_read<2>();   // at most two stores still reading: the one that last used this slot is not among them
      const uint32_t q = seq0 + nl, slot = q % COPY_SLOTS;
      const uint32_t sz = uint32_t(min((long long)COPY_CHUNK, bytes - (long long)nl * COPY_CHUNK));
      mbar_expect_tx(bars + slot * 8, sz);
      bulk_load(ring + slot * COPY_CHUNK, s8 + (long long)nl * COPY_CHUNK, sz, bars + slot * 8);
      ++nl;
    }
    const uint32_t q = seq0 + ns, slot = q % COPY_SLOTS, parity = (q / COPY_SLOTS) & 1u;
    if (!mbar_wait(bars + slot * 8, parity, abort_flag, status, ST_TIMEOUT_FULL)) {
      // give the loads already issued a bounded time to land before shared memory goes away
      const uint64_t t0 = globaltimer_ns();
      for (int j = ns; j < nl; ++j) {
        const uint32_t qq = seq0 + j;
        while (!mbar_try_wait(bars + (qq % COPY_SLOTS) * 8, (qq / COPY_SLOTS) & 1u)) {
          if (globaltimer_ns() - t0 > 2000000ull) { report(status, ST_TIMEOUT_DRAIN); break; }
        }
      }
      tma_store_wait<0>();
      return false;
    }
    fence_proxy_async_smem();
    const uint32_t sz = uint32_t(min((long long)COPY_CHUNK, bytes - (long long)ns * COPY_CHUNK));
    bulk_store(d8 + (long long)ns * COPY_CHUNK, ring + slot * COPY_CHUNK, sz);
    tma_store_commit();
    ++ns;
  }
  seq = seq0 + nt;
  tma_store_wait<0>();       // the block is in the gathered buffer
  fence_proxy_async_all();   // bulk-copy writes before the flag that publishes them
  return true;
}

__device__ __forceinline__ void copy_block_threads(const __nv_bfloat16* src, __nv_bfloat16* dst, long long ld, long long row_chunks,
                                                   int rows) {
  const long long total = (long long)rows * row_chunks;
  for (long long c = threadIdx.x; c < total; c += 4 * blockDim.x) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long cc = c + (long long)u * blockDim.x;
      if (cc < total) {
        const long long r = cc / row_chunks, k = cc % row_chunks;
        v[u] = *reinterpret_cast<const uint4*>(src + r * ld + k * 8);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long cc = c + (long long)u * blockDim.x;
      if (cc < total) {
        const long long r = cc / row_chunks, k = cc % row_chunks;
        *reinterpret_cast<uint4*>(dst + r * ld + k * 8) = v[u];
      }
    }
  }
}

__device__ __forceinline__ void tp_copy_role(const GemmParams& p, int cta, int ncopy, uint32_t ring, uint32_t bars,
                                             volatile int* abort_flag, const uint32_t slots) {
  if (threadIdx.x == 0) {
    for (uint32_t i = 0; i < slots; ++i) mbar_init(bars + i * 8, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  const int nA = (p.tp_mode & TP_AG) ? (p.ag.world - 1) * (p.ag.rows_per_shard / BM) : 0;
  const int nB = (p.tp_mode & TP_WG) ? (p.wg.world - (p.wg.skip_local ? 1 : 0)) * (p.wg.rows_per_shard / BM) : 0;
  uint32_t seq = 0;
  for (int idx = cta; idx < nA + nB; idx += ncopy) {
    const GatherSpec& g = idx < nA ? p.ag : p.wg;
    const int j = idx < nA ? idx : idx - nA;
    const int bps = g.rows_per_shard / BM;
    const int peer = (g.rank + (g.skip_local ? 1 : 0) + j / bps) % g.world;
    const int b = j % bps, blk = peer * bps + b;  // block inside the shard / inside the gathered operand
    if (blk * BM >= g.rows) continue;             // padding rows: nothing reads them
    TFB_BOUNDS(peer >= 0 && peer < g.world && blk >= 0, 11, blk, g.world * bps);
    const __nv_bfloat16* src = g.src[peer] + (long long)(g.src_is_full ? blk : b) * BM * g.ld;
    __nv_bfloat16* dst = g.dst + (long long)blk * BM * g.ld;
    if (g.ld == g.row_len) {
      // after a copy that ran out of time nothing more is published: the consumers' own bounded waits end the kernel
      if (threadIdx.x == 0 && !*abort_flag &&
          copy_block_bulk(src, dst, (long long)BM * g.row_len * 2, ring, bars, seq, abort_flag, p.status, slots)) {
        __threadfence();
        asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(g.ready + blk), "r"(g.epoch) : "memory");
      }
    } else {
      copy_block_threads(src, dst, g.ld, (long long)g.row_len / 8, BM);
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(g.ready + blk), "r"(g.epoch) : "memory");
      }
    }
  }
}

template <int BN>
struct SmemLayout {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STG_OFF = STAGES * STAGE_BYTES;   // epilogue staging slabs follow the operand stages
  // epilogue staging: one 32-row x 128-byte slab per epilogue warp, double-buffered where shared memory allows (the
  // 256-wide tile leaves room for one slab per warp next to its four operand stages)
  static constexpr int STG_BUFS = (BN == 256) ? 1 : 2;
  static constexpr int STG_BYTES = EPI_WARPS * STG_BUFS * 4096;
  static constexpr int BAR_OFF = STG_OFF + STG_BYTES;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;  // + barriers + alignment slack
};

// One 32-row strip of a tile, the columns of half `half`: tensor memory -> registers (alpha, bias, activation, residual) -> swizzled
// shared-memory slab of 32 rows x 128 bytes -> TMA store or fp32 reduce-add.  Executed by a whole warp.
template <int BN, int STG_BUFS>
__device__ __forceinline__ void staged_epilogue(const GemmParams& p, const CUtensorMap& tma_c, const PeerMaps& tma_peers, uint32_t taddr0, int n0,
                                                int slab_row0, int half, int lane, uint32_t stg_u32, int& sbuf, int cz) {
  const bool vec_ok_res = p.residual && ((p.ldr & 7) == 0) && ((reinterpret_cast<uintptr_t>(p.residual) & 15) == 0);
  // ---- staged epilogue: registers -> swizzled shared-memory slab -> TMA store / reduce-add ----
  const int row = slab_row0 + lane;
  const bool slab_live = slab_row0 < p.M;            // warp-uniform
  const uint32_t xr = uint32_t(lane & 7);
  if (p.out_mode == 0) {
#pragma unroll 1
    for (int c = half * (BN / 128); c < (half + 1) * (BN / 128); ++c) {
      const int col0 = n0 + c * 64;
      if (col0 >= p.N) break;
      uint32_t r0[32], r1[32];
      tmem_ld_32x32(taddr0 + c * 64, r0);
      tmem_ld_32x32(taddr0 + c * 64 + 32, r1);
      tmem_ld_wait();
      if (!slab_live) continue;
      float v[64];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        v[j] = __uint_as_float(r0[j]) * p.alpha;
        v[32 + j] = __uint_as_float(r1[j]) * p.alpha;
      }
      if (p.bias) {
#pragma unroll
        for (int j = 0; j < 64; ++j)
          if (col0 + j < p.N) v[j] += __bfloat162float(p.bias[col0 + j]);
      }
      if (p.act) {
#pragma unroll
        for (int j = 0; j < 64; ++j) v[j] = apply_act(v[j], p.act);
      }
      if (p.residual && row < p.M) {
        const __nv_bfloat16* rp = p.residual + (long long)row * p.ldr + col0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          if (vec_ok_res && col0 + q * 8 + 8 <= p.N) {
            const uint4 u = *reinterpret_cast<const uint4*>(rp + q * 8);
            const uint32_t uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const float2 f = unpack_bf16(uu[h]);
              v[q * 8 + h * 2] += f.x;
              v[q * 8 + h * 2 + 1] += f.y;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (col0 + q * 8 + j < p.N) v[q * 8 + j] += __bfloat162float(rp[q * 8 + j]);
          }
        }
      }
      if (lane == 0) tma_store_wait_read<STG_BUFS - 1>();   // the slab about to be rewritten has been read by its copy
      __syncwarp();
      const uint32_t slab = stg_u32 + sbuf * 4096 + lane * 128;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        st_shared_v4(slab + ((uint32_t(q) ^ xr) << 4), pack_bf16(v[q * 8 + 0], v[q * 8 + 1]), pack_bf16(v[q * 8 + 2], v[q * 8 + 3]),
                     pack_bf16(v[q * 8 + 4], v[q * 8 + 5]), pack_bf16(v[q * 8 + 6], v[q * 8 + 7]));
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (p.tp_mode & TP_RS) {
          // rows of shard d go to rank d's staging buffer, slot `rank`: one 32-row x 128-byte slab per copy, so the
          // bytes cross NVLink in whole lines (tile rows never straddle two shards: shards are multiples of 128 rows)
          const int d = slab_row0 / p.rs_rows_per_shard;
          tma_store_3d(&tma_peers.m[d], stg_u32 + sbuf * 4096, col0,
                       p.rs_rank * p.rs_rows_per_shard + (slab_row0 - d * p.rs_rows_per_shard), 0);
        } else {
          tma_store_3d(&tma_c, stg_u32 + sbuf * 4096, col0, slab_row0, 0);
        }
        tma_store_commit();
      }
      sbuf ^= (STG_BUFS - 1);
    }
  } else {
#pragma unroll 1
    for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
      const int col0 = n0 + c * 32;
      if (col0 >= p.N) break;
      uint32_t r[32];
      tmem_ld_32x32(taddr0 + c * 32, r);
      tmem_ld_wait();
      if (!slab_live) continue;
      if (lane == 0) tma_store_wait_read<STG_BUFS - 1>();
      __syncwarp();
      const uint32_t slab = stg_u32 + sbuf * 4096 + lane * 128;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        st_shared_v4(slab + ((uint32_t(q) ^ xr) << 4), __float_as_uint(__uint_as_float(r[q * 4]) * p.alpha),
                     __float_as_uint(__uint_as_float(r[q * 4 + 1]) * p.alpha), __float_as_uint(__uint_as_float(r[q * 4 + 2]) * p.alpha),
                     __float_as_uint(__uint_as_float(r[q * 4 + 3]) * p.alpha));
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (p.out_mode == 2) tma_reduce_add_3d(&tma_c, stg_u32 + sbuf * 4096, col0, slab_row0, cz);
        else tma_store_3d(&tma_c, stg_u32 + sbuf * 4096, col0, slab_row0, cz);
        tma_store_commit();
      }
      sbuf ^= (STG_BUFS - 1);
    }
  }
}

// The gated form on CTA pairs: columns 0..127 of the accumulator are "gate", 128..255 "up" of the same 128 outputs.  A warp takes 64 of them.
__device__ __forceinline__ void glu_epilogue(const GemmParams& p, const CUtensorMap& tma_c, uint32_t taddr0, int n0, int slab_row0, int half, int lane,
                                             uint32_t slab0) {
  const int col0 = n0 + half * 64;
  const bool store = slab_row0 < p.M && col0 < p.N;      // warp-uniform
  if (lane == 0) tma_store_wait_read<0>();               // the slab has been read by its last copy
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t g[32], u[32];
    tmem_ld_32x32(taddr0 + half * 64 + c * 32, g);
    tmem_ld_32x32(taddr0 + 128 + half * 64 + c * 32, u);
    tmem_ld_wait();
    uint32_t o[16];
#pragma unroll
    for (int j = 0; j < 16; ++j)
      o[j] = pack_bf16(apply_act(__uint_as_float(g[2 * j]), p.act) * __uint_as_float(u[2 * j]),
                       apply_act(__uint_as_float(g[2 * j + 1]), p.act) * __uint_as_float(u[2 * j + 1]));
#pragma unroll
    for (int q = 0; q < 4; ++q)
      st_shared_v4(slab0 + lane * 128 + ((uint32_t(c * 4 + q) ^ uint32_t(lane & 7)) << 4), o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
  }
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0 && store) {
    tma_store_3d(&tma_c, slab0, col0, slab_row0, 0);
    tma_store_commit();
  }
}

template <bool A_MN, bool B_MN, int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                 const __grid_constant__ CUtensorMap tma_c, const __grid_constant__ PeerMaps tma_peers, const GemmParams p) {
  using L = SmemLayout<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t smem_base = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  // bars[0..S) full, [S..2S) empty, [2S..2S+2) tmem_full, [2S+2..2S+4) tmem_empty
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = bar_full + STAGES * 8;
  const uint32_t bar_tfull = bar_empty + STAGES * 8;
  const uint32_t bar_tempty = bar_tfull + 2 * 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  constexpr uint32_t TMEM_COLS = 2 * BN;
  // copy CTAs take the lowest block indices so that they are scheduled first: a GEMM CTA may wait for a copy
  // CTA, never the other way round
  const int ncopy = (p.tp_mode & (TP_AG | TP_WG)) ? p.tp_copy_ctas : 0;
  const int nctas = int(gridDim.x) - ncopy;  // CTAs that run GEMM tiles
  const int cta = int(blockIdx.x) - ncopy;
  if (cta < 0) {
    tfb::pdl_sync();
    constexpr uint32_t kSlots = (STAGES * L::STAGE_BYTES / COPY_CHUNK) < COPY_MAX_SLOTS ? (STAGES * L::STAGE_BYTES / COPY_CHUNK)
                                                                                          : COPY_MAX_SLOTS;
    tp_copy_role(p, int(blockIdx.x), ncopy, smem_base, bar_full, abort_flag, kSlots);
    return;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar_full + s * 8, 1);
      mbar_init(bar_empty + s * 8, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_tfull + b * 8, 1);
      mbar_init(bar_tempty + b * 8, 32 * EPI_WARPS);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
    if (p.c_tma) tma_prefetch_desc(&tma_c);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  tfb::pdl_sync();   // set-up above touches no global memory; operands written by the previous kernel are read below

  const int total_kb = (p.K + BK - 1) / BK;
  const int num_work = p.tiles_m * p.tiles_n * (p.group_mode == 2 ? p.num_experts : p.splits);

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int w = cta; w < num_work && ok; w += nctas) {
        WorkItem it;
        if (!decode_work(p, w, total_kb, it)) continue;
        const int m0 = it.m0, n0 = it.n0 * BN, kb0 = it.kb0, kb1 = it.kb1;
        const int bz = p.group_mode == 1 ? it.expert : 0;
        auto wait_block = [&](const GatherSpec& g, int blk) -> bool {   // block `blk` of a gathered operand has landed locally
          if (g.skip_local && blk / (g.rows_per_shard / BM) == g.rank) return true;
          const uint64_t t0 = globaltimer_ns();
          uint32_t spins = 0;
          while (ld_acquire_gpu(g.ready + blk) < g.epoch) {
            if ((++spins & 255u) == 0u && (*abort_flag || globaltimer_ns() - t0 > TFB_WAIT_NS)) {
              report(p.status, ST_TIMEOUT_FLAG);
              *abort_flag = 1;
              return false;
            }
          }
          asm volatile("fence.proxy.async;" ::: "memory");  // the copy CTAs' writes -> visible to the TMA reads below
          return true;
        };
        if (p.tp_mode & TP_AG) {
          if (!wait_block(p.ag, m0 / BM)) { ok = false; break; }
        }
        if ((p.tp_mode & TP_WG) && !B_MN) {
          for (int r0 = n0; r0 < n0 + BN && r0 < p.N && ok; r0 += BM) ok = wait_block(p.wg, r0 / BM);
          if (!ok) break;
        }
        int last_blk = -1;
        for (int kb = kb0; kb < kb1; ++kb) {
          const int kbr = ((p.tp_mode & TP_WG) && B_MN) ? (kb + p.wg_k_shift) % total_kb : kb;   // local shard's rows first
          if ((p.tp_mode & TP_WG) && B_MN) {
            const int blk = kbr * BK / BM;
            if (blk != last_blk) {
              if (!wait_block(p.wg, blk)) { ok = false; break; }
              last_blk = blk;
            }
          }
          if (!mbar_wait(bar_empty + stage * 8, phase ^ 1, abort_flag, p.status, ST_TIMEOUT_EMPTY)) {
            ok = false;
            break;
          }
          const uint32_t fb = bar_full + stage * 8;
          mbar_expect_tx(fb, L::STAGE_BYTES);
          const uint32_t sa = smem_base + stage * L::STAGE_BYTES;
          const uint32_t sb = sa + L::A_BYTES;
          const int k0 = kbr * BK;
          if constexpr (!A_MN) {
            tma_load_2d(sa, &tma_a, fb, k0, m0);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d(sa + j * 8192, &tma_a, fb, m0 + j * 64, k0);
          }
          if constexpr (!B_MN) {
            tma_load_3d(sb, &tma_b, fb, k0, n0, bz);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) tma_load_3d(sb + j * 8192, &tma_b, fb, n0 + j * 64, k0, bz);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        // Unwinding: give copies already issued a bounded time to land before shared memory goes away.
        const uint64_t t0 = globaltimer_ns();
        for (int s = 0; s < STAGES; ++s) {
          const uint32_t par = (s < stage) ? phase : (phase ^ 1);
          while (!mbar_try_wait(bar_full + s * 8, par)) {
            if (globaltimer_ns() - t0 > 2000000ull) { report(p.status, ST_TIMEOUT_DRAIN); break; }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc(FMT_BF16, FMT_BF16, A_MN, B_MN, BM, BN);
      // One thread feeds the tensor core an instruction per 64 - 128 cycles: descriptors are a base plus the stage's offset (their
      // addresses count 16 bytes), and a plain product (every item the whole of K) decodes nothing.
      const uint32_t adesc0 = umma_desc_lo(smem_base, A_MN ? 8192 : 16), bdesc0 = umma_desc_lo(smem_base + L::A_BYTES, B_MN ? 8192 : 16);
      constexpr uint32_t ASTEP = A_MN ? 2048 >> 4 : 32 >> 4, BSTEP = B_MN ? 2048 >> 4 : 32 >> 4;
      const bool plain = p.group_mode == 0 && p.splits == 1;
      int stage = 0;
      uint32_t phase = 0;
      int abuf = 0;
      uint32_t aphase = 0;
      bool ok = true;
      for (int w = cta; w < num_work && ok; w += nctas) {
        int n_kb = total_kb;
        if (!plain) {
          WorkItem it;
          if (!decode_work(p, w, total_kb, it)) continue;
          n_kb = it.kb1 - it.kb0;
        }
        if (!mbar_wait(bar_tempty + abuf * 8, aphase ^ 1, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + abuf * BN;
        for (int kb = 0; kb < n_kb; ++kb) {
          if (!mbar_wait(bar_full + stage * 8, phase, abort_flag, p.status, ST_TIMEOUT_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t at = uint32_t(stage) * (L::STAGE_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_f16_ss_lo(tmem_d, adesc0 + at + k * ASTEP, bdesc0 + at + k * BSTEP, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit(bar_empty + stage * 8);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(bar_tfull + abuf * 8);
        abuf ^= 1;
        if (abuf == 0) aphase ^= 1;
      }
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    const int quad = warp & 3;  // TMEM lane quadrant this warp may read
    int abuf = 0;
    uint32_t aphase = 0;
    const bool vec_ok_bf16 = ((p.ldc & 7) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0);
    const bool vec_ok_f32 = ((p.ldc & 3) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0);
    const bool vec_ok_res =
        p.residual && ((p.ldr & 7) == 0) && ((reinterpret_cast<uintptr_t>(p.residual) & 15) == 0);
    const int ew = warp - 2;           // epilogue warp 0..7
    const int half = ew >> 2;          // which half of the tile's columns this warp drains
    const uint32_t stg_u32 = smem_base + L::STG_OFF + ew * (L::STG_BUFS * 4096);
    int sbuf = 0;
    for (int w = cta; w < num_work; w += nctas) {
      WorkItem it;
      if (!decode_work(p, w, total_kb, it)) continue;
      const int m0 = it.m0, n0 = it.n0 * BN;
      const long long c_off = p.group_mode == 2 ? (long long)it.expert * p.c_expert_stride : 0;
      if (!mbar_wait_warp(bar_tfull + abuf * 8, aphase, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) break;
      tc_fence_after();
      const int row = m0 + quad * 32 + lane;
      const uint32_t taddr0 = tmem_base + abuf * BN + (uint32_t(quad * 32) << 16);
      if (p.c_tma) {
        staged_epilogue<BN, L::STG_BUFS>(p, tma_c, tma_peers, taddr0, n0, m0 + quad * 32, half, lane, stg_u32, sbuf,
                                         p.group_mode == 2 ? it.expert : 0);
        tc_fence_before();
        mbar_arrive(bar_tempty + abuf * 8);
        abuf ^= 1;
        if (abuf == 0) aphase ^= 1;
        continue;
      }
#pragma unroll 1
      for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
        uint32_t r[32];
        tmem_ld_32x32(taddr0 + c * 32, r);
        tmem_ld_wait();
        const int col0 = n0 + c * 32;
        if (row >= p.M || col0 >= p.N) continue;
        const bool full = col0 + 32 <= p.N;
        if (p.out_mode == 0) {
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]) * p.alpha;
          if (p.bias) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (full || col0 + j < p.N) v[j] += __bfloat162float(p.bias[col0 + j]);
          }
          if (p.act) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = apply_act(v[j], p.act);
          }
          if (p.residual) {
            const __nv_bfloat16* rp = p.residual + (long long)row * p.ldr + col0;
            if (full && vec_ok_res) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint4 u = *reinterpret_cast<const uint4*>(rp + q * 8);
                const uint32_t uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                  const float2 f = unpack_bf16(uu[h]);
                  v[q * 8 + h * 2] += f.x;
                  v[q * 8 + h * 2 + 1] += f.y;
                }
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j < p.N) v[j] += __bfloat162float(rp[j]);
            }
          }
          __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)row * p.ldc + col0;
          if (p.tp_mode & TP_RS) {  // row belongs to shard d: store into rank d's staging slot for this rank
            const int d = row / p.rs_rows_per_shard;
            cp = p.rs_peer_c[d] + ((long long)p.rs_rank * p.rs_rows_per_shard + (row - d * p.rs_rows_per_shard)) * p.ldc + col0;
          }
          if (full && vec_ok_bf16) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint4 u;
              u.x = pack_bf16(v[q * 8 + 0], v[q * 8 + 1]);
              u.y = pack_bf16(v[q * 8 + 2], v[q * 8 + 3]);
              u.z = pack_bf16(v[q * 8 + 4], v[q * 8 + 5]);
              u.w = pack_bf16(v[q * 8 + 6], v[q * 8 + 7]);
              *reinterpret_cast<uint4*>(cp + q * 8) = u;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (col0 + j < p.N) cp[j] = __float2bfloat16(v[j]);
          }
        } else {
          float* cp = reinterpret_cast<float*>(p.C) + c_off + (long long)row * p.ldc + col0;
          if (p.out_mode == 1) {
            if (full && vec_ok_f32) {
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                float4 f = make_float4(__uint_as_float(r[q * 4]) * p.alpha, __uint_as_float(r[q * 4 + 1]) * p.alpha,
                                       __uint_as_float(r[q * 4 + 2]) * p.alpha, __uint_as_float(r[q * 4 + 3]) * p.alpha);
                *reinterpret_cast<float4*>(cp + q * 4) = f;
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j < p.N) cp[j] = __uint_as_float(r[j]) * p.alpha;
            }
          } else {
            if (full && vec_ok_f32) {
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(cp + q * 4),
                             "f"(__uint_as_float(r[q * 4]) * p.alpha), "f"(__uint_as_float(r[q * 4 + 1]) * p.alpha),
                             "f"(__uint_as_float(r[q * 4 + 2]) * p.alpha), "f"(__uint_as_float(r[q * 4 + 3]) * p.alpha)
                             : "memory");
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j < p.N) atomicAdd(cp + j, __uint_as_float(r[j]) * p.alpha);
            }
          }
        }
      }
      tc_fence_before();
      mbar_arrive(bar_tempty + abuf * 8);
      abuf ^= 1;
      if (abuf == 0) aphase ^= 1;
    }
    if (p.c_tma && lane == 0) tma_store_wait<0>();   // staged slabs must be out of shared memory before the CTA ends
  }

  // ------------------------------ teardown ------------------------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// The same product on CTA pairs: a cluster of two CTAs owns a 256 x 256 tile, each holds 128 rows of A, 128 of the 256 columns of B and its
// 128 rows of the accumulator, and one thread of the first CTA issues tcgen05.mma.cta_group::2 over both.  A k-block brings 32 KB
// into each SM instead of the 48 KB of a 128 x 256 tile, so that six of them fit in flight where four did: with short K (tiles of
// eight k-blocks) the single-CTA form waits for its loads behind the stores of the tile before.  (Measured there: without its
// stores 65536 x 2816 x 512 took 129 us instead of 166, with three stages and two staging slabs per warp 186.)
//   us, single-CTA -> pair: 65536 x 2816 x 512 nt 169 -> 152, 65536 x 512 x 1408 82 -> 72, 9472 x 32000 x 512 279 -> 250, 65536 x 512 x 2816 nn
//   143 -> 125, weight gradients 2816 x 512 x 65536 152 -> 129, 32000 x 512 x 9472 270 -> 227, 28672 x 4096 x 4096 893 -> 716, 5000 x 28672 x
//   4096 nt 876 -> 798 (1472 TFLOP/s).  Five stages with two slabs per warp are 2 - 5 % slower than six with one.
struct PairSmem {
  static constexpr int A_BYTES = BM * BK * 2, STAGE_BYTES = 2 * A_BYTES;
  static constexpr int STG_BUFS = 1, STG_BYTES = EPI_WARPS * STG_BUFS * 4096;
  static constexpr int STAGES = 6;
  static constexpr int STG_OFF = STAGES * STAGE_BYTES, BAR_OFF = STG_OFF + STG_BYTES;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

template <bool A_MN, bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const __grid_constant__ CUtensorMap tma_c,
                 const __grid_constant__ PeerMaps tma_peers, const GemmParams p) {
  using L = PairSmem;
  constexpr int BN = 256, ST = L::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t smem_base = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BAR_OFF);
  const uint32_t bar_full = smem_u32(bars);          // first CTA's: both CTAs' tiles of a k-block have landed
  const uint32_t bar_empty = bar_full + ST * 8;      // each CTA's: the instruction has read them
  const uint32_t bar_tfull = bar_empty + ST * 8;     // each CTA's: accumulator ready
  const uint32_t bar_tempty = bar_tfull + 2 * 8;     // first CTA's: drained by the epilogue warps of both
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * ST + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int npairs = int(gridDim.x) >> 1, pair = int(blockIdx.x) >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(bar_full + s * 8, 1);
      mbar_init(bar_empty + s * 8, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_tfull + b * 8, 1);
      mbar_init(bar_tempty + b * 8, 2 * EPI_WARPS);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
    tma_prefetch_desc(&tma_c);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), 2 * BN);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();      // the other CTA's barriers are set up
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  tfb::pdl_sync();

  const int total_kb = (p.K + BK - 1) / BK;
  const int num_work = p.tiles_m * p.tiles_n * p.splits;
  // work item -> tile (grouped raster, see decode_work) and k-blocks
  auto decode = [&](int w, int& m0, int& n0, int& kb0, int& kb1) {
    const int tile = w / p.splits, split = w - tile * p.splits;
    const int per_group = p.raster_gn * p.tiles_m;
    const int grp = tile / per_group, within = tile - grp * per_group;
    const int gn = min(p.raster_gn, p.tiles_n - grp * p.raster_gn);
    const int mi = within / gn;
    m0 = mi * (2 * BM) + int(rank) * BM;
    n0 = (grp * p.raster_gn + (within - mi * gn)) * (p.glu ? BN / 2 : BN);
    kb0 = split * p.kb_per_split;
    kb1 = min(total_kb, kb0 + p.kb_per_split);
  };

  if (warp == 0) {
    if (lane == 0) {
      const uint32_t full0 = map_cta(bar_full, 0);
      int stage = 0;
      uint32_t phase = 1;
      bool ok = true;
      for (int w = pair; w < num_work && ok; w += npairs) {
        int m0, n0, kb0, kb1;
        decode(w, m0, n0, kb0, kb1);
        const int nb = n0 + int(rank) * (p.glu ? p.glu : BM);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(bar_empty + stage * 8, phase, abort_flag, p.status, ST_TIMEOUT_EMPTY)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(bar_full + stage * 8, 2 * L::STAGE_BYTES);
          const uint32_t fb = full0 + stage * 8, sa = smem_base + stage * L::STAGE_BYTES, sb = sa + L::A_BYTES;
          const int k0 = kb * BK;
          if constexpr (!A_MN) {
            tma_load_2d_pair(sa, &tma_a, fb, k0, m0);
          } else {
            tma_load_2d_pair(sa, &tma_a, fb, m0, k0);
            tma_load_2d_pair(sa + 8192, &tma_a, fb, m0 + 64, k0);
          }
          if constexpr (!B_MN) {
            tma_load_2d_pair(sb, &tma_b, fb, k0, nb);
          } else {
            tma_load_2d_pair(sb, &tma_b, fb, nb, k0);
            tma_load_2d_pair(sb + 8192, &tma_b, fb, nb + 64, k0);
          }
          if (++stage == ST) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {   // copies in flight land before shared memory goes away
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) {}
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = umma_idesc(FMT_BF16, FMT_BF16, A_MN, B_MN, 2 * BM, BN);
      const uint32_t adesc0 = umma_desc_lo(smem_base, A_MN ? 8192 : 16), bdesc0 = umma_desc_lo(smem_base + L::A_BYTES, B_MN ? 8192 : 16);
      constexpr uint32_t ASTEP = A_MN ? 2048 >> 4 : 32 >> 4, BSTEP = B_MN ? 2048 >> 4 : 32 >> 4;
      int stage = 0, abuf = 0;
      uint32_t phase = 0, aphase = 1;
      bool ok = true;
      for (int w = pair; w < num_work && ok; w += npairs) {
        int n_kb = total_kb;
        if (p.splits > 1) {
          int m0, n0, kb0, kb1;
          decode(w, m0, n0, kb0, kb1);
          n_kb = kb1 - kb0;
        }
        if (!mbar_wait(bar_tempty + abuf * 8, aphase, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + abuf * BN;
        for (int kb = 0; kb < n_kb; ++kb) {
          if (!mbar_wait(bar_full + stage * 8, phase, abort_flag, p.status, ST_TIMEOUT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint32_t at = uint32_t(stage) * (L::STAGE_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_f16_ss_pair(tmem_d, adesc0 + at + k * ASTEP, bdesc0 + at + k * BSTEP, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit_pair(bar_empty + stage * 8);
          if (++stage == ST) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit_pair(bar_tfull + abuf * 8);
        abuf ^= 1;
        if (abuf == 0) aphase ^= 1;
      }
    }
  } else {
    const int quad = warp & 3, ew = warp - 2, half = ew >> 2;
    const uint32_t stg_u32 = smem_base + L::STG_OFF + ew * (L::STG_BUFS * 4096), tempty0 = map_cta(bar_tempty, 0);
    int sbuf = 0, abuf = 0;
    uint32_t aphase = 0;
    for (int w = pair; w < num_work; w += npairs) {
      int m0, n0, kb0, kb1;
      decode(w, m0, n0, kb0, kb1);
      if (!mbar_wait_warp(bar_tfull + abuf * 8, aphase, abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) break;
      tc_fence_after();
      const uint32_t taddr0 = tmem_base + abuf * BN + (uint32_t(quad * 32) << 16);
      if (p.glu) glu_epilogue(p, tma_c, taddr0, n0, m0 + quad * 32, half, lane, stg_u32);
      else staged_epilogue<BN, L::STG_BUFS>(p, tma_c, tma_peers, taddr0, n0, m0 + quad * 32, half, lane, stg_u32, sbuf, 0);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(tempty0 + abuf * 8);
      abuf ^= 1;
      if (abuf == 0) aphase ^= 1;
    }
    if (lane == 0) tma_store_wait<0>();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();      // neither CTA leaves while the other may read its shared memory or arrive on its barriers
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * BN);
  }
}

// -------------------------------------------------------------------------------------------------
// host launcher
// -------------------------------------------------------------------------------------------------
template <bool A_MN, bool B_MN, int BN>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const PeerMaps& tpeers, const GemmParams& p,
                  int grid, cudaStream_t st) {
  using L = SmemLayout<BN>;
  static DeviceOnce once;
  auto kern = gemm_bf16_kernel<A_MN, B_MN, BN>;
  if (int e = ensure_dyn_smem(once, kern, L::TOTAL)) return e;
  tfb::launch_k(kern, grid, GEMM_THREADS, L::TOTAL, st, ta, tb, tc, tpeers, p);
  return int(cudaGetLastError());
}

template <bool A_MN, bool B_MN>
static int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const GemmParams& p, int pairs, cudaStream_t st) {
  using L = PairSmem;
  static DeviceOnce once;
  static const PeerMaps none = {};
  auto kern = gemm_pair_kernel<A_MN, B_MN>;
  if (int e = ensure_dyn_smem(once, kern, L::TOTAL)) return e;
  tfb::launch_k(kern, 2 * pairs, GEMM_THREADS, L::TOTAL, st, ta, tb, tc, none, p);
  return int(cudaGetLastError());
}

}  // namespace tfb

struct TfbGemmGroup {
  int mode;                    // 0 dense, 1 rows grouped (B has a leading expert dim), 2 reduction grouped (C has one)
  int num_experts;
  const int* expert_of_mtile;  // mode 1 (device)
  const int* seg_start;        // mode 2 (device, [E + 1])
  long long b_expert_stride;   // mode 1: elements between consecutive experts' B matrices
  long long c_expert_stride;   // mode 2: elements between consecutive experts' C matrices
};

struct TfbGemmTp {
  int mode;               // bits: 1 all-gather -> GEMM, 2 GEMM -> reduce-scatter, 4 weight gather -> GEMM
  int rank, world;        // tensor-parallel group (bits 1, 2)
  int copy_ctas;          // bits 1, 4: CTAs that move data instead of multiplying
  int epoch;              // bit 1: value of a ready flag once its block has landed
  int* ready;             // bit 1: local int[M / 128]
  const void* peer_a;     // bit 1: device array [world] of gathered-A base pointers
  const void* peer_c;     // bit 2: device array [world] of staging-buffer base pointers
  const void* const* peer_c_host;   // bit 2, optional: the same addresses in host memory; with them (and world <= 8) the
                                    // partial tiles leave through TMA stores instead of per-thread stores
  // bit 4: B is the local gather buffer of a weight whose row shards ([wg_rows / wg_world, ldb] each, 128-row blocks)
  // live on the wg_world ranks of the data-parallel group
  int wg_rank, wg_world, wg_epoch, wg_rows;   // wg_rows: padded row count, a multiple of 128 * wg_world
  int* wg_ready;          // local int[wg_rows / 128]
  const void* wg_src;     // device array [wg_world] of shard base pointers
  int wg_skip_local;      // 1: the caller has already copied this rank's shard into B (the copy CTAs then move remote rows only)
};

// ---------------------------------------------------------------------------------------------------------------------
// Small-M path (decode batches): a product with few output tiles cannot fill the machine, and split-K needs an fp32
// accumulation target.  The partial products go into a per-device fp32 workspace with TMA reduce-add, and a finalize
// kernel applies bias / activation / residual and writes the requested type.  The workspace is allocated once
// (256 MB: up to 256 rows x 262144 columns); a shape that needs more takes the single-wave path instead.
constexpr long long SPLITK_WS_ELEMS = 64ll << 20;

// One workspace per device, allocated at the first small-M product outside a stream capture (an allocation inside a
// capture would invalidate it: a product that arrives first during capture takes the ordinary single-wave path).
// Products of one device are expected to be issued from one stream at a time, as the inference engine does; two streams
// running small-M products concurrently on the same device would share the buffer.
static float* splitk_workspace(cudaStream_t stream) {
  static float* ws[64] = {};
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (!ws[dev]) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
      (void)cudaGetLastError();
      return nullptr;
    }
    void* q = nullptr;
    if (cudaMalloc(&q, SPLITK_WS_ELEMS * sizeof(float)) != cudaSuccess) {
      (void)cudaGetLastError();
      return nullptr;
    }
    // The workspace is all zero between products: cleared once here, and the finalize kernel clears what it has read.
    if (cudaMemset(q, 0, SPLITK_WS_ELEMS * sizeof(float)) != cudaSuccess) {
      (void)cudaGetLastError();
      (void)cudaFree(q);
      return nullptr;
    }
    ws[dev] = static_cast<float*>(q);
  }
  return ws[dev];
}

__global__ void __launch_bounds__(256) splitk_finalize_kernel(float* __restrict__ ws, long long ldw, void* __restrict__ C, long long ldc,
                                                              const __nv_bfloat16* __restrict__ bias,
                                                              const __nv_bfloat16* __restrict__ residual, long long ldr, int M, int N,
                                                              int act, int out_fp32) {
  tfb::pdl_sync();
  const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * 4;      // 4 consecutive columns
  if (i >= (long long)M * ldw) return;
  const int m = int(i / ldw), n = int(i % ldw);
  if (n >= N) return;
  const float4 a = *reinterpret_cast<const float4*>(ws + i);
  *reinterpret_cast<float4*>(ws + i) = make_float4(0.f, 0.f, 0.f, 0.f);     // leave the workspace clear for the next product
  float v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (n + j < N) {
      if (bias) v[j] += __bfloat162float(bias[n + j]);
      v[j] = tfb::apply_act(v[j], act);
      if (residual) v[j] += __bfloat162float(residual[(long long)m * ldr + n + j]);
      if (out_fp32) static_cast<float*>(C)[(long long)m * ldc + n + j] = v[j];
      else static_cast<__nv_bfloat16*>(C)[(long long)m * ldc + n + j] = __float2bfloat16(v[j]);
    }
  }
}

// Few rows: the product streams the weights once and is bound by how evenly the work items cover the SMs.  The split count whose item
// count (tiles x splits) fills whole waves best, keeping at least 8 k-blocks per split; the partials are accumulated in fp32 and finished in a
// second kernel.  `fill`: the share of the waves that the tiles alone fill.
static int few_row_splits(int M, int N, int K, int sms, double* fill) {
  using namespace tfb;
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + (N > 128 ? 255 : 127)) / (N > 128 ? 256 : 128));
  const int total_kb = (K + BK - 1) / BK;
  int best_s = 1;
  double best_eff = 0.0, eff1 = double(tiles) / double((tiles + sms - 1) / sms * sms);
  for (int sp = 1; K >= 16 * BK && sp <= 16 && sp * 8 <= total_kb; ++sp) {
    const long long items = tiles * sp;
    const double eff = double(items) / double((items + sms - 1) / sms * sms);
    if (eff > best_eff + 0.02) { best_eff = eff; best_s = sp; }
  }
  if (fill) *fill = eff1;
  return best_eff < eff1 + 0.1 ? 1 : best_s;          // the workspace pass costs about a tenth of a weight-streaming product
}

// Products of few rows: whether the streaming form of gemm_rows.cu (tiles of 128 weight rows) is faster than this file's kernels with their
// split over K.  us, this file / streaming / streaming with the weights fetched ahead (w_static):
//   - Short K: a block holds many whole tiles, and its time is their drains.  32000 x 512 at 16 / 64 rows 11.1 / 11.8 / 11.8 and 11.3 / 17.0 / 16.2;
//     50304 x 768 19.3 / 20.4 / 18.4 and 19.9 / 25.1 / 22.8.
//   - Where this file's tiles fill their waves without a split, one to a block, theirs is one drain: 32000 x 1024 at 8 / 64 rows 16.7 / 18.0 / 16.3
//     and 16.4 / 21.9 / 20.5, 32000 x 2048 at 64 26.7 / 33.6 / 31.1 (but 32000 x 4096, which it splits, 72 / 54 / 51).
//   - Many blocks to a tile: they meet in memory, more of it with more rows.  4096 x 4096 at 16 / 64 rows 13.7 / 12.8 / 12.6 and 16.0 / 18.0 / 17.2,
//     2048 x 8192 at 32 rows 13.9 / 14.9 / 15.2, 6144 x 4096 at 64 18.8 / 19.5 / 18.5, 8192 x 2048 17.8 / 17.1 / 15.9.
//   - Without the early fetch the longer streams win nothing while this file's kernels fill the machine: 4096 x 14336 at 16 rows 26.1 / 26.4 / 23.9,
//     8192 x 8192 28.9 / 29.6 / 25.7; from 16384 weight rows on they do not (28672 x 4096 at 16 / 64 / 128 rows 48.6 / 45.4 / 42.1, 63 / 49 / 47
//     and 86 / 57 / 56).
static bool rows_pay(int M, int N, int K, long long tiles, int w_static) {
  const int KB = (K + tfb::BK - 1) / tfb::BK;
  if (KB < (M <= 16 && w_static ? 12 : 16)) return false;
  double fill;
  if ((M > 16 || !w_static) && few_row_splits(M, N, K, tfb::sm_count(), &fill) == 1 && fill >= 0.8) return false;
  if (M > 64) return tiles >= 128;
  if (w_static) return M <= 16 || tiles >= 48;
  return (M <= 16 || tiles >= 64) && (KB <= 64 || tiles >= 128);
}

static int gemm_impl(const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn, void* C,
                     long long ldc, int M, int N, int K, const void* bias, const void* residual, long long ldr,
                     float alpha, int act, int out_mode, int max_ctas, const TfbGemmGroup* grp, int* status,
                     void* stream, const TfbGemmTp* tp = nullptr, int force_splits = 0, int w_static = 0) {
  using namespace tfb;
  if (M <= 0 || N <= 0 || K <= 0) return TFB_ERR_ARG;
  if (out_mode != 0 && (bias || residual || act)) return TFB_ERR_ARG;
  if (!grp && !tp && !a_mn && !b_mn && out_mode != 2 && max_ctas <= 0 && M <= 128) {
    int rc0 = gemm_skinny(A, lda, B, ldb, C, ldc, M, N, K, bias, residual, ldr, alpha, act, out_mode == 1, stream);
    if (rc0 == TFB_NOT_TAKEN && rows_pay(M, N, K, (N + 127) / 128, w_static))
      rc0 = gemm_rows(A, lda, B, ldb, nullptr, nullptr, -1, 0, C, ldc, M, N, K, K, bias, residual, ldr, alpha, act, out_mode == 1, w_static, status,
                      stream);
    if (rc0 != TFB_NOT_TAKEN) return rc0;
  }
  const int gmode = grp ? grp->mode : 0;
  const int E = (gmode != 0) ? grp->num_experts : 1;
  if (gmode == 2 && out_mode == 0) return TFB_ERR_ARG;
  if (gmode == 0 && !tp && out_mode != 2 && M <= 256 && K >= 16 * BK) {
    const long long ldw = (N + 3) / 4 * 4;
    const int all_sms = (max_ctas > 0 && max_ctas < sm_count()) ? max_ctas : sm_count();
    const int best_s = few_row_splits(M, N, K, all_sms, nullptr);
    if (best_s > 1 && (long long)M * ldw <= SPLITK_WS_ELEMS) {
      cudaStream_t st0 = static_cast<cudaStream_t>(stream);
      if (float* ws = splitk_workspace(st0)) {
        if (int rc0 = gemm_impl(A, lda, a_mn, B, ldb, b_mn, ws, ldw, M, N, K, nullptr, nullptr, 0, alpha, 0, 2, max_ctas, nullptr, status,
                                stream, nullptr, best_s))
          return rc0;
        const long long quads = (long long)M * ldw / 4;
        tfb::launch_k(splitk_finalize_kernel, int((quads + 255) / 256), 256, 0, st0, ws, ldw, C, ldc, static_cast<const __nv_bfloat16*>(bias),
                                                                          static_cast<const __nv_bfloat16*>(residual), ldr, M, N, act,
                                                                          out_mode == 1);
        return int(cudaGetLastError());
      }
    }
  }
  int BN = (N > 128) ? 256 : 128;
  int sms = sm_count();
  if (max_ctas > 0 && max_ctas < sms) sms = max_ctas;
  {
    // prefer the narrower tile when it puts more SMs to work and still fits into one wave; when the narrow tiling would
    // need a second wave (8192 x 512: 256 tiles of 128 columns) the wide one finishes in a single wave and wins by
    // 12 - 27 % (measured: 13.3 against 15.2 us at K = 512, 28.8 against 39.7 us at K = 2816)
    const long long tm = (M + BM - 1) / BM;
    const long long t256 = tm * ((N + 255) / 256), t128 = tm * ((N + 127) / 128);
    static const int narrow_env = [] { const char* e = getenv("TFB_GEMM_NARROW"); return e ? atoi(e) : 1; }();
    if (narrow_env && BN == 256 && gmode != 2 && out_mode != 2 && t256 < sms && t128 > t256 && t128 <= sms) BN = 128;
  }
  static const int raster_env = [] { const char* e = getenv("TFB_GEMM_RASTER"); return e ? atoi(e) : -1; }();
  // Tiles of 256 columns of a plain product with more than one tile row run on CTA pairs, except
  //   - where few k-blocks leave the set-up of the cluster in sight: one wave of at most 12 (us, pairs / single CTAs: 777 x 2816 x 512 9.2 / 8.6, 1024 x
  //     3072 x 768 10.7 / 10.0; 512 x 6144 x 4096 27.5 / 30.4), or at most 4 (4096 x 4096 x 129 accumulated 22.2 / 19.7; 300 instead of 129
  //     23.2 / 24.6);
  //   - where their larger tiles take a wave more, and a wave on pairs at 0.85 of the time does not make up for it (4662 x 1000 x 776, 2 waves against
  //     1, 24.3 / 18.0; 4662 x 3072 x 768, 4 against 3, 22.7 / 21.5; 4662 x 4096 x 14336, 5 against 4, 395 / 369; 777 x 28672 x 4096, 7 against
  //     6, 160 / 160) - but not for one or two tile rows over long K, bound by the weights that single CTAs read once more (300 x 28672 x
  //     4096, 4 against 3, 88 / 110).
  bool want_pair = BN == 256 && gmode == 0 && !tp && M > BM && sms >= 2;
  if (want_pair) {
    const int kbs = (K + BK - 1) / BK, pairs = sms / 2;
    const long long tm2 = (M + 2 * BM - 1) / (2 * BM), tn = (N + BN - 1) / BN, tm1 = (M + BM - 1) / BM;
    const long long waves2 = (tm2 * tn + pairs - 1) / pairs, waves1 = (tm1 * tn + sms - 1) / sms;
    if (kbs <= 4 || (waves2 == 1 && kbs <= 12) || (waves2 * 17 > waves1 * 20 && (tm2 > 2 || kbs < 32 || waves1 == 1))) want_pair = false;
  }
  CUtensorMap ta, tb;
  int rc;
  if (!a_mn) rc = make_tmap_2d(&ta, A, 2, K, M, lda * 2, BK, BM);
  else rc = make_tmap_2d(&ta, A, 2, M, K, lda * 2, 64, BK);
  if (rc) return rc;
  if (want_pair) {
    CUtensorMap tb2, tc2;
    const int esz = out_mode == 0 ? 2 : 4;
    rc = !b_mn ? make_tmap_2d(&tb2, B, 2, K, N, ldb * 2, BK, BM) : make_tmap_2d(&tb2, B, 2, N, K, ldb * 2, 64, BK);
    if (rc) return rc;
    if ((reinterpret_cast<uintptr_t>(C) & 15) == 0 && (ldc * esz) % 16 == 0 &&
        make_tmap_3d(&tc2, C, esz, N, M, 1, ldc * esz, (unsigned long long)ldc * esz * M, 128 / esz, 32, 1) == 0) {
      GemmParams p = {};
      p.M = M; p.N = N; p.K = K;
      p.C = C; p.ldc = ldc;
      p.bias = static_cast<const __nv_bfloat16*>(bias);
      p.residual = static_cast<const __nv_bfloat16*>(residual);
      p.ldr = ldr;
      p.alpha = alpha; p.act = act; p.out_mode = out_mode;
      p.tiles_m = (M + 2 * BM - 1) / (2 * BM);
      p.tiles_n = (N + BN - 1) / BN;
      p.num_experts = 1;
      p.rs_world = 1;
      p.c_tma = 1;
      p.status = status;
      // tile order as below, in groups of eight tile columns where B is wide
      p.raster_gn = raster_env != 0 && p.tiles_n > 12 && p.tiles_m >= 2 ? (raster_env > 0 ? raster_env : 8) : p.tiles_n;
      const int total_kb = (K + BK - 1) / BK, tiles = p.tiles_m * p.tiles_n, pairs = sms / 2;
      int splits = 1;
      if (force_splits > 0 && out_mode == 2) splits = force_splits;
      else if (out_mode == 2 && tiles < pairs) splits = max(1, min(pairs / tiles, (total_kb + 7) / 8));   // one wave, at least 8 k-blocks per split
      p.kb_per_split = (total_kb + splits - 1) / splits;
      p.splits = (total_kb + p.kb_per_split - 1) / p.kb_per_split;
      const int grid = int(min((long long)tiles * p.splits, (long long)pairs));
      cudaStream_t st = static_cast<cudaStream_t>(stream);
      switch ((a_mn ? 2 : 0) | (b_mn ? 1 : 0)) {
        case 0: return launch_pair<false, false>(ta, tb2, tc2, p, grid, st);
        case 1: return launch_pair<false, true>(ta, tb2, tc2, p, grid, st);
        case 2: return launch_pair<true, false>(ta, tb2, tc2, p, grid, st);
        default: return launch_pair<true, true>(ta, tb2, tc2, p, grid, st);
      }
    }
  }
  const int EB = gmode == 1 ? E : 1;
  const unsigned long long bes = gmode == 1 ? (unsigned long long)grp->b_expert_stride * 2 : (unsigned long long)ldb * 2 * (b_mn ? K : N);
  if (!b_mn) rc = make_tmap_3d(&tb, B, 2, K, N, EB, ldb * 2, bes, BK, BN, 1);
  else rc = make_tmap_3d(&tb, B, 2, N, K, EB, ldb * 2, bes, 64, BK, 1);
  if (rc) return rc;

  GemmParams p;
  p.M = M; p.N = N; p.K = K;
  p.C = C; p.ldc = ldc;
  // C tensor map for the staged epilogue: 32-row x 128-byte boxes.  Needs a 16-byte aligned base and row pitch.
  CUtensorMap tc;
  memset(&tc, 0, sizeof(tc));
  PeerMaps tpeers;
  memset(&tpeers, 0, sizeof(tpeers));
  p.c_tma = 0;
  {
    const int esz = out_mode == 0 ? 2 : 4;
    const bool aligned = (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (ldc * esz) % 16 == 0 &&
                         (gmode != 2 || (grp->c_expert_stride * esz) % 16 == 0);
    const bool rs = tp && (tp->mode & TP_RS);
    if (aligned && rs && tp->peer_c_host && tp->world <= RS_TMA_MAX_WORLD && out_mode == 0 && (ldc * 2) % 16 == 0) {
      const int rps = M / tp->world;
      bool ok = true;
      for (int d = 0; d < tp->world && ok; ++d)
        ok = (reinterpret_cast<uintptr_t>(tp->peer_c_host[d]) & 15) == 0 &&
             make_tmap_3d(&tpeers.m[d], tp->peer_c_host[d], 2, N, (unsigned long long)tp->world * rps, 1, ldc * 2,
                          (unsigned long long)ldc * 2 * tp->world * rps, 64, 32, 1) == 0;
      if (ok) p.c_tma = 1;
    }
    if (aligned && !rs) {
      const unsigned long long zs = gmode == 2 ? (unsigned long long)grp->c_expert_stride * esz : (unsigned long long)ldc * esz * M;
      if (make_tmap_3d(&tc, C, esz, N, M, gmode == 2 ? E : 1, ldc * esz, zs, 128 / esz, 32, 1) == 0) p.c_tma = 1;
    }
  }
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.ldr = ldr;
  p.alpha = alpha; p.act = act; p.out_mode = out_mode;
  p.tiles_m = (M + BM - 1) / BM;
  p.tiles_n = (N + BN - 1) / BN;
  p.status = status;
  p.group_mode = gmode; p.num_experts = E;
  p.expert_of_mtile = grp ? grp->expert_of_mtile : nullptr;
  p.seg_start = grp ? grp->seg_start : nullptr;
  p.c_expert_stride = grp ? grp->c_expert_stride : 0;
  p.tp_mode = 0; p.tp_copy_ctas = 0;
  memset(&p.ag, 0, sizeof(p.ag));
  memset(&p.wg, 0, sizeof(p.wg));
  p.wg_n_shift = -1; p.wg_k_shift = 0;
  p.glu = 0;
  p.rs_rank = 0; p.rs_world = 1; p.rs_rows_per_shard = M; p.rs_peer_c = nullptr;
  if (tp) {
    if (gmode != 0 || tp->mode < 1 || tp->mode > 7 || (tp->mode & (TP_AG | TP_RS)) == (TP_AG | TP_RS)) return TFB_ERR_ARG;
    if (tp->mode & (TP_AG | TP_WG)) {
      if (tp->copy_ctas < 1 || tp->copy_ctas >= sms) return TFB_ERR_ARG;
      p.tp_copy_ctas = tp->copy_ctas;
      sms -= tp->copy_ctas;
    }
    if (tp->mode & (TP_AG | TP_RS)) {
      if (tp->world < 1 || M % (tp->world * BM) || a_mn || out_mode != 0) return TFB_ERR_ARG;
    }
    if (tp->mode & TP_AG) {
      if (K % 8 || !tp->ready || !tp->peer_a) return TFB_ERR_ARG;
      p.ag.rank = tp->rank; p.ag.world = tp->world; p.ag.rows_per_shard = M / tp->world; p.ag.row_len = K;
      p.ag.epoch = tp->epoch; p.ag.rows = M; p.ag.src_is_full = 1; p.ag.skip_local = 1; p.ag.ready = tp->ready;
      p.ag.src = static_cast<const __nv_bfloat16* const*>(tp->peer_a);
      p.ag.dst = const_cast<__nv_bfloat16*>(static_cast<const __nv_bfloat16*>(A));
      p.ag.ld = lda;
    }
    if (tp->mode & TP_RS) {
      if (!tp->peer_c) return TFB_ERR_ARG;
      p.rs_rank = tp->rank; p.rs_world = tp->world; p.rs_rows_per_shard = M / tp->world;
      p.rs_peer_c = static_cast<__nv_bfloat16* const*>(tp->peer_c);
    }
    if (tp->mode & TP_WG) {
      // gathered B: rows = N (K-major B) or K (MN-major B), sharded in 128-row blocks over the data-parallel group
      const int rows = b_mn ? K : N, row_len = b_mn ? N : K;
      if (tp->wg_world < 1 || tp->wg_rows < rows || tp->wg_rows % (tp->wg_world * BM) || row_len % 8 || out_mode == 2 ||
          !tp->wg_ready || !tp->wg_src)
        return TFB_ERR_ARG;
      p.wg.rank = tp->wg_rank; p.wg.world = tp->wg_world; p.wg.rows_per_shard = tp->wg_rows / tp->wg_world;
      p.wg.row_len = row_len; p.wg.epoch = tp->wg_epoch; p.wg.rows = rows; p.wg.src_is_full = 0; p.wg.skip_local = tp->wg_skip_local ? 1 : 0;
      p.wg.ready = tp->wg_ready;
      p.wg.src = static_cast<const __nv_bfloat16* const*>(tp->wg_src);
      p.wg.dst = const_cast<__nv_bfloat16*>(static_cast<const __nv_bfloat16*>(B));
      p.wg.ld = ldb;
      if (!b_mn) p.wg_n_shift = (tp->wg_rank * (p.wg.rows_per_shard / BN)) % p.tiles_n;
      else p.wg_k_shift = (tp->wg_rank * (p.wg.rows_per_shard / BK)) % ((K + BK - 1) / BK);
    }
    p.tp_mode = tp->mode;
  }
  {
    // tile order (see decode_work): row-major unless B is wide; the activation gather / reduce-scatter orders follow the
    // row blocks and stay row-major; a gathered K-major weight is always walked in column groups
    const int wide = (BN == 256) ? 8 : 16;
    p.raster_gn = p.tiles_n;
    if (gmode != 2 && !(p.tp_mode & (TP_AG | TP_RS))) {
      if ((p.tp_mode & TP_WG) && p.wg_n_shift >= 0) p.raster_gn = raster_env == 0 ? 1 : min(wide, p.tiles_n);
      else if (raster_env != 0 && p.tiles_n > wide + wide / 2 && p.tiles_m >= 4) p.raster_gn = raster_env > 0 ? raster_env : wide;
    }
    if (p.raster_gn < 1) p.raster_gn = 1;
  }
  const int total_kb = (K + BK - 1) / BK;
  const int tiles = p.tiles_m * p.tiles_n;
  int splits = 1;
  if (force_splits > 0 && out_mode == 2 && gmode == 0) {
    splits = force_splits;
  } else if (out_mode == 2 && gmode == 0 && tiles < sms) {
    splits = sms / tiles;                       // round down: all work items must fit in one wave
    const int max_splits = (total_kb + 7) / 8;  // keep at least 8 k-blocks (512 of K) per split
    if (splits > max_splits) splits = max_splits;
    if (splits < 1) splits = 1;
  }
  p.kb_per_split = (total_kb + splits - 1) / splits;
  p.splits = (total_kb + p.kb_per_split - 1) / p.kb_per_split;
  const long long work = (long long)tiles * (gmode == 2 ? E : p.splits);
  const int grid = int(work < sms ? work : sms) + p.tp_copy_ctas;   // copy CTAs take the lowest block indices
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int key = (a_mn ? 2 : 0) | (b_mn ? 1 : 0);
  if (BN == 256) {
    switch (key) {
      case 0: return launch<false, false, 256>(ta, tb, tc, tpeers, p, grid, st);
      case 1: return launch<false, true, 256>(ta, tb, tc, tpeers, p, grid, st);
      case 2: return launch<true, false, 256>(ta, tb, tc, tpeers, p, grid, st);
      default: return launch<true, true, 256>(ta, tb, tc, tpeers, p, grid, st);
    }
  } else {
    switch (key) {
      case 0: return launch<false, false, 128>(ta, tb, tc, tpeers, p, grid, st);
      case 1: return launch<false, true, 128>(ta, tb, tc, tpeers, p, grid, st);
      case 2: return launch<true, false, 128>(ta, tb, tc, tpeers, p, grid, st);
      default: return launch<true, true, 128>(ta, tb, tc, tpeers, p, grid, st);
    }
  }
}

// C[M,N] (ldc) = act(alpha * A.B + bias) + residual.
//   a_mn = 0: A is [M,K] with K contiguous (row pitch lda elements); a_mn = 1: A is stored [K,M], M contiguous.
//   b_mn = 0: B is [N,K] with K contiguous (weight layout [out,in]);  b_mn = 1: B is stored [K,N], N contiguous.
//   out_mode 0: bf16 store; 1: fp32 store; 2: fp32 atomic accumulate (C += ...), the only mode that allows split-K.
//   max_ctas > 0 limits the persistent grid (leaves SMs free for a concurrent communication kernel).
TFB_API int tfb_gemm_bf16(const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn, void* C,
                          long long ldc, int M, int N, int K, const void* bias, const void* residual, long long ldr,
                          float alpha, int act, int out_mode, int max_ctas, int* status, void* stream) {
  return gemm_impl(A, lda, a_mn, B, ldb, b_mn, C, ldc, M, N, K, bias, residual, ldr, alpha, act, out_mode, max_ctas,
                   nullptr, status, stream);
}

// C [M, F] = act(A . B[0..F)^T) * (A . B[F..2F)^T): the gated projection of a feed-forward without its [M, 2F] product in memory.  Whole passes,
// product and gating kernel -> this: four prompts of 1000 - 4000 tokens at the 8b widths 37.4 -> 35.7 ms, scoring 2 x 2500 tokens 17.7 ->
// 17.4, 64 single-token steps 67.3 -> 62.9, 16 sequences of the 50m shape 20.0 -> 19.2.
// TFB_ERR_ARG where no kernel takes it (the caller runs the two).
TFB_API int tfb_gemm_glu(const void* A, long long lda, const void* B, long long ldb, void* C, long long ldc, int M, int F, int K, int act, int w_static,
                         int* status, void* stream) {
  using namespace tfb;
  if (M <= 0 || F <= 0 || F % 8 || K <= 0 || act < 1 || act > 4) return TFB_ERR_ARG;
  if (M <= BM) {
    int rc = gemm_skinny_glu(A, lda, B, ldb, C, ldc, M, F, K, act, stream);
    // above 32 rows the exchange of the halves in the epilogue costs more than the gating kernel (64 sequences of the 8b widths: 104 against 101 ms a pass)
    if (rc == TFB_NOT_TAKEN && M <= 32 && rows_pay(M, 2 * F, K, (F + 63) / 64, w_static)) rc = gemm_rows_glu(A, lda, B, ldb, C, ldc, M, F, K, act, w_static, status, stream);
    return rc == TFB_NOT_TAKEN ? int(TFB_ERR_ARG) : rc;
  }
  CUtensorMap ta, tb, tc;
  if ((reinterpret_cast<uintptr_t>(C) & 15) || ldc % 8 || sm_count() < 2) return TFB_ERR_ARG;
  // Its tiles of 256 x 128 outputs have to fill their waves on pairs: us, product and gating kernel / this: F x K = 1408 x 512 at 300 rows (0.3 waves)
  // 9.2 / 11.1, 3072 x 768 at 300 (0.65) 10.7 / 12.5, 5632 x 2048 at 300 (1.2) 22.7 / 28.9; 14336 x 4096 at 300 (3.03) 116 / 90, 8192 x 1024 at 129 (0.9)
  // 16.5 / 15.0.  Up to 256 rows over long K the other path has a pass over its split sums: 5632 x 2048 at 129 (0.6) 30.9 / 19.4.
  const long long tiles = (long long)((M + 2 * BM - 1) / (2 * BM)) * ((F + BM - 1) / BM), pairs = sm_count() / 2;
  if (tiles * 4 < (tiles + pairs - 1) / pairs * pairs * 3 && (M > 2 * BM || K < 16 * BK || tiles * 5 < pairs)) return TFB_ERR_ARG;
  if (int rc = make_tmap_2d(&ta, A, 2, K, M, lda * 2, BK, BM)) return rc;
  if (int rc = make_tmap_2d(&tb, B, 2, K, 2ull * F, ldb * 2, BK, BM)) return rc;
  if (int rc = make_tmap_3d(&tc, C, 2, F, M, 1, ldc * 2, (unsigned long long)ldc * 2 * M, 64, 32, 1)) return rc;
  GemmParams p = {};
  p.M = M; p.N = F; p.K = K;
  p.C = C; p.ldc = ldc;
  p.alpha = 1.f; p.act = act; p.glu = F;
  p.tiles_m = (M + 2 * BM - 1) / (2 * BM);
  p.tiles_n = (F + BM - 1) / BM;
  p.num_experts = 1; p.rs_world = 1; p.c_tma = 1;
  p.status = status;
  p.raster_gn = p.tiles_n > 12 && p.tiles_m >= 2 ? 8 : p.tiles_n;
  p.splits = 1;
  p.kb_per_split = (K + BK - 1) / BK;
  return launch_pair<false, false>(ta, tb, tc, p, min(p.tiles_m * p.tiles_n, sm_count() / 2), static_cast<cudaStream_t>(stream));
}

// The same for weights of a model that serves: the caller promises that the kernel launched just before this one on the stream does not
// write B, so that a product of few rows may begin to fetch it before that kernel has ended.
TFB_API int tfb_gemm_bf16_static(const void* A, long long lda, const void* B, long long ldb, void* C, long long ldc, int M, int N, int K,
                                 const void* bias, const void* residual, long long ldr, int out_mode, int* status, void* stream) {
  return gemm_impl(A, lda, 0, B, ldb, 0, C, ldc, M, N, K, bias, residual, ldr, 1.f, 0, out_mode, 0, nullptr, status, stream, nullptr, 0, 1);
}

// Grouped (mixture-of-experts) form; see TfbGemmGroup.  Mode 1: M counts the padded rows of all experts, B is
// [E, N, K] (or [E, K, N] with b_mn).  Mode 2: K counts the padded rows, C is [E, M, N] fp32 (out_mode 1 or 2).
TFB_API int tfb_gemm_bf16_grouped(const void* A, long long lda, int a_mn, const void* B, long long ldb, int b_mn,
                                  void* C, long long ldc, int M, int N, int K, float alpha, int out_mode,
                                  const TfbGemmGroup* grp, int* status, void* stream) {
  if (!grp || grp->mode < 1 || grp->mode > 2 || grp->num_experts < 1) return TFB_ERR_ARG;
  return gemm_impl(A, lda, a_mn, B, ldb, b_mn, C, ldc, M, N, K, nullptr, nullptr, 0, alpha, 0, out_mode, 0, grp,
                   status, stream);
}

// Fused compute + collective forms (see TfbGemmTp and tp_fused.cu).  Bit 1: C[M, N] = gathered A [M, K] . B^T where
// A's row shards live on the W tensor-parallel ranks.  Bit 2: C is ignored; partial products go to the peers' staging
// buffers (row pitch ldc) and are summed by tfb_tp_reduce.  Bit 4: B is the local gather buffer of a weight whose row
// shards live on the data-parallel ranks (tp->wg_src); the shards are pulled while the tiles of the local shard run.
// `residual` ([M, ldr] bf16, added in the epilogue) is allowed when bit 2 is clear.
TFB_API int tfb_gemm_bf16_tp(const void* A, long long lda, const void* B, long long ldb, int b_mn, void* C,
                             long long ldc, int M, int N, int K, const void* residual, long long ldr,
                             const TfbGemmTp* tp, int* status, void* stream) {
  if (!tp || tp->mode < 1 || tp->mode > 7) return TFB_ERR_ARG;
  if (residual && (tp->mode & 2)) return TFB_ERR_ARG;
  return gemm_impl(A, lda, 0, B, ldb, b_mn, C, ldc, M, N, K, nullptr, residual, ldr, 1.0f, 0, 0, 0, nullptr, status,
                   stream, tp);
}
