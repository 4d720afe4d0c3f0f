// RMSNorm / LayerNorm forward and backward, fused with the residual add.
//
// All of these are bound by HBM: every activation is read once and written once, 128 bits at a time, and the row stays in
// registers between the statistics pass and the scale pass.  Rows of up to 1024 entries belong to a warp each (no barrier, and
// the loads of the warp's next row are in flight while it finishes this one), wider rows to a block of 256 threads: a warp that
// holds 4096 entries needs 166 registers a lane, which leaves 12 % of the warps resident and the loads unhidden (5000 x 4096
// forward: 58 us by warps, 18 us by blocks, 13 us of HBM time).  The backward accumulates the weight gradient in registers
// over all rows that a thread visits and flushes it once with fp32 atomics into the fp32 gradient buffer.
//
// Replaces the reference's one-thread-per-row kernels (src/backend/gpu_compute_cuda.cpp:219
// rmsnorm_kernel, :617 layernorm_kernel) and its CPU fused residual+norm
// (src/backend/gpu_compute_vulkan.cpp:1749-1761 vk_rms_norm_add).
#include "tfb_host.h"
#include "tfb_ptx.cuh"

namespace tfb {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = unpack_bf16(w[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16(f[0], f[1]);
  u.y = pack_bf16(f[2], f[3]);
  u.z = pack_bf16(f[4], f[5]);
  u.w = pack_bf16(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}

__device__ __forceinline__ void cvt8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = unpack_bf16(w[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

// y = norm(x + res) * w (+ b);  h_out = x + res (optional);  stats: rstd (and mean for LayerNorm).
// One warp per row (H <= 256 NCHUNK).
template <int NCHUNK, bool LAYERNORM>
__global__ void __launch_bounds__(256) norm_fwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                       const __nv_bfloat16* __restrict__ res,
                                                       const __nv_bfloat16* __restrict__ w,
                                                       const __nv_bfloat16* __restrict__ b,
                                                       __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ h_out,
                                                       float* __restrict__ rstd_out, float* __restrict__ mean_out,
                                                       int rows, int H, float eps) {
  tfb::pdl_sync();
  const int lane = threadIdx.x & 31;
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int row = warp_global; row < rows; row += nwarps) {
    const long long off = (long long)row * H;
    float v[NCHUNK][8];
    float s = 0.f, ss = 0.f;
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      const int col = (c * 32 + lane) * 8;
      if (col < H) {
        load8(x + off + col, v[c]);
        if (res) {
          float r[8];
          load8(res + off + col, r);
#pragma unroll
          for (int i = 0; i < 8; ++i) v[c][i] += r[i];
        }
        if (h_out) {
          store8(h_out + off + col, v[c]);
          // statistics are taken on the bf16-rounded residual stream so forward and backward agree
#pragma unroll
          for (int i = 0; i < 8; ++i) v[c][i] = __bfloat162float(__float2bfloat16(v[c][i]));
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          s += v[c][i];
          ss += v[c][i] * v[c][i];
        }
      }
    }
    s = warp_sum(s);
    ss = warp_sum(ss);
    float mean = 0.f, rstd;
    if (LAYERNORM) {
      mean = s / H;
      rstd = rsqrtf(fmaxf(ss / H - mean * mean, 0.f) + eps);
    } else {
      rstd = rsqrtf(ss / H + eps);
    }
    if (lane == 0) {
      if (rstd_out) rstd_out[row] = rstd;
      if (LAYERNORM && mean_out) mean_out[row] = mean;
    }
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      const int col = (c * 32 + lane) * 8;
      if (col < H) {
        float wv[8], o[8];
        load8(w + col, wv);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = (v[c][i] - mean) * rstd * wv[i];
        if (LAYERNORM && b) {
          float bv[8];
          load8(b + col, bv);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += bv[i];
        }
        store8(y + off + col, o);
      }
    }
  }
}

// dx = rstd * (g - xhat * mean(g * xhat) [- mean(g)])  with g = dy * w, xhat = (h - mean) * rstd, plus the incoming
// residual-stream gradient `dres`;  dw += sum_rows dy * xhat (db += sum_rows dy).
// WIDE = false: a warp per row, eight rows at a time in a block (H <= 256 NCHUNK).  WIDE = true: the block's 256 threads share a row
// (H <= 2048 NCHUNK); the row's two sums meet in shared memory, in one of two slots so that a row costs one barrier.
// The loads of the next row are issued before the sums of this one are reduced.  The weight gradient of the block's rows
// meets in shared memory (plain stores, one slice per warp: fp32 atomics on shared memory are a compare-and-swap loop, and
// with them layer norm of 4662 x 768 took 33 us, 13 us without) and leaves with one atomic per column.
template <int NCHUNK, bool LAYERNORM, bool WIDE>
__global__ void __launch_bounds__(256) norm_bwd_kernel(const __nv_bfloat16* __restrict__ dy,
                                                       const __nv_bfloat16* __restrict__ h,
                                                       const __nv_bfloat16* __restrict__ w,
                                                       const float* __restrict__ rstd_in,
                                                       const float* __restrict__ mean_in,
                                                       const __nv_bfloat16* __restrict__ dres,
                                                       __nv_bfloat16* __restrict__ dx, float* __restrict__ dw,
                                                       float* __restrict__ db, int rows, int H) {
  tfb::pdl_sync();
  extern __shared__ float red[];                      // gradient slices: [8][H], WIDE: [H]
  __shared__ float sums[2][2][8];
  constexpr int TPR = WIDE ? 256 : 32;                // threads per row
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = WIDE ? int(threadIdx.x) : lane;       // place in the row
  const int first = WIDE ? int(blockIdx.x) : int(blockIdx.x) * 8 + warp;
  const int step = WIDE ? int(gridDim.x) : int(gridDim.x) * 8;
  float dw_acc[NCHUNK][8], db_acc[LAYERNORM ? NCHUNK : 1][8];
#pragma unroll
  for (int c = 0; c < NCHUNK; ++c)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      dw_acc[c][i] = 0.f;
      if (LAYERNORM) db_acc[c][i] = 0.f;
    }
  uint4 wr[NCHUNK];
#pragma unroll
  for (int c = 0; c < NCHUNK; ++c) {
    const int col = (c * TPR + t) * 8;
    if (col < H) wr[c] = *reinterpret_cast<const uint4*>(w + col);
  }
  uint4 dyn[NCHUNK], hn[NCHUNK], rn[NCHUNK];
  float rstd_n = 0.f, mean_n = 0.f;
  auto fetch = [&](int row) {
    const long long off = (long long)row * H;
    rstd_n = rstd_in[row];
    if (LAYERNORM) mean_n = mean_in[row];
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      const int col = (c * TPR + t) * 8;
      if (col < H) {
        dyn[c] = *reinterpret_cast<const uint4*>(dy + off + col);
        hn[c] = *reinterpret_cast<const uint4*>(h + off + col);
        if (dres) rn[c] = *reinterpret_cast<const uint4*>(dres + off + col);
      }
    }
  };
  if (first < rows) fetch(first);
  int slot = 0;
  for (int row = first; row < rows; row += step, slot ^= 1) {
    const long long off = (long long)row * H;
    const float rstd = rstd_n, mean = mean_n;
    uint4 dyr[NCHUNK], hr[NCHUNK], rr[NCHUNK];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      const int col = (c * TPR + t) * 8;
      if (col < H) {
        dyr[c] = dyn[c];
        hr[c] = hn[c];
        rr[c] = rn[c];
        float d[8], xh[8], wv[8];
        cvt8(dyr[c], d);
        cvt8(hr[c], xh);
        cvt8(wr[c], wv);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          xh[i] = (xh[i] - mean) * rstd;
          dw_acc[c][i] += d[i] * xh[i];
          if (LAYERNORM) db_acc[c][i] += d[i];
          const float g = d[i] * wv[i];
          s1 += g * xh[i];
          s2 += g;
        }
      }
    }
    if (row + step < rows) fetch(row + step);
    s1 = warp_sum(s1);
    if (LAYERNORM) s2 = warp_sum(s2);
    if (WIDE) {
      if (lane == 0) {
        sums[slot][0][warp] = s1;
        sums[slot][1][warp] = s2;
      }
      __syncthreads();
      s1 = s2 = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        s1 += sums[slot][0][i];
        s2 += sums[slot][1][i];
      }
    }
    s1 /= H;
    s2 = LAYERNORM ? s2 / H : 0.f;
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      const int col = (c * TPR + t) * 8;
      if (col < H) {
        float d[8], xh[8], wv[8], o[8];
        cvt8(dyr[c], d);
        cvt8(hr[c], xh);
        cvt8(wr[c], wv);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xn = (xh[i] - mean) * rstd;
          o[i] = rstd * (d[i] * wv[i] - xn * s1 - s2);
        }
        if (dres) {
          float r[8];
          cvt8(rr[c], r);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += r[i];
        }
        store8(dx + off + col, o);
      }
    }
  }
  for (int pass = 0; pass < (LAYERNORM && db ? 2 : 1); ++pass) {
    float* dst = pass == 0 ? dw : db;
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      const int col = (c * TPR + t) * 8;
      if (col < H) {
        const float(&a)[8] = pass == 0 ? dw_acc[c] : db_acc[LAYERNORM ? c : 0];
        float4* r = reinterpret_cast<float4*>(red + (WIDE ? 0 : warp * H) + col);
        r[0] = make_float4(a[0], a[1], a[2], a[3]);
        r[1] = make_float4(a[4], a[5], a[6], a[7]);
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < H; i += 256) {
      float v = red[i];                               // WIDE: every column has one thread in the block
      if (!WIDE) {
#pragma unroll
        for (int k = 1; k < 8; ++k) v += red[k * H + i];
      }
      atomicAdd(dst + i, v);
    }
    __syncthreads();
  }
}

// out[n] += sum over rows of x[m, n]: the gradient of a bias.  Bound by reading x once: a block takes 64 columns (eight threads a row,
// 32 rows at a time, FLIGHT of them in flight per thread), a cluster of BLOCKS shares the rows.  The sums meet in a fixed order - lanes,
// warps, blocks over distributed shared memory - so that the same input gives the same bits; blocks that meet in atomics are 10 - 40 %
// faster and do not (us, atomics -> this: 131 x 768 1.8 -> 2.2, 4662 x 768 3.0 -> 4.1, 4662 x 3072 6.5 -> 8.3, 65536 x 3072 59 -> 61; fp32 copy and
// torch's sum 9.1, 25.7, 61, 667).
constexpr int CS_ROWS = 32;
template <int BLOCKS, int FLIGHT>
__global__ void __cluster_dims__(1, BLOCKS, 1) __launch_bounds__(256) col_sum_kernel(const __nv_bfloat16* __restrict__ x, long long ldx,
                                                                                    float* __restrict__ out, int rows, int N) {
  tfb::pdl_sync();
  __shared__ float red[8][64], part[64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c0 = (threadIdx.x & 7) * 8;
  const int col = blockIdx.x * 64 + c0;
  constexpr int STEP = BLOCKS * CS_ROWS;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (col < N) {
    for (int row = blockIdx.y * CS_ROWS + int(threadIdx.x >> 3); row < rows; row += FLIGHT * STEP) {
      uint4 v[FLIGHT];
#pragma unroll
      for (int u = 0; u < FLIGHT; ++u)
        if (row + u * STEP < rows) v[u] = *reinterpret_cast<const uint4*>(x + (long long)(row + u * STEP) * ldx + col);
#pragma unroll
      for (int u = 0; u < FLIGHT; ++u) {
        if (row + u * STEP >= rows) break;
        float f[8];
        cvt8(v[u], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += f[i];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 8);
    acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 16);
  }
  if (lane < 8) {
#pragma unroll
    for (int i = 0; i < 8; ++i) red[warp][c0 + i] = acc[i];
  }
  __syncthreads();
  if (threadIdx.x < 64) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) v += red[k][threadIdx.x];
    if (BLOCKS == 1) {
      if (blockIdx.x * 64 + int(threadIdx.x) < N) out[blockIdx.x * 64 + threadIdx.x] += v;
    } else {
      part[threadIdx.x] = v;
    }
  }
  if (BLOCKS == 1) return;
  cluster_sync();
  if (blockIdx.y == 0 && threadIdx.x < 64 && blockIdx.x * 64 + int(threadIdx.x) < N) {
    const uint32_t mine = smem_u32(&part[threadIdx.x]);
    float v[BLOCKS], sum = 0.f;
#pragma unroll
    for (int k = 0; k < BLOCKS; ++k) v[k] = ld_shared_cluster_f32(map_cta(mine, k));
#pragma unroll
    for (int k = 0; k < BLOCKS; ++k) sum += v[k];
    out[blockIdx.x * 64 + threadIdx.x] += sum;
  }
  cluster_sync();      // a block's shared memory stays until it has been read
}

// Wide rows (more than 1024 entries): one CTA per row, so that a 4096-wide row is two 16-byte loads per thread.
template <int NCH, bool LAYERNORM>
__global__ void __launch_bounds__(256) norm_fwd_rowblock_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                                                                const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ b,
                                                                __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ h_out,
                                                                float* __restrict__ rstd_out, float* __restrict__ mean_out, int rows, int H,
                                                                float eps) {
  tfb::pdl_sync();
  __shared__ float red[2][8];
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long off = (long long)row * H;
  float v[NCH][8], wv[NCH][8];
  float s = 0.f, ss = 0.f;
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int col = (c * 256 + threadIdx.x) * 8;
    if (col < H) {
      load8(x + off + col, v[c]);
      load8(w + col, wv[c]);
    }
  }
  if (res) {
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const int col = (c * 256 + threadIdx.x) * 8;
      if (col < H) {
        float r[8];
        load8(res + off + col, r);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[c][i] += r[i];
      }
    }
  }
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int col = (c * 256 + threadIdx.x) * 8;
    if (col < H) {
      if (h_out) {
        store8(h_out + off + col, v[c]);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[c][i] = __bfloat162float(__float2bfloat16(v[c][i]));
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        s += v[c][i];
        ss += v[c][i] * v[c][i];
      }
    }
  }
  s = warp_sum(s);
  ss = warp_sum(ss);
  if (lane == 0) {
    red[0][warp] = s;
    red[1][warp] = ss;
  }
  __syncthreads();
  s = ss = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    s += red[0][i];
    ss += red[1][i];
  }
  float mean = 0.f, rstd;
  if (LAYERNORM) {
    mean = s / H;
    rstd = rsqrtf(fmaxf(ss / H - mean * mean, 0.f) + eps);
  } else {
    rstd = rsqrtf(ss / H + eps);
  }
  if (threadIdx.x == 0) {
    if (rstd_out) rstd_out[row] = rstd;
    if (LAYERNORM && mean_out) mean_out[row] = mean;
  }
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int col = (c * 256 + threadIdx.x) * 8;
    if (col < H) {
      float o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] = (v[c][i] - mean) * rstd * wv[c][i];
      if (LAYERNORM && b) {
        float bv[8];
        load8(b + col, bv);
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] += bv[i];
      }
      store8(y + off + col, o);
    }
  }
}

template <bool LN>
static int launch_fwd(const void* x, const void* res, const void* w, const void* b, void* y, void* h_out, float* rstd,
                      float* mean, int rows, int H, float eps, cudaStream_t st) {
  if (H % 8 || H > 8192) return TFB_ERR_ARG;
  auto X = static_cast<const __nv_bfloat16*>(x);
  auto R = static_cast<const __nv_bfloat16*>(res);
  auto W = static_cast<const __nv_bfloat16*>(w);
  auto B = static_cast<const __nv_bfloat16*>(b);
  auto Y = static_cast<__nv_bfloat16*>(y);
  auto Ho = static_cast<__nv_bfloat16*>(h_out);
#define TFB_GO(KERN, blocks) tfb::launch_k_rows(rows, KERN, blocks, 256, 0, st, X, R, W, B, Y, Ho, rstd, mean, rows, H, eps)
  const int warps8 = (rows + 7) / 8;
  if (H <= 512) TFB_GO((norm_fwd_kernel<2, LN>), warps8);
  else if (H <= 1024) TFB_GO((norm_fwd_kernel<4, LN>), warps8);
  else if (H <= 2048) TFB_GO((norm_fwd_rowblock_kernel<1, LN>), rows);
  else if (H <= 4096) TFB_GO((norm_fwd_rowblock_kernel<2, LN>), rows);
  else TFB_GO((norm_fwd_rowblock_kernel<4, LN>), rows);
#undef TFB_GO
  return int(cudaGetLastError());
}

template <bool LN>
static int launch_bwd(const void* dy, const void* h, const void* w, const float* rstd, const float* mean,
                      const void* dres, void* dx, float* dw, float* db, int rows, int H, cudaStream_t st) {
  if (H % 8 || H > 8192) return TFB_ERR_ARG;
  auto DY = static_cast<const __nv_bfloat16*>(dy);
  auto Hh = static_cast<const __nv_bfloat16*>(h);
  auto W = static_cast<const __nv_bfloat16*>(w);
  auto DR = static_cast<const __nv_bfloat16*>(dres);
  auto DX = static_cast<__nv_bfloat16*>(dx);
#define TFB_GO(NC, WIDE, blocks) \
  tfb::launch_k(norm_bwd_kernel<NC, LN, WIDE>, blocks, 256, size_t(H) * (WIDE ? 4 : 32), st, DY, Hh, W, rstd, mean, DR, DX, dw, db, rows, H)
  // blocks that stay for many rows: each adds one atomic per column of dw at its end
  const int warps8 = min((rows + 7) / 8, sm_count() * 4);
  if (H <= 512) TFB_GO(2, false, warps8);
  else if (H <= 1024) TFB_GO(4, false, warps8);
  else if (H <= 2048) TFB_GO(1, true, min(rows, sm_count() * 4));
  else if (H <= 4096) TFB_GO(2, true, min(rows, sm_count() * 2));
  else TFB_GO(4, true, min(rows, sm_count()));
#undef TFB_GO
  return int(cudaGetLastError());
}

}  // namespace tfb

// y = rmsnorm(x + res) * w; h_out (optional) receives x + res; rstd [rows] fp32 is saved for backward.
TFB_API int tfb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out, float* rstd, int rows,
                            int H, float eps, void* stream) {
  return tfb::launch_fwd<false>(x, res, w, nullptr, y, h_out, rstd, nullptr, rows, H, eps,
                                static_cast<cudaStream_t>(stream));
}
// dx = d rmsnorm / d h (+ dres); dw (fp32) accumulates.
TFB_API int tfb_rmsnorm_bwd(const void* dy, const void* h, const void* w, const float* rstd, const void* dres, void* dx,
                            float* dw, int rows, int H, void* stream) {
  return tfb::launch_bwd<false>(dy, h, w, rstd, nullptr, dres, dx, dw, nullptr, rows, H,
                                static_cast<cudaStream_t>(stream));
}
TFB_API int tfb_layernorm_fwd(const void* x, const void* res, const void* w, const void* b, void* y, void* h_out,
                              float* rstd, float* mean, int rows, int H, float eps, void* stream) {
  return tfb::launch_fwd<true>(x, res, w, b, y, h_out, rstd, mean, rows, H, eps, static_cast<cudaStream_t>(stream));
}
TFB_API int tfb_layernorm_bwd(const void* dy, const void* h, const void* w, const float* rstd, const float* mean,
                              const void* dres, void* dx, float* dw, float* db, int rows, int H, void* stream) {
  return tfb::launch_bwd<true>(dy, h, w, rstd, mean, dres, dx, dw, db, rows, H, static_cast<cudaStream_t>(stream));
}
// out [N] fp32 += column sums of x [rows, N] bf16 (row pitch ldx); N and ldx multiples of 8, x aligned to 16 bytes.
TFB_API int tfb_col_sum(const void* x, long long ldx, float* out, int rows, int N, void* stream) {
  using namespace tfb;
  if (rows < 0 || N <= 0 || N % 8 || ldx % 8 || (reinterpret_cast<uintptr_t>(x) & 15)) return TFB_ERR_ARG;
  if (rows == 0) return TFB_OK;
  auto X = static_cast<const __nv_bfloat16*>(x);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int gx = (N + 63) / 64;
  // one block per 64 columns while its few turns take less time than a cluster's meeting (512 x 768 2.9 us against 2.8, 131 x 768 2.2
  // against 2.7); clusters of four where their number is large (8192 x 6144 18 us against 21); more in flight where it is small (16384 x 768 8
  // against 10)
#define TFB_GO(BLOCKS, FLIGHT) tfb::launch_k(col_sum_kernel<BLOCKS, FLIGHT>, dim3(gx, BLOCKS), 256, 0, st, X, ldx, out, rows, N)
  if (rows <= 512) TFB_GO(1, 8);
  else if (gx > 64) TFB_GO(4, 8);
  else if (gx > 16) TFB_GO(8, 8);
  else TFB_GO(8, 16);
#undef TFB_GO
  return int(cudaGetLastError());
}
