// Products of few rows with packed weights: out[M, N] = x[M, K] . dequant(W)[N, K]^T + bias + residual, M <= 16, formats and layout of
// gemm_wq.cu.  The codes go from global memory to registers, become bf16 there and are the A operand of mma.sync at once: a lane owns
// 16 consecutive k of a row in every k-block of 64 (its quarter of the row's unit-major codes) and calls them the k slots of four
// consecutive steps, for the weights and for x alike.  No ring, no barrier, no second kernel: eight warps take the k-blocks of 16 or 32
// weight rows in turn and meet once in shared memory.  The codes of the next k-block are in flight behind the arithmetic of this one;
// those of the first are fetched before the previous kernel of the stream has ended where the weights do not change (w_static).
//
// What bounds it: the stream at 8 bits, the decoding at 4; from 9 rows on also what every block reads of x.  The tensor-memory form of
// gemm_rows.cu hands every k-block through five barriers and takes 0.45 us per 128 x 64 codes and SM whatever the format.  us, that form ->
// this, int8: 28672 x 4096 at 1 / 8 / 16 rows 49.0 / 48.9 / 49.0 -> 33.1 / 33.8 / 45.8 (117 MB: 18), 4096 x 14336 28.1 / 28.1 / 28.1 -> 22.4 /
// 23.1 / 32.0, 6144 x 4096 16.0 / 16.1 / 16.1 -> 10.0 / 9.9 / 12.9, 4096 x 4096 13.1 -> 7.6 / 7.8 / 10.0; int4 28672 x 4096 at 8 rows 47.3 -> 24.1;
// at 32 rows it was no faster (28672 x 4096 55.4 against 50.9).
#include "tfb_host.h"
#include "tfb_mma.cuh"
#include "tfb_ptx.cuh"
#include "wq_decode.cuh"

namespace tfb {

struct SkinnyWqArgs {
  const __nv_bfloat16* x;
  long long ldx;
  const uint8_t* codes;
  const uint16_t* scales;
  __nv_bfloat16* out;
  long long ldo;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  long long ldr;
  int M, N, K, KB, group, w_static;
};

constexpr int SW_WARPS = 8;

template <int FMT, int RT>
struct WqRows {                          // a lane's 16 codes of 2 RT rows and their scales
  static constexpr int WORDS = FMT == 0 || FMT == 2 ? 4 : FMT == 4 ? 1 : 2;
  uint32_t w[2 * RT][WORDS];
  uint32_t s[2 * RT];
  // blob: codes of the 128-row tile at this k-block; row: first row of the lane inside it (rows row, row + 8, ...)
  __device__ __forceinline__ void load(const uint8_t* blob, const uint16_t* sc, int row, int q, int spr) {
#pragma unroll
    for (int i = 0; i < 2 * RT; ++i) {
      const int r = row + i * 8;
      if constexpr (FMT == 0 || FMT == 2) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(blob + (q * 128 + r) * 16));
        w[i][0] = v.x; w[i][1] = v.y; w[i][2] = v.z; w[i][3] = v.w;
      } else if constexpr (FMT == 4) {
        w[i][0] = __ldg(reinterpret_cast<const uint32_t*>(blob + ((q >> 1) * 128 + r) * 8 + (q & 1) * 4));
      } else {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(blob + ((q >> 1) * 128 + r) * 16 + (q & 1) * 8));
        w[i][0] = v.x; w[i][1] = v.y;
      }
      s[i] = __ldg(sc + r * spr + (spr == 2 ? q >> 1 : 0));
    }
  }
  __device__ __forceinline__ void decode(int i, uint32_t (&o)[16]) const {      // o[0..7]: pairs of consecutive k
    uint32_t c[8] = {};
#pragma unroll
    for (int j = 0; j < WORDS; ++j) c[j] = w[i][j];
    wq_convert<FMT>(c, s[i], o);
  }
};

template <int FMT, int RT, int NT>
__global__ void __launch_bounds__(SW_WARPS * 32) skinny_wq_kernel(const SkinnyWqArgs p) {
  __shared__ float red[SW_WARPS][RT * 16][NT * 8 + 1];
  constexpr int CODE_BYTES = 128 * wq_row_bytes(FMT);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int n0 = blockIdx.x * RT * 16, spr = 64 / p.group, row = (n0 & 127) + g;
  const uint8_t* blob = p.codes + (long long)(n0 >> 7) * p.KB * CODE_BYTES;
  const uint16_t* sc = p.scales + (long long)(n0 >> 7) * p.KB * 128 * spr;
  float acc[RT][NT][4];
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[r][t][0] = acc[r][t][1] = acc[r][t][2] = acc[r][t][3] = 0.f;
  WqRows<FMT, RT> next;
  int kb = warp;
  auto fetch = [&](int k) { next.load(blob + (long long)k * CODE_BYTES, sc + (long long)k * 128 * spr, row, q, spr); };
  if (p.w_static && kb < p.KB) fetch(kb);
  pdl_sync();
  if (!p.w_static && kb < p.KB) fetch(kb);
  for (; kb < p.KB; kb += SW_WARPS) {
    const WqRows<FMT, RT> cur = next;
    if (kb + SW_WARPS < p.KB) fetch(kb + SW_WARPS);
    const int k = kb * 64 + q * 16;
    uint32_t xv[NT][8];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const bool live = t * 8 + g < p.M;
      const __nv_bfloat16* xr = p.x + (t * 8 + g) * p.ldx + k;
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
      const uint4 a = live && k < p.K ? *reinterpret_cast<const uint4*>(xr) : zero;
      const uint4 b = live && k + 8 < p.K ? *reinterpret_cast<const uint4*>(xr + 8) : zero;
      xv[t][0] = a.x; xv[t][1] = a.y; xv[t][2] = a.z; xv[t][3] = a.w;
      xv[t][4] = b.x; xv[t][5] = b.y; xv[t][6] = b.z; xv[t][7] = b.w;
    }
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      uint32_t lo[16], hi[16];                        // rows g and g + 8 of the tile
      cur.decode(2 * r, lo);
      cur.decode(2 * r + 1, hi);
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const uint32_t a[4] = {lo[2 * s], hi[2 * s], lo[2 * s + 1], hi[2 * s + 1]};
#pragma unroll
        for (int t = 0; t < NT; ++t) mma_bf16(acc[r][t], a, xv[t][2 * s], xv[t][2 * s + 1]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) red[warp][r * 16 + g + (e >> 1) * 8][t * 8 + q * 2 + (e & 1)] = acc[r][t][e];
  __syncthreads();
  for (int i = threadIdx.x; i < RT * 16 * NT * 8; i += SW_WARPS * 32) {
    const int m = i / (RT * 16), n = i % (RT * 16);
    if (m >= p.M || n0 + n >= p.N) continue;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < SW_WARPS; ++w) v += red[w][n][m];
    if (p.bias) v += __bfloat162float(p.bias[n0 + n]);
    if (p.residual) v += __bfloat162float(p.residual[m * p.ldr + n0 + n]);
    p.out[m * p.ldo + n0 + n] = __float2bfloat16(v);
  }
}

template <int FMT>
static void launch_skinny_wq(const SkinnyWqArgs& p, cudaStream_t st) {
  // 32 rows a block halve what is read of x; 16 where that would leave SMs with fewer than two blocks
  const bool two = p.N >= 2 * 32 * sm_count();
  const int blocks = (p.N + (two ? 31 : 15)) / (two ? 32 : 16);
#define TFB_GO(NT)                                                                                     \
  do {                                                                                                 \
    if (two) launch_k_pdl(skinny_wq_kernel<FMT, 2, NT>, blocks, SW_WARPS * 32, 0, st, p);               \
    else launch_k_pdl(skinny_wq_kernel<FMT, 1, NT>, blocks, SW_WARPS * 32, 0, st, p);                   \
  } while (0)
  if (p.M <= 8) TFB_GO(1);
  else TFB_GO(2);
#undef TFB_GO
}

}  // namespace tfb

// x [M, ldx] bf16 (K a multiple of 8, rows on 16-byte boundaries), codes and scales tile-major with the rows padded to a multiple of 128 and
// Kw >= K entries, a multiple of 64.  bias [N], residual [M, ldr]: bf16 or null.  w_static: the kernel launched just before does not write the weights.
TFB_API int tfb_skinny_wq(const void* x, long long ldx, const void* codes, const void* scales, int fmt, int group, void* out, long long ldo, int M, int N,
                          int K, int Kw, const void* bias, const void* residual, long long ldr, int w_static, void* stream) {
  using namespace tfb;
  using bf16 = __nv_bfloat16;
  if (M <= 0 || M > 16 || N <= 0 || K <= 0 || K % 8 || ldx % 8 || (reinterpret_cast<uintptr_t>(x) & 15) || fmt < 0 || fmt > 4 ||
      (group != 32 && group != 64) || Kw % 64 || Kw < K || (reinterpret_cast<uintptr_t>(codes) & 15) || (reinterpret_cast<uintptr_t>(scales) & 1))
    return TFB_ERR_ARG;
  const SkinnyWqArgs p{static_cast<const bf16*>(x), ldx, static_cast<const uint8_t*>(codes), static_cast<const uint16_t*>(scales), static_cast<bf16*>(out),
                       ldo, static_cast<const bf16*>(bias), static_cast<const bf16*>(residual), ldr, M, N, K, Kw / 64, group, w_static};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (fmt) {
    case 0: launch_skinny_wq<0>(p, st); break;
    case 1: launch_skinny_wq<1>(p, st); break;
    case 2: launch_skinny_wq<2>(p, st); break;
    case 3: launch_skinny_wq<3>(p, st); break;
    default: launch_skinny_wq<4>(p, st); break;
  }
  return int(cudaGetLastError());
}
