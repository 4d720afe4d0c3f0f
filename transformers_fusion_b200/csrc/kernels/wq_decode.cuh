// Packed weight formats (see gemm_wq.cu for the layout): codes of a staged tile -> bf16 values in registers.
#pragma once
#include <cuda_fp16.h>

#include "tfb_ptx.cuh"

namespace tfb {

__host__ __device__ constexpr int wq_row_bytes(int fmt) { return fmt == 0 || fmt == 2 ? 64 : (fmt == 4 ? 16 : 32); }

__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint2 ld_shared_v2(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t ld_shared_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t ld_shared_u16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}
// two e4m3 bytes (low 16 bits of v) -> two floats, through the hardware e4m3x2 -> f16x2 conversion
__device__ __forceinline__ float2 e4m3x2_to_f2(uint32_t v) {
  uint32_t h2;
  const uint16_t lo = uint16_t(v);
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(lo));
  return __half22float2(*reinterpret_cast<const __half2*>(&h2));
}

// Loads the codes of 32 consecutive k of one weight row (half h of row r) from the staged blob into registers.
template <int FMT>
__device__ __forceinline__ void wq_load_codes(uint32_t raw, int r, int h, uint32_t (&w)[8]) {
  if (FMT == 0 || FMT == 2) {                      // 64-byte rows, 4 units of 16 bytes: units 2h, 2h + 1
    const uint4 a = ld_shared_v4(raw + ((2 * h) * 128 + r) * 16), b = ld_shared_v4(raw + ((2 * h + 1) * 128 + r) * 16);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
  } else if (FMT == 1 || FMT == 3) {               // 32-byte rows, 2 units of 16 bytes: unit h
    const uint4 a = ld_shared_v4(raw + (h * 128 + r) * 16);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
  } else {                                         // 16-byte rows, 2 units of 8 bytes: unit h
    const uint2 a = ld_shared_v2(raw + (h * 128 + r) * 8);
    w[0] = a.x; w[1] = a.y;
  }
}

// Decodes the 32 codes held in w, scales them and packs them as 16 bf16x2 words in k order.  `sbits` is the bf16 scale.
// Every path yields exactly round_to_bf16(code_value * scale), the value the fp32 oracle computes:
//   int8     the byte (biased by 128) is placed in byte 1 of 0x47000000, which reads as the float 2^15 + u; one FMA with
//            the scale and the constant -(2^15 + 128) * scale (exact: 257 * 128 times an 8-bit mantissa) gives b * scale
//   int4 / ternary   the code is OR-ed into the bf16 128.0 (0x4300 | u = 128 + u exactly), a packed bf16 subtract removes
//            128 + zero_point and a packed bf16 multiply applies the scale: two values per instruction, no final pack
template <int FMT>
__device__ __forceinline__ void wq_convert(const uint32_t (&w)[8], uint32_t sbits, uint32_t (&o)[16]) {
  const float s = __uint_as_float(sbits << 16);
  const uint32_t s2u = sbits | (sbits << 16);
  const __nv_bfloat162 s2 = *reinterpret_cast<const __nv_bfloat162*>(&s2u);
  auto bf2 = [&](uint32_t magic_or_codes, uint32_t offset_bits) -> uint32_t {
    const __nv_bfloat162 v = __hmul2(__hsub2(*reinterpret_cast<const __nv_bfloat162*>(&magic_or_codes),
                                             *reinterpret_cast<const __nv_bfloat162*>(&offset_bits)), s2);
    return *reinterpret_cast<const uint32_t*>(&v);
  };
  if (FMT == 0) {
    const float c = -32896.f * s;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t x = w[i] ^ 0x80808080u;
      const float f0 = fmaf(__uint_as_float(__byte_perm(x, 0x47000000u, 0x7504)), s, c);
      const float f1 = fmaf(__uint_as_float(__byte_perm(x, 0x47000000u, 0x7514)), s, c);
      const float f2 = fmaf(__uint_as_float(__byte_perm(x, 0x47000000u, 0x7524)), s, c);
      const float f3 = fmaf(__uint_as_float(__byte_perm(x, 0x47000000u, 0x7534)), s, c);
      o[2 * i] = pack_bf16(f0, f1);
      o[2 * i + 1] = pack_bf16(f2, f3);
    }
  } else if (FMT == 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) o[4 * i + j] = bf2(((w[i] >> (4 * j)) & 0x000F000Fu) | 0x43004300u, 0x43084308u);
    }
  } else if (FMT == 2) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 a = e4m3x2_to_f2(w[i]), b = e4m3x2_to_f2(w[i] >> 16);
      o[2 * i] = pack_bf16(a.x * s, a.y * s);
      o[2 * i + 1] = pack_bf16(b.x * s, b.y * s);
    }
  } else if (FMT == 3) {
    // e2m1 nibble s|ee|m placed as an fp16 with exponent field ee and top mantissa bit m is the value / 2^14
    // (zero, the subnormal 0.5 and the normals alike), so one multiply by 2^14 * scale finishes the job
    const float s14 = s * 16384.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t y = (w[i] >> (4 * j)) & 0x000F000Fu;
        const uint32_t h2 = ((y & 0x00070007u) << 9) | ((y & 0x00080008u) << 12);
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h2));
        o[4 * i + j] = pack_bf16(f.x * s14, f.y * s14);
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) o[8 * i + j] = bf2(((w[i] >> (2 * j)) & 0x00030003u) | 0x43004300u, 0x43014301u);
    }
  }
}

}  // namespace tfb
