// Pieces of the feature map Phi shared by the tensor-memory kernels: rows of a token tile and products of two 8-wide blocks.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace fm {
namespace tc {

__device__ __forceinline__ uint32_t hmul2_u32(uint32_t a, uint32_t b) {
  __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<uint32_t*>(&r);
}

// Row `row` of a 128-byte-swizzled tile with 128-byte rows: 16-byte chunk cc.
__device__ __forceinline__ uint4 sw_chunk(const uint8_t* tile, int row, int cc) {
  return *reinterpret_cast<const uint4*>(tile + row * 128 + ((cc ^ (row & 7)) << 4));
}

// 64 features x[8a+mi] * x[8b+ri] of token row l of a raw [token][64] tile -> 32 packed registers (register 4 mi + j holds
// ri = 2j, 2j + 1).  `dbl`: x[8a+mi] is doubled (exact), for an off-diagonal unit.
__device__ __forceinline__ void apply_pair_slab(uint32_t (&r)[32], const uint8_t* raw, int l, int a, int b, bool dbl) {
  uint4 xa4 = sw_chunk(raw, l, a);
  const uint4 xb4 = sw_chunk(raw, l, b);
  if (dbl) {
    const uint32_t two = 0x40004000u;  // bf16x2 (2, 2)
    xa4.x = hmul2_u32(xa4.x, two); xa4.y = hmul2_u32(xa4.y, two); xa4.z = hmul2_u32(xa4.z, two); xa4.w = hmul2_u32(xa4.w, two);
  }
  const uint32_t xa[4] = {xa4.x, xa4.y, xa4.z, xa4.w};
#pragma unroll
  for (int mi = 0; mi < 8; ++mi) {
    const uint32_t pr = xa[mi >> 1];
    const uint32_t bc = (mi & 1) ? __byte_perm(pr, pr, 0x3232) : __byte_perm(pr, pr, 0x1010);
    r[4 * mi + 0] = hmul2_u32(bc, xb4.x);
    r[4 * mi + 1] = hmul2_u32(bc, xb4.y);
    r[4 * mi + 2] = hmul2_u32(bc, xb4.z);
    r[4 * mi + 3] = hmul2_u32(bc, xb4.w);
  }
}

}  // namespace tc
}  // namespace fm
