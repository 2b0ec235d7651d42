// Expansion of packed codes to the 16-bit integers (code - zero) the delta MMAs multiply with.
#pragma once

#include <cuda_bf16.h>

#include "dz_common.cuh"

namespace dz {

// The pair (code_lo - zero, code_hi - zero) as fp16 (DT = 0) or bf16 (DT = 1) from the
// BITS-wide fields at bit P of both half-words of w, without shifting: OR-ing the field
// into the mantissa of 2^(m-P) (m = 10 / 7 mantissa bits) gives 2^(m-P) + code (the field
// has weight 2^-P there), and one subtraction of 2^(m-P) + zero leaves the exact small
// integer.  Needs P + BITS <= m.
template <int BITS, int P, int DT>
__device__ __forceinline__ uint32_t code_pair(uint32_t w) {
  constexpr uint32_t kMant = DT == 0 ? 10u : 7u;
  constexpr uint32_t kExpBias = DT == 0 ? 15u : 127u;
  static_assert(P + BITS <= (DT == 0 ? 10 : 7), "field must sit inside the mantissa");
  constexpr uint32_t kMask = ((((1u << BITS) - 1u) << P)) * 0x00010001u;
  constexpr uint32_t kMagic = ((kExpBias + kMant - P) << kMant) * 0x00010001u;
  constexpr uint32_t kBiasBits =
      (((kExpBias + kMant - P) << kMant) | ((1u << (BITS - 1)) << P)) * 0x00010001u;
  uint32_t t;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(t) : "r"(w), "n"(kMask), "n"(kMagic));
  uint32_t b = kBiasBits;
  if (DT == 0) {
    __half2 hv = __hsub2(*reinterpret_cast<__half2*>(&t), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&hv);
  } else {
    __nv_bfloat162 hv =
        __hsub2(*reinterpret_cast<__nv_bfloat162*>(&t), *reinterpret_cast<__nv_bfloat162*>(&b));
    return *reinterpret_cast<uint32_t*>(&hv);
  }
}
// the 8 (4-bit) or 16 (2-bit) kept values of one packed word -> 4 / 8 pairs
template <int DT>
__device__ __forceinline__ void expand_word4(uint32_t w, uint32_t* o) {
  if (DT == 0) {
    const uint32_t s = w >> 8;
    o[0] = code_pair<4, 0, 0>(w);
    o[1] = code_pair<4, 4, 0>(w);
    o[2] = code_pair<4, 0, 0>(s);
    o[3] = code_pair<4, 4, 0>(s);
  } else {   // 7 mantissa bits hold one nibble at a time
    o[0] = code_pair<4, 0, 1>(w);
    o[1] = code_pair<4, 0, 1>(w >> 4);
    o[2] = code_pair<4, 0, 1>(w >> 8);
    o[3] = code_pair<4, 0, 1>(w >> 12);
  }
}
template <int DT>
__device__ __forceinline__ void expand_word2(uint32_t w, uint32_t* o) {
  if (DT == 0) {
    const uint32_t s = w >> 10;
    o[0] = code_pair<2, 0, 0>(w);
    o[1] = code_pair<2, 2, 0>(w);
    o[2] = code_pair<2, 4, 0>(w);
    o[3] = code_pair<2, 6, 0>(w);
    o[4] = code_pair<2, 8, 0>(w);
    o[5] = code_pair<2, 0, 0>(s);
    o[6] = code_pair<2, 2, 0>(s);
    o[7] = code_pair<2, 4, 0>(s);
  } else {
    const uint32_t s = w >> 6, u = w >> 12;
    o[0] = code_pair<2, 0, 1>(w);
    o[1] = code_pair<2, 2, 1>(w);
    o[2] = code_pair<2, 4, 1>(w);
    o[3] = code_pair<2, 0, 1>(s);
    o[4] = code_pair<2, 2, 1>(s);
    o[5] = code_pair<2, 4, 1>(s);
    o[6] = code_pair<2, 0, 1>(u);
    o[7] = code_pair<2, 2, 1>(u);
  }
}

}  // namespace dz
