// The chunkwise recurrences with head sizes of 128 on the 5th-generation tensor cores (dz_recurrent_tc.cu).
#pragma once

#include "dz_elem.cuh"

namespace dz {

struct RecurrentParams {
  const void* x;                         // rows [q | k | v | g], heads * 128 columns each
  int64_t row_stride;
  int rows;
  int k_off, v_off, g_off;
  void* out;                             // [rows, heads * 128]
  float* S;                              // pool [slots, heads, 128, 128]
  const int* slots;
  const int* q_starts;
  const int* ctx_lens;
  int heads;
  int* status;                           // first error: the first word of the call's workspace
  // matrix memory: gates, denominator, head norm and output gate
  const float* pre_if;                   // [rows, 2 heads]
  const float* b_if;
  float cap, scale;
  float *n, *m;
  const float* norm_w;
  float eps;
  // constant decay: the output before the norm goes to `out`
  const float* powers;                   // [heads, 65] w^0 ... w^64
};

constexpr size_t kRecStatusBytes = 256;  // workspace of a chunkwise call: [status word | tickets]

int launch_recurrent_tc(const RecurrentParams& p, bool matrix_memory, int dtype, int num_seqs, cudaStream_t st);

__device__ __forceinline__ float log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float soft_cap(float x, float cap) { return cap * tanhf(x / cap); }
// Whether both of a pair are at least -40 (a NaN is not).
template <typename T> __device__ __forceinline__ bool above_m40(uint32_t w);
template <> __device__ __forceinline__ bool above_m40<__half>(uint32_t w) {
  return __hbge2(*reinterpret_cast<__half2*>(&w), __float2half2_rn(-40.f));
}
template <> __device__ __forceinline__ bool above_m40<__nv_bfloat16>(uint32_t w) {
  return __hbge2(*reinterpret_cast<__nv_bfloat162*>(&w), __float2bfloat162_rn(-40.f));
}
// SiLU of eight values.  Two share a reciprocal, the special function unit being the bound.  Below -40, where the product
// of two denominators may overflow, and with a NaN, which would reach its neighbour, each divides by its own.
template <typename T> __device__ __forceinline__ uint4 silu8(const uint4& v) {
  uint32_t w[4] = {v.x, v.y, v.z, v.w};
  if (above_m40<T>(v.x) && above_m40<T>(v.y) && above_m40<T>(v.z) && above_m40<T>(v.w)) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = Cvt<T>::up(w[j]);
      const float a = 1.f + __expf(-f.x), b = 1.f + __expf(-f.y), r = __fdividef(1.f, a * b);
      w[j] = Cvt<T>::down(f.x * (r * b), f.y * (r * a));
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = Cvt<T>::up(w[j]);
      w[j] = Cvt<T>::down(__fdividef(f.x, 1.f + __expf(-f.x)), __fdividef(f.y, 1.f + __expf(-f.y)));
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

}  // namespace dz
