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
// SiLU of eight values.  Two share a reciprocal, the special function unit being the bound; below -40, where it is
// less than 2e-16, it is zero, and the product of two denominators stays finite.
template <typename T> __device__ __forceinline__ uint4 silu8(const uint4& v) {
  uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = Cvt<T>::up(w[j]);
    const float a = 1.f + __expf(-fmaxf(f.x, -40.f)), b = 1.f + __expf(-fmaxf(f.y, -40.f));
    const float r = __fdividef(1.f, a * b);
    w[j] = Cvt<T>::down((f.x < -40.f ? 0.f : f.x) * (r * b), (f.y < -40.f ? 0.f : f.y) * (r * a));
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

}  // namespace dz
