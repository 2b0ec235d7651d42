// Compressor kernels: the steps of the reference's offline compression that are not plain
// dense linear algebra, for one linear layer's delta W [N, K] (float32):
//
//   sparsegpt_block_kernel   one 128-column block of SparseGPT.fasterprune with prunen:prunem =
//                            2:4 (deltazip/core/sparsegpt.py:98-146): per group of four columns
//                            the two entries with the smallest w^2 / Hinv_ii^2 are pruned, every
//                            entry goes through the symmetric per-row quantiser
//                            (deltazip/core/quant.py:9-18), and the quantisation / pruning error
//                            of column i is fed forward into the block's later columns through
//                            row i of the upper Cholesky factor of H^-1 (:139-141).  Rows of W are
//                            independent; eight lanes own one row, a group of four columns belongs to one lane, and
//                            the block of Hinv sits in shared memory.
//                            Outputs Q (quantised block) and Err ((w - q) / Hinv_ii per column),
//                            from which the caller forms the update of the columns behind the
//                            block, W[:, i2:] -= Err @ Hinv[i1:i2, i2:] (:146), a plain GEMM.
//   triangular_inverse_kernel  the 128-wide diagonal blocks of an upper triangular matrix inverted, all in one launch.
//   split_update_kernel      the operands of that GEMM as sums of three bf16 numbers each, for tensor cores.
//   pack_gptq_kernel         QuantLinear.pack (deltazip/nn_modules/qlinear.py:83-183) for one
//                            quantisation group: codes round((W + zero*scale) / fp16(scale))
//                            packed along K into int32 words, zero points (minus one) packed
//                            along N, scales as fp16 -- the GPTQ-layout tensors the reference
//                            stores, bit for bit.
//
// Arithmetic follows the reference's float32 operations one by one (IEEE division, products and
// differences rounded separately, round-half-even), so that results can be compared bit for bit
// with the reference run on the same inputs wherever no long accumulation is involved.
#include <cuda_bf16.h>

#include "dz_common.cuh"

namespace dz {
namespace {

constexpr int kCBlock = 128;

// a / b correctly rounded for many a and one b, y = 1 / b correctly rounded: two corrections of a * y by the exact remainder.
// After the first q is within one unit of the last place, and the second then rounds correctly (Markstein, IBM J. Res. Dev.
// 34, 1990; Muller et al., Handbook of Floating-Point Arithmetic, 4.7).  That holds while no remainder underflows and
// nothing overflows: `ok` of the operands, which the caller has to look at before it uses the quotients.  (A zero's sign is
// not kept.)
struct Divisor {
  float b, y;
};
__device__ __forceinline__ bool divides(float b) { return fabsf(b) > 1e-12f && fabsf(b) < 1e8f; }
__device__ __forceinline__ bool divided(float a) { return fabsf(a) < 1e24f && (fabsf(a) > 1e-28f || a == 0.f); }
__device__ __forceinline__ Divisor divisor(float b) { return Divisor{b, __fdiv_rn(1.f, b)}; }
template <bool FAST>
__device__ __forceinline__ float quotient(float a, const Divisor& d, bool& ok) {
  if (!FAST) return __fdiv_rn(a, d.b);
  ok = ok && divided(a);
  float q = __fmul_rn(a, d.y);
  q = __fmaf_rn(__fmaf_rn(-q, d.b, a), d.y, q);
  return __fmaf_rn(__fmaf_rn(-q, d.b, a), d.y, q);
}

// One group of four columns of a row: ranked by w^2 / d^2, the two smallest pruned (ties: the lower column first, as a stable
// selection does), each quantised (quant.py:9-18: q = clamp(round(w / scale) + zero, 0, maxq), scale * (q - zero)) and its
// error fed forward to the group's later columns.  False: a division was outside the range of the quick form.
struct Group {
  float q[4], err[4], loss[4];
};
template <bool FAST>
__device__ __forceinline__ bool settle_group(const float (&w0)[4], const float (&h)[4][4], const Divisor (&diag)[4],
                                             const Divisor (&square)[4], const Divisor& scale, float zero, float maxq, Group& g) {
  bool ok = true;
  float w[4], rank[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    w[e] = w0[e];
    rank[e] = quotient<FAST>(__fmul_rn(w[e], w[e]), square[e], ok);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    int smaller = 0;
#pragma unroll
    for (int o = 0; o < 4; ++o) smaller += (rank[o] < rank[e] || (rank[o] == rank[e] && o < e)) ? 1 : 0;
    const float code = rintf(quotient<FAST>(smaller < 2 ? 0.f : w[e], scale, ok)) + zero;
    g.q[e] = __fmul_rn(scale.b, fminf(fmaxf(code, 0.f), maxq) - zero);
    const float diff = w[e] - g.q[e];
    g.err[e] = quotient<FAST>(diff, diag[e], ok);
    g.loss[e] = __fmul_rn(diff, diff);
    // W1[:, i:] -= err * Hinv1[i, i:] (the column itself is not read again)
#pragma unroll
    for (int o = e + 1; o < 4; ++o) w[o] = __fsub_rn(w[o], __fmul_rn(g.err[e], h[e][o]));
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) g.loss[e] = quotient<FAST>(g.loss[e], square[e], ok);
  return ok;
}

// W1: [N, ldw] block start (column i1), count <= 128 columns.  Lane t of a row's T holds the groups G = T J + t: columns
// 4 T J + 4 t + 0..3.  The chain -- rank, quantise, error, next column -- stays inside the lane that owns a group, the rows
// of a warp side by side; its four errors then go to the row's other lanes, which take them off their later groups.
// `w[0]` is the group of the current J (registers move down by one a J, so that the loop over the 32 groups is one body
// of code).  Bound by the latency of that chain, which the divisions by the grid and by the diagonal make up: CUDA's
// own, whose slow path a pruned entry's zero takes, cost 51 us a block of 4096 rows (T = 4), the quick form with a test for
// each 43, with one test a group 33, and 31 with T = 8, two warps to a scheduler (T = 16: 37; a warp to a row, 73).
constexpr int kRowLanes = 8, kBlockRows = 32;   // rows of a block: one block an SM for 4096 rows, three fit
__global__ void __launch_bounds__(kRowLanes * kBlockRows)
sparsegpt_block_kernel(const float* W, long long ldw, const float* __restrict__ hinv, long long ldh,
                       const float* __restrict__ scale, const float* __restrict__ zero, float maxq, int N, int count,
                       float* Q, long long ldq, float* __restrict__ Err, long long lde, float* __restrict__ loss) {
  extern __shared__ __align__(16) float s_h[];             // [128][128]; what lies below a group of four is not read
  if ((ldh & 3) == 0 && ((size_t)hinv & 15) == 0) {
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(s_h);
    for (int i = threadIdx.x; i < kCBlock * kCBlock / 4; i += blockDim.x) {
      const int r = i / (kCBlock / 4), c = i % (kCBlock / 4) * 4;
      if (c + 3 >= r && c < count)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(base + i * 16), "l"(hinv + (size_t)r * ldh + c) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    for (int i = threadIdx.x; i < kCBlock * kCBlock; i += blockDim.x) {
      const int r = i / kCBlock, c = i % kCBlock;
      if (c >= r && c < count) s_h[i] = hinv[(size_t)r * ldh + c];
    }
  }
  __syncthreads();
  constexpr int T = kRowLanes, kGroups = kCBlock / (4 * T);
  const int t = threadIdx.x & (T - 1);
  const int place = blockIdx.x * kBlockRows + threadIdx.x / T;
  const bool live = place < N;
  const size_t row = live ? place : N - 1;                 // (whole warps take part in the exchange)
  const Divisor sc = divisor(scale[row]);
  const float zp = zero[row];
  float w[kGroups][4];
#pragma unroll
  for (int j = 0; j < kGroups; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = 4 * T * j + 4 * t + e;
      w[j][e] = c < count ? W[row * ldw + c] : 0.f;
    }
  float row_loss = 0.f;
  for (int J = 0; 4 * T * J < count; ++J) {
    const int c0 = 4 * T * J + 4 * t;                      // this lane's group
    float hb[4][4];
    Divisor diag[4], square[4];
    bool ranged = divides(sc.b);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 v = *reinterpret_cast<const float4*>(s_h + (c0 + e) * kCBlock + c0);
      hb[e][0] = v.x; hb[e][1] = v.y; hb[e][2] = v.z; hb[e][3] = v.w;
      diag[e] = divisor(hb[e][e]);
      square[e] = divisor(__fmul_rn(hb[e][e], hb[e][e]));
      ranged = ranged && divides(diag[e].b) && divides(square[e].b);
    }
    for (int owner = 0; owner < T && 4 * T * J + 4 * owner < count; ++owner) {
      Group g;
      // (every lane goes through it; the owner's results count)
      if (!(settle_group<true>(w[0], hb, diag, square, sc, zp, maxq, g) && ranged) && t == owner)
        settle_group<false>(w[0], hb, diag, square, sc, zp, maxq, g);
      float e4[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) e4[e] = __shfl_sync(0xffffffffu, g.err[e], owner, T);
      if (t == owner && live) {
        row_loss += (g.loss[0] + g.loss[1]) + (g.loss[2] + g.loss[3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          Q[row * ldq + c0 + e] = g.q[e];
          Err[row * lde + c0 + e] = g.err[e];
        }
      }
      const float* h = s_h + (4 * T * J + 4 * owner) * kCBlock + c0;
#pragma unroll
      for (int j = 0; j < kGroups; ++j) {
        if (4 * T * (J + j) >= count) break;
        if (j == 0 && t <= owner) continue;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 v = *reinterpret_cast<const float4*>(h + e * kCBlock + 4 * T * j);
          w[j][0] = __fsub_rn(w[j][0], __fmul_rn(e4[e], v.x));
          w[j][1] = __fsub_rn(w[j][1], __fmul_rn(e4[e], v.y));
          w[j][2] = __fsub_rn(w[j][2], __fmul_rn(e4[e], v.z));
          w[j][3] = __fsub_rn(w[j][3], __fmul_rn(e4[e], v.w));
        }
      }
    }
#pragma unroll
    for (int j = 0; j + 1 < kGroups; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) w[j][e] = w[j + 1][e];
  }
#pragma unroll
  for (int o = 1; o < T; o *= 2) row_loss += __shfl_xor_sync(0xffffffffu, row_loss, o);
  if (t == 0 && live && loss) loss[row] += row_loss * 0.5f;
}

// Diagonal blocks of 128 (the last may be smaller) of an upper triangular matrix inverted into `X`, whose other entries are
// left alone.  Eight lanes own a column of the inverse, lane t the rows 8 m + t, and go up it: an entry once known is
// handed to the other lanes, which take its share off their rows' sums -- sixteen independent sums a lane, so that a
// step's latency is one exchange and one multiply-add, not a chain of them (four lanes with a sum each: 122 us for the 32
// blocks of 4096 columns).  `acc[0]` belongs to the current m; sums move down by one each eight rows.
constexpr int kInvLanes = 8, kInvRows = kCBlock / kInvLanes, kInvLd = kCBlock + 2;     // (eight rows: eight pairs of banks)
__global__ void __launch_bounds__(kInvLanes * kCBlock)
triangular_inverse_kernel(const double* __restrict__ R, long long ldr, int k, double* __restrict__ X, long long ldx) {
  extern __shared__ double s[];                            // R, and below its diagonal the inverse, transposed
  __shared__ double s_diag[kCBlock];                       // diagonal of the inverse
  const int b0 = blockIdx.x * kCBlock, n = min(kCBlock, k - b0);
  for (int i = threadIdx.x; i < kCBlock * kCBlock; i += blockDim.x) {
    const int r = i / kCBlock, c = i % kCBlock;
    if (c >= r) s[r * kInvLd + c] = c < n ? R[(size_t)(b0 + r) * ldr + b0 + c] : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < kCBlock) s_diag[threadIdx.x] = (int)threadIdx.x < n ? 1.0 / s[threadIdx.x * (kInvLd + 1)] : 0.0;
  __syncthreads();
  const int t = threadIdx.x & 7, col = threadIdx.x >> 3;
  double acc[kInvRows];
#pragma unroll
  for (int m = 0; m < kInvRows; ++m) acc[m] = 0.0;
  for (int M = kInvRows - 1; M >= 0; --M) {
    for (int o = kInvLanes - 1; o >= 0; --o) {
      const int l = 8 * M + o;
      double x = l == col ? s_diag[l] : acc[0] * s_diag[l];          // (of lane o; zero below the diagonal: no sum yet)
      x = __shfl_sync(0xffffffffu, x, o, kInvLanes);
      if (t == o && l < col) s[col * kInvLd + l] = x;
      if (t < o) acc[0] -= s[(8 * M + t) * kInvLd + l] * x;
#pragma unroll
      for (int m = 1; m < kInvRows; ++m) {
        if (m > M) break;
        acc[m] -= s[(8 * (M - m) + t) * kInvLd + l] * x;
      }
    }
#pragma unroll
    for (int m = 0; m + 1 < kInvRows; ++m) acc[m] = acc[m + 1];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n * n; i += blockDim.x) {
    const int r = i / n, c = i % n;
    X[(size_t)(b0 + r) * ldx + b0 + c] = c > r ? s[c * kInvLd + r] : c == r ? s_diag[r] : 0.0;
  }
}

// W -= E U on the tensor cores: a float is the sum of three bf16 numbers h + m + l (8 + 8 + 8 bits), and of the nine
// products the six of 2^-16 and more count, largest last: l h + m m + h l + m h + h m + h h is one bf16 GEMM with sums in 32
// bits over six times the columns.  Rows of A [n, 6 count] are [l m h m h h] of E, the rows of B [6 count, c]
// [h m l h m h] of U.  For a block of 128 columns the product's error against 64 bits is below that of a 32-bit GEMM (4096
// rows: 1.2e-7 and 2.0e-7 of its norm; over 512 columns it would not be: 4.7e-7 and 4.1e-7, sums being cut, not rounded).
// 4096 rows and 2048 columns behind the block: 55 us as a 32-bit GEMM, 16 so and 4 for this kernel, bound by its bytes.
//   Range.  bf16 has the exponents of a float, so below 2^-109 a third part loses bits, and infinities leave NaN in the
// others.  A row of E whose largest entry is outside [2^-64, 2^32], or not a number, is given zeros as operands and taken off
// its row of W here, in 32 bits.  Of the other rows the parts' absolute error, 2^-134, is 2^-70 of the largest entry, and U's,
// times E, below 2^-102.  A finite entry that rounds to infinity keeps the largest bf16 number as its first part.
__device__ __forceinline__ void split3(float x, __nv_bfloat16* v) {
  v[0] = __float2bfloat16_rn(x);
  if (__hisinf(v[0]) && fabsf(x) <= 3.4028235e38f) v[0] = __ushort_as_bfloat16(x > 0.f ? 0x7f7f : 0xff7f);
  const float r = x - __bfloat162float(v[0]);
  v[1] = __float2bfloat16_rn(r);
  v[2] = __float2bfloat16_rn(r - __bfloat162float(v[1]));
}
// four entries into their six places, `part_of` giving the part of each
template <typename F>
__device__ __forceinline__ void store_parts(const float (&x)[4], __nv_bfloat16* dst, long long step, F part_of) {
  __nv_bfloat16 v[4][3];
#pragma unroll
  for (int q = 0; q < 4; ++q) split3(x[q], v[q]);
#pragma unroll
  for (int p = 0; p < 6; ++p) {
    const int part = part_of(p);
    __nv_bfloat162 lo, hi;
    lo.x = v[0][part]; lo.y = v[1][part];
    hi.x = v[2][part]; hi.y = v[3][part];
    *reinterpret_cast<uint2*>(dst + p * step) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
  }
}
// A warp takes a row of E, then quads of U.  W (may be null: every row is split): [n, c], the columns behind the block.
__global__ void __launch_bounds__(256)
split_update_kernel(const float* __restrict__ E, long long lde, int n, int count, const float* __restrict__ U, long long ldu, int c,
                    float* W, long long ldw, __nv_bfloat16* __restrict__ A, __nv_bfloat16* __restrict__ B) {
  const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
  for (int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < n; row += warps) {
    const float* src = E + row * lde;
    bool in = true, large = false, any = false;
    if (W) {
      for (int i = lane; i < count; i += 32) {
        const float x = fabsf(src[i]);
        in = in && x <= 0x1p32f;                             // (false for a NaN)
        large = large || x >= 0x1p-64f;
        any = any || x != 0.f;
      }
      in = __all_sync(0xffffffffu, in) && (__any_sync(0xffffffffu, large) || !__any_sync(0xffffffffu, any));
    }
    for (int col = 4 * lane; col < count; col += 128) {
      float x[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) x[q] = in ? src[col + q] : 0.f;
      store_parts(x, A + (long long)row * 6 * count + col, count, [](int p) { return p == 0 ? 2 : p == 1 || p == 3 ? 1 : 0; });
    }
    if (!in)
      for (int j = lane; j < c; j += 32) {
        float sum = 0.f;
        for (int i = 0; i < count; ++i) sum = fmaf(src[i], U[i * ldu + j], sum);
        W[row * ldw + j] -= sum;
      }
  }
  const long long quads = c / 4, all = count * quads;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < all; i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / quads, col = i % quads * 4;
    float x[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) x[q] = U[row * ldu + col + q];
    store_parts(x, B + row * c + col, (long long)count * c, [](int p) { return p == 2 ? 2 : p == 1 || p == 4 ? 1 : 0; });
  }
}

// one thread per packed word: grid covers [K*bits/32, N]
__global__ void pack_gptq_kernel(const float* __restrict__ Wq, const float* __restrict__ scale,
                                 const float* __restrict__ zero, int N, int K, int bits,
                                 int32_t* __restrict__ qweight, int32_t* __restrict__ qzeros,
                                 __half* __restrict__ scales) {
  const int per = 32 / bits;
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  const int kw = blockIdx.y;
  if (n >= N) return;
  const float sc = scale[n], zp = zero[n];
  const __half sh = __float2half_rn(sc);
  const float scf = __half2float(sh);
  const float sz = __fmul_rn(zp, sc);
  uint32_t word = 0;
  for (int j = 0; j < per; ++j) {
    const float v = Wq[(size_t)n * K + (size_t)kw * per + j];
    const int code = (int)rintf(__fdiv_rn(v + sz, scf));
    word |= ((uint32_t)code) << (bits * j);
  }
  qweight[(size_t)kw * N + n] = (int32_t)word;
  if (kw == 0) {
    scales[n] = sh;
    if (n % per == 0) {
      uint32_t z = 0;
      for (int j = 0; j < per && n + j < N; ++j)
        z |= ((uint32_t)(zero[n + j] - 1.f)) << (bits * j);
      qzeros[n / per] = (int32_t)z;
    }
  }
}

// per-row symmetric grid (quant.py:48-86 with perchannel, sym, no mse): one warp per row
__global__ void find_params_kernel(const float* __restrict__ W, int N, int K, float maxq,
                                   float* __restrict__ scale, float* __restrict__ zero) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= N) return;
  float mn = 0.f, mx = 0.f;
  for (int c = lane; c < K; c += 32) {
    const float v = W[(size_t)row * K + c];
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if (lane == 0) {
    mx = fmaxf(fabsf(mn), mx);
    if (mn < 0.f) mn = -mx;
    if (mn == 0.f && mx == 0.f) { mn = -1.f; mx = 1.f; }
    scale[row] = __fdiv_rn(mx - mn, maxq);
    zero[row] = (maxq + 1.f) * 0.5f;
  }
}

}  // namespace
}  // namespace dz

using namespace dz;

extern "C" {

int dz_quant_find_params(const float* W, int N, int K, int bits, float* scale, float* zero, void* stream) {
  if (!W || !scale || !zero || N <= 0 || K <= 0) return DZ_ERR_INVALID_ARG;
  if (bits != 2 && bits != 4 && bits != 8) return DZ_ERR_SHAPE;
  find_params_kernel<<<(N + 7) / 8, 256, 0, (cudaStream_t)stream>>>(W, N, K, (float)((1 << bits) - 1), scale, zero);
  DZ_CUDA_OK(cudaGetLastError());
  return DZ_OK;
}

int dz_sparsegpt_block_strided(const float* W_block, int64_t ldw, const float* hinv_block, int64_t ldh,
                               const float* scale, const float* zero, int bits, int N, int count, float* Q,
                               int64_t ldq, float* Err, int64_t lde, float* loss, void* stream) {
  if (!W_block || !hinv_block || !scale || !zero || !Q || !Err) return DZ_ERR_INVALID_ARG;
  if (N <= 0 || count <= 0 || count > kCBlock || (count & 3) || ldq < count || lde < count) return DZ_ERR_SHAPE;
  if (bits != 2 && bits != 4 && bits != 8) return DZ_ERR_SHAPE;
  constexpr int kSmem = kCBlock * kCBlock * sizeof(float);
  DZ_CUDA_OK(cudaFuncSetAttribute(sparsegpt_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  sparsegpt_block_kernel<<<(N + kBlockRows - 1) / kBlockRows, kRowLanes * kBlockRows, kSmem, (cudaStream_t)stream>>>(
      W_block, ldw, hinv_block, ldh, scale, zero, (float)((1 << bits) - 1), N, count, Q, ldq, Err, lde, loss);
  DZ_CUDA_OK(cudaGetLastError());
  return DZ_OK;
}

int dz_sparsegpt_block(const float* W_block, int64_t ldw, const float* hinv_block, int64_t ldh,
                       const float* scale, const float* zero, int bits, int N, int count, float* Q,
                       float* Err, float* loss, void* stream) {
  return dz_sparsegpt_block_strided(W_block, ldw, hinv_block, ldh, scale, zero, bits, N, count, Q, count, Err, count,
                                    loss, stream);
}

int dz_triangular_inverse_blocks(const double* R, int64_t ldr, int k, double* X, int64_t ldx, void* stream) {
  if (!R || !X) return DZ_ERR_INVALID_ARG;
  if (k <= 0 || ldr < k || ldx < k) return DZ_ERR_SHAPE;
  constexpr int kSmem = kCBlock * kInvLd * sizeof(double);
  DZ_CUDA_OK(cudaFuncSetAttribute(triangular_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  triangular_inverse_kernel<<<(k + kCBlock - 1) / kCBlock, kInvLanes * kCBlock, kSmem, (cudaStream_t)stream>>>(R, ldr, k, X, ldx);
  DZ_CUDA_OK(cudaGetLastError());
  return DZ_OK;
}

int dz_split_update_rows(const float* E, int64_t lde, int n, int count, const float* U, int64_t ldu, int c, float* W, int64_t ldw,
                         void* A, void* B, void* stream) {
  if (!E || !U || !A || !B) return DZ_ERR_INVALID_ARG;
  if (n <= 0 || count <= 0 || c <= 0 || (count & 3) || (c & 3) || lde < count || ldu < c || (W && ldw < c)) return DZ_ERR_SHAPE;
  if (((uintptr_t)A | (uintptr_t)B) & 7) return DZ_ERR_ALIGNMENT;
  const long long quads = max((long long)n * 32, (long long)count * (c / 4));
  const int blocks = (int)min(quads / 256 + 1, 2048ll);
  split_update_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(E, lde, n, count, U, ldu, c, W, ldw, (__nv_bfloat16*)A,
                                                                (__nv_bfloat16*)B);
  DZ_CUDA_OK(cudaGetLastError());
  return DZ_OK;
}

int dz_split_update(const float* E, int64_t lde, int n, int count, const float* U, int64_t ldu, int c, void* A, void* B,
                    void* stream) {
  return dz_split_update_rows(E, lde, n, count, U, ldu, c, nullptr, 0, A, B, stream);
}

int dz_pack_gptq(const float* Wq, const float* scale, const float* zero, int N, int K, int bits,
                 int32_t* qweight, int32_t* qzeros, uint16_t* scales, void* stream) {
  if (!Wq || !scale || !zero || !qweight || !qzeros || !scales) return DZ_ERR_INVALID_ARG;
  if (bits != 2 && bits != 4 && bits != 8) return DZ_ERR_SHAPE;
  const int per = 32 / bits;
  if (N <= 0 || K <= 0 || K % per || N % per) return DZ_ERR_SHAPE;
  const dim3 grid((N + 255) / 256, K / per);
  pack_gptq_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(Wq, scale, zero, N, K, bits, qweight, qzeros,
                                                           reinterpret_cast<__half*>(scales));
  DZ_CUDA_OK(cudaGetLastError());
  return DZ_OK;
}

}  // extern "C"
