// Chunkwise matrix-memory (dz_mlstm.cu) and constant-decay (dz_lightning.cu) recurrences for heads of 128 x 128 on
// the 5th-generation tensor cores: a CTA walks one (sequence, head) in chunks of 128 tokens.  With e(t, s) the
// weight of token s in the output of token t, w_s its weight in the state at the end of the chunk, in_t and `decay`
// those of the state before it,
//   P = (Q K^T) * e        O = P V + in * (Q S)        S' = decay S + (w V)^T K (kept transposed: rows are v's columns)
// are four products per chunk, 56 MMAs of 128 x 128 x 16.  The state, P and w V, held in 32 bits, enter them as hi +
// lo pairs of the 16-bit type; the state itself stays in 32 bits in registers.
//
// Bound by the sixteen warps: of about 17 thousand cycles a chunk (one warp's clock, 1965 MHz) SiLU takes 8.7 (constant
// decay; the special function unit); in the matrix memory w V and the sums for n and q.n take 3, the weights of P and the
// scaling of O 3, the output with its norm and gate 9.  Waits for the products come to 0.4 and 0.9.
// Measured against the warp-MMA kernels of 64 tokens at a time, bf16: matrix memory, 4 prompts of up to 2048 tokens x
// 32 heads, 565 -> 170 us; constant decay, 5 prompts of up to 1500 x 16 heads, continued, 260 -> 135 us.
//
// Tensor memory (128 columns each): scores, then P in their place | O | the update | w V.
// Shared memory: a ring of four tiles of 128 x 128 (q, k, v, q, ...) and S as the product with q reads it.
// Roles: 16 warps work on what lies between the products -- a thread owns a row (lane) and 32 of its columns --, two
// bring tiles in, one issues the MMAs, one computes the gates' weights a chunk ahead.  While a step of the 16
// runs, the tensor cores do another product: scores and Q S under w V, the update under P, P V under the state's
// update.  All waits are bounded.
#include <cuda.h>

#include <type_traits>

#include "dz_recurrent_tc.cuh"
#include "dz_tc.cuh"

namespace dz {
namespace {

constexpr int kTok = 128, kDim = 128;                    // tokens of a chunk; head size of q, k and v
constexpr int kSlab = kTok * 128, kTileBytes = 2 * kSlab;    // a tile: two slabs of 64 columns, 128-byte swizzle
constexpr int kSlots = 4;
// Twenty warps, the most that leave a thread 96 registers (32 of a worker's hold the state): the workers, one that
// issues, with gates one that computes the weights, the rest bring tiles in.
constexpr int kWorkWarps = 16, kIssueWarp = 19, kThreadsRec = 20 * 32;
constexpr int kLoaders = 64;
constexpr int kTQk = 0, kTO = 128, kTU = 256, kTW = 384;     // columns of tensor memory
constexpr float kDenEps = 1e-6f;
constexpr size_t kSmemRec = (kSlots + 2) * kTileBytes + 1024;

struct alignas(16) ChunkWeights {        // read as vectors, and two of them lie side by side
  float a[kTok], mx[kTok];               // matrix memory: e(t, s) = scale exp(a_s - mx_t)
  float em[kTok];                        // and the least denominator
  float in[kTok], w[kTok];
  float decay;
};

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void warp_umma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 db;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}" ::"r"(d),
      "r"(a), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void cp_async16_u32(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
struct Sum { float hi, lo; };            // hi + lo, lo below hi's last place
// (Knuth's two-sum: hi takes the rounded sum, lo what the rounding left.)
__device__ __forceinline__ Sum add(Sum a, Sum b) {
  const float s = a.hi + b.hi, t = s - a.hi, lo = ((a.hi - (s - t)) + (b.hi - t)) + (a.lo + b.lo), hi = s + lo;
  return {hi, lo - (hi - s)};
}
__device__ __forceinline__ float apart(Sum a, Sum b) { return (a.hi - b.hi) + (a.lo - b.lo); }
template <typename T> __device__ __forceinline__ float lds_one(uint32_t a) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return Cvt<T>::one(*reinterpret_cast<T*>(&v));
}

template <typename T, bool MEMORY>
__global__ void __launch_bounds__(kThreadsRec, 1) recurrent_chunk_tc_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                            const RecurrentParams p) {
  constexpr int DT = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t b_full[kSlots], b_empty[kSlots], b_wfull[2], b_wempty[2], b_qk, b_inter, b_u, b_pv, b_k, b_w,
      b_p, b_s, b_ofree;
  __shared__ ChunkWeights s_cw[2];
  __shared__ __align__(16) float s_n[kDim], s_nw[kDim];
  __shared__ float s_np[4][kDim], s_nq[4][kTok], s_den[4][kTok], s_sq[4][kTok];
  __shared__ float s_pw[2 * kTok + 1];                   // w^i at [128 + i], zero before it
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int head = blockIdx.x, seq = blockIdx.y;
  pdl_wait();
  pdl_launch();
  const int q0 = p.q_starts[seq], qn = p.q_starts[seq + 1] - q0, ctx = p.ctx_lens[seq], slot = p.slots[seq];
  if (qn <= 0) return;
  const int chunks = (qn + kTok - 1) / kTok;
  const uint32_t s_ring = (smem_u32(smem_dyn) + 1023u) & ~1023u, s_hi = s_ring + kSlots * kTileBytes, s_lo = s_hi + kTileBytes;
  volatile int* abort_flag = &s_abort;
  float* S = p.S + ((size_t)slot * p.heads + head) * kDim * kDim;

  if (tid == 0) {
    for (int i = 0; i < kSlots; ++i) {
      mbar_init(smem_u32(&b_full[i]), kLoaders);
      mbar_init(smem_u32(&b_empty[i]), 1 + kWorkWarps);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&b_wfull[i]), 32);
      mbar_init(smem_u32(&b_wempty[i]), kWorkWarps);
    }
    for (uint64_t* b : {&b_qk, &b_inter, &b_u, &b_pv}) mbar_init(smem_u32(b), 1);
    for (uint64_t* b : {&b_k, &b_w, &b_p, &b_s, &b_ofree}) mbar_init(smem_u32(b), kWorkWarps);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
  }
  if (warp == kIssueWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "n"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if constexpr (MEMORY) {
    if (tid < kDim) s_nw[tid] = p.norm_w[(size_t)head * kDim + tid];
    if (tid < kDim) s_n[tid] = ctx > 0 ? p.n[((size_t)slot * p.heads + head) * kDim + tid] : 0.f;
  } else {
    for (int j = tid; j <= 2 * kTok; j += kThreadsRec) { // past the table: w^64 w^(i - 64)
      const int i = j - kTok;
      const float* pw = p.powers + (size_t)head * 65;
      s_pw[j] = i < 0 ? 0.f : i <= 64 ? pw[i] : pw[64] * pw[i - 64];
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;

  if (warp < kWorkWarps) {
    // ---- between the products: row r, columns [c0, c0 + 32) ----
    const int h = warp >> 2, r = (warp & 3) * 32 + lane, c0 = h * 32;
    const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    auto signal = [&](uint64_t* b) {                     // what this warp wrote or read is done
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(b));
    };
    float acc[32];                                       // S[c0 + j][r]
#pragma unroll
    for (int j = 0; j < 32; ++j) acc[j] = ctx > 0 ? S[(size_t)(c0 + j) * kDim + r] : 0.f;
    auto publish = [&]() {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split_pair<T>(acc[c * 8 + 2 * j], acc[c * 8 + 2 * j + 1], hi[j], lo[j]);
        const uint32_t at = swizzled(r, h * 4 + c, kSlab);
        sts128(s_hi + at, make_uint4(hi[0], hi[1], hi[2], hi[3]));
        sts128(s_lo + at, make_uint4(lo[0], lo[1], lo[2], lo[3]));
      }
      fence_proxy_async();
      tc_fence_before();
      signal(&b_s);
    };
    if (ctx > 0) publish();
    // byte of element (token 0, column r) of a tile; the swizzle of token s is (s & 7) << 4
    const uint32_t col = (uint32_t)((r >> 6) * kSlab + (r & 7) * 2), col_chunk = (uint32_t)((r & 63) >> 3);
    for (int i = 0; i < chunks; ++i) {
      const int base = i * kTok, len = min(kTok, qn - base), nq = 3 * i, nk = nq + 1, nv = nq + 2;
      const bool state = i > 0 || ctx > 0;
      const ChunkWeights& cw = s_cw[i & 1];
      if constexpr (MEMORY) bar_wait(&b_wfull[i & 1], (i >> 1) & 1, abort_flag, p.status);
      // Each tile has a barrier of its own: copies complete in any order, and only a wait on a copy's own barrier makes
      // its bytes visible.
      if constexpr (MEMORY) {
        for (int n = nq; n <= nv; ++n) bar_wait(&b_full[n & 3], (n >> 2) & 1, abort_flag, p.status);
        __syncwarp();
      }
      if constexpr (!MEMORY) {                           // q, k and v go through SiLU in place
        for (int n = nq; n <= nv; ++n) {
          bar_wait(&b_full[n & 3], (n >> 2) & 1, abort_flag, p.status);
          __syncwarp();
          const uint32_t at = s_ring + (n & 3) * kTileBytes;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int e = tid + j * kWorkWarps * 32;
            const uint32_t a = at + swizzled(e >> 4, e & 15, kSlab);
            sts128(a, silu8<T>(lds128(a)));
          }
          fence_proxy_async();
          if (n == nk) signal(&b_k);
        }
        named_bar_sync(1, kWorkWarps * 32);
      }
      // w V, transposed: this row's column of v
      const uint32_t v_at = s_ring + (nv & 3) * kTileBytes + col;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int s = c0 + g * 16 + 2 * j;
          float2 w;
          if constexpr (MEMORY) w = *reinterpret_cast<const float2*>(cw.w + s);
          else w = make_float2(s_pw[kTok + len - 1 - s], s_pw[kTok + len - 2 - s]);
          const float a = lds_one<T>(v_at + s * 128 + ((col_chunk ^ (uint32_t)((2 * j) & 7)) << 4));
          const float b = lds_one<T>(v_at + s * 128 + 128 + ((col_chunk ^ (uint32_t)((2 * j + 1) & 7)) << 4));
          split_pair<T>(a * w.x, b * w.y, hi[j], lo[j]);
        }
        tmem_st8(lanes + kTW + c0 + g * 8, hi);
        tmem_st8(lanes + kTW + c0 + 16 + g * 8, lo);
      }
      tmem_wait_st();
      tc_fence_before();
      signal(&b_w);
      signal(&b_empty[nv & 3]);
      if constexpr (MEMORY) {
        const uint32_t k_at = s_ring + (nk & 3) * kTileBytes + col;
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 w = *reinterpret_cast<const float4*>(cw.w + c0 + j);
          const float wj[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            sum = fmaf(wj[e], lds_one<T>(k_at + (c0 + j + e) * 128 + ((col_chunk ^ (uint32_t)((j + e) & 7)) << 4)), sum);
        }
        s_np[h][r] = sum;
        const uint32_t q_at = s_ring + (nq & 3) * kTileBytes;
        float dot = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 v = lds128(q_at + swizzled(r, h * 4 + c, kSlab));
          const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = Cvt<T>::up(u[j]), m = *reinterpret_cast<const float2*>(s_n + c0 + c * 8 + 2 * j);
            dot = fmaf(f.x, m.x, dot);
            dot = fmaf(f.y, m.y, dot);
          }
        }
        s_nq[h][r] = dot;
      }
      signal(&b_empty[nq & 3]);
      signal(&b_empty[nk & 3]);

      // P
      bar_wait(&b_qk, i & 1, abort_flag, p.status);
      __syncwarp();
      tc_fence_after();
      float den = 0.f;
      if (h <= (warp & 3)) {
        float own = 0.f;
        if constexpr (MEMORY) own = cw.mx[r];
        float u[32];                                     // hi and lo take the place of these columns
        tmem_ld32(lanes + kTQk + c0, u);
        tmem_wait_ld();
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t hi[8], lo[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float f[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int s = c0 + g * 16 + 2 * j + e;
              float w;
              if constexpr (MEMORY) {
                w = __expf(cw.a[s] - own) * p.scale;
                w = s <= r ? w : 0.f;
              } else {
                w = s_pw[kTok + r - s];
              }
              f[e] = u[g * 16 + 2 * j + e] * w;
              den += f[e];
            }
            split_pair<T>(f[0], f[1], hi[j], lo[j]);
          }
          tmem_st8(lanes + kTQk + c0 + g * 8, hi);
          tmem_st8(lanes + kTQk + c0 + 16 + g * 8, lo);
        }
      } else {                                           // tokens behind every row of this warp
        tmem_st16_zero(lanes + kTQk + c0);
        tmem_st16_zero(lanes + kTQk + c0 + 16);
      }
      if constexpr (MEMORY) s_den[h][r] = den;
      if (state) {
        bar_wait(&b_inter, (ctx > 0 ? i : i - 1) & 1, abort_flag, p.status);
        __syncwarp();
        tc_fence_after();
        float in;
        if constexpr (MEMORY) in = cw.in[r];
        else in = s_pw[kTok + r + 1];
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t u[16];
          tmem_ld16(lanes + kTO + c0 + g * 16, u);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) u[j] = __float_as_uint(__uint_as_float(u[j]) * in);
          tmem_st16(lanes + kTO + c0 + g * 16, u);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      signal(&b_p);

      // the state
      bar_wait(&b_u, i & 1, abort_flag, p.status);
      __syncwarp();
      tc_fence_after();
      float decay;
      if constexpr (MEMORY) decay = cw.decay;
      else decay = s_pw[kTok + len];
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint32_t u[16];
        tmem_ld16(lanes + kTU + c0 + g * 16, u);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[g * 16 + j] = fmaf(acc[g * 16 + j], decay, __uint_as_float(u[j]));
      }
      if (i + 1 < chunks) publish();

      // the output
      const bool row_ok = r < len;
      T* op = (T*)p.out + (size_t)(q0 + base + (row_ok ? r : 0)) * p.heads * kDim + (size_t)head * kDim + c0;
      float inv = 1.f;
      uint4 gate[MEMORY ? 4 : 1];
      if constexpr (MEMORY) {
        const T* gp = (const T*)p.x + (size_t)(q0 + base + (row_ok ? r : 0)) * p.row_stride + p.g_off + (size_t)head * kDim + c0;
#pragma unroll
        for (int c = 0; c < 4; ++c) gate[c] = reinterpret_cast<const uint4*>(gp)[c];
        named_bar_sync(1, kWorkWarps * 32);              // everyone's parts of n, q.n and the sums of P
        float nq_sum = 0.f, ds = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) { nq_sum += s_nq[k][r]; ds += s_den[k][r]; }
        if (h == 0) s_n[r] = fmaf(s_n[r], decay, (s_np[0][r] + s_np[1][r]) + (s_np[2][r] + s_np[3][r]));
        inv = 1.f / (fmaxf(fabsf(fmaf(cw.in[r], nq_sum, ds)), cw.em[r]) + kDenEps);
        signal(&b_wempty[i & 1]);
      }
      bar_wait(&b_pv, i & 1, abort_flag, p.status);
      __syncwarp();
      tc_fence_after();
      float o[32];
      tmem_ld32(lanes + kTO + c0, o);
      tmem_wait_ld();
      tc_fence_before();
      signal(&b_ofree);
      if constexpr (MEMORY) {
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          o[j] *= inv;
          ss += o[j] * o[j];
        }
        s_sq[h][r] = ss;
        named_bar_sync(1, kWorkWarps * 32);
        const float rms = 1.f / sqrtf(((s_sq[0][r] + s_sq[1][r]) + (s_sq[2][r] + s_sq[3][r])) / (float)kDim + p.eps);
        if (row_ok) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint32_t g[4] = {gate[c].x, gate[c].y, gate[c].z, gate[c].w};
            float f[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 e = Cvt<T>::up(g[j]);
              const int k = c * 8 + 2 * j;
              f[2 * j] = o[k] * rms * s_nw[c0 + k] / (1.f + __expf(-e.x));
              f[2 * j + 1] = o[k + 1] * rms * s_nw[c0 + k + 1] / (1.f + __expf(-e.y));
            }
            store8<T>(op + c * 8, f);
          }
        }
      } else if (row_ok) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float f[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = o[c * 8 + j];
          store8<T>(op + c * 8, f);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 32; ++j) S[(size_t)(c0 + j) * kDim + r] = acc[j];
    if constexpr (MEMORY) {
      if (h == 0) p.n[((size_t)slot * p.heads + head) * kDim + r] = s_n[r];
    }
  } else if (warp < kWorkWarps + kLoaders / 32) {
    // ---- tiles q, k, v of every chunk: TMA, or copies that leave absent tokens zero ----
    const int t = tid - kWorkWarps * 32;
    const T* x = (const T*)p.x + (size_t)q0 * p.row_stride + (size_t)head * kDim;
    for (int n = 0; n < 3 * chunks; ++n) {
      const int which = n % 3, tok0 = n / 3 * kTok, off = which == 0 ? 0 : which == 1 ? p.k_off : p.v_off;
      const uint32_t dst = s_ring + (n & 3) * kTileBytes, full = smem_u32(&b_full[n & 3]);
      bar_wait(&b_empty[n & 3], ((n >> 2) & 1) ^ 1, abort_flag, p.status);
      if (tok0 + kTok <= qn) {
        if (t == 0) {
          mbar_expect_tx(full, kTileBytes);
          for (int i = 0; i < 2; ++i) tma_load_2d(dst + i * kSlab, &map_x, off + head * kDim + i * 64, q0 + tok0, full);
        } else {
          mbar_arrive(full);
        }
        continue;
      }
#pragma unroll 4
      for (int e = t; e < kTok * 16; e += kLoaders) {
        const int r = e >> 4, c = e & 15;
        const bool ok = tok0 + r < qn;
        cp_async16_u32(dst + swizzled(r, c, kSlab), x + off + (size_t)(ok ? tok0 + r : 0) * p.row_stride + c * 8, ok);
      }
      cp_async_commit();
      cp_async_wait<0>();
      fence_proxy_async();
      mbar_arrive(full);
    }
  } else if (warp == kIssueWarp) {
    // ---- MMA issue ----
    const uint32_t id = make_idesc<DT>(kDim, false), id_mn = id | (1u << 16);    // the second: B as [k][n]
    for (int i = 0; i < chunks; ++i) {
      const int nq = 3 * i, nk = nq + 1, nv = nq + 2, published = ctx > 0 ? i : i - 1;
      const uint32_t q = s_ring + (nq & 3) * kTileBytes, k = s_ring + (nk & 3) * kTileBytes, v = s_ring + (nv & 3) * kTileBytes;
      if constexpr (MEMORY) {
        // the scores go where P V reads P: MMAs into different accumulators keep no order by themselves
        if (i > 0) bar_wait(&b_pv, (i - 1) & 1, abort_flag, p.status);
        bar_wait(&b_full[nq & 3], (nq >> 2) & 1, abort_flag, p.status);
        bar_wait(&b_full[nk & 3], (nk >> 2) & 1, abort_flag, p.status);
      } else {                                           // signalled by warps that have waited for P V
        bar_wait(&b_k, i & 1, abort_flag, p.status);
      }
      __syncwarp();
      tc_fence_after();
      const uint32_t dq = desc_lo(q), dk = desc_lo(k);
#pragma unroll
      for (int j = 0; j < 8; ++j) {                      // 16 columns: 32 bytes; four of them to a slab
        const uint32_t o = (uint32_t)((j >> 2) * (kSlab >> 4) + (j & 3) * 2);
        warp_umma_ss(tmem + kTQk, dq + o, dk + o, id, j > 0);
      }
      warp_umma_commit(smem_u32(&b_qk));
      if (i > 0) bar_wait(&b_ofree, (i - 1) & 1, abort_flag, p.status);
      if (published >= 0) {
        bar_wait(&b_s, published & 1, abort_flag, p.status);
        __syncwarp();
        tc_fence_after();
        const uint32_t dh = desc_lo(s_hi), dl = desc_lo(s_lo);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t o = (uint32_t)((j >> 2) * (kSlab >> 4) + (j & 3) * 2);
          warp_umma_ss(tmem + kTO, dq + o, dh + o, id, j > 0);
          warp_umma_ss(tmem + kTO, dq + o, dl + o, id, 1);
        }
        warp_umma_commit(smem_u32(&b_inter));
      }
      warp_umma_commit(smem_u32(&b_empty[nq & 3]));
      bar_wait(&b_w, i & 1, abort_flag, p.status);
      __syncwarp();
      tc_fence_after();
      const uint32_t dkm = desc_lo_mn(k, kSlab), dvm = desc_lo_mn(v, kSlab);
#pragma unroll
      for (int j = 0; j < 8; ++j) {                      // 16 tokens: 2048 bytes of a tile
        const uint32_t a = tmem + kTW + (j >> 1) * 32 + (j & 1) * 8;
        warp_umma_ts(tmem + kTU, a + 16, dkm + j * 128, id_mn, j > 0);      // lo while the sums are smaller
        warp_umma_ts(tmem + kTU, a, dkm + j * 128, id_mn, 1);
      }
      warp_umma_commit(smem_u32(&b_u));
      warp_umma_commit(smem_u32(&b_empty[nk & 3]));
      bar_wait(&b_p, i & 1, abort_flag, p.status);
      __syncwarp();
      tc_fence_after();
      const uint32_t first = published >= 0 ? 1u : 0u;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t a = tmem + kTQk + (j >> 1) * 32 + (j & 1) * 8;
        warp_umma_ts(tmem + kTO, a, dvm + j * 128, id_mn, j > 0 ? 1u : first);
        warp_umma_ts(tmem + kTO, a + 16, dvm + j * 128, id_mn, 1);
      }
      warp_umma_commit(smem_u32(&b_pv));
      warp_umma_commit(smem_u32(&b_empty[nv & 3]));
    }
  } else if constexpr (MEMORY) {
    // ---- the chunk's weights; a lane holds four tokens.  A sum of 128 gates is kept as hi + lo, weights are taken
    // against the chunk's last maximum: what a weight's logarithm is off by does not grow with the sums ----
    Sum m = {ctx > 0 ? p.m[(size_t)slot * p.heads + head] : 0.f, 0.f};
    for (int i = 0; i < chunks; ++i) {
      const int base = i * kTok, len = min(kTok, qn - base), t = 4 * lane;
      ChunkWeights& cw = s_cw[i & 1];
      Sum F[4], a[4];
      float gi[4], M[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        gi[j] = -INFINITY;                               // absent tokens add nothing and forget nothing
        F[j] = {0.f, 0.f};
        if (t + j < len) {
          const float* pre = p.pre_if + (size_t)(q0 + base + t + j) * 2 * p.heads + head;
          gi[j] = soft_cap(pre[0] + p.b_if[head], p.cap);
          F[j].hi = log_sigmoid(soft_cap(pre[p.heads] + p.b_if[p.heads + head], p.cap));
        }
      }
#pragma unroll
      for (int j = 1; j < 4; ++j) F[j] = add(F[j], F[j - 1]);
      Sum sum = F[3];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const Sum up = {__shfl_up_sync(0xffffffffu, sum.hi, o), __shfl_up_sync(0xffffffffu, sum.lo, o)};
        if (lane >= o) sum = add(sum, up);
      }
      const Sum before = {__shfl_up_sync(0xffffffffu, sum.hi, 1), __shfl_up_sync(0xffffffffu, sum.lo, 1)};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (lane > 0) F[j] = add(F[j], before);
        a[j] = t + j < len ? add({gi[j], 0.f}, {-F[j].hi, -F[j].lo}) : Sum{-INFINITY, 0.f};
        M[j] = j > 0 ? fmaxf(M[j - 1], a[j].hi) : a[j].hi;     // (a row may take any M near its largest)
      }
      float mx = M[3];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, mx, o);
        if (lane >= o) mx = fmaxf(mx, up);
      }
      float top = __shfl_up_sync(0xffffffffu, mx, 1);
      top = lane > 0 ? fmaxf(top, m.hi) : m.hi;
#pragma unroll
      for (int j = 0; j < 4; ++j) M[j] = fmaxf(M[j], top);
      // the last one goes into m: with the lo of whose hi it is
      Sum ML = {__shfl_sync(0xffffffffu, M[3], 31), 0.f};
#pragma unroll
      for (int j = 0; j < 4; ++j) ML.lo = a[j].hi == ML.hi ? a[j].lo : ML.lo;
      const unsigned holders = __ballot_sync(0xffffffffu, a[0].hi == ML.hi || a[1].hi == ML.hi || a[2].hi == ML.hi || a[3].hi == ML.hi);
      ML.lo = __shfl_sync(0xffffffffu, ML.lo, holders ? __ffs(holders) - 1 : 0);
      if (!holders) ML.lo = m.lo;
      const Sum FL = {__shfl_sync(0xffffffffu, F[3].hi, 31), __shfl_sync(0xffffffffu, F[3].lo, 31)};
      bar_wait(&b_wempty[i & 1], ((i >> 1) & 1) ^ 1, abort_flag, p.status);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float rel = apart(a[j], ML);
        cw.a[t + j] = rel;
        cw.mx[t + j] = (M[j] - ML.hi) - ML.lo;
        cw.in[t + j] = expf((m.hi - M[j]) + m.lo) * p.scale;
        cw.em[t + j] = expf(-((F[j].hi + M[j]) + F[j].lo));
        cw.w[t + j] = expf(rel);
      }
      if (lane == 0) cw.decay = expf(apart(m, ML));
      m = add(FL, ML);
      mbar_arrive(smem_u32(&b_wfull[i & 1]));
    }
    if (lane == 0) p.m[(size_t)slot * p.heads + head] = m.hi;
  }

  tc_fence_before();
  __syncthreads();
  if (s_abort) {                                         // let copies and MMAs under way end
    const unsigned long long t0 = globaltimer();
    while (globaltimer() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == kIssueWarp) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
  }
}

template <typename T>
int run(const RecurrentParams& p, bool matrix_memory, int num_seqs, cudaStream_t st) {
  CUtensorMap map_x;
  const int rc = make_map(&map_x, p.x, p.rows, (int)p.row_stride, kTok, std::is_same<T, __nv_bfloat16>::value);
  if (rc) return rc;
  auto kern = matrix_memory ? recurrent_chunk_tc_kernel<T, true> : recurrent_chunk_tc_kernel<T, false>;
  DZ_CUDA_OK(allow_smem(kern, kSmemRec));
  DZ_CUDA_OK(launch_ex(kern, dim3(p.heads, num_seqs), dim3(kThreadsRec), kSmemRec, 1, st, map_x, p));
  return DZ_OK;
}

}  // namespace

int launch_recurrent_tc(const RecurrentParams& p, bool matrix_memory, int dtype, int num_seqs, cudaStream_t st) {
  return dtype == DZ_DTYPE_BF16 ? run<__nv_bfloat16>(p, matrix_memory, num_seqs, st)
                                : run<__half>(p, matrix_memory, num_seqs, st);
}

}  // namespace dz
