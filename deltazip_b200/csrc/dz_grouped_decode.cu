// Decode attention where several query heads share a key/value head: paged cache, one query token per
// sequence, head size 128.
//
// Bound: the cache's bytes.  On CUDA cores eight heads cost 16 multiply-adds and conversions per byte, which
// held the kernel at a seventh of the copy bandwidth; here the heads are the rows of a warp MMA, so a 16-key tile
// costs 48 of them whatever the head count.
//   scores   S[heads, 8 keys] += Q K^T: the eight heads are rows 0-7 of the 16-row operand.  The order of the 128
//            products of a score is free, so a lane's 16-byte piece of a key row serves two MMAs as it lies.
//   output   O[heads, 128] += P V: a 32-bit weight is the sum of three 16-bit parts, hi, mid and lo.  Rows 0-7 of two
//            MMAs carry half of hi each, rows 8-15 mid and lo; V comes transposed by ldmatrix.  (No row of an MMA
//            mixes hi with a part that may be zero: an infinity in V stays one.)
// A CTA is four warps over the keys of one (sequence, key/value head, split), 16 keys per warp and step, each warp
// with a ring of three tiles of its own (cp.async, no barrier but the warp's): two CTAs of 96 KB per SM keep 128 KB
// of the cache in flight.  Chunks of a row are stored in an order that depends on the row (swizzle), so that
// neither the 16-byte reads of K nor ldmatrix meet a bank twice.
// Measured, 64 sequences x 64 query heads on 8, 938 keys in the mean (246 MB, 38 us at the copy bandwidth): 50.8 us
// (weights of two parts, 16 to 22 bits: 47.3), the form on CUDA cores 272; 32 heads on 8, 2560 keys: 0.85 of the copy
// bandwidth.
#include "dz_grouped_decode.cuh"

namespace dz {
namespace {

constexpr int kWarps = 4, kStages = 3, kTile = 16;             // keys per warp and step
constexpr int kRowBytes = kGroupedDim * 2, kHalfStage = kTile * kRowBytes, kStageBytes = 2 * kHalfStage;
constexpr int kRingBytes = kStages * kStageBytes;
constexpr size_t kSmem = (size_t)kWarps * kRingBytes;
static_assert(kRingBytes >= kGroupedHeads * kGroupedDim * 4, "a warp's ring also holds its output");

// Where 16-byte chunk c of row r lies: rows r, r + 1 in different halves of the banks, any eight consecutive
// rows in eight different chunks.
__device__ __forceinline__ int chunk_at(int r, int c) { return r * kRowBytes + ((c ^ ((r & 1) << 2 | (r >> 1 & 3))) << 4); }

// Two weights in [0, 1] times `kScale` as half + half + mid + lo: 24 bits, all of a weight's (fp16: of weights above
// 2^-16; below, what is lost is at most 2^-40, which no sum of weights around 1 can hold).
template <typename T> constexpr float kScale = 1.f;
template <> constexpr float kScale<__half> = 32768.f;
template <typename T>
__device__ __forceinline__ void split_weights(float a, float b, uint32_t& half, uint32_t& mid, uint32_t& lo) {
  a *= 0.5f * kScale<T>;
  b *= 0.5f * kScale<T>;
  half = Cvt<T>::down(a, b);
  const float2 h = Cvt<T>::up(half);
  split_pair<T>(2.f * (a - h.x), 2.f * (b - h.y), mid, lo);
}

template <typename T>
__global__ void __launch_bounds__(kWarps * 32, 2)
grouped_decode_kernel(GroupedDecode p) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ float s_m[kWarps][kGroupedHeads], s_l[kWarps][kGroupedHeads];
  __shared__ int s_last;
  const int seq = blockIdx.y, split = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int ratio = p.heads / p.kv_heads, parts = (ratio + kGroupedHeads - 1) / kGroupedHeads;
  const int kvh = blockIdx.x / parts, h0 = kvh * ratio + blockIdx.x % parts * kGroupedHeads;
  const int live = min(kGroupedHeads, (kvh + 1) * ratio - h0);
  pdl_wait();
  pdl_launch();
  const int len = p.lens[seq] + p.more, lo = p.window > 0 ? max(0, len - p.window) : 0;
  // A step of the CTA takes a tile for each of its warps: no split has fewer keys, and those left without any end here.
  // (The count may come from the table's width, of which a short sequence fills little: 8 heads on 1, 300 keys in a table
  // for 16384, 25.5 us with every split merged, 7.6 so.)
  constexpr int kStep = kWarps * kTile;
  const int per = max(((len - lo + p.splits - 1) / p.splits + kTile - 1) / kTile * kTile, kStep);
  const int splits = max(1, (len - lo + per - 1) / per);
  if (split >= splits) return;
  const int t0 = lo + split * per, t1 = min(len, t0 + per);
  const int* table = p.tables + (size_t)seq * p.ring_blocks;
  const T* kc = (const T*)p.k_cache;
  const T* vc = (const T*)p.v_cache;
  uint8_t* ring = smem + warp * kRingBytes;

  // cache row of key t0 + 16 * tile + (lane & 15); keys past the end repeat the last one
  auto row_of = [&](int tile) {
    const int k = min(t0 + tile * kTile + (lane & 15), t1 - 1), b = k / p.block_size;
    return ((uint32_t)table[b % p.ring_blocks] * p.block_size + (k - b * p.block_size)) * p.kv_heads + kvh;
  };
  auto issue = [&](int stage, int tile, uint32_t row) {
    const int c = lane & 15, keys = t1 - t0 - tile * kTile;    // values past the end are zero, as their weights are
#pragma unroll
    for (int j = 0; j < kTile / 2; ++j) {
      const int r = 2 * j + (lane >> 4);
      const size_t at = (size_t)__shfl_sync(0xffffffffu, row, r) * kGroupedDim + c * 8;
      uint8_t* dst = ring + stage * kStageBytes + chunk_at(r, c);
      cp_async16(dst, kc + at, true);
      cp_async16(dst + kHalfStage, vc + at, r < keys);
    }
  };
  const int tiles = t1 > t0 ? (t1 - t0 + kTile - 1) / kTile : 0;
  uint32_t next = 0;                                           // row of the tile that is requested next
  if (warp < tiles) next = row_of(warp);
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    const int tile = warp + s * kWarps;
    if (tile < tiles) {
      issue(s, tile, next);
      if (tile + kWarps < tiles) next = row_of(tile + kWarps);
    }
    cp_async_commit();
  }

  uint4 q[4];                                                  // head g's components 32 c + 8 t ... + 7
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    q[c] = make_uint4(0, 0, 0, 0);
    if (g < live)
      q[c] = *reinterpret_cast<const uint4*>((const T*)p.q + (size_t)seq * p.q_stride + (size_t)(h0 + g) * kGroupedDim +
                                             c * 32 + t * 8);
  }
  const int head = h0 + min(g, live - 1);
  // Scores are kept as they are, not times log2 e: a mask of the type's lowest value has to stay finite.
  const float* bias = p.bias ? p.bias + (size_t)head * p.bias_len : nullptr;
  const float far_bias = bias ? bias[p.bias_len - 1] : 0.f;
  // one warp of one split starts with the sink in its sum (which is kept per lane: the head's first one)
  const bool sink = p.sink && split == 0 && warp == 0;
  float m = sink ? p.sink[head] : -INFINITY, l = sink && t == 0 ? 1.f : 0.f;
  float o[16][4];                                              // [8 components][head g: 2 of hi; 2 of mid and lo]
#pragma unroll
  for (int j = 0; j < 16; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] = 0.f;

  int stage = 0;
  for (int tile = warp; tile < tiles; tile += kWarps) {
    cp_async_wait<kStages - 2>();
    __syncwarp();
    {
      const int ahead = tile + (kStages - 1) * kWarps;
      if (ahead < tiles) {
        issue(stage == 0 ? kStages - 1 : stage - 1, ahead, next);
        if (ahead + kWarps < tiles) next = row_of(ahead + kWarps);
      }
      cp_async_commit();
    }
    const uint8_t* ks = ring + stage * kStageBytes;
    const int k0 = t0 + tile * kTile;
    float x[2][2];                                             // keys k0 + 8 i + 2 t + {0, 1}
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint4 k = *reinterpret_cast<const uint4*>(ks + chunk_at(i * 8 + g, 4 * c + t));
        const uint32_t a0[4] = {q[c].x, 0, q[c].y, 0}, a1[4] = {q[c].z, 0, q[c].w, 0};
        mma16816<T>(s[0], a0, k.x, k.y);
        mma16816<T>(s[1], a1, k.z, k.w);
      }
      float b[2] = {far_bias, far_bias};
      if (bias && len - 1 - (k0 + kTile - 1) < p.bias_len - 1) {         // distances that have a bias of their own
#pragma unroll
        for (int e = 0; e < 2; ++e) b[e] = bias[min(max(len - 1 - (k0 + i * 8 + 2 * t + e), 0), p.bias_len - 1)];
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) x[i][e] = fmaf(s[0][e] + s[1][e], p.scale, b[e]);
    }
    if (k0 + kTile > t1) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (k0 + i * 8 + 2 * t + e >= t1) x[i][e] = -INFINITY;
    }
    float mx = fmaxf(fmaxf(x[0][0], x[0][1]), fmaxf(x[1][0], x[1][1]));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mn = fmaxf(m, mx), ms = mn == -INFINITY ? 0.f : mn;
    if (__any_sync(0xffffffffu, mn != m)) {
      const float c = __expf(m - ms);
      l *= c;
#pragma unroll
      for (int j = 0; j < 16; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[j][e] *= c;
      m = mn;
    }
    uint32_t a[4], a2[4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float w0 = __expf(x[i][0] - ms), w1 = __expf(x[i][1] - ms);
      l += w0 + w1;
      split_weights<T>(w0, w1, a[2 * i], a[2 * i + 1], a2[2 * i + 1]);
      a2[2 * i] = a[2 * i];
    }
    const uint8_t* vs = ks + kHalfStage;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      uint32_t b[4];
      ldsm4_t(b, vs + chunk_at(lane & 15, 2 * j + (lane >> 4)));
      mma16816<T>(o[2 * j], a, b[0], b[1]);
      mma16816<T>(o[2 * j + 1], a, b[2], b[3]);
      mma16816<T>(o[2 * j], a2, b[0], b[1]);
      mma16816<T>(o[2 * j + 1], a2, b[2], b[3]);
    }
    stage = stage == kStages - 1 ? 0 : stage + 1;
  }
  cp_async_wait<0>();
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  __syncwarp();                                                // the warp's ring becomes its output [heads, 128]
  float* own = reinterpret_cast<float*>(ring);
  // where the values held an infinity, hi's products are the result and the other parts' may be anything
  auto whole = [](float hi, float rest) { return (isfinite(hi) ? hi + rest : hi) * (1.f / kScale<T>); };
#pragma unroll
  for (int j = 0; j < 16; ++j)
    *reinterpret_cast<float2*>(own + g * kGroupedDim + j * 8 + 2 * t) = make_float2(whole(o[j][0], o[j][2]), whole(o[j][1], o[j][3]));
  if (t == 0) {
    s_m[warp][g] = m;
    s_l[warp][g] = l;
  }
  __syncthreads();

  // four components of a head per thread and round
  const size_t column = (size_t)seq * p.heads + h0;
  float2* const ml = reinterpret_cast<float2*>(p.partial + (size_t)gridDim.y * p.heads * p.splits * kGroupedDim);
  auto store = [&](int h, int d, const float (&a)[4], float sum) {
    uint2 v = make_uint2(Cvt<T>::down(a[0] / sum, a[1] / sum), Cvt<T>::down(a[2] / sum, a[3] / sum));
    if (p.empty_is_zero && !(sum > 0.f)) v = make_uint2(0, 0);
    *reinterpret_cast<uint2*>((T*)p.out + (column + h) * kGroupedDim + d) = v;
  };
  for (int i = threadIdx.x * 4; i < live * kGroupedDim; i += kWarps * 32 * 4) {
    const int h = i / kGroupedDim, d = i % kGroupedDim;
    float mm = -INFINITY, sum = 0.f, a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, s_m[w][h]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float c = s_m[w][h] == -INFINITY ? 0.f : __expf(s_m[w][h] - mm);
      const float4 v = *reinterpret_cast<const float4*>(smem + w * kRingBytes + (size_t)i * 4);
      sum += s_l[w][h] * c;
      a[0] += v.x * c;
      a[1] += v.y * c;
      a[2] += v.z * c;
      a[3] += v.w * c;
    }
    if (splits == 1) {
      store(h, d, a, sum);
    } else {
      const size_t at = (column + h) * p.splits + split;
      *reinterpret_cast<float4*>(p.partial + at * kGroupedDim + d) = make_float4(a[0], a[1], a[2], a[3]);
      if (d == 0) ml[at] = make_float2(mm, sum);
    }
  }
  if (splits == 1) return;
  // the last split of this column to finish merges all of them; nothing waits
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    int* ticket = p.tickets + (size_t)seq * gridDim.x + blockIdx.x;
    s_last = atomicAdd(ticket, 1) == splits - 1;
    if (s_last) *ticket = 0;                                   // ready for the next launch
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int i = threadIdx.x * 4; i < live * kGroupedDim; i += kWarps * 32 * 4) {
    const int h = i / kGroupedDim, d = i % kGroupedDim;
    const size_t at = (column + h) * p.splits;
    float mm = -INFINITY, sum = 0.f, a[4] = {0.f, 0.f, 0.f, 0.f};
    for (int s = 0; s < splits; ++s) mm = fmaxf(mm, __ldcg(&ml[at + s]).x);
#pragma unroll 4
    for (int s = 0; s < splits; ++s) {
      const float2 w = __ldcg(&ml[at + s]);
      const float4 v = __ldcg(reinterpret_cast<const float4*>(p.partial + (at + s) * kGroupedDim + d));
      const float c = w.x == -INFINITY ? 0.f : __expf(w.x - mm);
      sum += w.y * c;
      a[0] += v.x * c;
      a[1] += v.y * c;
      a[2] += v.z * c;
      a[3] += v.w * c;
    }
    store(h, d, a, sum);
  }
}

}  // namespace

int launch_grouped_decode(const GroupedDecode& p, int num_seqs, int dtype, cudaStream_t st) {
  const dim3 grid(grouped_decode_columns(p.heads, p.kv_heads), num_seqs, p.splits);
  DZ_DISPATCH16(dtype, DZ_CUDA_OK(allow_smem(grouped_decode_kernel<T>, kSmem));
                DZ_CUDA_OK(launch_ex(grouped_decode_kernel<T>, grid, dim3(kWarps * 32), kSmem, 1, st, p)));
  return DZ_OK;
}

}  // namespace dz
