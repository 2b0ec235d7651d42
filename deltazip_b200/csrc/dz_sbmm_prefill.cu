// y += x dequant(delta_slot)^T for prompt batches (hundreds to thousands of tokens, few slots).
//
// A prompt's tokens share one slot, so the tokens of a slot form long runs of the sorted batch.  A run is cut into
// equal blocks of at most 176 tokens; a tile of work is a token block times F (1 or 2) groups of 128 output
// features, over the whole of K.  The features are the MMA's rows, the block's tokens its columns: the packed codes
// of a (feature group, 128 k) unit are expanded to the compressed A operand in tensor memory once per token block
// instead of once per 32-token window, and B is the x tile as TMA brings it -- columns past the end of the run are
// computed and not stored, so no row has to be masked or copied.
//
// With F = 2 an x tile serves 256 features: x is what a unit moves most of (45 KB of x to 6 KB of codes).  F = 1 is for
// an odd number of feature groups.
//
// Measured on the four projections of a 7B decoder layer, 1999 tokens in seven runs, 4-bit: 4670 -> 1259 us with the
// dense products (about 550 of them), against one pass of the decode kernel per 128 tokens.
//
// Roles: a TMA producer (x), a bulk-copy producer (packed stages), F MMA issuers, two warpgroups that expand, two
// that drain one accumulator each and add it to y.  All waits are bounded.
#include <cuda.h>
#include <type_traits>

#include "dz_elem.cuh"
#include "dz_expand.cuh"
#include "dz_tc.cuh"

namespace dz {
namespace {

constexpr int kPTokens = 176;                  // most columns of a token block
constexpr int kPBoxRows = 88;                  // rows of one TMA copy of x (one or two per half-tile)
constexpr int kPThreads = 20 * 32;             // 4 service warps, 2 x 4 expanding, 2 x 4 draining
constexpr int kPXHalf = kPTokens * 128, kPXStages = 3, kPXBytes = 2 * kPXHalf;    // a unit's two half-tiles of 64 k
constexpr int kPRStages = 8;
constexpr int kPTmemCols = 512;
// tensor memory: two accumulators, four buffers of expanded A (32 columns) and of metadata (4)
constexpr int kPAcc1 = 192, kPACol = 368, kPECol = 496;
__host__ __device__ constexpr int p_raw_bytes(int bits) { return 128 * 64 * bits / 8; }
__host__ __device__ constexpr int p_stage_bytes(int bits) { return p_raw_bytes(bits) + 2048; }
constexpr int p_smem_bytes(int bits) { return kPXStages * kPXBytes + kPRStages * p_stage_bytes(bits) + 1024; }

struct PParams {
  int M, K, num_slots, num_kblocks, num_kunits;
  int groups, F;                               // feature groups of 128, of which a tile takes F (groups % F == 0)
  long long ldy;
  const uint8_t *qweight, *meta, *scales;
  long long qstride, mstride, sstride;
  const uint8_t* seg;
  void* y;
  int* status;
  int tokens_sorted;
};

// Token blocks of a run of n tokens, and the tokens of each but the last.
__device__ __forceinline__ int run_blocks(int n) { return (n + kPTokens - 1) / kPTokens; }
__device__ __forceinline__ int block_tokens(int n) {
  const int nb = run_blocks(n);
  return ((n + nb - 1) / nb + 15) & ~15;
}

struct PTile {
  int slot, row0, rows, group0;                // sorted rows [row0, row0 + rows), feature groups from group0
};
// Tile v: token blocks in slot order, feature groups fastest.
__device__ __forceinline__ PTile tile_at(int v, const PParams& p, const int* first, const int* begin, const int* end) {
  const int per = p.groups / p.F;
  const int b = v / per;
  int lo = 0, hi = p.num_slots;                // the last slot with first[slot] <= b
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (first[mid] <= b) lo = mid; else hi = mid;
  }
  const int n = end[lo] - begin[lo], each = block_tokens(n);
  PTile t;
  t.slot = lo;
  t.row0 = begin[lo] + (b - first[lo]) * each;
  t.rows = min(each, end[lo] - t.row0);        // > 0: each <= 176, and one block fewer of 176 would not hold the run
  t.group0 = (v - b * per) * p.F;
  return t;
}

template <int BITS, int DT>
__global__ void __launch_bounds__(kPThreads, 1)
sbmm_prefill_kernel(const __grid_constant__ CUtensorMap map_x, const PParams p) {
  using T = typename std::conditional<DT == 0, __half, __nv_bfloat16>::type;
  extern __shared__ uint8_t smem_dyn[];
  __shared__ __align__(8) uint64_t s_xfull[kPXStages], s_xempty[kPXStages], s_rfull[kPRStages], s_rempty[kPRStages],
      s_aready[4], s_afree[4], s_accfull[2], s_accempty[2];
  __shared__ int s_begin[kPrefillMaxSlots], s_end[kPrefillMaxSlots], s_first[kPrefillMaxSlots + 1];
  __shared__ int s_tok[2][kPTokens];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t s_x = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  const uint32_t s_r = s_x + kPXStages * kPXBytes;
  volatile int* abort_flag = &s_abort;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kPXStages; ++i) { mbar_init(smem_u32(&s_xfull[i]), 1); mbar_init(smem_u32(&s_xempty[i]), p.F); }
    for (int i = 0; i < kPRStages; ++i) { mbar_init(smem_u32(&s_rfull[i]), 1); mbar_init(smem_u32(&s_rempty[i]), 128); }
    for (int i = 0; i < 4; ++i) { mbar_init(smem_u32(&s_aready[i]), 128); mbar_init(smem_u32(&s_afree[i]), 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&s_accfull[i]), 1); mbar_init(smem_u32(&s_accempty[i]), 128); }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)),
                 "n"(kPTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  // ---- the batch: where each slot's run begins and ends, and its first token block ----
  const SegHeader* hdr = reinterpret_cast<const SegHeader*>(p.seg);
  const SegLayout lay = seg_layout(p.M, p.num_slots);
  const int* perm = reinterpret_cast<const int*>(p.seg + lay.perm);
  const int* slot_of = reinterpret_cast<const int*>(p.seg + lay.slot_of);
  const bool bad = hdr->capacity_M != p.M || hdr->num_slots != p.num_slots || (p.tokens_sorted && !hdr->sorted);
  if (bad && blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(p.status, 0, (int)DZ_ERR_INVALID_ARG);
  for (int i = threadIdx.x; i < p.num_slots; i += kPThreads) s_begin[i] = s_end[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < p.M && !bad; i += kPThreads) {
    const int s = slot_of[i];
    if (s < 0 || s >= p.num_slots) continue;
    if (i == 0 || slot_of[i - 1] != s) s_begin[s] = i;
    if (i + 1 == p.M || slot_of[i + 1] != s) s_end[s] = i + 1;
  }
  __syncthreads();
  if (warp == 0) {
    int run = 0;
    for (int s0 = 0; s0 < p.num_slots; s0 += 32) {
      const int n = s0 + lane < p.num_slots ? run_blocks(s_end[s0 + lane] - s_begin[s0 + lane]) : 0;
      int sum = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
      }
      if (s0 + lane < p.num_slots) s_first[s0 + lane] = run + sum - n;
      run += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) s_first[p.num_slots] = run;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem_base;
  const int total = s_first[p.num_slots] * (p.groups / p.F);
  const int F = p.F;

  if (warp == 0) {
    // ---- x ----
    Ring rx(kPXStages, 1);
    for (int v = blockIdx.x; v < total; v += gridDim.x) {
      const PTile t = tile_at(v, p, s_first, s_begin, s_end);
      const int boxes = t.rows > kPBoxRows ? 2 : 1;
      for (int ku = 0; ku < p.num_kunits; ++ku) {
        const int nhalf = min(2, p.num_kblocks - ku * 2);
        bar_wait(&s_xempty[rx.idx], rx.par, abort_flag, p.status);
        __syncwarp();
        const uint32_t full = smem_u32(&s_xfull[rx.idx]);
        warp_mbar_expect_tx(full, nhalf * boxes * kPBoxRows * 128);
        for (int h = 0; h < nhalf; ++h)
          for (int b = 0; b < boxes; ++b)
            warp_tma_load_2d(s_x + rx.idx * kPXBytes + h * kPXHalf + b * (kPBoxRows * 128), &map_x, (ku * 2 + h) * kBlockK,
                             t.row0 + b * kPBoxRows, full);
        rx.advance();
      }
    }
  } else if (warp == 2) {
    // ---- packed stages: (unit, feature group) ----
    Ring rr(kPRStages, 1);
    for (int v = blockIdx.x; v < total; v += gridDim.x) {
      const PTile t = tile_at(v, p, s_first, s_begin, s_end);
      const uint8_t* qs = p.qweight + (size_t)t.slot * p.qstride;
      const uint8_t* ms = p.meta + (size_t)t.slot * p.mstride;
      for (int ku = 0; ku < p.num_kunits; ++ku) {
        const int nhalf = min(2, p.num_kblocks - ku * 2);
        for (int f = 0; f < F; ++f) {
          bar_wait(&s_rempty[rr.idx], rr.par, abort_flag, p.status);
          __syncwarp();
          const uint32_t full = smem_u32(&s_rfull[rr.idx]), dst = s_r + rr.idx * p_stage_bytes(BITS);
          const size_t blk = (size_t)(t.group0 + f) * p.num_kblocks + (size_t)ku * 2;
          warp_mbar_expect_tx(full, nhalf * (codes_block_bytes(BITS) + kMetaBlockBytes));
          warp_bulk_load(dst, qs + blk * codes_block_bytes(BITS), nhalf * codes_block_bytes(BITS), full);
          warp_bulk_load(dst + p_raw_bytes(BITS), ms + blk * kMetaBlockBytes, nhalf * kMetaBlockBytes, full);
          rr.advance();
        }
      }
    }
  } else if (warp == 1 || (warp == 3 && F == 2)) {
    // ---- MMA issue: with two feature groups a warp for each (one warp takes 900 cycles to a unit of two groups,
    // waits and commits included, and the MMAs of 176 columns 700; their accumulators are independent) ----
    const int mine = F == 2 ? warp >> 1 : 0;
    Ring rx(kPXStages, 0);
    int stage = mine, tiles = 0;
    const int whole = p.num_kblocks / 2;
    for (int v = blockIdx.x; v < total; v += gridDim.x, ++tiles) {
      const PTile t = tile_at(v, p, s_first, s_begin, s_end);
      const uint32_t idesc = make_idesc<DT>((t.rows + 15) & ~15, true);
      // F = 2: group f in accumulator f; F = 1: tiles alternate between the accumulators
      const int acc = F == 2 ? mine : tiles & 1, use = F == 2 ? tiles : tiles >> 1;
      const uint32_t d = tmem + acc * kPAcc1;
      bar_wait(&s_accempty[acc], (use & 1) ^ 1, abort_flag, p.status);
      for (int ku = 0; ku < p.num_kunits; ++ku, stage += F) {
        const int buf = (stage & 1) + 2 * ((stage >> 1) & 1);
        bar_wait(&s_xfull[rx.idx], rx.par, abort_flag, p.status);
        bar_wait(&s_aready[buf], (stage >> 2) & 1, abort_flag, p.status);
        __syncwarp();
        tc_fence_after();
        const uint32_t b0 = desc_lo(s_x + rx.idx * kPXBytes), b1 = b0 + (kPXHalf >> 4);
        const uint32_t a = tmem + kPACol + buf * 32, e = tmem + kPECol + buf * 4;
        if (ku < whole) {                                // (a branch between the MMAs would cost them their uniform registers)
          warp_umma_ts_sp(d, a, b0, e, idesc, ku > 0);
          warp_umma_ts_sp(d, a + 8, b0 + 4, e, idesc | 1, 1);
          warp_umma_ts_sp(d, a + 16, b1, e + 2, idesc, 1);
          warp_umma_ts_sp(d, a + 24, b1 + 4, e + 2, idesc | 1, 1);
        } else {                                         // K ends with half a unit
          warp_umma_ts_sp(d, a, b0, e, idesc, ku > 0);
          warp_umma_ts_sp(d, a + 8, b0 + 4, e, idesc | 1, 1);
        }
        warp_umma_commit(smem_u32(&s_afree[buf]));
        warp_umma_commit(smem_u32(&s_xempty[rx.idx]));
        rx.advance();
      }
      warp_umma_commit(smem_u32(&s_accfull[acc]));
    }
  } else if (warp >= 4 && warp < 12) {
    // ---- expansion: warpgroup w takes the stages of its parity ----
    const int w = (warp - 4) >> 2, q = warp & 3, r = q * 32 + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(q * 32) << 16);
    int n = 0;                                 // stages this warpgroup has expanded
    int stage = 0;                             // of this CTA, before the current tile
    for (int v = blockIdx.x; v < total; v += gridDim.x) {
      const PTile t = tile_at(v, p, s_first, s_begin, s_end);
      const int count = p.num_kunits * F;
      for (int i = (stage & 1) == w ? 0 : 1; i < count; i += 2, ++n) {
        const int ku = F == 2 ? i >> 1 : i;
        const bool both = ku * 2 + 1 < p.num_kblocks;
        const int s = stage + i, ri = s % kPRStages, buf = w + 2 * (n & 1);
        bar_wait(&s_rfull[ri], (s / kPRStages) & 1, abort_flag, p.status);
        bar_wait(&s_afree[buf], ((n >> 1) & 1) ^ 1, abort_flag, p.status);
        __syncwarp();
        tc_fence_after();
        const uint32_t raw = s_r + ri * p_stage_bytes(BITS);
        uint32_t mw[4] = {0, 0, 0, 0};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (h == 1 && !both) break;
          uint32_t o[16];
          if (BITS == 4) {
            const uint4 cw = lds128(raw + h * 2048 + r * 16);
            const uint32_t wv[4] = {cw.x, cw.y, cw.z, cw.w};
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) expand_word4<DT>(wv[i4], o + i4 * 4);
          } else {
            const uint2 cw = lds64(raw + h * 1024 + r * 8);
            expand_word2<DT>(cw.x, o);
            expand_word2<DT>(cw.y, o + 8);
          }
          tmem_st16(lane_addr + kPACol + buf * 32 + h * 16, o);
          const uint2 m2 = lds64(raw + p_raw_bytes(BITS) + h * 1024 + r * 8);
          mw[h * 2] = m2.x;
          mw[h * 2 + 1] = m2.y;
        }
        tmem_st4(lane_addr + kPECol + buf * 4, mw[0], mw[1], mw[2], mw[3]);
        mbar_arrive(smem_u32(&s_rempty[ri]));
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(smem_u32(&s_aready[buf]));
      }
      stage += count;
    }
  } else if (warp >= 12) {
    // ---- warpgroup d drains accumulator d into y ----
    const int d = (warp - 12) >> 2, q = warp & 3, r = q * 32 + lane;
    const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + d * kPAcc1;
    auto drain_sync = [&]() {                            // this warpgroup
      if (d == 0) named_bar_sync(1, 128);
      else named_bar_sync(2, 128);
    };
    T* const y = reinterpret_cast<T*>(p.y);
    int tiles = 0, uses = 0;
    for (int v = blockIdx.x; v < total; v += gridDim.x) {
      const PTile t = tile_at(v, p, s_first, s_begin, s_end);
      const bool mine = F == 2 || (tiles & 1) == d;
      ++tiles;
      if (!mine) continue;
      const int n = (t.group0 + (F == 2 ? d : 0)) * kTileN + r;
      const float sc = __half2float(*reinterpret_cast<const __half*>(p.scales + (size_t)t.slot * p.sstride + (size_t)n * 2));
      // A lane works on two features of every second token (its own sums and its neighbour's), so that y moves 32 bits
      // at a time; 64 tokens of it are on their way before the sums are complete and from there on.
      constexpr int kAhead = 4;
      const int odd = lane & 1;
      int* const tok = s_tok[d];
      drain_sync();                        // the tile before has been read
      for (int i = r; i < t.rows; i += 128) tok[i] = perm[t.row0 + i];
      drain_sync();
      uint32_t old[kAhead][8];
      auto fetch = [&](uint32_t (&o)[8], int c) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int at = c + 2 * i + odd;
          o[i] = at < t.rows ? *reinterpret_cast<const uint32_t*>(y + (size_t)tok[at] * p.ldy + (n - odd)) : 0;
        }
      };
#pragma unroll
      for (int g = 0; g < kAhead; ++g) fetch(old[g], g * 16);
      bar_wait(&s_accfull[d], uses & 1, abort_flag, p.status);
      ++uses;
      __syncwarp();
      tc_fence_after();
      for (int c0 = 0; c0 < t.rows; c0 += 16 * kAhead) {
#pragma unroll
        for (int g = 0; g < kAhead; ++g) {
          const int c = c0 + g * 16;
          if (c >= t.rows) break;
          uint32_t u[16];
          tmem_ld16(acc + c, u);
          tmem_wait_ld();
          if (c + 16 >= t.rows) {
            tc_fence_before();
            mbar_arrive(smem_u32(&s_accempty[d]));
          }
          uint32_t now[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float a = sc * __uint_as_float(u[2 * i]), b = sc * __uint_as_float(u[2 * i + 1]);
            const float got = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
            const float2 before = Cvt<T>::up(old[g][i]);
            now[i] = odd ? Cvt<T>::down(before.x + got, before.y + b) : Cvt<T>::down(before.x + a, before.y + got);
          }
          fetch(old[g], c + 16 * kAhead);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int at = c + 2 * i + odd;
            if (at < t.rows) *reinterpret_cast<uint32_t*>(y + (size_t)tok[at] * p.ldy + (n - odd)) = now[i];
          }
        }
      }
    }
  }

  // ---- teardown ----
  tc_fence_before();
  __syncthreads();
  if (s_abort) {
    // copies still in flight get a bounded time to land before the shared memory is released
    const unsigned long long t0 = globaltimer();
    while (globaltimer() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kPTmemCols) : "memory");
  }
}

}  // namespace

int launch_sbmm_prefill(const dz_sbmm_args& a, const void* xsrc, int sms, cudaStream_t st) {
  const int dt = a.dtype == DZ_DTYPE_BF16 ? 1 : 0;
  CUtensorMap map_x;
  int rc = make_map(&map_x, xsrc, a.M, a.K, kPBoxRows, dt);
  if (rc) return rc;
  PParams p;
  p.M = a.M; p.K = a.K; p.num_slots = a.num_slots;
  p.num_kblocks = a.K / kBlockK;
  p.num_kunits = (p.num_kblocks + 1) / 2;
  p.groups = a.N / kTileN;
  // One feature group only where their number is odd: with two an x tile serves both and two warps issue (12288 x 4096,
  // 2048 tokens of one slot: 125 us, with one 148; 4096 x 4096, whose 192 tiles fill 1.3 waves: 68 and 70; with 48
  // tiles, 513 tokens, still 64 against 69).
  p.F = p.groups % 2 == 0 ? 2 : 1;
  p.ldy = a.y_stride ? a.y_stride : a.N;
  p.qweight = (const uint8_t*)a.qweight; p.meta = (const uint8_t*)a.meta; p.scales = (const uint8_t*)a.scales;
  p.qstride = a.qweight_stride; p.mstride = a.meta_stride; p.sstride = a.scales_stride;
  p.seg = (const uint8_t*)a.segments;
  p.y = a.y;
  p.status = reinterpret_cast<int*>((uint8_t*)a.workspace + kWsStatus);
  p.tokens_sorted = a.tokens_sorted != 0;
  const size_t smem = a.bits == 2 ? p_smem_bytes(2) : p_smem_bytes(4);
  using Kern = void (*)(const CUtensorMap, const PParams);
  static const Kern kerns[4] = {sbmm_prefill_kernel<2, 0>, sbmm_prefill_kernel<4, 0>, sbmm_prefill_kernel<2, 1>,
                                sbmm_prefill_kernel<4, 1>};
  Kern kern = kerns[(a.bits == 4 ? 1 : 0) + 2 * dt];
  DZ_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<sms, kPThreads, smem, st>>>(map_x, p);
  DZ_CUDA_OK(cudaGetLastError());
  return DZ_OK;
}

}  // namespace dz
