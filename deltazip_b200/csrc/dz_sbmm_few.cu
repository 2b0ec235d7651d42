// The SBMM of a few tokens (at most 16):  y = x W^T + x dequant(delta_slot)^T as in dz_sbmm_tc.cu, split by features alone.
//
// With a few tokens a call is 5 to 20 us of streaming, and what it costs beside that counts as much.  The form for larger
// batches splits a tile of 128 features along k over several CTAs, which then settle it through parked partial sums and
// counters (4 to 5 of its 16 us at 4096 x 4096), and holds a whole SM's shared memory, so that the next call's CTAs cannot
// be there before it ends.  Here a CTA takes a slice of 16 features over all of k: nothing is settled between CTAs, no
// workspace, two CTAs fit an SM beside each other or the next call's beside this one's.  Sixteen features are no M for
// tcgen05.mma (64 at least), and at 16 tokens its products would not be the bound: these are warp MMAs, 16 x 8 x 16 for W
// and 2:4-sparse 16 x 8 x 32 for the deltas.
//
//   Warps.  Eight warps share a slice's blocks of 64 k.  Each streams its own blocks through its own ring of 2 KB stages
//   (cp.async, D - 1 of them ahead, no barrier with any other warp): a stage is a block of W, or that of up to five present
//   deltas' codes and metadata.  At the end of a slice the warps' sums meet in shared memory, in the warps' order.
//   Order of k.  Within a block of 64 k lane t of a quad has, for m = 0 and 1, the eight k from 32 (t >> 1) + 16 m +
//   8 (t & 1): one 16-byte piece of a row of W and of x, four operand pairs, two dense MMAs.  The sparse MMA wants a group
//   of four k halved between two lanes, so lanes t and t ^ 1 swap half of their x once a block; lane pair u = t >> 1 then
//   holds the groups of word 2u + m of a row's codes as the MMA's groups 2i + u (i = 0..3), and lane t as owner of groups
//   t and t + 4 of the codes finds them in word 2 (t & 1) + m as pairs t >> 1 and 2 + (t >> 1).  Metadata of two
//   words interleaves by nibbles.
//   Columns.  Tokens keep the batch's order; of x a delta's MMA sees the rows of its own tokens, the others as zero.
// Which calls take it, and what both forms measured: sbmm_few_supported.
#include <cuda_bf16.h>

#include <type_traits>

#include "dz_common.cuh"
#include "dz_expand.cuh"
#include "dz_tc.cuh"

namespace dz {
namespace {

constexpr int kPerStage = 5;                   // deltas of a stage
constexpr int kFewMax = 16;                    // tokens, and so present deltas

struct FewParams {
  int M, N, K, num_slots, delta_only, tokens_sorted, accumulate, stable;
  long long ldy, qstride, mstride, sstride;
  const uint8_t *x, *w, *qweight, *meta, *scales, *seg;
  void* y;
  int* status;
};

__device__ __forceinline__ void few_copy16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
template <int DT>
__device__ __forceinline__ void mma_dense(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if (DT == 0)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 2:4-sparse; the metadata of lanes 2 SEL and 2 SEL + 1 of a quad is read
template <int DT, int SEL>
__device__ __forceinline__ void mma_sparse(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, const uint32_t* b, uint32_t e) {
  if (DT == 0)
    asm("mma.sp::ordered_metadata.sync.aligned.m16n8k32.row.col.f32.f16.f16.f32 "
        "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9, %10, %11}, {%0, %1, %2, %3}, %12, %13;"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(e), "n"(SEL));
  else
    asm("mma.sp::ordered_metadata.sync.aligned.m16n8k32.row.col.f32.bf16.bf16.f32 "
        "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9, %10, %11}, {%0, %1, %2, %3}, %12, %13;"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(e), "n"(SEL));
}

// The (code - zero) pairs `at` and 2 + `at` of words 2v and 2v + 1 of a row's block (4-bit), or `at`, 2 + `at`, 4 + `at` and
// 6 + `at` of word v (2-bit): a[m][i], operand pair i of MMA m.  fp16 takes a field where it lies in the low byte of a
// half-word, so lanes differ in masks alone; bf16's shorter mantissa needs the field at the bottom, so there lanes shift.
template <int BITS, int DT>
struct Fields {
  uint32_t mask[2], magic[2], bias[2];
  int shift;
  __device__ __forceinline__ explicit Fields(int at) {
    shift = BITS * at;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t P = 4 * i + BITS * at;                  // (4-bit: i = 0 only)
      mask[i] = (((1u << BITS) - 1u) << P) * 0x00010001u;
      magic[i] = ((25u - P) << 10) * 0x00010001u;
      bias[i] = (((25u - P) << 10) | ((1u << (BITS - 1)) << P)) * 0x00010001u;
    }
  }
  __device__ __forceinline__ uint32_t field(uint32_t w, int i) const {
    uint32_t t;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(t) : "r"(w), "r"(mask[i]), "r"(magic[i]));
    const __half2 v = __hsub2(*reinterpret_cast<__half2*>(&t), *reinterpret_cast<const __half2*>(&bias[i]));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  __device__ __forceinline__ void operator()(uint32_t w0, uint32_t w1, uint32_t (*a)[2]) const {
    if (BITS == 4 && DT == 0) {
      a[0][0] = field(w0, 0);
      a[0][1] = field(w0 >> 8, 0);
      a[1][0] = field(w1, 0);
      a[1][1] = field(w1 >> 8, 0);
    } else if (BITS == 4) {
      const uint32_t v0 = w0 >> shift, v1 = w1 >> shift;
      a[0][0] = code_pair<4, 0, 1>(v0);
      a[0][1] = code_pair<4, 0, 1>(v0 >> 8);
      a[1][0] = code_pair<4, 0, 1>(v1);
      a[1][1] = code_pair<4, 0, 1>(v1 >> 8);
    } else if (DT == 0) {
      const uint32_t v = w0 >> 8;
      a[0][0] = field(w0, 0);
      a[0][1] = field(w0, 1);
      a[1][0] = field(v, 0);
      a[1][1] = field(v, 1);
    } else {
      const uint32_t v = w0 >> shift, u = v >> 8;
      a[0][0] = code_pair<2, 0, 1>(v);
      a[0][1] = code_pair<2, 4, 1>(v);
      a[1][0] = code_pair<2, 0, 1>(u);
      a[1][1] = code_pair<2, 4, 1>(u);
    }
  }
};

// Bytes of a stage and stages of a warp's ring for slices of RT x 16 features: sixteen warps of an SM have 192 KB in all
// cases.  A warp's sums take the place of the stage that it has read last.
__host__ __device__ constexpr int few_stage(int rt) { return rt * 16 * 128; }
__host__ __device__ constexpr int few_depth(int rt) { return rt == 1 ? 6 : 3; }
constexpr int few_smem(int rt, int warps) { return warps * few_depth(rt) * few_stage(rt); }

// NB: blocks of eight tokens; RT: tiles of 16 features of a slice
template <int BITS, int DT, int NB, int RT, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 16 / WARPS) sbmm_few_kernel(const FewParams p) {
  constexpr int D = few_depth(RT), kFewWarps = WARPS, kSlice = 16 * RT, kStage = few_stage(RT);
  constexpr int kCodeBytes = kSlice * 4 * BITS, kMetaSlice = kSlice * 8;
  constexpr int kWin = kCodeBytes + kMetaSlice;                // one delta's part of a stage
  constexpr int kPieces = kWin / 16, kRounds = (kPieces + 31) / 32;
  static_assert(kPerStage * kWin <= kStage && 8 * NB * kSlice * 4 <= kStage, "stage");
  extern __shared__ __align__(128) uint8_t s_few[];
  __shared__ int s_slot[kFewMax], s_win[kFewMax];              // slot of each token, of each present delta
  __shared__ const uint8_t* s_from[kFewMax][2];                // codes and metadata of each present delta
  __shared__ int s_sum[WARPS];                                 // byte offset of each warp's sums
  static_assert(16 / WARPS * (few_smem(RT, WARPS) + 2 * sizeof(int) * kFewMax + sizeof(s_from) + sizeof(s_sum) + 1024) <= 228 * 1024,
                "sixteen warps an SM (1 KB of a CTA's shared memory is the system's)");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;

  if (!p.stable) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }
  int nwin = 0;
  if (p.seg) {
    const SegHeader* hdr = reinterpret_cast<const SegHeader*>(p.seg);
    const SegLayout lay = seg_layout(p.M, p.num_slots);
    const bool bad = hdr->capacity_M != p.M || hdr->num_slots != p.num_slots || (p.tokens_sorted && !hdr->sorted);
    nwin = min(reinterpret_cast<const int*>(p.seg + lay.block_begin)[1], kFewMax);
    if (threadIdx.x < kFewMax) {
      const int i = threadIdx.x;
      if (i < nwin) {
        const int slot = reinterpret_cast<const Window*>(p.seg + lay.windows)[i].slot;
        s_win[i] = slot;
        s_from[i][0] = p.qweight + (size_t)slot * p.qstride;
        s_from[i][1] = p.meta + (size_t)slot * p.mstride;
      }
      if (i < p.M) {
        const int tok = reinterpret_cast<const int*>(p.seg + lay.perm)[i];
        if ((unsigned)tok < (unsigned)kFewMax) s_slot[tok] = reinterpret_cast<const int*>(p.seg + lay.slot_of)[i];
      }
    }
    if (bad) {                                                 // (the same in every thread)
      if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(p.status, 0, (int)DZ_ERR_INVALID_ARG);
      // a grid that ended before its predecessor would let its successor start beside that
      if (p.stable) asm volatile("griddepcontrol.wait;" ::: "memory");
      return;
    }
    __syncthreads();
  }

  const int slices = p.N / kSlice, kbs = p.K / kBlockK;
  const size_t row_bytes = (size_t)p.K * 2;
  const int parts = (p.delta_only ? 0 : 1) + (nwin + kPerStage - 1) / kPerStage;     // stages of a block of k
  const int w_parts = p.delta_only ? 0 : 1;
  const uint32_t ring = smem_u32(s_few) + warp * D * kStage;

  // ---- copies: this warp's stages in order, slice by slice, block by block ----
  int c_slice = blockIdx.x, c_kb = warp, c_part = 0, c_at = 0;
  const uint8_t* const w_lane = p.w + (size_t)(lane >> 3) * row_bytes + (lane & 7) * 16;
  const uint32_t w_dst = (lane >> 3) * 128 + (((lane & 7) ^ (((lane >> 3) & 1) * 2)) << 4);
  auto request = [&]() {
    if (c_slice < slices && c_kb < kbs && parts > 0) {
      const uint32_t dst = ring + c_at * kStage;
      if (c_part < w_parts) {
        const uint8_t* src = w_lane + (size_t)c_slice * kSlice * row_bytes + (size_t)c_kb * 128;
#pragma unroll
        for (int j = 0; j < 4 * RT; ++j) few_copy16(dst + w_dst + j * 512, src + j * 4 * row_bytes);
      } else {
        const int first = (c_part - w_parts) * kPerStage, count = min(kPerStage, nwin - first);
        const int tile = c_slice * kSlice / kTileN, sub = c_slice * kSlice % kTileN;
        const size_t blk = (size_t)tile * kbs + c_kb;
#pragma unroll
        for (int j = 0; j < kRounds; ++j) {
          const int piece = lane + 32 * j, role = piece * 16 < kCodeBytes ? 0 : 1;
          const size_t off = role ? blk * kMetaBlockBytes + sub * 8 + piece * 16 - kCodeBytes
                                  : blk * codes_block_bytes(BITS) + sub * 4 * BITS + piece * 16;
          if (piece < kPieces)
            for (int i = 0; i < count; ++i) few_copy16(dst + i * kWin + piece * 16, s_from[first + i][role] + off);
        }
      }
      if (++c_part == parts) {
        c_part = 0;
        c_kb += kFewWarps;
        if (c_kb >= kbs) { c_kb = warp; c_slice += gridDim.x; }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (++c_at == D) c_at = 0;
  };
#pragma unroll
  for (int i = 0; i < D - 1; ++i) request();
  if (p.stable) {                                              // x and y depend on the predecessor
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }

  // this lane's tokens as columns of B: rows of x (those past the batch repeat the last one) and their slots
  const uint8_t* xr[NB];
  uint32_t owners[NB];                                         // bit w: the token is of present delta w
#pragma unroll
  for (int nb = 0; nb < NB; ++nb) {
    const int tok = min(nb * 8 + g, p.M - 1);
    xr[nb] = p.x + (size_t)tok * row_bytes + 64 * (t >> 1) + 16 * (t & 1);
    owners[nb] = 0;
    for (int w = 0; w < nwin; ++w) owners[nb] |= (s_slot[tok] == s_win[w] ? 1u : 0u) << w;
  }
  uint4 xn[NB][2];                                             // the next block's
  auto load_x = [&](int kb) {
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int m = 0; m < 2; ++m) xn[nb][m] = *reinterpret_cast<const uint4*>(xr[nb] + (size_t)kb * 128 + m * 32);
  };
  if (warp < kbs) load_x(warp);

  const Fields<BITS, DT> fields(t >> 1);
  const uint32_t w_at = g * 128 + (((4 * (t >> 1) + (t & 1)) ^ ((g & 1) * 2)) << 4);
  const uint32_t code_at = BITS == 4 ? g * 16 + (t & 1) * 8 : g * 8 + (t & 1) * 4;
  // (of two tiles of 16 rows lanes 2 and 3 of a quad have the second's metadata, 128 bytes further; they take their two
  // words in the other order, so that a read meets every bank once)
  const uint32_t meta_at = RT == 1 ? kCodeBytes + g * 8 : (uint32_t)(kCodeBytes + (g + 16 * (t >> 1)) * 8) ^ (t & 2 ? 64 : 0);
  const uint32_t meta_sel = t & 1 ? 0x7351 : 0x6240;
  int at = 0;                                                  // stage
  for (int slice = blockIdx.x; slice < slices; slice += gridDim.x) {
    float base[RT][NB][4], delta[RT][NB][4];
#pragma unroll
    for (int i = 0; i < RT * NB * 4; ++i) (&base[0][0][0])[i] = (&delta[0][0][0])[i] = 0.f;
    for (int kb = warp; kb < kbs; kb += kFewWarps) {
      uint4 x[NB][2];
#pragma unroll
      for (int i = 0; i < 2 * NB; ++i) (&x[0][0])[i] = (&xn[0][0])[i];
      load_x(kb + kFewWarps < kbs ? kb + kFewWarps : warp);
      auto next_stage = [&]() {
        asm volatile("cp.async.wait_group %0;" ::"n"(D - 2) : "memory");
        __syncwarp();                                          // every lane's copies are there, and the last stage read
        request();
        const uint32_t st = ring + at * kStage;
        if (++at == D) at = 0;
        return st;
      };
      if (w_parts) {
        const uint32_t st = next_stage();
#pragma unroll
        for (int m = 0; m < 2; ++m) {
#pragma unroll
          for (int rt = 0; rt < RT; ++rt) {
            const uint32_t w = ((st + w_at) ^ (m * 32)) + rt * 2048;
            const uint4 a = lds128(w), b = lds128(w + 1024);
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
              mma_dense<DT>(base[rt][nb], a.x, b.x, a.y, b.y, x[nb][m].x, x[nb][m].y);
              mma_dense<DT>(base[rt][nb], a.z, b.z, a.w, b.w, x[nb][m].z, x[nb][m].w);
            }
          }
        }
      }
      if (nwin > 0) {
        uint32_t half[NB][2][4];                               // half t & 1 of the lane pair's groups
        const bool odd = t & 1;
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            const uint4 v = x[nb][m];
            const uint32_t r0 = __shfl_xor_sync(0xffffffffu, odd ? v.x : v.y, 1), r1 = __shfl_xor_sync(0xffffffffu, odd ? v.z : v.w, 1);
            half[nb][m][0] = odd ? r0 : v.x;
            half[nb][m][1] = odd ? r1 : v.z;
            half[nb][m][2] = odd ? v.y : r0;
            half[nb][m][3] = odd ? v.w : r1;
          }
        for (int first = 0; first < nwin; first += kPerStage) {
          const uint32_t st = next_stage();
          const int count = min(kPerStage, nwin - first);
          // U deltas at a time: the words of all are requested before the first is expanded
          auto products = [&](auto unroll, const int i) {
            constexpr int U = decltype(unroll)::value;
            uint32_t c[U][2 * RT][2];
            uint2 md[U][2];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const uint32_t win = st + (i + u) * kWin;
#pragma unroll
              for (int r = 0; r < 2 * RT; ++r) {
                if (BITS == 4) {
                  const uint2 v = lds64(win + code_at + r * 128);
                  c[u][r][0] = v.x;
                  c[u][r][1] = v.y;
                } else {
                  c[u][r][0] = lds32(win + code_at + r * 64);
                  c[u][r][1] = 0;
                }
              }
#pragma unroll
              for (int r = 0; r < 2; ++r) md[u][r] = lds64((win + meta_at) ^ (r * 64));   // words m and 2 + m, rows g and
            }                                                                             // g + 8 in their halves
#pragma unroll
            for (int u = 0; u < U; ++u) {
              uint32_t e[2];
#pragma unroll
              for (int m = 0; m < 2; ++m) {
                const uint2 w = md[u][m];
                const uint32_t even = (w.x & 0x0f0f0f0fu) | ((w.y << 4) & 0xf0f0f0f0u);
                const uint32_t odds = ((w.x >> 4) & 0x0f0f0f0fu) | (w.y & 0xf0f0f0f0u);
                e[m] = __byte_perm(even, odds, meta_sel);
              }
              uint32_t b[NB][2][4];
#pragma unroll
              for (int nb = 0; nb < NB; ++nb) {
                const uint32_t keep = (uint32_t)((int)(owners[nb] << (31 - first - i - u)) >> 31);
#pragma unroll
                for (int k = 0; k < 8; ++k) (&b[nb][0][0])[k] = (&half[nb][0][0])[k] & keep;
              }
#pragma unroll
              for (int rt = 0; rt < RT; ++rt) {
                uint32_t a[2][2][2];
                fields(c[u][2 * rt][0], c[u][2 * rt][1], a[0]);
                fields(c[u][2 * rt + 1][0], c[u][2 * rt + 1][1], a[1]);
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                  for (int m = 0; m < 2; ++m) {
                    if (rt == 0) mma_sparse<DT, 0>(delta[rt][nb], a[0][m][0], a[1][m][0], a[0][m][1], a[1][m][1], b[nb][m], e[m]);
                    else mma_sparse<DT, 1>(delta[rt][nb], a[0][m][0], a[1][m][0], a[0][m][1], a[1][m][1], b[nb][m], e[1 - m]);
                  }
              }
            }
          };
          int i = 0;
          for (; i + 1 < count; i += 2) products(std::integral_constant<int, 2>(), i);
          if (i < count) products(std::integral_constant<int, 1>(), i);
        }
      }
    }
    // ---- the warps' sums, with their deltas' scales: [column][row], in the stage that the warp requests next ----
    __syncwarp();                                              // (every lane has read it; nothing is under way to it)
    const int mine_at = (warp * D + c_at) * kStage;
    float* const mine = reinterpret_cast<float*>(s_few + mine_at);
    if (lane == 0) s_sum[warp] = mine_at;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int tok = nb * 8 + 2 * t + c, slot = p.seg && tok < p.M ? s_slot[tok] : -1;
#pragma unroll
        for (int r = 0; r < 2 * RT; ++r) {
          const int row = g + 8 * r;
          float v = base[r >> 1][nb][2 * (r & 1) + c];
          if (slot >= 0) {
            const unsigned short sc = *reinterpret_cast<const unsigned short*>(p.scales + (size_t)slot * p.sstride +
                                                                               (size_t)(slice * kSlice + row) * 2);
            v = fmaf(__half2float(__ushort_as_half(sc)), delta[r >> 1][nb][2 * (r & 1) + c], v);
          }
          mine[tok * kSlice + row] = v;
        }
      }
    __syncthreads();
    for (int i = threadIdx.x; i < p.M * kSlice; i += 32 * kFewWarps) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < kFewWarps; ++w) v += reinterpret_cast<const float*>(s_few + s_sum[w])[i];
      store_out<DT>(p.y, (size_t)(i / kSlice) * p.ldy + slice * kSlice + i % kSlice, v, p.accumulate);
    }
    __syncthreads();
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

}  // namespace

// Whether a call takes this form: few tokens, an output that is not pushed to other GPUs (their flags are per tile of 128
// features), and not too much delta work.  A CTA's warps go through all of k, delta by delta, where the larger form splits k
// over CTAs and hands the products to tcgen05.mma.sp: k times deltas (at most min(tokens, slots)) is the chain here, the
// whole delta work the chip's load, and twice the columns make both twice as long.  With one slice an SM the chain has the
// SM to itself and may be longer; at equal times this form is the better one, as its launch encodes no tensor maps.  Times in
// us, larger form against this one, fp16 4-bit, weights and slots not in L2, device time in a graph (2-bit codes and bf16 lie
// on the same side):
//   base product alone    1 row   4096 x 4096 17.1, 8.6   12288 x 4096 35.4, 18.8   22016 x 4096 40.4, 30.9   32000 x 4096 55.4, 41.5
//                         16 rows             17.5, 10.2              36.1, 20.8               40.9, 35.1               56.7, 46.2
//   8 tokens, by deltas   11264 x 2048 3: 20.5, 17.8 (4: 22.1, 21.1; 6: 25.4, 28.7)    6144 x 2048 4: 15.4, 14.5 (6: 17.7, 19.1)
//                         4096 x 4096 2: 16.3, 15.1 (3: 17.0, 16.9; 4: 18.0, 19.2)     12288 x 4096 1: 29.8, 25.6 (4: 36.9, 37.5)
//                         5120 x 5120 1: 19.5, 17.3 (2: 20.5, 21.3)     22016 x 4096 (1: 46.1, 45.7; 2: 49.3, 53.4)
//     one slice an SM     2048 x 2048 8: 13.3, 11.7    1024 x 4096 4: 13.5, 12.9 (6: 14.5, 16.7)    2048 x 5632 3: 15.1, 15.1 (4: 15.6, 16.9)
//                         1024 x 6144 1: 13.9, 12.6 (but 1280 x 8192 1: 14.6, 15.8)
//   16 tokens             2048 x 2048 4: 11.9, 10.3 (8: 13.3, 13.5)     4096 x 4096 1: 15.7, 15.6 (2: 16.2, 18.4)
//                         1024 x 4096 2: 13.1, 12.8 (3: 13.3, 13.7)     2048 x 5632 1: 14.4, 14.2 (but 1024 x 6144 1: 13.9, 14.7)
// Of 1596 measured calls on this side of the line seven are faster in the larger form, by 3 % at most (1024 x 6144, 2 deltas);
// by the product of deltas and weights alone 1280 x 8192 with 6 deltas took 29.4 where the larger form takes 17.9.
bool sbmm_few_supported(const dz_sbmm_args& a, bool base_only, int sms) {
  if (a.M > kFewMax || a.push) return false;
  if (base_only) return true;
  const long long deltas = min(a.M, a.num_slots), chain = deltas * a.K, work = chain * a.N;
  if (a.M > 8) return a.K <= 5632 && chain <= 8192 && work <= 1ll << 24;
  return a.K <= 6144 && chain <= (a.N / 16 <= sms ? 17000 : 8192) && work <= 70000000ll;
}

int launch_sbmm_few(const dz_sbmm_args& a, bool base_only, int sms, int* status, cudaStream_t st) {
  FewParams p;
  p.M = a.M; p.N = a.N; p.K = a.K; p.num_slots = a.num_slots;
  p.delta_only = !base_only && !a.w_base;
  p.tokens_sorted = base_only || a.tokens_sorted;
  p.accumulate = (a.flags & DZ_SBMM_ACCUMULATE) ? 1 : 0;
  p.stable = (a.flags & DZ_SBMM_INPUTS_STABLE) ? 1 : 0;
  p.ldy = a.y_stride ? a.y_stride : a.N;
  p.qstride = a.qweight_stride; p.mstride = a.meta_stride; p.sstride = a.scales_stride;
  p.x = (const uint8_t*)a.x; p.w = (const uint8_t*)a.w_base;
  p.qweight = (const uint8_t*)a.qweight; p.meta = (const uint8_t*)a.meta; p.scales = (const uint8_t*)a.scales;
  p.seg = base_only ? nullptr : (const uint8_t*)a.segments;
  p.y = a.y;
  p.status = status;
  const int dt = a.dtype == DZ_DTYPE_BF16, nb = a.M > 8;
  using Kern = void (*)(const FewParams);
#define DZ_FEW(NB, RT, W) \
  sbmm_few_kernel<2, 0, NB, RT, W>, sbmm_few_kernel<4, 0, NB, RT, W>, sbmm_few_kernel<2, 1, NB, RT, W>, sbmm_few_kernel<4, 1, NB, RT, W>
  static const Kern kerns[24] = {DZ_FEW(1, 1, 8), DZ_FEW(2, 1, 8), DZ_FEW(1, 2, 8), DZ_FEW(2, 2, 8), DZ_FEW(1, 2, 4), DZ_FEW(2, 2, 4)};
#undef DZ_FEW
  // Slices of 32 features, with half the work per delta that does not grow with the features (metadata, masking x), where
  // two CTAs an SM have one each; narrower ones keep more SMs busy (one token, one delta: 2048 x 2048 6.7 us with 16, 7.1
  // with 32; 4096 x 4096 12.8 and 12.3; 6144 x 2048 13.3 and 9.4; 12288 x 4096 32.1 and 25.9).  Two CTAs of eight warps an SM; four of four where the slices are more than those.
  const int rt = a.N / 16 > 2 * sms ? 2 : 1, slices = a.N / (16 * rt), warps = slices > 2 * sms ? 4 : 8;
  // Three of those, held down to that by their shared memory, where rounds of three end sooner than rounds of four: with
  // four some SMs get four CTAs and others two.  Base products of 9 rows, three always (four did not fit) and so: 11264 x
  // 2048 10.7 us both, 22016 x 4096 35.4 and 34.4 (four: 38.6), 15360 x 5120 39.6 and 28.2, 32000 x 4096 50.9 and 44.3.
  auto rounds = [&](int per_sm) { return (slices + per_sm * sms - 1) / (per_sm * sms); };
  const int per_sm = warps == 8 ? 2 : 3 * rounds(3) < 4 * rounds(4) ? 3 : 4;
  const int kidx = (a.bits == 4) + 2 * dt + 4 * nb + 8 * (rt - 1) + (warps == 4 ? 8 : 0);   // (four warps: slices of 32)
  constexpr int kAFourth = 228 * 1024 / 4;
  const int smem = per_sm == 3 ? kAFourth : few_smem(rt, warps);
  Kern kern = kerns[kidx];
  static bool attr_set[64][24] = {};
  int dev = 0;
  DZ_CUDA_OK(cudaGetDevice(&dev));
  bool& set = attr_set[dev & 63][kidx];
  if (!set) {
    DZ_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, max(smem, kAFourth)));
    set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(min(slices, per_sm * sms));
  cfg.blockDim = dim3(32 * warps);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  DZ_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, p));
  return DZ_OK;
}

}  // namespace dz
