// Decode attention where several query heads share a key/value head (dz_grouped_decode.cu).
#pragma once

#include "dz_elem.cuh"

namespace dz {

struct GroupedDecode {
  const void* q;                         // rows [query heads * 128 | ...], one per sequence
  int64_t q_stride;                      // elements between rows
  void* out;                             // [sequences, heads * 128]
  const void* k_cache;                   // [slots, kv_heads, 128]
  const void* v_cache;
  const int* tables;                     // [sequences, ring_blocks]; position t is in block (t / block_size) % ring_blocks
  int ring_blocks, block_size;
  const int* lens;                       // [sequences]; the sequence has lens[s] + more keys, the newest is the query's own
  int more;
  int heads, kv_heads;
  float scale;
  int window;                            // keys a query sees, 0: all
  const float* bias;                     // [heads, bias_len] per distance (the last one for all farther ones), or nullptr
  int bias_len;
  const float* sink;                     // [heads] one more score without a key, or nullptr
  int empty_is_zero;                     // a row without a sum gets zero, otherwise 0 / 0
  int splits;
  float* partial;                        // splits > 1: kGroupedDim + 2 floats per (sequence, head, split)
  int* tickets;                          // ... and one per (sequence, CTA column), zero between launches
};

constexpr int kGroupedDim = 128;         // head size of keys and values
constexpr int kGroupedHeads = 8;         // query heads of a CTA
inline int grouped_decode_columns(int heads, int kv_heads) {
  return kv_heads * ((heads / kv_heads + kGroupedHeads - 1) / kGroupedHeads);
}
// Scratch of `splits` > 1 behind the tickets, any address.
inline size_t grouped_decode_partial_bytes(int num_seqs, int heads, int splits) {
  return (size_t)num_seqs * heads * splits * (kGroupedDim + 2) * 4 + 16;
}
inline float* grouped_decode_partial(void* scratch) { return (float*)(((uintptr_t)scratch + 15) & ~(uintptr_t)15); }
int launch_grouped_decode(const GroupedDecode& p, int num_seqs, int dtype, cudaStream_t st);

}  // namespace dz
