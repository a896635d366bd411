// Element masks of partial list entries in the forward kernels.
#pragma once
#include "attn_common.cuh"
#include "internal.h"

namespace kvx {

// Mask bits of query token r for the 128 keys from c0 of a partial list entry without an element mask (the pool of masks was
// used up: rare).  Not inlined: what it needs then lives in no register of the tile loop, and the loop is shorter (the
// instruction fetch of a loop this long is not free: 4 x 4k tokens 372 -> 358 us).
static __device__ __noinline__ uint4 fwd_keep_slow(const FwdArgs* a, int b, int r, int c0) {
  const bool row_valid = r < a->tok.q_len;
  const RowBounds rb = load_bounds(a->mask, b, min(r, a->tok.q_len - 1));
  int q_seg = KVAX_B200_PADDING_SEGMENT_ID, q_pos = 0;
  if (row_valid) {
    q_seg = __ldg(a->tok.q_seg + (long long)b * a->tok.q_len + r);
    q_pos = query_position(a->tok, b, r);
  }
  const int32_t* kv_seg = a->tok.kv_seg + (long long)b * a->tok.kv_len;
  const int32_t* kv_pos = a->tok.sequential ? nullptr : a->tok.kv_pos + (long long)b * a->tok.kv_len;
  uint32_t w[4];
#pragma unroll
  for (int ch = 0; ch < 4; ++ch)
    w[ch] = keep_bits32<false>(rb, c0 + ch * 32, a->tok.kv_len, row_valid, q_seg, q_pos, kv_seg + c0 + ch * 32,
                               kv_pos ? kv_pos + c0 + ch * 32 : nullptr);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Element mask of partial list entry e for query token r, row `row` of the list's query tile: worked out once by the list
// builder for every head (16 bytes per row), else by the function above.
__device__ __forceinline__ uint4 fwd_keep(const FwdArgs& a, uint32_t e, int b, int r, int row) {
  return (e & kBitmapBit) ? __ldg(entry_bitmap(a.list, e) + row) : fwd_keep_slow(&a, b, r, int(e & a.list.tile_mask) * kTile);
}

// Masked scores become -inf.
__device__ __forceinline__ void mask_scores(uint32_t (&v)[4][32], const uint4 keep) {
  const uint32_t w[4] = {keep.x, keep.y, keep.z, keep.w};
#pragma unroll
  for (int ch = 0; ch < 4; ++ch) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[ch][j] = ((w[ch] >> j) & 1u) ? v[ch][j] : 0xff800000u;
  }
}

}  // namespace kvx
