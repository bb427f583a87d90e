// Segment ids in the flash-attention kernels.
//
// A query sees the keys of its own segment only.  Two things keep packed sequences at the cost of what their rows see:
//   * lvb_segment_ranges reduces every block of 128 ids to its (lowest, highest) id, and a CTA leaves out the leading (and without a causal
//     part the trailing) blocks whose range does not meet its own: nothing in them can be equal, whatever the order of the ids.
//   * a warp looks at the ids of a block once, one id per lane and 32 columns, and makes a word of visible columns per row from a ballot per
//     distinct id among its rows (packed sequences: one or two).  A block whose ids are all those of the warp's rows needs no words at all.
// Ids are compared as unsigned numbers: padding rows (negative ids) lie after all others, where packing puts them.
//
// What bounded the kernels before was the mask itself: every thread read 128 ids per block and tested every column for three conditions (about
// 15 us per block of 256 queries x 128 keys against 4 us without ids), on every block up to the diagonal.  Per layer on a B200: 2 x 3000 tokens
// in five documents each, 16 heads of 128 over 8, forward 519 -> 84 us, backward 488 -> 218 us; 16 prompts of up to 1024 tokens, 32 heads over
// 8, forward 810 -> 282 us.  The ranges take 2.6 us.
#pragma once
#include "common.cuh"

namespace lvb {
namespace seg {

constexpr int kBlock = 128;

// One warp: the first and last of the blocks lo .. hi whose range meets own; (hi + 1, lo - 1) when there is none
__device__ __forceinline__ int2 meeting_blocks(const uint2* __restrict__ ranges, uint2 own, int lo, int hi, int lane) {
  int first = hi + 1, last = lo - 1;
  for (int j0 = lo; j0 <= hi; j0 += 32) {
    const int j = j0 + lane;
    bool meets = false;
    if (j <= hi) {
      const uint2 r = __ldg(ranges + j);
      meets = r.x <= own.y && own.x <= r.y;
    }
    const uint32_t m = __ballot_sync(0xffffffffu, meets);
    if (m != 0u) {
      if (first > hi) first = j0 + __ffs(m) - 1;
      last = j0 + 31 - __clz(m);
    }
  }
  return make_int2(first, last);
}

// Bits lo .. hi of a word (either bound may lie outside it)
__device__ __forceinline__ uint32_t bit_range(int lo, int hi) {
  if (hi < 0 || lo > 31 || lo > hi) return 0u;
  return (0xffffffffu << max(lo, 0)) & (0xffffffffu >> (31 - min(hi, 31)));
}

// same[i]: the columns 32 i + 0 .. 31 whose id (ids[i], one per lane) is this row's.  Returns whether every row of the warp sees them all.
template <int N>
__device__ __forceinline__ bool same_segment(int mine, const int (&ids)[N], uint32_t (&same)[N]) {
  const int first = __shfl_sync(0xffffffffu, mine, 0);
  bool all = mine == first;
#pragma unroll
  for (int i = 0; i < N; ++i) all = all && ids[i] == first;
  if (__all_sync(0xffffffffu, all)) {
#pragma unroll
    for (int i = 0; i < N; ++i) same[i] = 0xffffffffu;
    return true;
  }
  uint32_t todo = 0xffffffffu;
  while (todo != 0u) {
    const int id = __shfl_sync(0xffffffffu, mine, __ffs(todo) - 1);
    const bool hit = mine == id;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const uint32_t m = __ballot_sync(0xffffffffu, ids[i] == id);
      if (hit) same[i] = m;
    }
    todo &= ~__ballot_sync(0xffffffffu, hit);
  }
  return false;
}

}  // namespace seg
}  // namespace lvb
