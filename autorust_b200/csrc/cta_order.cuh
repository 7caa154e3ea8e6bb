// The order in which the CTAs of a (tiles, batch x head) grid take their work, shared by the attention kernels.
//
// The hardware starts CTAs in the order of their linear index.  With the tiles of one head behind one another, the
// last CTAs to start are those of the last heads, heavy and light ones alike, and a launch of one to a few waves ends
// on whatever heavy CTA started last.  Here the heads are walked in groups whose streamed operands fit the L2
// together; inside a group the tile index is outermost, and each kernel counts its tiles from the heaviest (the far
// end of a causal triangle, a full tile before a partial one), so that a group ends on its lightest CTAs.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace ar {

// Streamed operands of the heads that are walked together: a quarter of the 126 MB L2, whose two halves may each hold
// a copy.  Heads beyond that would stream from memory once per tile instead of once per group.
constexpr size_t HEAD_GROUP_BYTES = (size_t)32 << 20;

// Heads per group when every head streams `bytes_per_head` (K/V heads shared by a GQA group count once).  Launches of
// more than eight rounds keep the heads one by one: their end weighs little, and a head whose CTAs run side by side
// reads its operands from nearby rows of L2 at about the same time (B=4 H=32 S=8192 D=128 INT8, 4096 CTAs: 3.11 ms head by
// head, 3.25 ms in groups of ten).
inline int head_group_for(size_t bytes_per_head, int heads, long long ctas) {
  if (ctas > 8 * 148) return 1;
  const size_t fit = HEAD_GROUP_BYTES / (bytes_per_head ? bytes_per_head : 1);
  return fit < 1 ? 1 : fit < (size_t)heads ? (int)fit : heads;
}

#ifdef __CUDACC__
// This CTA's tile (0 = first to run) and head in a grid of (tiles, heads).
__device__ __forceinline__ void cta_order(int head_group, int& tile, int& head) {
  const uint32_t lin = blockIdx.y * gridDim.x + blockIdx.x;
  const uint32_t per = (uint32_t)head_group * gridDim.x;
  const uint32_t grp = lin / per, in_grp = lin - grp * per;
  const uint32_t heads = min((uint32_t)head_group, gridDim.y - grp * (uint32_t)head_group);
  const uint32_t t = in_grp / heads;
  tile = (int)t;
  head = (int)(grp * (uint32_t)head_group + in_grp - t * heads);
}
#endif

}  // namespace ar
