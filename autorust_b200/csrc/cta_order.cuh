// The order in which the CTAs of a (tiles, batch x head) problem take their work, shared by the attention kernels.
//
// The hardware starts CTAs in the order of their linear index.  With the tiles of one head behind one another, the
// last CTAs to start are those of the last heads, heavy and light ones alike, and a launch of one to a few rounds ends
// on whatever heavy CTA started last.  A grouped grid walks the heads in groups whose streamed operands fit the L2
// together; inside a group the tile index is outermost, and each kernel counts its tiles from the heaviest (the far
// end of a causal triangle, a full tile before a partial one), so that a group ends on its lightest CTAs.
//   plain:    grid (tiles, heads)
//   grouped:  grid (heads of a group, tiles, groups)
// The order is in the shape of the grid, so that a kernel reads tile and head from its block index wherever it needs
// them: with one computed from a linear index they stay in registers, which cost the D = 128 forward kernels 12 bytes
// of spills and 3 % (B=4 H=32 S=8192 INT8 3.11 -> 3.25 ms).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace ar {

// Streamed operands of the heads that are walked together: a quarter of the 126 MB L2, whose two halves may each hold
// a copy.  Heads beyond that would stream from memory once per tile instead of once per group.
constexpr size_t HEAD_GROUP_BYTES = (size_t)32 << 20;
enum { EVEN_TILES, PARTIAL_TILE, CAUSAL_TILES };  // how the tiles of a launch differ in weight

struct CtaGrid {
  dim3 grid;
  int grouped;
};
// `bytes_per_head`: what every head streams past its tiles (K/V heads shared by a GQA group count once); `split` neighbouring CTAs
// share a tile.  Plain stay launches of more than eight rounds of CTAs, whose end weighs little, those whose tiles all weigh
// the same, and those of one round with a partial tile: the order gains them nothing, and the heads that run side by side
// should be few (bf16 D = 128, B=1 H=8 S=8192: 225 us plain, 231 grouped; H=32 831 and 852).  A causal launch of one round
// is still better off with its heavy CTAs side by side (B=1 H=32/8 S=512: 14.8 us, 15.5 plain).  Measured with a limit of 28
// rounds as well, 54 shapes of 8 to 28 rounds each: with a partial tile no difference (-2 to +3 %), under a causal mask 5 %
// faster in the mean, but up to 5 % slower at S=8000.
inline CtaGrid cta_grid(size_t bytes_per_head, int heads, int tiles, int uneven, int split = 1) {
  int group = 1;
  const long long ctas = (long long)tiles * heads;
  if (uneven && tiles > 1 && (uneven == CAUSAL_TILES || ctas * split > 148) && ctas <= 8 * 148 && tiles <= 65535) {
    const size_t fit = HEAD_GROUP_BYTES / (bytes_per_head ? bytes_per_head : 1);
    for (int d = fit < (size_t)heads ? (int)fit : heads; d > 1 && group == 1; d--)  // the largest divisor that fits
      if (heads % d == 0) group = d;
  }
  if (group == 1) return {dim3((unsigned)(tiles * split), (unsigned)heads, 1), 0};
  return {dim3((unsigned)(group * split), (unsigned)tiles, (unsigned)(heads / group)), 1};
}

#ifdef __CUDACC__
__device__ __forceinline__ int cta_tiles(int grouped, int split = 1) {
  return (int)(grouped ? gridDim.y : gridDim.x / (uint32_t)split);
}
// This CTA's tile (0 = first to run).
__device__ __forceinline__ int cta_tile(int grouped, int split = 1) {
  return (int)(grouped ? blockIdx.y : blockIdx.x / (uint32_t)split);
}
__device__ __forceinline__ int cta_head(int grouped, int split = 1) {
  return (int)(grouped ? blockIdx.z * (gridDim.x / (uint32_t)split) + blockIdx.x / (uint32_t)split : blockIdx.y);
}
#endif

}  // namespace ar
