// blocks.cuh -- a grid's columns dealt out to the CTAs that keep them on chip.
#pragma once
#include <algorithm>
#include <cstdint>

namespace bsp {

struct BlockSplit {
  int nbx, nby;  // blocks along i, j: block (bi, bj) has i in [nx bi / nbx, nx (bi + 1) / nbx)
  int w, h;      // columns of the largest block along i, j
};
// The split into at most `ctas` blocks of columns with the fewest cells (a halo
// cell counted as half) in its largest block.
inline BlockSplit split_blocks(int nx, int ny, int ctas) {
  BlockSplit best{1, 1, nx, ny};
  double least = 1e30;
  for (int x = 1; x <= std::min(nx, ctas); ++x) {
    const int y = std::min(ny, ctas / x), w = (nx + x - 1) / x, h = (ny + y - 1) / y;
    const double cost = (double)w * h + (w + h);
    if (cost < least) {
      least = cost;
      best = BlockSplit{x, y, w, h};
    }
  }
  return best;
}

}  // namespace bsp
