// Width of the products' tiles (gemm_tc.cu) and the slices of dL/dC's contraction
// (tensor_vjp.cu), which are chosen for the width that the product then takes.
#pragma once

#include <stdint.h>

namespace smx {
namespace tc {

// Columns per tile: the width with the least rounds of tiles on the SMs x time of a
// round, which measured 69, 73 and 115 - 140 us for 64, 128 and 256 columns (split
// BF16, K = 6016: a narrow tile still loads the 128 rows of A; FP16 pairs 64, 68 and
// 109).  Columns and rounds that are not filled cost as much as full ones: 10000 x 300
// outputs take 136 us with 128 columns (2 rounds) and 212 with 256 (2), 65536 x 400 take
// 878 (14) and 785 (7), 10000 x 100 take 127 with 64 (2) and 76 with 128 (1).
struct TileChoice {
  int columns;
  int64_t cost;  // 100 per round of 128-column tiles
};
inline TileChoice choose_tile(int64_t row_tiles, int N, int sms) {
  TileChoice best{0, 0};
  for (int bn : {256, 128, 64}) {
    const int64_t tiles = row_tiles * ((N + bn - 1) / bn);
    const int64_t cost = (tiles + sms - 1) / sms * (bn == 256 ? 177 : bn == 128 ? 100 : 94);
    if (!best.columns || cost < best.cost) best = TileChoice{bn, cost};
  }
  return best;
}

// Slices of a contraction that gives [M x N] values: the count of up to 16 with the
// least time, a slice's share of the contraction being 1 / slices (a count is only
// raised for 2 % and more).
inline int choose_slices(int64_t M, int N, int sms) {
  int best = 1;
  double cost = 1e30;
  for (int s = 1; s <= 16; ++s) {
    const double c = double(choose_tile((M + 127) / 128 * s, N, sms).cost) / s;
    if (c < 0.98 * cost) cost = c, best = s;
  }
  return best;
}

}  // namespace tc
}  // namespace smx
