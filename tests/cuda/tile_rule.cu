// Prints for every (M, N) of the command line the tile width, the slices and, per count of
// slices, the rounds x weight / slices of the width that the product would take.
#include <stdio.h>
#include <stdlib.h>

#include "tile_rule.h"

int main(int argc, char** argv) {
  for (int i = 1; i + 1 < argc; i += 2) {
    const long M = atol(argv[i]), N = atol(argv[i + 1]);
    printf("%d %d", smx::tc::choose_tile((M + 127) / 128, int(N), 152).columns, smx::tc::choose_slices(M, int(N), 152));
    for (int s = 1; s <= 16; ++s)
      printf(" %.6f", double(smx::tc::choose_tile((M + 127) / 128 * s, int(N), 152).cost) / s);
    printf("\n");
  }
}
