/* The tile order of the TMA stencil kernels (st_tiles.h): every tile of a grid is
   some block's, once; and on the longest grids, where 32-bit products of the strips
   could wrap, a block's tile lies on the grid and its number leads back to it. */
#include <stdio.h>
#include <stdlib.h>
#include <vector>

#include "st_tiles.h"

static int check_all(int tx, int ty, int layers)
{
  const long total = (long)tx * ty * layers;
  std::vector<char> seen(total, 0);
  for (long b = 0; b < total; b++) {
    int x, y, l;
    st_tile((unsigned)b, tx, ty, layers, st_strip(tx, ty), &x, &y, &l);
    if (x < 0 || x >= tx || y < 0 || y >= ty || l < 0 || l >= layers) return 1;
    char& s = seen[((long)l * ty + y) * tx + x];
    if (s) return 1;
    s = 1;
  }
  return 0;
}

/* a grid of one tile in x and y: block b is layer b */
static int check_column(long layers)
{
  const long probes[] = {0, 1, layers / 3, layers / 2 + 1, 268435455, 268435456, 268435457, 536870912, layers - 1};
  for (long b : probes) {
    if (b >= layers) continue;
    int x, y, l;
    st_tile((unsigned)b, 1, 1, (int)layers, st_strip(1, 1), &x, &y, &l);
    if (x || y || l != b) return 1;
  }
  return 0;
}

int main()
{
  unsigned r = 1;
  auto next = [&](int m) { r = r * 1664525u + 1013904223u; return 1 + (int)((r >> 8) % m); };
  for (int t = 0; t < 3000; t++) {
    const int tx = next(40), ty = next(40), l = next(30);
    if (check_all(tx, ty, l)) return printf("tiles %d x %d, %d layers\n", tx, ty, l), 1;
  }
  for (long l : {200000000L, 268435457L, 300000000L, 600000000L, 2147483647L})
    if (check_column(l)) return printf("a column of %ld layers\n", l), 1;
  printf("ok\n");
  return 0;
}
