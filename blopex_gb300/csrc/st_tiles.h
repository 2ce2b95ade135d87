/* st_tiles.h -- the order of the tiles of the TMA stencil kernels (operators.cu):
   strips of about ST_STRIP tiles, z before the next strip, so that the CTAs that
   share halo planes run within a few columns of each other. */
#ifndef ST_TILES_H
#define ST_TILES_H

#ifdef __CUDACC__
#define ST_HD __host__ __device__ __forceinline__
#else
#define ST_HD inline
#endif

#define ST_STRIP 16

/* tile rows of a strip; no more than there are, so that a strip's tiles times the
   layers never exceed the grid (and its 31 bits) */
static inline int st_strip(int tiles_x, int tiles_y)
{
  const int strip = tiles_x < ST_STRIP ? ST_STRIP / tiles_x : 1;
  return strip < tiles_y ? strip : tiles_y;
}

/* block b of tiles_x x tiles_y x layers: its tile column and row, and its layer */
static ST_HD void st_tile(unsigned b, int tiles_x, int tiles_y, int layers, int strip, int* x, int* y, int* layer)
{
  const unsigned per = (unsigned)tiles_x * strip * layers;
  const int s0 = (int)(b / per) * strip;
  const unsigned rest = b % per, in_strip = (unsigned)tiles_x * (strip < tiles_y - s0 ? strip : tiles_y - s0);
  const int tile = (int)(rest % in_strip);
  *layer = (int)(rest / in_strip);
  *x = tile % tiles_x;
  *y = s0 + tile / tiles_x;
}

#endif
