/* cg_steric_tiles.h -- how the steric kernels split a chain (host; plain C, so
 * that it can be tested without a GPU).
 *
 * Rows come in tiles of up to 32 on the grid's x axis, columns in chunks on its y
 * axis, which the hardware limits to 65,535.  A chunk is 1,024 columns (one pass of
 * a tile's threads, four columns each), or as many passes as keep the chunks to 32.
 * Where fewer than two CTAs per SM would run so, chunks of 256 columns, a column a
 * thread, and then tiles of fewer rows spread the FP64 terms of the near pairs, ~4 k
 * cycles each for a warp, over more SMs, as long as the chunks fit the y axis and the
 * tiles' sums their buffer (n_beads + 32 doubles): 300 beads all within e 33 us, 120 in
 * tiles of 32 rows throughout; 100 moved beads of 1,000, e seven spacings, 40 and 170. */
#ifndef CG_STERIC_TILES_H
#define CG_STERIC_TILES_H

#define CG_STERIC_ROWS 32
#define CG_STERIC_THREADS 256
#define CG_STERIC_MAX_CHUNKS 65535

/* Columns per chunk and (*rows) rows per tile for n_rows rows against n_beads columns
 * on n_sm SMs. */
static inline long long cg_steric_split(long long n_beads, long long n_rows, int n_sm, int* rows) {
  const long long t = CG_STERIC_THREADS, narrow = (n_beads + t - 1) / t;
  long long tiles = (n_rows + CG_STERIC_ROWS - 1) / CG_STERIC_ROWS;
  long long wide = ((n_beads + 31) / 32 + t - 1) / t * t;
  *rows = CG_STERIC_ROWS;
  if (wide < 4 * t) wide = 4 * t;
  if (tiles * ((n_beads + wide - 1) / wide) >= 2LL * n_sm || narrow > CG_STERIC_MAX_CHUNKS ||
      tiles * narrow > n_beads + 32)
    return wide;
  while (*rows > 1 && tiles * narrow < 2LL * n_sm) {
    const long long more = (n_rows + *rows / 2 - 1) / (*rows / 2);
    if (more * narrow > n_beads + 32) break;
    *rows /= 2;
    tiles = more;
  }
  return t;
}

#endif
