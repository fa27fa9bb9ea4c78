/* cg_steric_tiles.h -- how the steric kernels split a chain (host; plain C, so
 * that it can be tested without a GPU).
 *
 * Rows come in tiles of 32 on the grid's x axis, columns in chunks on its y axis,
 * which the hardware limits to 65,535.  A chunk is 1,024 columns (one pass of a
 * tile's threads, four columns each), or as many passes as keep the chunks to
 * 32.  Where fewer than two CTAs per SM would run so, chunks of 256 columns, a
 * column a thread, spread the FP64 terms of the few near pairs, ~4 k cycles each,
 * over more warps.  They are taken as long as they fit the y axis and the buffer
 * of the tiles' sums (n_beads + 32 doubles). */
#ifndef CG_STERIC_TILES_H
#define CG_STERIC_TILES_H

#define CG_STERIC_ROWS 32
#define CG_STERIC_THREADS 256
#define CG_STERIC_MAX_CHUNKS 65535

/* Columns per chunk for tiles of rows against n_beads columns on n_sm SMs. */
static inline long long cg_steric_chunk(long long n_beads, long long tiles, int n_sm) {
  const long long t = CG_STERIC_THREADS, narrow = (n_beads + t - 1) / t;
  long long wide = ((n_beads + 31) / 32 + t - 1) / t * t;
  if (wide < 4 * t) wide = 4 * t;
  if (tiles * ((n_beads + wide - 1) / wide) < 2LL * n_sm && narrow <= CG_STERIC_MAX_CHUNKS &&
      tiles * narrow <= n_beads + 32)
    return t;
  return wide;
}

#endif
