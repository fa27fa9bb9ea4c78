/* cg_exact.h -- an exact sum of FP64 terms in fixed point (host and device; plain C,
 * so that it can be tested without a GPU).
 *
 * Eleven limbs of 20 bits, from 2^-160 up, in 32-bit integers: a term's 53 bits go to
 * four of them (cgx_split), and sums of the limbs by any number of threads in any
 * order are the same integers.  A limb holds the parts of 2,047 terms besides one
 * carried form (cgx_carry).  Terms are taken from 2^-108 up to 2^32. */
#ifndef CG_EXACT_H
#define CG_EXACT_H

#include <string.h>

#ifdef __CUDACC__
#define CGX_FN __host__ __device__ __forceinline__
#else
#define CGX_FN static inline
#endif

#define CGX_LIMBS 11
#define CGX_TERMS 2047

/* The parts v[0..3] of the FP64 number with these bits and the index of the first
 * one's limb; -1 where the number is outside the range (and for zeros, infinities and
 * NaN). */
CGX_FN int cgx_split(unsigned long long bits, int v[4]) {
  const unsigned p = (unsigned)(bits >> 52 & 0x7FF) - (1075u - 160u); /* place of the last bit, from 2^-160 */
  if (p > 139u) return -1;
  const unsigned i = p / 20u, sh = p - 20u * i;
  const unsigned long long m = (bits & 0xFFFFFFFFFFFFFull) | 1ull << 52, r = m >> (20u - sh);
  const int sign = bits >> 63 ? -1 : 0;
  v[0] = (int)((unsigned)m << sh & 0xFFFFFu);
  v[1] = (int)((unsigned)r & 0xFFFFFu);
  v[2] = (int)((unsigned)(r >> 20) & 0xFFFFFu);
  v[3] = (int)(unsigned)(r >> 40);
  for (int k = 0; k < 4; k++) v[k] = (v[k] ^ sign) - sign;
  return (int)i;
}

/* The limbs in [0, 2^20) but the last, which holds the sign. */
CGX_FN void cgx_carry(int* L) {
  for (int i = 0; i + 1 < CGX_LIMBS; i++) {
    const int c = L[i] >> 20;
    L[i] -= c * (1 << 20);
    L[i + 1] += c;
  }
}

/* The limbs' sum, rounded once (to nearest, ties to even). */
CGX_FN double cgx_value(const int* L) {
  long long c = 0;
  for (int i = 0; i < CGX_LIMBS; i++) c = (c + L[i]) >> 20;
  const int sign = (int)(c >> 63);
  unsigned long long g[4] = {0, 0, 0, 0}; /* groups of 60 bits, the uppermost first */
  c = 0;
  for (int i = 0; i < CGX_LIMBS; i++) {
    c += (L[i] ^ sign) - sign;
    g[3 - i / 3] |= (unsigned long long)(c & 0xFFFFF) << (20 * (i % 3));
    c >>= 20;
  }
  g[0] |= (unsigned long long)c << 40;
  int w = 20;
  unsigned long long rest = g[3];
  if (!g[0]) { g[0] = g[1]; g[1] = g[2]; g[2] = g[3]; rest = 0; w = -40; }
  if (!g[0]) { g[0] = g[1]; g[1] = g[2]; g[2] = 0; w -= 60; }
  if (!g[0]) { g[0] = g[1]; g[1] = 0; w -= 60; }
  if (!g[0]) return 0.0;
#ifdef __CUDA_ARCH__
  const int z = __clzll((long long)g[0]);
#else
  const int z = __builtin_clzll(g[0]);
#endif
  /* the leading 64 bits; the bits below them in the last one, below the rounding's */
  const unsigned long long low = z <= 60 ? g[1] >> (60 - z) : g[1] << (z - 60);
  const unsigned long long lost = z <= 60 ? g[1] & ((1ull << (60 - z)) - 1) : 0ull;
  const double d = (double)(g[0] << z | low | ((lost | g[2] | rest) ? 1ull : 0ull));
  unsigned long long bits;
  memcpy(&bits, &d, 8);
  bits += (unsigned long long)(long long)(w - z) << 52; /* times 2^(w - z) */
  if (sign) bits |= 1ull << 63;
  double out;
  memcpy(&out, &bits, 8);
  return out;
}

#endif
