// cg_energy.cuh -- FP64 energy terms of one bead and one voxel, shared by
// the per-replica energy kernel and the drift guard.
//
// The energy is the one whose differences are the per-move dE: SSWLC elastic
// energy (SSWLC.compute_E, chromo/polymers.pyx:1348-1381), the single-site
// binding free energy whose differences are binding_dE
// (chromo/polymers.pyx:1383-1538), and the field energy in the form whose
// differences are the per-move field dE (chromo/fields.pyx:1675-1875).
#pragma once
#include <cooperative_groups.h>

#include "cg_device.cuh"
#include "cg_kernels.h"
#include "cg_move.cuh"

namespace cg {

// Partial sums of one replica's energy over a range of beads and voxels.
struct EnergyParts {
  double el, bi, fe, sx;                // elastic, binding, field, chi-free sum S
  long long dbl[CG_MAX_BINDERS];        // doubly bound beads per binder
};

// Bond i - 1 -> i (i > 0) and the binding free energy of bead i.
template <typename Pos>
__device__ __forceinline__ void bead_energy(const KArgs& a, const RepDev& rd, long long i, EnergyParts& p) {
  const V4<Pos>* r4 = reinterpret_cast<const V4<Pos>*>(a.r4) + rd.bead_off;
  const V4<Pos>* t34 = reinterpret_cast<const V4<Pos>*>(a.t34) + rd.bead_off;
  const double* bonds = a.bonds + rd.bead_off * 6;
  if (i > 0) {
    double r0[3], r1[3], a0[3], a1[3], dr[3], dp[3], bend[3];
    ld3(r4, i - 1, r0); ld3(r4, i, r1); ld3(t34, i - 1, a0); ld3(t34, i, a1);
    Bond<double> b = load_bond<double>(bonds, i - 1);
    for (int j = 0; j < 3; j++) dr[j] = r1[j] - r0[j];
    double par = a0[0] * dr[0] + a0[1] * dr[1] + a0[2] * dr[2];
    for (int j = 0; j < 3; j++) dp[j] = dr[j] - a0[j] * par;
    for (int j = 0; j < 3; j++) bend[j] = a1[j] + (-a0[j] - b.eta * dp[j]);
    p.el += e_pair(b, bend, par, dp);
    if (rd.twist) {  // SSTWLC.compute_E, chromo/polymers.pyx:2250-2285
      const V4<Pos>* t24 = reinterpret_cast<const V4<Pos>*>(a.t24) + rd.bead_off;
      p.el += twist_bond_energy(a.twist + 2 * (rd.bead_off + i - 1), frame_of(t24[i - 1], t34[i - 1]),
                                frame_of(t24[i], t34[i]));
    }
  }
  const unsigned sw = a.states[rd.bead_off + i], mw = a.marks[rd.bead_off + i];
  int tot = 0;
  for (int b = 0; b < rd.nb; b++) {
    int s = (int)((sw >> (8 * b)) & 0xFF), nm = (int)((mw >> (8 * b)) & 0xFF);
    double me = rd.mu[b] > 0 ? rd.mu[b] * (-rd.mu_adjust + 2) : rd.mu[b] * rd.mu_adjust;
    p.bi += bind_f(rd, b, nm, s) - (double)s * me;
    tot += s;
    p.dbl[b] += s == 2;
  }
  if (rd.max_binders != -1 && tot > rd.max_binders) p.bi += kEHugePoly * (double)(tot - rd.max_binders);
}

// Field terms of voxel v (UniformDensityField only).
__device__ __forceinline__ void voxel_energy(const KArgs& a, const RepDev& rd, long long v, EnergyParts& p) {
  const long long* grid = a.grid + rd.vox_off * a.ncol;
  double V = rd.has_access ? a.access_vol[rd.vox_off + v] : rd.vol_bin;
  double rho[CG_MAX_BINDERS];
  for (int b = 0; b < rd.nb; b++) rho[b] = ((double)grid[v * a.ncol + 1 + b] * kFxInv) / V;
  for (int b = 0; b < rd.nb; b++) p.fe += rd.pref[b] * rho[b] * rho[b];
  for (int b = 0; b < rd.nb; b++)
    for (int e = 0; e < rd.nb; e++) p.fe += rd.xpref[b * CG_MAX_BINDERS + e] * rho[b] * rho[e];
  double vf = ((double)grid[v * a.ncol] * kFxInv) / V * rd.bead_vol;
  double sv = (V / rd.bead_vol) * vf * vf;
  // S: the chi-free sum over the voxels at or below vf_limit (a voxel above
  // it costs 1e99 vf, which does not depend on chi)
  if (!(vf > rd.vf_limit)) p.sx += sv;
  p.fe += vf > rd.vf_limit ? kEHugeField * vf : rd.chi * sv;
}

// ---------------------------------------------------------------- sums of one replica
// The energies, the exchange's S and the derivative terms are sums over one
// replica's beads and voxels.  A replica is taken by a cluster of 1 to 8 CTAs
// (cg_sim::sum_log), whose partial sums meet in distributed shared memory and are
// added in rank order: no workspace, the same bits every time.  FP64 runs at 1/64 of
// the FP32 rate here, so the loops hold only the FP64 operations the sums need: rows
// of empty voxels are skipped (two thirds of a 40^3 grid of a 5,000-bead chain), the
// volume factors are applied once to the sums of products of fixed-point values
// (uniform volumes), vf > vf_limit is an integer comparison, products are FMAs, and
// each bond's bead before it comes from the neighbouring lane, already converted (64
// chains of 5,000 beads: energies 53 us, 2.05 ms with a CTA per replica and five
// divisions a voxel).
constexpr int kSumThreads = 256;

// A CTA's replica and its part of the replica's beads or voxels: one of 2^log_ctas.
struct SumPart {
  int rep, rank, log_ctas;
  explicit __device__ __forceinline__ SumPart(int log)
      : rep((int)(blockIdx.x >> log)), rank((int)(blockIdx.x & ((1u << log) - 1u))), log_ctas(log) {}
  __device__ __forceinline__ void of(long long n, long long& lo, long long& hi) const {
    const long long per = (n + (1 << log_ctas) - 1) >> log_ctas;
    lo = rank * per;
    hi = lo + per < n ? lo + per : n;
  }
};

// Launch of one of the sum kernels, instantiated for whole replicas (a CTA each) and for
// replicas split over a cluster of 2^log_ctas CTAs.
template <class... P, class... A>
static void launch_sums(void (*whole)(KArgs, int, P...), void (*split)(KArgs, int, P...), const KArgs& a, int log_ctas,
                        cudaStream_t s, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = 1u << log_ctas;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)a.n_reps << log_ctas);
  c.blockDim = dim3(kSumThreads);
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = log_ctas > 0 ? 1 : 0;
  cudaLaunchKernelEx(&c, log_ctas > 0 ? split : whole, a, log_ctas, P(args)...);
}

// The warps' sums in sh added in warp order, then (SPLIT) the CTAs' in rank order, valid
// in the first 16 threads of rank 0.  Without SPLIT many replicas share the FP64 pipes,
// and zero sums are left out; with it few CTAs run, and loads and additions without
// branches are sooner done (derivative terms of one 1,000-bead chain, 8 CTAs: 12.3 us,
// 14.4 with the branches).
template <bool SPLIT>
__device__ __forceinline__ double over_ctas(double (*sh)[16]) {
  constexpr int kWarps = kSumThreads / 32;
  double t = 0;
  if (!SPLIT) {
    if (threadIdx.x < 16)
      #pragma unroll 1
      for (int w = 0; w < kWarps; w++)
        if (!is_zero64(sh[w][threadIdx.x])) t += sh[w][threadIdx.x];
    return t;
  }
  namespace cgr = cooperative_groups;
  cgr::cluster_group cl = cgr::this_cluster();
  constexpr int kMaxCtas = 8;
  const int ctas = (int)cl.num_blocks();
  if (threadIdx.x < 16) {
#pragma unroll
    for (int w = 0; w < kWarps; w++) t += sh[w][threadIdx.x];
    sh[0][threadIdx.x] = t;
  }
  cl.sync();
  if (cl.block_rank() == 0 && threadIdx.x < 16) {
    double part[kMaxCtas];
#pragma unroll
    for (int r = 1; r < kMaxCtas; r++) part[r] = r < ctas ? cl.map_shared_rank(&sh[0][0], r)[threadIdx.x] : 0.0;
#pragma unroll
    for (int r = 1; r < kMaxCtas; r++)
      if (r < ctas) t += part[r];
  }
  cl.sync();  // no CTA leaves while its sums are read
  return t;
}

// 16 sums over the CTAs of a cluster, valid in the first 16 threads of rank 0
// (thread k: sum k).  Every thread of the cluster calls it.  Within a warp the
// lanes halve the set of sums they carry at each step (16 FP64 additions
// instead of 80).
template <bool SPLIT>
__device__ __forceinline__ double cluster_sums(double (&v)[16], double (*sh)[16]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  bool any = SPLIT;  // of few beads or voxels most warps hold zeros
#pragma unroll
  for (int k = 0; k < 16; k++) any = any || !is_zero64(v[k]);
  if (SPLIT || __any_sync(kFull, any)) {
#pragma unroll
    for (int h = 8, o = 16; h >= 1; h >>= 1, o >>= 1) {
      const bool up = lane & o;
#pragma unroll
      for (int k = 0; k < h; k++) {
        const double keep = up ? v[k + h] : v[k], give = up ? v[k] : v[k + h];
        v[k] = keep + __shfl_xor_sync(kFull, give, o);
      }
    }
    v[0] += __shfl_xor_sync(kFull, v[0], 1);
  } else {
    v[0] = 0.0;
  }
  // lane l holds sum (bits 4, 3, 2, 1 of l as bits 3, 2, 1, 0)
  if (!(lane & 1)) sh[warp][lane >> 1] = v[0];
  __syncthreads();
  return over_ctas<SPLIT>(sh);
}
// The sum of one number over the CTAs of a cluster, by the additions of cluster_sums,
// valid in thread 0 of rank 0.
template <bool SPLIT>
__device__ __forceinline__ double cluster_sum(double v, double (*sh)[16]) {
  const bool any = !is_zero64(v);
  if (SPLIT || __any_sync(kFull, any))
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  else
    v = 0.0;
  if ((threadIdx.x & 31) < 16) sh[threadIdx.x >> 5][threadIdx.x & 31] = v;
  __syncthreads();
  return over_ctas<SPLIT>(sh);
}

// The line of vf_limit in fixed-point bead weights, uniform volumes: the volume
// fraction, as the FP64 expression of voxel_energy gives it, is not above the limit
// for weights up to `sure` and above it beyond `over`; the few between take the
// expression itself (it does not decrease with the weight).
struct Limit {
  long long sure, over;
};
__device__ __forceinline__ bool weight_is_over(const RepDev& rd, long long n) {
  return ((double)n * kFxInv) / rd.vol_bin * rd.bead_vol > rd.vf_limit;
}
__device__ __forceinline__ Limit limit_of(const RepDev& rd) {
  const double est = rd.vf_limit / rd.bead_vol * rd.vol_bin * kFxScale;
  if (!(est < 4e18)) return Limit{0x7FFFFFFFFFFFFFFFLL, 0x7FFFFFFFFFFFFFFFLL};
  if (!(est > 0)) {  // limits of 0 and below: only empty voxels, or none
    const long long w = weight_is_over(rd, 0) ? -1 : 0;
    return Limit{w, w};
  }
  const long long lo = (long long)(est * (1 - 4e-15)) - 2, hi = (long long)(est * (1 + 4e-15)) + 2;
  return Limit{lo < 0 ? 0 : lo, hi};
}
static __device__ __noinline__ bool near_limit(const RepDev& rd, long long n) { return weight_is_over(rd, n); }
__device__ __forceinline__ bool above_limit(const RepDev& rd, const Limit& lim, long long n) {
  return n > lim.sure && (n > lim.over || near_limit(rd, n));
}
// The largest weight not above the limit.
__device__ __forceinline__ long long weight_at_limit(const RepDev& rd) {
  Limit l = limit_of(rd);
  while (l.over - l.sure > 1) {
    const long long mid = l.sure + (l.over - l.sure) / 2;
    if (weight_is_over(rd, mid)) l.over = mid;
    else l.sure = mid;
  }
  return l.sure;
}

// One CTA's part of a replica's voxels: f(voxel, row) for its thread's rows, or
// (SKIP) for those of them that are not empty; g() after every kRowsInFlight.
constexpr int kRowsInFlight = 4;
template <bool SKIP, class F, class G>
__device__ __forceinline__ void for_each_row(const KArgs& a, const RepDev& rd, SumPart part, const F& f, const G& g) {
  const long long* grid = a.grid + rd.vox_off * a.ncol;
  long long v0, v1;
  part.of(rd.n_vox, v0, v1);
  constexpr int U = kRowsInFlight;
  for (long long v = v0 + threadIdx.x; v < v1; v += U * kSumThreads) {
    long long row[U][4];
#pragma unroll
    for (int u = 0; u < U; u++) {
      row[u][0] = row[u][1] = row[u][2] = row[u][3] = 0;
      const long long w = v + u * kSumThreads;
      if (w < v1) load_row(grid + w * a.ncol, a.ncol, row[u]);
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (SKIP ? (row[u][0] | row[u][1] | row[u][2] | row[u][3]) != 0 : v + u * kSumThreads < v1)
        f(v + u * kSumThreads, row[u]);
    g();
  }
}
template <bool SKIP, class F>
__device__ __forceinline__ void for_each_row(const KArgs& a, const RepDev& rd, SumPart part, const F& f) {
  for_each_row<SKIP>(a, rd, part, f, [] {});
}

// Non-uniform volumes: an empty voxel adds nothing, unless its volume is not
// positive (0 / 0 is the energy's value there).
__device__ __forceinline__ bool empty_voxel(const KArgs& a, const RepDev& rd, long long v, const long long (&row)[4]) {
  return (row[0] | row[1] | row[2] | row[3]) == 0 && a.access_vol[rd.vox_off + v] > 0;
}

// Sum of products x y of fixed-point values 0 <= x, y < 2^52, exactly: of the
// products of their 26-bit halves, sum ll + lh 2^26 + hh 2^52 (squares: lh holds
// x_l x_h once).  Three or four 32 x 32 + 64-bit integer multiply-adds, where
// FP64 takes two conversions and an FMA, each ~65 cycles of a quarter SM.  The
// 64-bit sums hold kFxRows products.  40^3 voxels, two binders, with the
// read-back: derivative terms of 64 replicas 124 -> 64 us, energies of 256
// replicas 523 -> 327 us (held to 84 registers, 3 CTAs per SM instead of 2: 98
// and 343 us).
struct FxSum {
  unsigned long long ll, lh, hh;
};
constexpr int kFxRows = 2048;  // lh of x y: two products below 2^52 each
__device__ __forceinline__ void fx_split(long long x, unsigned& l, unsigned& h) {
  l = (unsigned)x & 0x3FFFFFFu;
  h = (unsigned)((unsigned long long)x >> 26);
}
__device__ __forceinline__ void fx_square(FxSum& s, unsigned l, unsigned h) {
  s.ll += (unsigned long long)l * l;
  s.lh += (unsigned long long)l * h;
  s.hh += (unsigned long long)h * h;
}
__device__ __forceinline__ void fx_product(FxSum& s, unsigned l0, unsigned h0, unsigned l1, unsigned h1) {
  s.ll += (unsigned long long)l0 * l1;
  s.lh += (unsigned long long)l0 * h1;
  s.lh += (unsigned long long)h0 * l1;
  s.hh += (unsigned long long)h0 * h1;
}
// The sum in FP64 (one conversion, of its leading 64 bits); `shift` is 26, or 27
// for squares.
template <bool SPLIT>
__device__ __forceinline__ double fx_value(const FxSum& s, int shift) {
  if (!SPLIT && !(s.ll | s.lh | s.hh)) return 0.0;
  unsigned long long lo = s.ll, hi = s.lh >> (64 - shift), t = s.lh << shift;
  lo += t;
  hi += lo < t ? 1 : 0;
  t = s.hh << 52;
  lo += t;
  hi += (s.hh >> 12) + (lo < t ? 1 : 0);
  const int z = hi ? __clzll((long long)hi) : 64;
  const unsigned long long top = z == 64 ? lo : (z ? hi << z | lo >> (64 - z) : hi);
  const double d = __ull2double_rn(top);
  return z == 64 ? d : __longlong_as_double(__double_as_longlong(d) + ((long long)(64 - z) << 52));
}

// Sums of products of the fixed-point columns over a replica's voxels
// (uniform volumes): bead weight squared at or below the limit, binder columns
// squared and in pairs (01, 02, 12).  What the integer sums cannot hold -- a
// column of 2^52 (4,096 beads in one voxel) or more, full 64-bit sums -- and the
// rows above the limit go to FP64 sums in shared memory, a column per thread.
struct GridSums {
  FxSum s00, sbb[CG_MAX_BINDERS], sx[3];
  int left;    // outer iterations until the 64-bit sums are emptied
  bool rest;   // the FP64 sums are in use
};
enum { kRest00, kRestBB, kRestX = kRestBB + CG_MAX_BINDERS, kRestOver = kRestX + 3, kRestVf, kRests };
typedef double RestSums[kRests][kSumThreads];

__device__ __forceinline__ void init_sums(GridSums& s, RestSums& rest) {
  s = GridSums{};
  s.left = kFxRows / kRowsInFlight;
  for (int k = 0; k < kRests; k++) rest[k][threadIdx.x] = 0.0;
}
// The integer sums as FP64, in the order of kRest00 .. kRestX + 2.
template <bool SPLIT, class F>
__device__ __forceinline__ void sum_values(const GridSums& s, int nb, const F& f) {
  f(kRest00, fx_value<SPLIT>(s.s00, 27));
#pragma unroll
  for (int b = 0; b < CG_MAX_BINDERS; b++) f(kRestBB + b, b < nb ? fx_value<SPLIT>(s.sbb[b], 27) : 0.0);
  f(kRestX, nb > 1 ? fx_value<SPLIT>(s.sx[0], 26) : 0.0);
  f(kRestX + 1, nb > 2 ? fx_value<SPLIT>(s.sx[1], 26) : 0.0);
  f(kRestX + 2, nb > 2 ? fx_value<SPLIT>(s.sx[2], 26) : 0.0);
}
static __device__ __noinline__ void add_row_f64(RestSums& rest, long long gmax, double vol, double bead_vol,
                                                long long r0, long long r1, long long r2, long long r3) {
  const int t = threadIdx.x;
  const double g0 = (double)r0, g[3] = {(double)r1, (double)r2, (double)r3};
  double& s00 = rest[r0 <= gmax ? kRest00 : kRestOver][t];
  s00 = __fma_rn(g0, g0, s00);
  if (r0 > gmax) rest[kRestVf][t] += (g0 * kFxInv) / vol * bead_vol;
  for (int b = 0; b < 3; b++) rest[kRestBB + b][t] = __fma_rn(g[b], g[b], rest[kRestBB + b][t]);
  rest[kRestX][t] = __fma_rn(g[0], g[1], rest[kRestX][t]);
  rest[kRestX + 1][t] = __fma_rn(g[0], g[2], rest[kRestX + 1][t]);
  rest[kRestX + 2][t] = __fma_rn(g[1], g[2], rest[kRestX + 2][t]);
}
__device__ __forceinline__ void add_row(const RepDev& rd, long long gmax, const long long (&row)[4], GridSums& s,
                                        RestSums& rest) {
  if (row[0] > gmax || (unsigned long long)(row[0] | row[1] | row[2] | row[3]) >> 52) {
    add_row_f64(rest, gmax, rd.vol_bin, rd.bead_vol, row[0], row[1], row[2], row[3]);
    s.rest = true;
    return;
  }
  unsigned l[4], h[4];
#pragma unroll
  for (int k = 0; k < 4; k++) fx_split(row[k], l[k], h[k]);
  fx_square(s.s00, l[0], h[0]);
  fx_square(s.sbb[0], l[1], h[1]);
  if (rd.nb > 1) {
    fx_square(s.sbb[1], l[2], h[2]);
    fx_product(s.sx[0], l[1], h[1], l[2], h[2]);
  }
  if (rd.nb > 2) {
    fx_square(s.sbb[2], l[3], h[3]);
    fx_product(s.sx[1], l[1], h[1], l[3], h[3]);
    fx_product(s.sx[2], l[2], h[2], l[3], h[3]);
  }
}
// Called after every outer iteration: empties full integer sums.
template <bool SPLIT>
__device__ __forceinline__ void drain_sums(int nb, GridSums& s, RestSums& rest) {
  if (--s.left) return;
  sum_values<SPLIT>(s, nb, [&](int k, double x) { rest[k][threadIdx.x] += x; });
  s = GridSums{};
  s.left = kFxRows / kRowsInFlight;
  s.rest = true;
}
// The sums of one CTA's part of a replica: out[kRest00 .. kRestVf].
template <bool SPLIT>
__device__ __forceinline__ void grid_sums(const KArgs& a, const RepDev& rd, SumPart part, long long gmax, RestSums& rest,
                                          double (&out)[kRests]) {
  GridSums s;
  init_sums(s, rest);
  const int nb = rd.nb;
  for_each_row<true>(a, rd, part, [&](long long, const long long (&row)[4]) { add_row(rd, gmax, row, s, rest); },
                     [&] { drain_sums<SPLIT>(nb, s, rest); });
  out[kRestOver] = out[kRestVf] = 0.0;
  sum_values<SPLIT>(s, nb, [&](int k, double x) { out[k] = x; });
  if (s.rest)
#pragma unroll
    for (int k = 0; k < kRests; k++) out[k] += rest[k][threadIdx.x];
}

// Elastic energy of bond i - 1 -> i from the two beads' vectors in FP64.
__device__ __forceinline__ double bond_energy(const double* b, const double r0[3], const double r1[3],
                                              const double a0[3], const double a1[3]) {
  const double2 q0 = *reinterpret_cast<const double2*>(b), q1 = *reinterpret_cast<const double2*>(b + 2);
  const double eb = q0.x, g = q0.y, ep = q1.x, epp = q1.y, eta = b[4];
  double dr[3], dp[3], bend[3];
  for (int j = 0; j < 3; j++) dr[j] = r1[j] - r0[j];
  const double par = __fma_rn(a0[2], dr[2], __fma_rn(a0[1], dr[1], a0[0] * dr[0]));
  for (int j = 0; j < 3; j++) dp[j] = __fma_rn(-a0[j], par, dr[j]);
  for (int j = 0; j < 3; j++) bend[j] = __fma_rn(-eta, dp[j], a1[j] - a0[j]);
  const double b2 = __fma_rn(bend[2], bend[2], __fma_rn(bend[1], bend[1], bend[0] * bend[0]));
  const double p2 = __fma_rn(dp[2], dp[2], __fma_rn(dp[1], dp[1], dp[0] * dp[0]));
  const double x = par - g;
  return 0.5 * __fma_rn(eb, b2, __fma_rn(ep, x * x, epp * p2));
}

// One CTA's part of a replica's beads: elastic (and twist) energy, binding free
// energy from the replica's table `bf` ([binder][marks][state], the chemical
// potential's term included), doubly bound beads per binder, and the sites
// bound beyond max_binders.  A warp takes 31 bonds a pass: lane l holds bead
// i0 + l, converted once, and its bond to lane l - 1's bead.
template <typename Pos>
__device__ __forceinline__ void bead_sums(const KArgs& a, const RepDev& rd, SumPart part, const double* bf, double& el,
                                          double& bi, int (&dbl)[CG_MAX_BINDERS], long long& excess) {
  const V4<Pos>* r4 = reinterpret_cast<const V4<Pos>*>(a.r4) + rd.bead_off;
  const V4<Pos>* t34 = reinterpret_cast<const V4<Pos>*>(a.t34) + rd.bead_off;
  const V4<Pos>* t24 = reinterpret_cast<const V4<Pos>*>(a.t24) + rd.bead_off;
  const double* bonds = a.bonds + rd.bead_off * 6;
  long long b0, b1;
  part.of(rd.n_beads, b0, b1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // lane 0's bead is the one before the pass's first
  for (long long i0 = b0 - 1 + 31LL * warp; i0 + 1 < b1; i0 += 31LL * (kSumThreads / 32)) {
    const long long i = i0 + lane;
    const bool have = i >= 0 && i < b1;
    double r[3] = {0, 0, 0}, t[3] = {0, 0, 0}, rp[3], tp[3];
    if (have) {
      ld3(r4, i, r);
      ld3(t34, i, t);
    }
    for (int j = 0; j < 3; j++) {
      rp[j] = __shfl_up_sync(kFull, r[j], 1);
      tp[j] = __shfl_up_sync(kFull, t[j], 1);
    }
    if (!have || lane == 0) continue;
    if (i > 0) {
      el += bond_energy(bonds + 6 * (i - 1), rp, r, tp, t);
      if (rd.twist)  // SSTWLC.compute_E, chromo/polymers.pyx:2250-2285
        el += twist_bond_energy(a.twist + 2 * (rd.bead_off + i - 1), frame_of(t24[i - 1], t34[i - 1]),
                                frame_of(t24[i], t34[i]));
    }
    const unsigned sw = a.states[rd.bead_off + i], mw = a.marks[rd.bead_off + i];
    int tot = 0;
#pragma unroll
    for (int b = 0; b < CG_MAX_BINDERS; b++)
      if (b < rd.nb) {
        const int s = (int)((sw >> (8 * b)) & 0xFF), nm = (int)((mw >> (8 * b)) & 0xFF);
        bi += bf[(b * (CG_MAX_MARK + 1) + nm) * (CG_MAX_MARK + 1) + s];
        tot += s;
        dbl[b] += s == 2;
      }
    if (rd.max_binders != -1 && tot > rd.max_binders) excess += tot - rd.max_binders;
  }
}

// The replica's binding table with the chemical potential's term
// (polymers.pyx:1494-1537), by the CTA's threads.
__device__ __forceinline__ void fill_bind_table(const RepDev& rd, double* bf) {
  for (int k = threadIdx.x; k < CG_MAX_BINDERS * (CG_MAX_MARK + 1) * (CG_MAX_MARK + 1); k += blockDim.x) {
    const int b = k / ((CG_MAX_MARK + 1) * (CG_MAX_MARK + 1)), s = k % (CG_MAX_MARK + 1);
    const double me = rd.mu[b] > 0 ? rd.mu[b] * (-rd.mu_adjust + 2) : rd.mu[b] * rd.mu_adjust;
    bf[k] = rd.bind_f[k] - (double)s * me;
  }
}

// one block; deterministic tree reduction, the total valid in warp 0
__device__ __forceinline__ double block_total(double v, double* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double t = 0;
  if (threadIdx.x < 32) {
    t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
    t = warp_sum(t);
  }
  return t;
}

}  // namespace cg
