// cg_grad.cu -- derivatives of the FP64 replica energy (no counterpart in the
// reference, which has no derivatives).
//
// The energy is the one cg_energy reports: SSWLC elastic energy
// (chromo/polymers.pyx:1348-1381), binding free energy (:1383-1538) and the
// field energy in the form whose differences are the per-move field dE
// (chromo/fields.pyx:1675-1875):
//   E_field = sum_v [ sum_b pref_b rho_b^2 + sum_bc xpref_bc rho_b rho_c
//                     + (vf > vf_limit ? 1e99 vf : chi (V / V_bead) vf^2) ]
//             + sum_b intra_b #(beads with state_b == 2),
// rho_b = (sum_i w_i(v) s_ib) / V and vf = (sum_i w_i(v)) V_bead / V, w_i(v)
// the trilinear weight of bead i at voxel v.
//
// gradient_kernel: dE/dr_i = elastic (the two bonds at bead i) + field
// (sum over the bead's eight voxels of dE_v/dw_i(v) dw_i(v)/dr_i).
// terms_kernel: the sums whose linear combinations are dE/d(chi, mu, eps)
// and the reweighting observables, optionally added (with their outer
// products) to per-replica running sums over sampled configurations.
#include <cuda_runtime.h>

#include <algorithm>

#include "cg_energy.cuh"

namespace cg {

// Derivatives of E_pair of bond (bead j -> bead j+1), dr = r_{j+1} - r_j, a0 / a1
// the t3 tangents at j / j+1 taken as free vectors.  With par = a0.dr,
// dp = P dr (P = I - a0 a0^T), bend = a1 - a0 - eta dp:
//   dE/ddr = -eta eb P bend + ep (par - gamma) a0 + epp P dp,
//   dE/da1 = eb bend,
//   dE/da0 = eb (eta (par bend + (a0.bend) dr) - bend) + ep (par - gamma) dr
//            - epp (par dp + (a0.dp) dr).
__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
  return __fma_rn(a[2], b[2], __fma_rn(a[1], b[1], a[0] * b[0]));
}
__device__ __forceinline__ void bond_grad(const double* bp, const double a0[3], const double a1[3],
                                          const double dr[3], bool tangents, double g[3], double g0[3],
                                          double g1[3]) {
  const double2 q0 = *reinterpret_cast<const double2*>(bp), q1 = *reinterpret_cast<const double2*>(bp + 2);
  const double eb = q0.x, gamma = q0.y, ep = q1.x, epp = q1.y, eta = bp[4];
  const double par = dot3(a0, dr);
  double dp[3], bend[3];
  for (int j = 0; j < 3; j++) dp[j] = __fma_rn(-a0[j], par, dr[j]);
  for (int j = 0; j < 3; j++) bend[j] = __fma_rn(-eta, dp[j], a1[j] - a0[j]);
  const double ab = dot3(a0, bend), ad = dot3(a0, dp);
  const double ee = eta * eb, px = ep * (par - gamma);
  // -ee (bend - a0 ab) + px a0 + epp (dp - a0 ad) = -ee bend + epp dp + (ee ab + px - epp ad) a0
  const double c = __fma_rn(ee, ab, __fma_rn(-epp, ad, px));
  for (int j = 0; j < 3; j++) g[j] = __fma_rn(-ee, bend[j], __fma_rn(epp, dp[j], c * a0[j]));
  if (tangents) {
    const double cb = __fma_rn(ee, par, -eb), cp = -epp * par;
    for (int j = 0; j < 3; j++) {
      g1[j] = eb * bend[j];
      g0[j] = __fma_rn(cb, bend[j], __fma_rn(c, dr[j], cp * dp[j]));
    }
  }
}

// One coordinate's voxels (lower, upper) and its fraction of the way between
// them, in FP64 (the construction of voxel_axes).  The quotient by the voxel
// width is a product and an FMA remainder, corrected to floor(x / d), comparisons
// and roundings in integer steps; coordinates and boxes that wrap_near leaves
// out take the plain form.
struct AxisCell {
  double r;
  int ind;
};
static __device__ __noinline__ AxisCell far_cell(double pos, double width, double d, double inv) {
  const double x = pymod(pos + 0.5 * width, width) - 0.5 * d;
  double q = floor(x * inv);
  double r = __fma_rn(-q, d, x);
  if (r < 0) {
    q -= 1;
    r = __fma_rn(-q, d, x);
  } else if (r >= d) {
    const double r1 = __fma_rn(-(q + 1), d, x);
    if (r1 >= 0) { q += 1; r = r1; }
  }
  return AxisCell{r, (int)q};
}
__device__ __forceinline__ double cell_of(double pos, double width, double d, double inv, float iw, int n, int& lo,
                                          int& hi) {
  double m;
  AxisCell c;
  if (wrap_near(pos + 0.5 * width, width, iw, m)) {
    const double x = m - 0.5 * d;  // -1/2 <= x / d < n
    const int ind = floor_index(x * inv);
    c.ind = ind;
    c.r = __fma_rn(ind < 0 ? 1.0 : -whole_double(ind), d, x);
    const long long bits = __double_as_longlong(c.r);
    const int fix = bits < 0 && (bits << 1) != 0 ? -1 : (bits >= __double_as_longlong(d) ? 1 : 0);
    if (fix) {
      const double r1 = __fma_rn(-(double)(ind + fix), d, x);
      if (fix < 0 || r1 >= 0) {
        c.ind = ind + fix;
        c.r = r1;
      }
    }
  } else {
    c = far_cell(pos, width, d, inv);
  }
  const int li = c.ind == -1 ? n - 1 : c.ind;
  lo = li < 0 ? 0 : (li >= n ? n - 1 : li);
  hi = lo + 1 == n ? 0 : lo + 1;
  return c.r * inv;
}

// dE_v/dw at one voxel of a replica with non-uniform volumes (states in sw).
__device__ __forceinline__ double voxel_slope(const KArgs& a, const RepDev& rd, long long v, unsigned sw) {
  const long long* row = a.grid + (rd.vox_off + v) * a.ncol;
  const double V = a.access_vol[rd.vox_off + v];
  double rho[CG_MAX_BINDERS];
  for (int b = 0; b < rd.nb; b++) rho[b] = ((double)row[1 + b] * kFxInv) / V;
  const double vf = ((double)row[0] * kFxInv) / V * rd.bead_vol;
  double phi = vf > rd.vf_limit ? kEHugeField * rd.bead_vol / V : 2 * rd.chi * vf;
  for (int b = 0; b < rd.nb; b++) {
    const int s = (int)((sw >> (8 * b)) & 0xFF);
    if (!s) continue;
    double pb = 2 * rd.pref[b] * rho[b];
    for (int c = 0; c < rd.nb; c++) pb += (rd.xpref[b * CG_MAX_BINDERS + c] + rd.xpref[c * CG_MAX_BINDERS + b]) * rho[c];
    phi += (double)s * pb / V;
  }
  return phi;
}

// dE/dr (and dE/dt3) of every bead.  FP64 runs at 1/64 of the FP32 rate here, so
// the kernel is bound by its FP64 operations (~150 a bead): a warp takes 30
// beads a pass, each lane converting one bead and evaluating the bond to the
// next lane's, whose derivatives come back by shuffles (every bond once); with
// uniform volumes dE_v/dw is a linear combination of the voxel's fixed-point
// columns whose coefficients depend on the bead's states only (a table of the
// CTA), and the eight corners are contracted axis by axis.  Five divisions a
// corner and every bond twice took 680 us for 64 chains of 5,000 beads with the
// read-back; one pass a warp and conversions, comparisons and roundings on the
// FP64 pipe 229, now 183.
template <typename Pos, typename Out>
__global__ void __launch_bounds__(128) gradient_kernel(KArgs a, Out* out, Out* out_t3) {
  __shared__ double tab[64][CG_MAX_BINDERS];  // binder columns' coefficients for packed states (2 bits each)
  __shared__ double k0_sh, huge_sh, inv_sh[3];
  __shared__ float iw_sh[3];
  __shared__ long long gmax_sh;
  const int rep = blockIdx.y;
  const RepDev& rd = a.reps[rep];
  const long long N = rd.n_beads;
  constexpr int kBeads = 30;  // beads a warp writes per pass
  if (blockIdx.x * (long long)(blockDim.x / 32) * kBeads >= N) return;
  const bool field = rd.field_kind == 2, uniform = field && !rd.has_access;
  if (field) {
    const double u = 1.0 / rd.vol_bin;  // the columns as fx_double gives them
    if (uniform)
      for (int k = threadIdx.x; k < 64 * CG_MAX_BINDERS; k += blockDim.x) {
        const int code = k / CG_MAX_BINDERS, c = k % CG_MAX_BINDERS;
        double t = 0;
        if (c < rd.nb)
          for (int b = 0; b < rd.nb; b++) {
            const int s = (code >> (2 * b)) & 3;
            double pb = rd.xpref[b * CG_MAX_BINDERS + c] + rd.xpref[c * CG_MAX_BINDERS + b];
            if (b == c) pb += 2 * rd.pref[b];
            if (s) t += (double)s * pb;
          }
        tab[code][c] = t * (u * u);
      }
    if (threadIdx.x < 3) {
      const double width[3] = {rd.wx, rd.wy, rd.wz};
      const int n[3] = {rd.nx, rd.ny, rd.nz};
      inv_sh[threadIdx.x] = (double)n[threadIdx.x] / width[threadIdx.x];
      iw_sh[threadIdx.x] = (float)(1.0 / width[threadIdx.x]);
    }
    if (threadIdx.x == 64) {
      k0_sh = 2 * rd.chi * rd.bead_vol * u;
      huge_sh = kEHugeField * rd.bead_vol / rd.vol_bin;
    }
    if (threadIdx.x == 96) gmax_sh = uniform ? weight_at_limit(rd) : 0;
  }
  __syncthreads();
  const V4<Pos>* r4 = reinterpret_cast<const V4<Pos>*>(a.r4) + rd.bead_off;
  const V4<Pos>* t34 = reinterpret_cast<const V4<Pos>*>(a.t34) + rd.bead_off;
  const double* bonds = a.bonds + rd.bead_off * 6;
  const unsigned* st = a.states + rd.bead_off;
  const long long* grid = a.grid + rd.vox_off * a.ncol;
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const bool tangents = out_t3 != nullptr;
  for (long long i0 = ((long long)blockIdx.x * wpb + (threadIdx.x >> 5)) * kBeads - 1; i0 + 1 < N;
       i0 += (long long)gridDim.x * wpb * kBeads) {
    const long long i = i0 + lane;
    const bool have = i >= 0 && i < N;
    double r[3] = {0, 0, 0}, t[3] = {0, 0, 0};
    if (have) {
      ld3(r4, i, r);
      ld3(t34, i, t);
    }
    double dr[3], tn[3], g[3] = {0, 0, 0}, g0[3] = {0, 0, 0}, g1[3] = {0, 0, 0};
    for (int j = 0; j < 3; j++) {
      dr[j] = __shfl_down_sync(kFull, r[j], 1) - r[j];
      tn[j] = __shfl_down_sync(kFull, t[j], 1);
    }
    if (have && lane < 31 && i + 1 < N) bond_grad(bonds + 6 * i, t, tn, dr, tangents, g, g0, g1);
    // bond (i-1 -> i): + dE/ddr, dE/da1; bond (i -> i+1): - dE/ddr, dE/da0
    double gr[3], gt[3];
    for (int j = 0; j < 3; j++) {
      gr[j] = __shfl_up_sync(kFull, g[j], 1) - g[j];
      gt[j] = __shfl_up_sync(kFull, g1[j], 1) + g0[j];
    }
    if (!have || lane == 0 || lane > kBeads) continue;
    if (field) {
      int lo[3], hi[3];
      const double inv[3] = {inv_sh[0], inv_sh[1], inv_sh[2]};
      const double fx = cell_of(r[0], rd.wx, rd.dx, inv[0], iw_sh[0], rd.nx, lo[0], hi[0]);
      const double fy = cell_of(r[1], rd.wy, rd.dy, inv[1], iw_sh[1], rd.ny, lo[1], hi[1]);
      const double fz = cell_of(r[2], rd.wz, rd.dz, inv[2], iw_sh[2], rd.nz, lo[2], hi[2]);
      const unsigned sw = st[i];
      const int code = (int)((sw & 3u) | ((sw >> 6) & 12u) | ((sw >> 12) & 48u));
      double phi[8];
#pragma unroll
      for (int l = 0; l < 8; l++) {
        const long long v = (l & 1 ? hi[0] : lo[0]) +
                            (long long)rd.nx * ((l & 2 ? hi[1] : lo[1]) + (long long)rd.ny * (l & 4 ? hi[2] : lo[2]));
        if (uniform) {
          long long row[4];
          load_row(grid + v * a.ncol, a.ncol, row);
          double p = row[0] > gmax_sh ? huge_sh : k0_sh * fx_double(row[0]);
#pragma unroll
          for (int c = 0; c < CG_MAX_BINDERS; c++)
            if (row[1 + c]) p = __fma_rn(tab[code][c], fx_double(row[1 + c]), p);
          phi[l] = p;
        } else {
          phi[l] = voxel_slope(a, rd, v, sw);
        }
      }
      // along x: slopes d and values e on the four (y, z) edges; then y, z
      double d[4], e[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        d[k] = phi[2 * k + 1] - phi[2 * k];
        e[k] = __fma_rn(fx, d[k], phi[2 * k]);
      }
      const double dx0 = __fma_rn(fy, d[1] - d[0], d[0]), dx1 = __fma_rn(fy, d[3] - d[2], d[2]);
      const double ey0 = e[1] - e[0], ey1 = e[3] - e[2];
      const double ez0 = __fma_rn(fy, ey0, e[0]), ez1 = __fma_rn(fy, ey1, e[2]);
      gr[0] = __fma_rn(inv[0], __fma_rn(fz, dx1 - dx0, dx0), gr[0]);
      gr[1] = __fma_rn(inv[1], __fma_rn(fz, ey1 - ey0, ey0), gr[1]);
      gr[2] = __fma_rn(inv[2], ez1 - ez0, gr[2]);
    }
    Out* o = out + 3 * (rd.bead_off + i);
    for (int j = 0; j < 3; j++) o[j] = (Out)gr[j];
    if (tangents) {
      Out* ot = out_t3 + 3 * (rd.bead_off + i);
      for (int j = 0; j < 3; j++) ot[j] = (Out)gt[j];
    }
  }
}

// Terms T[14] of one replica: [0] S = sum_(vf <= limit) (V / V_bead) vf^2,
// [1..3] sum_v rho_b^2, [4..6] sum_v rho_0 rho_1, rho_0 rho_2, rho_1 rho_2,
// [7..9] #(state_b == 2), [10..12] sum_i s_ib, [13] sum_v (W / V)^2 with W the
// bead weight of the voxel.  acc (or null): running sums [T, T T^T, count].
// A CTA or (SPLIT) a cluster per replica (see cg_energy.cuh).
template <bool SPLIT>
__global__ void __launch_bounds__(kSumThreads)
    terms_kernel(KArgs a, int log_ctas, double* terms, double* acc) {
  __shared__ double sh[kSumThreads / 32][16];
  __shared__ double T[16];
  __shared__ RestSums rest;
  __shared__ long long gmax_sh;
  const SumPart part(log_ctas);
  const int rep = part.rep, rank = part.rank;
  const RepDev& rd = a.reps[rep];
  const bool field = rd.field_kind == 2, uniform = field && !rd.has_access;
  if (threadIdx.x == 0) gmax_sh = uniform ? weight_at_limit(rd) : 0;
  __syncthreads();
  int dbl[CG_MAX_BINDERS] = {0, 0, 0};
  long long sum[CG_MAX_BINDERS] = {0, 0, 0};
  {
    const unsigned* st = a.states + rd.bead_off;
    long long b0, b1;
    part.of(rd.n_beads, b0, b1);
    for (long long i = b0 + threadIdx.x; i < b1; i += blockDim.x) {
      const unsigned sw = st[i];
#pragma unroll
      for (int b = 0; b < CG_MAX_BINDERS; b++)
        if (b < rd.nb) {
          const int s = (int)((sw >> (8 * b)) & 0xFF);
          dbl[b] += s == 2;
          sum[b] += s;
        }
    }
  }
  double g[kRests] = {}, dens2 = 0;
  if (uniform) {
    grid_sums<SPLIT>(a, rd, part, gmax_sh, rest, g);
  } else if (field) {
    for_each_row<false>(a, rd, part, [&](long long v, const long long (&row)[4]) {
      if (empty_voxel(a, rd, v, row)) return;
      const double V = a.access_vol[rd.vox_off + v];
      double rho[CG_MAX_BINDERS] = {0, 0, 0};
#pragma unroll
      for (int b = 0; b < CG_MAX_BINDERS; b++)
        if (b < rd.nb) rho[b] = ((double)row[1 + b] * kFxInv) / V;
      const double dens = ((double)row[0] * kFxInv) / V;
      const double vf = dens * rd.bead_vol;
      if (vf <= rd.vf_limit) g[kRest00] += (V / rd.bead_vol) * vf * vf;
      for (int b = 0; b < CG_MAX_BINDERS; b++) g[kRestBB + b] += rho[b] * rho[b];
      g[kRestX + 0] += rho[0] * rho[1];
      g[kRestX + 1] += rho[0] * rho[2];
      g[kRestX + 2] += rho[1] * rho[2];
      dens2 += dens * dens;
    });
  }
  double v[16] = {g[kRest00], g[kRestBB], g[kRestBB + 1], g[kRestBB + 2], g[kRestX], g[kRestX + 1], g[kRestX + 2],
                  (double)dbl[0], (double)dbl[1], (double)dbl[2], (double)sum[0], (double)sum[1], (double)sum[2],
                  uniform ? g[kRest00] + g[kRestOver] : dens2, 0.0, 0.0};
  double t = cluster_sums<SPLIT>(v, sh);
  if (rank != 0) return;
  if (threadIdx.x < kTerms) {
    const int k = threadIdx.x;
    if (uniform) {
      const double u = kFxInv / rd.vol_bin, c = u * rd.bead_vol;
      if (k == 0) t *= (rd.vol_bin / rd.bead_vol) * (c * c);
      else if (k < 7 || k == 13) t *= u * u;
    }
    T[k] = t;
    if (terms) terms[rep * kTerms + k] = t;
  }
  __syncthreads();
  if (acc) {
    double* A = acc + (long long)rep * kAccPerRep;
    if (threadIdx.x < kTerms) A[threadIdx.x] += T[threadIdx.x];
    for (int k = threadIdx.x; k < kTerms * kTerms; k += blockDim.x)
      A[kTerms + k] += T[k / kTerms] * T[k % kTerms];
    if (threadIdx.x == 0) A[kTerms + kTerms * kTerms] += 1.0;
  }
}

}  // namespace cg

// CTAs of 4 warps, 30 beads a warp and pass; passes per warp so that about one
// wave of CTAs (5 per SM) remains, up to 8: a CTA's constants take ~200 FP64
// operations, a pass ~170 a warp.  64 chains of 5,000 beads with the read-back:
// one pass a warp 210 us, two waves of CTAs 195, one 183.
static dim3 gradient_grid(const cg::KArgs& a, long long max_beads, int n_sm) {
  const long long passes = (max_beads + 29) / 30;
  const long long per =
      std::min<long long>(8, std::max<long long>(1, passes * a.n_reps / (4 * 5 * std::max(1, n_sm))));
  long long bx = (passes + 4 * per - 1) / (4 * per);
  if (bx < 1) bx = 1;
  return dim3((unsigned)bx, (unsigned)a.n_reps);
}

void cg_launch_gradient(const cg::KArgs& a, bool fp64, float* out, long long max_beads, int n_sm,
                        cudaStream_t s) {
  const dim3 grid = gradient_grid(a, max_beads, n_sm);
  if (fp64) cg::gradient_kernel<double, float><<<grid, 128, 0, s>>>(a, out, nullptr);
  else cg::gradient_kernel<float, float><<<grid, 128, 0, s>>>(a, out, nullptr);
}

void cg_launch_gradient64(const cg::KArgs& a, bool fp64, double* out, double* out_t3, long long max_beads,
                          int n_sm, cudaStream_t s) {
  const dim3 grid = gradient_grid(a, max_beads, n_sm);
  if (fp64) cg::gradient_kernel<double, double><<<grid, 128, 0, s>>>(a, out, out_t3);
  else cg::gradient_kernel<float, double><<<grid, 128, 0, s>>>(a, out, out_t3);
}

namespace cg {
// Global bead b (replicas concatenated) of FP64 [total_beads x 3] arrays into
// the resident 4-vector storage.
template <typename Pos>
__global__ void store_chains_kernel(KArgs a, long long total, const double* r, const double* t3) {
  V4<Pos>* r4 = reinterpret_cast<V4<Pos>*>(a.r4);
  V4<Pos>* t34 = reinterpret_cast<V4<Pos>*>(a.t34);
  for (long long b = blockIdx.x * (long long)blockDim.x + threadIdx.x; b < total;
       b += (long long)gridDim.x * blockDim.x) {
    if (r) r4[b] = V4<Pos>{(Pos)r[3 * b], (Pos)r[3 * b + 1], (Pos)r[3 * b + 2], (Pos)0};
    if (t3) t34[b] = V4<Pos>{(Pos)t3[3 * b], (Pos)t3[3 * b + 1], (Pos)t3[3 * b + 2], (Pos)0};
  }
}
}  // namespace cg

void cg_launch_store_chains(const cg::KArgs& a, bool fp64, long long total, const double* r, const double* t3,
                            cudaStream_t s) {
  long long blocks = (total + 255) / 256;
  if (blocks > 152 * 8) blocks = 152 * 8;
  if (blocks < 1) blocks = 1;
  if (fp64) cg::store_chains_kernel<double><<<(unsigned)blocks, 256, 0, s>>>(a, total, r, t3);
  else cg::store_chains_kernel<float><<<(unsigned)blocks, 256, 0, s>>>(a, total, r, t3);
}

void cg_launch_terms(const cg::KArgs& a, int log_ctas, double* terms, double* acc, cudaStream_t s) {
  cg::launch_sums(cg::terms_kernel<false>, cg::terms_kernel<true>, a, log_ctas, s, terms, acc);
}
